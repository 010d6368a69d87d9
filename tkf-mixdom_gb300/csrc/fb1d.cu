// fb1d.cu -- batched 1D alignment-conditioned forward-backward.
//
// Along a fixed alignment the pair HMM is an ordinary HMM over the alignment
// columns (dp/hmm.py:127-250, 471-607): column l emits through the states of
// its type only (dp/hmm.py:854-1082), alpha_l = (alpha_{l-1} chi) .* e_l.
// One CTA per pair, in two phases:
//   recursions   one warp walks the columns forward and another backward at the
//                same time; a lane owns one state (two above 32) with its column
//                or row of chi in registers, the vector passes through shared
//                memory, and the power-of-two rescaling after every column
//                (exact, the exponents kept as integers) takes its maximum by one
//                warp reduction: no barrier, about 200 clocks a column;
//   counts       every thread owns entries of the expected transitions, in
//                Kahan-compensated float32 registers, and walks the columns from
//                the last to the first through tiles of both vectors in shared
//                memory (the order of an entry's additions is that of the
//                backward walk, so the sums do not depend on the split).
// What bounds it is the recursions' chain: column by column a product of N
// multiply-adds, a maximum and a rescaling.  With one 128-thread CTA walking the
// columns forward, then backward and counting every pair of states between its
// barriers (each thread taking the float64 exponential of the column's scale),
// 256 alignments of 40-500 columns took 1.51 ms at 17 states; now 0.18 ms, and 64 of
// 60-400 at 42 states 0.26 ms instead of 1.99, with the same bits.
// Emission tables come as linear per-column rows [sum L][N]; a second
// kernel builds them from an alignment and the per-group tables the 2D path
// uses.
#include "pairhmm.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

extern "C" __attribute__((visibility("hidden"))) void phmm_internal_set_error(const char *msg);

namespace fb1 {

constexpr int MAXN = 64;         // states
constexpr int TILE = 16;         // columns staged for the counts at a time
constexpr int EXPN = -(1 << 28); // exponent of an all-zero vector
constexpr double LN2 = 0.69314718055994530942;

struct Meta {
    int64_t off;   // first column
    int32_t L;
    int32_t pad;
};

__device__ __forceinline__ int exp2_of(float m) {   // m * 2^-e in [0.5, 1) for m > 0
    int e;
    frexpf(m, &e);
    return e;
}

// The largest of the warp's values and 0 (compared as integers: the values are not negative).
__device__ __forceinline__ float warp_max(float v) {
    return __int_as_float(__reduce_max_sync(0xffffffffu, max(__float_as_int(v), 0)));
}

// v * 2^-e
__device__ __forceinline__ float scale_down(float v, int e) {
    return (e >= -126 && e <= 126) ? v * __int_as_float((127 - e) << 23) : ldexpf(v, -e);
}

// Rescales a vector held NR states to a lane by the power of two of its largest
// entry; returns the exponent, cum plus its own (EXPN once a vector is all zero).
template <int NR>
__device__ __forceinline__ int rescale(float (&v)[NR], int cum) {
    float mx = v[0];
    if (NR > 1) mx = fmaxf(mx, v[NR - 1]);
    mx = warp_max(mx);
    const int b = __float_as_int(mx) >> 23;
    const int e = mx > 0.f ? (b > 0 && b < 255 ? b - 126 : exp2_of(mx)) : 0;
#pragma unroll
    for (int z = 0; z < NR; ++z) v[z] = mx > 0.f ? scale_down(v[z], e) : 0.f;
    return (mx > 0.f && cum > EXPN) ? cum + e : EXPN;
}

struct Args {
    const Meta *meta;
    int N, chi_per_pair, init, fin;
    const float *chi, *emit;
    float *alpha, *beta;    // rescaled vectors by column
    int *aexp, *bexp;       // their exponents
    double *ll, *n;
    float *post;
    int32_t *status;
};

// The dot products of a lane's NR states: c[z][.] against the vector in shared
// memory (padded with zeros to NB), one term after the other.
template <int NB, int NR>
__device__ __forceinline__ void dots(const float *vec, const float (&c)[NR][NB], float (&s)[NR]) {
#pragma unroll
    for (int z = 0; z < NR; ++z) s[z] = 0.f;
#pragma unroll
    for (int j4 = 0; j4 < NB / 4; ++j4) {
        const float4 f = ((const float4 *)vec)[j4];
#pragma unroll
        for (int z = 0; z < NR; ++z) {
            s[z] = fmaf(f.x, c[z][4 * j4], s[z]);
            s[z] = fmaf(f.y, c[z][4 * j4 + 1], s[z]);
            s[z] = fmaf(f.z, c[z][4 * j4 + 2], s[z]);
            s[z] = fmaf(f.w, c[z][4 * j4 + 3], s[z]);
        }
    }
}

// NB: bound of N (a multiple of 4); NR: states per lane of the recursions; NT:
// threads; EPT: entries of the counts per thread (EPT NT >= NB NB).
template <int NB, int NR, int NT, int EPT>
__global__ void __launch_bounds__(NT)
fb1d_kernel(const __grid_constant__ Args A) {
    constexpr int AHEAD = 4;                    // columns the emissions are loaded ahead
    static_assert(EPT * NT >= NB * NB, "every entry has a thread");
    extern __shared__ float smf[];              // chi [N][N], then two tiles [TILE][N] of both vectors
    __shared__ __align__(16) float vec[2][2][NB];   // direction, column parity
    __shared__ float scale[2][TILE];            // 2^(exponents - log2 P) of the transitions, of the posteriors
    __shared__ double s_lp2;
    __shared__ int s_ok;
    __shared__ float s_f[2];                    // scales of the last column's alpha and the first's beta
    const int p = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const Meta m = A.meta[p];
    const int N = A.N, NN = N * N, L = m.L;
    float *chi = smf;
    const float *chig = A.chi + (A.chi_per_pair ? (int64_t)p * NN : 0);
    for (int idx = tid; idx < NN; idx += NT) chi[idx] = chig[idx];
    double *nt = A.n + (int64_t)p * NN;
    __syncthreads();
    if (L == 0) {   // empty alignment: S -> E directly
        const float c = chi[A.init * N + A.fin];
        if (tid == 0) {
            A.ll[p] = c > 0.f ? log((double)c) : -1e30;
            if (!(c > 0.f)) atomicOr(A.status + p, PHMM_ST_ZERO_LL);
        }
        for (int idx = tid; idx < NN; idx += NT) nt[idx] = (idx == A.init * N + A.fin) ? 1.0 : 0.0;
        return;
    }
    const float *em = A.emit + m.off * N;
    float *al = A.alpha + m.off * N, *be = A.beta + m.off * N;
    int *ae = A.aexp + m.off, *bx = A.bexp + m.off;

    if (warp < 2) {
        // ---- the recursions: warp 0 forward, warp 1 backward
        const bool fwd = warp == 0;
        float c[NR][NB], v[NR], w[NR];
        int k[NR];
#pragma unroll
        for (int z = 0; z < NR; ++z) {
            k[z] = lane + 32 * z;
#pragma unroll
            for (int j = 0; j < NB; ++j)
                c[z][j] = (k[z] < N && j < N) ? (fwd ? chi[j * N + k[z]] : chi[k[z] * N + j]) : 0.f;
        }
        auto put = [&](int par, const float (&x)[NR]) {   // the vector into shared memory
#pragma unroll
            for (int z = 0; z < NR; ++z)
                if (k[z] < NB) vec[warp][par][k[z]] = x[z];
            __syncwarp();
        };
        auto load = [&](const float *row, bool in, float (&x)[NR]) {
#pragma unroll
            for (int z = 0; z < NR; ++z) x[z] = (in && k[z] < N) ? __ldg(row + k[z]) : 0.f;
        };
        float e[AHEAD][NR];
        int cum;
        if (fwd) {
#pragma unroll
            for (int u = 0; u < AHEAD; ++u) load(em + (int64_t)u * N, u < L, e[u]);
            cum = 0;
            for (int l0 = 0; l0 < L; l0 += AHEAD) {
#pragma unroll
                for (int u = 0; u < AHEAD; ++u) {
                    const int l = l0 + u;
                    if (l >= L) break;
                    if (l == 0) {
#pragma unroll
                        for (int z = 0; z < NR; ++z) v[z] = k[z] < N ? chi[A.init * N + k[z]] : 0.f;
                    } else {
                        dots<NB, NR>(vec[0][l & 1], c, v);
                    }
#pragma unroll
                    for (int z = 0; z < NR; ++z) v[z] = v[z] * e[u][z];
                    load(em + (int64_t)(l + AHEAD) * N, l + AHEAD < L, e[u]);
                    cum = rescale<NR>(v, cum);
                    put((l + 1) & 1, v);
#pragma unroll
                    for (int z = 0; z < NR; ++z)
                        if (k[z] < N) al[(int64_t)l * N + k[z]] = v[z];
                    if (lane == 0) ae[l] = cum;
                }
            }
            double pz = 0.0, part[NR];
#pragma unroll
            for (int z = 0; z < NR; ++z) {
                part[z] = k[z] < N ? (double)v[z] * (double)chi[k[z] * N + A.fin] : 0.0;
                for (int o = 16; o > 0; o >>= 1) part[z] += __shfl_xor_sync(0xffffffffu, part[z], o);
                pz += part[z];
            }
            const bool ok = pz > 0.0 && cum > EXPN;
            if (lane == 0) {
                const double lp2 = ok ? log2(pz) + (double)cum : 0.0;   // log2 P
                s_lp2 = lp2;
                s_ok = ok;
                A.ll[p] = ok ? lp2 * LN2 : -1e30;
                if (!ok) atomicOr(A.status + p, PHMM_ST_ZERO_LL);
            }
        } else {
#pragma unroll
            for (int u = 0; u < AHEAD; ++u) load(em + (int64_t)(L - 1 - u) * N, L - 1 - u >= 0, e[u]);
#pragma unroll
            for (int z = 0; z < NR; ++z) v[z] = k[z] < N ? chi[k[z] * N + A.fin] : 0.f;
            cum = rescale<NR>(v, 0);
            for (int l0 = L - 1; l0 >= 0; l0 -= AHEAD) {
#pragma unroll
                for (int u = 0; u < AHEAD; ++u) {
                    const int l = l0 - u;       // v = b_l
                    if (l < 0) break;
#pragma unroll
                    for (int z = 0; z < NR; ++z)
                        if (k[z] < N) be[(int64_t)l * N + k[z]] = v[z];
                    if (lane == 0) bx[l] = cum;
#pragma unroll
                    for (int z = 0; z < NR; ++z) w[z] = e[u][z] * v[z];
                    load(em + (int64_t)(l - AHEAD) * N, l - AHEAD >= 0, e[u]);
                    if (l == 0) break;
                    put(l & 1, w);
                    dots<NB, NR>(vec[1][l & 1], c, v);   // b_{l-1}
                    cum = rescale<NR>(v, cum);
                }
            }
        }
    }
    __syncthreads();
    if (!s_ok) {
        for (int idx = tid; idx < NN; idx += NT) nt[idx] = 0.0;
        return;
    }
    // ---- the counts
    const double lp2 = s_lp2;
    float *ta = smf + NN, *tw = ta + TILE * N;  // a_l and w_{l+1} = e_{l+1} b_{l+1} of the tile's columns
    if (tid < 2) s_f[tid] = (float)exp2((double)(tid == 0 ? ae[L - 1] : bx[0]) - lp2);
    __syncthreads();
    float ch[EPT], cs[EPT], cc[EPT];
    int es[EPT], ek[EPT];
    auto add = [&](float &s, float &c, float v, float f) {   // Kahan, of the product v f
        const float y = fmaf(v, f, -c), t = s + y;
        c = (t - s) - y;
        s = t;
    };
#pragma unroll
    for (int z = 0; z < EPT; ++z) {
        const int idx = tid + z * NT;
        es[z] = idx < NN ? idx / N : 0;
        ek[z] = idx < NN ? idx % N : 0;
        ch[z] = idx < NN ? chi[idx] : 0.f;
        // the step to the final state: a_{L-1}[s] chi[s][final] / P
        cs[z] = idx < NN && ek[z] == A.fin ? __fmul_rn(al[(int64_t)(L - 1) * N + es[z]] * ch[z], s_f[0]) : 0.f;
        cc[z] = 0.f;
    }
    for (int top = L - 1; top >= 0; top -= TILE) {   // columns top, top - 1, ...
        const int n = min(TILE, top + 1);
        __syncthreads();
        if (tid < 2 * TILE) {
            const int i = tid % TILE, l = top - i, ln = tid < TILE ? l + 1 : l;
            if (i < n) scale[tid / TILE][i] = ln < L ? (float)exp2((double)ae[l] + (double)bx[ln] - lp2) : 0.f;
        }
        for (int q = tid; q < n * N; q += NT) {
            const int i = q / N, k = q - i * N, l = top - i;
            ta[q] = al[(int64_t)l * N + k];
            tw[q] = l + 1 < L ? em[(int64_t)(l + 1) * N + k] * be[(int64_t)(l + 1) * N + k] : 0.f;
        }
        __syncthreads();
        if (A.post)
            for (int q = tid; q < n * N; q += NT) {
                const int i = q / N, k = q - i * N, l = top - i;
                A.post[(m.off + l) * N + k] = ta[q] * be[(int64_t)l * N + k] * scale[1][i];
            }
        // n[s][k] += a_l[s] chi[s][k] w_{l+1}[k] 2^(A_l + B_{l+1} - log2 P)
        for (int i = top == L - 1 ? 1 : 0; i < n; ++i) {
            const float f = scale[0][i];
            const float *a = ta + i * N, *w = tw + i * N;
#pragma unroll
            for (int z = 0; z < EPT; ++z) {
                const float v = a[es[z]] * ch[z] * w[ek[z]];
                if (v != 0.f) add(cs[z], cc[z], v, f);
            }
        }
    }
#pragma unroll
    for (int z = 0; z < EPT; ++z) {
        const int idx = tid + z * NT;
        if (idx >= NN) break;
        // the step from the initial state: chi[init][k] e_0[k] b_0[k] / P
        if (es[z] == A.init) add(cs[z], cc[z], ch[z] * (em[ek[z]] * be[ek[z]]), s_f[1]);
        nt[idx] = (double)cs[z] - (double)cc[z];
    }
}

template <int NB, int NR, int NT, int EPT>
cudaError_t launch(const Args &a, int P, cudaStream_t st) {
    const size_t smem = sizeof(float) * ((size_t)a.N * a.N + 2 * TILE * a.N);
    fb1d_kernel<NB, NR, NT, EPT><<<P, NT, smem, st>>>(a);
    return cudaGetLastError();
}

// Per-column emissions of an alignment: column l of type c (1 M, 2 I, 3 D)
// emits through the states of type c with the per-group tables of the 2D
// path (M: table_M[g][anc][desc]; I: table_I[g][desc]; D: table_D[g][anc]);
// other states (and S, E) get 0.
struct EmitDesc {
    int N;
    int8_t type[MAXN];
    int8_t group[MAXN];
};

// One warp per column, a lane per state; blockIdx.y takes columns of its own.
__global__ void __launch_bounds__(256)
emit1d_kernel(const __grid_constant__ EmitDesc ed, const Meta *__restrict__ meta, const uint8_t *__restrict__ cols,
              const uint8_t *__restrict__ anc, const uint8_t *__restrict__ desc, const float *__restrict__ tM,
              const float *__restrict__ tI, const float *__restrict__ tD, int per_pair, int G,
              float *__restrict__ emit, int32_t *__restrict__ status) {
    const int p = blockIdx.x, lane = threadIdx.x & 31;
    const Meta m = meta[p];
    const int N = ed.N;
    const float *M_ = tM + (per_pair ? (int64_t)p * G * 441 : 0);
    const float *I_ = tI + (per_pair ? (int64_t)p * G * 21 : 0);
    const float *D_ = tD + (per_pair ? (int64_t)p * G * 21 : 0);
    for (int l = blockIdx.y * 8 + (threadIdx.x >> 5); l < m.L; l += gridDim.y * 8) {
        const int c = cols[m.off + l];
        int a = anc[m.off + l], b = desc[m.off + l];
        if (a > 20 || b > 20) {
            if (lane == 0) atomicOr(status + p, PHMM_ST_BAD_RESIDUE);
            a = a > 20 ? 20 : a;
            b = b > 20 ? 20 : b;
        }
        for (int s = lane; s < N; s += 32) {
            float v = 0.f;
            if (c == ed.type[s]) {
                const int g = ed.group[s];
                if (c == 1) v = M_[g * 441 + a * 21 + b];
                else if (c == 2) v = I_[g * 21 + b];
                else if (c == 3) v = D_[g * 21 + a];
            }
            emit[(m.off + l) * N + s] = v;
        }
    }
}

// Expected emission counts of the alignments: the posterior of every state at a
// column of its type, summed by the state's group and the column's characters.
// A warp per column; blockIdx.y takes columns of its own.
__global__ void __launch_bounds__(256)
count1d_kernel(const __grid_constant__ EmitDesc ed, const Meta *__restrict__ meta, const uint8_t *__restrict__ cols,
               const uint8_t *__restrict__ anc, const uint8_t *__restrict__ desc, const float *__restrict__ post, int G,
               double *__restrict__ cM, double *__restrict__ cI, double *__restrict__ cD) {
    const int p = blockIdx.x, lane = threadIdx.x & 31, N = ed.N;
    const Meta m = meta[p];
    for (int l = blockIdx.y * 8 + (threadIdx.x >> 5); l < m.L; l += gridDim.y * 8) {
        const int c = cols[m.off + l], a = min((int)anc[m.off + l], 20), b = min((int)desc[m.off + l], 20);
        for (int s = lane; s < N; s += 32) {
            if (c != ed.type[s] || c < 1 || c > 3) continue;
            const double v = (double)post[(m.off + l) * N + s];
            const int64_t g = (int64_t)p * G + ed.group[s];
            if (c == 1) atomicAdd(cM + g * 441 + a * 21 + b, v);
            else if (c == 2) atomicAdd(cI + g * 21 + b, v);
            else atomicAdd(cD + g * 21 + a, v);
        }
    }
}

}  // namespace fb1

static int fb1_fail(int code, const char *msg) {
    phmm_internal_set_error(msg);
    return code;
}

static size_t fb1_align(size_t v) { return (v + 255) & ~(size_t)255; }

static int fb1_layout(int P, const int32_t *L_host, const int64_t *off_host, int N, size_t *cols_out,
                      size_t *o_alpha, size_t *o_aexp, size_t *total) {
    size_t cols = 0;
    for (int p = 0; p < P; ++p) {
        if (L_host[p] < 0 || off_host[p] < 0) return fb1_fail(PHMM_E_ARG, "phmm_fb1d: negative length or offset");
        cols = std::max(cols, (size_t)(off_host[p] + L_host[p]));
    }
    const size_t o_meta = 0;
    *o_alpha = fb1_align(o_meta + sizeof(fb1::Meta) * (size_t)P);
    *o_aexp = fb1_align(*o_alpha + 2 * sizeof(float) * cols * N);   // alpha, then beta
    *total = fb1_align(*o_aexp + 2 * sizeof(int) * cols);
    *cols_out = cols;
    return PHMM_OK;
}

extern "C" int phmm_fb1d_workspace_bytes(const phmm_fb1d_batch *b, size_t *bytes) {
    if (!b || !bytes) return fb1_fail(PHMM_E_ARG, "phmm_fb1d_workspace_bytes: null argument");
    *bytes = 0;
    if (b->n_pairs <= 0) return PHMM_OK;
    if (!b->L_host || !b->off_host) return fb1_fail(PHMM_E_ARG, "phmm_fb1d: null host length or offset array");
    size_t cols, oa, oe, total;
    int rc = fb1_layout(b->n_pairs, b->L_host, b->off_host, b->n_states, &cols, &oa, &oe, &total);
    if (rc) return rc;
    *bytes = total;
    return PHMM_OK;
}

extern "C" int phmm_fb1d(const phmm_fb1d_batch *b, void *workspace, size_t workspace_bytes, double *ll_out,
                         double *n_trans, float *posteriors, int32_t *status_out, void *stream) {
    using namespace fb1;
    if (!b) return fb1_fail(PHMM_E_ARG, "phmm_fb1d: null batch");
    const int P = b->n_pairs, N = b->n_states;
    if (P < 0) return fb1_fail(PHMM_E_ARG, "phmm_fb1d: negative n_pairs");
    if (P == 0) return PHMM_OK;
    if (N < 2 || N > MAXN) return fb1_fail(PHMM_E_ARG, "phmm_fb1d: n_states must be in 2..64");
    if (b->init_state < 0 || b->init_state >= N || b->final_state < 0 || b->final_state >= N)
        return fb1_fail(PHMM_E_ARG, "phmm_fb1d: bad init or final state");
    if (!b->L_host || !b->off_host || !b->emit || !b->chi || !ll_out || !n_trans || !status_out || !workspace)
        return fb1_fail(PHMM_E_ARG, "phmm_fb1d: null pointer");
    if ((uintptr_t)workspace & 255) return fb1_fail(PHMM_E_ARG, "phmm_fb1d: workspace must be 256-byte aligned");
    size_t cols, oa, oe, total;
    int rc = fb1_layout(P, b->L_host, b->off_host, N, &cols, &oa, &oe, &total);
    if (rc) return rc;
    if (workspace_bytes < total) return fb1_fail(PHMM_E_ARG, "phmm_fb1d: workspace too small");
    std::vector<Meta> meta(P);
    for (int p = 0; p < P; ++p) meta[p] = Meta{b->off_host[p], b->L_host[p], 0};
    cudaStream_t st = (cudaStream_t)stream;
    char *ws = (char *)workspace;
    cudaError_t e = cudaMemcpyAsync(ws, meta.data(), sizeof(Meta) * P, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(status_out, 0, sizeof(int32_t) * P, st);
    if (e != cudaSuccess) return fb1_fail(PHMM_E_CUDA, cudaGetErrorString(e));
    Args a;
    a.meta = (const Meta *)ws;
    a.N = N;
    a.chi_per_pair = b->chi_per_pair;
    a.init = b->init_state;
    a.fin = b->final_state;
    a.chi = b->chi;
    a.emit = b->emit;
    a.alpha = (float *)(ws + oa);
    a.beta = a.alpha + cols * N;
    a.aexp = (int *)(ws + oe);
    a.bexp = a.aexp + cols;
    a.ll = ll_out;
    a.n = n_trans;
    a.post = posteriors;
    a.status = status_out;
    // one state per recursion lane up to 32 states, two above; the bounds keep the padding of the products small
    if (N <= 8) e = launch<8, 1, 64, 1>(a, P, st);
    else if (N <= 20) e = launch<20, 1, 256, 2>(a, P, st);
    else if (N <= 32) e = launch<32, 1, 256, 4>(a, P, st);
    else if (N <= 44) e = launch<44, 2, 256, 8>(a, P, st);
    else e = launch<64, 2, 256, 16>(a, P, st);
    if (e != cudaSuccess) return fb1_fail(PHMM_E_CUDA, cudaGetErrorString(e));
    return PHMM_OK;
}

extern "C" int phmm_fb1d_emissions(const phmm_model_desc *model, int32_t n_pairs, const int32_t *L_host,
                                   const int64_t *off_host, const uint8_t *cols, const uint8_t *anc,
                                   const uint8_t *desc, const float *emit_M, const float *emit_I,
                                   const float *emit_D, int32_t emit_per_pair, void *workspace,
                                   size_t workspace_bytes, float *emit, int32_t *status_out, void *stream) {
    using namespace fb1;
    if (!model || !model->state_types || !model->state_group)
        return fb1_fail(PHMM_E_ARG, "phmm_fb1d_emissions: bad model description");
    const int N = model->n_states, G = model->n_groups;
    if (N < 2 || N > MAXN) return fb1_fail(PHMM_E_ARG, "phmm_fb1d_emissions: n_states must be in 2..64");
    if (n_pairs < 0) return fb1_fail(PHMM_E_ARG, "phmm_fb1d_emissions: negative n_pairs");
    if (n_pairs == 0) return PHMM_OK;
    if (!L_host || !off_host || !cols || !anc || !desc || !emit_M || !emit_I || !emit_D || !emit || !workspace ||
        !status_out)
        return fb1_fail(PHMM_E_ARG, "phmm_fb1d_emissions: null pointer");
    if (workspace_bytes < sizeof(Meta) * (size_t)n_pairs)
        return fb1_fail(PHMM_E_ARG, "phmm_fb1d_emissions: workspace too small");
    EmitDesc ed;
    std::memset(&ed, 0, sizeof(ed));
    ed.N = N;
    for (int s = 0; s < N; ++s) {
        ed.type[s] = model->state_types[s];
        ed.group[s] = (int8_t)model->state_group[s];
        if (model->state_group[s] < 0 || model->state_group[s] >= G)
            return fb1_fail(PHMM_E_ARG, "phmm_fb1d_emissions: state group out of range");
    }
    std::vector<Meta> meta(n_pairs);
    for (int p = 0; p < n_pairs; ++p) {
        if (L_host[p] < 0 || off_host[p] < 0) return fb1_fail(PHMM_E_ARG, "phmm_fb1d_emissions: negative length");
        meta[p] = Meta{off_host[p], L_host[p], 0};
    }
    cudaStream_t st = (cudaStream_t)stream;
    cudaError_t e = cudaMemcpyAsync(workspace, meta.data(), sizeof(Meta) * n_pairs, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(status_out, 0, sizeof(int32_t) * n_pairs, st);
    if (e != cudaSuccess) return fb1_fail(PHMM_E_CUDA, cudaGetErrorString(e));
    int most = 1;
    for (const Meta &m : meta) most = std::max(most, (int)m.L);
    emit1d_kernel<<<dim3(n_pairs, std::min(16, (most + 31) / 32)), 256, 0, st>>>(ed, (const Meta *)workspace, cols, anc, desc, emit_M, emit_I, emit_D,
                                          emit_per_pair, G, emit, status_out);
    e = cudaGetLastError();
    if (e != cudaSuccess) return fb1_fail(PHMM_E_CUDA, cudaGetErrorString(e));
    return PHMM_OK;
}

extern "C" int phmm_fb1d_counts(const phmm_model_desc *model, int32_t n_pairs, const int32_t *L_host,
                                const int64_t *off_host, const uint8_t *cols, const uint8_t *anc, const uint8_t *desc,
                                const float *posteriors, void *workspace, size_t workspace_bytes, double *cnt_M,
                                double *cnt_I, double *cnt_D, void *stream) {
    using namespace fb1;
    if (!model || !model->state_types || !model->state_group)
        return fb1_fail(PHMM_E_ARG, "phmm_fb1d_counts: bad model description");
    const int N = model->n_states, G = model->n_groups;
    if (N < 2 || N > MAXN) return fb1_fail(PHMM_E_ARG, "phmm_fb1d_counts: n_states must be in 2..64");
    if (n_pairs < 0) return fb1_fail(PHMM_E_ARG, "phmm_fb1d_counts: negative n_pairs");
    if (n_pairs == 0) return PHMM_OK;
    if (!L_host || !off_host || !cols || !anc || !desc || !posteriors || !workspace || !cnt_M || !cnt_I || !cnt_D)
        return fb1_fail(PHMM_E_ARG, "phmm_fb1d_counts: null pointer");
    if (workspace_bytes < sizeof(Meta) * (size_t)n_pairs)
        return fb1_fail(PHMM_E_ARG, "phmm_fb1d_counts: workspace too small");
    EmitDesc ed;
    std::memset(&ed, 0, sizeof(ed));
    ed.N = N;
    for (int s = 0; s < N; ++s) {
        ed.type[s] = model->state_types[s];
        ed.group[s] = (int8_t)model->state_group[s];
        if (model->state_group[s] < 0 || model->state_group[s] >= G)
            return fb1_fail(PHMM_E_ARG, "phmm_fb1d_counts: state group out of range");
    }
    std::vector<Meta> meta(n_pairs);
    int most = 1;
    for (int p = 0; p < n_pairs; ++p) {
        if (L_host[p] < 0 || off_host[p] < 0) return fb1_fail(PHMM_E_ARG, "phmm_fb1d_counts: negative length");
        meta[p] = Meta{off_host[p], L_host[p], 0};
        most = std::max(most, (int)L_host[p]);
    }
    cudaStream_t st = (cudaStream_t)stream;
    const size_t PG = (size_t)n_pairs * G;
    cudaError_t e = cudaMemcpyAsync(workspace, meta.data(), sizeof(Meta) * n_pairs, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(cnt_M, 0, sizeof(double) * PG * 441, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(cnt_I, 0, sizeof(double) * PG * 21, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(cnt_D, 0, sizeof(double) * PG * 21, st);
    if (e != cudaSuccess) return fb1_fail(PHMM_E_CUDA, cudaGetErrorString(e));
    count1d_kernel<<<dim3(n_pairs, std::min(16, (most + 31) / 32)), 256, 0, st>>>(
        ed, (const Meta *)workspace, cols, anc, desc, posteriors, G, cnt_M, cnt_I, cnt_D);
    e = cudaGetLastError();
    if (e != cudaSuccess) return fb1_fail(PHMM_E_CUDA, cudaGetErrorString(e));
    return PHMM_OK;
}
