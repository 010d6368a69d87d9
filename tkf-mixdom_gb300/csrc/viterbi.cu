// viterbi.cu -- batched 2D pair-HMM Viterbi with traceback (dp/hmm.py:1976-2040).
//
// V[i][j][k] = max_s (V[pred(k)][s] + logchi[s][k]) + logemit_k(x_i, y_j) in
// float64 log space, pred by the type of k (M: (i-1,j-1), I: (i,j-1), D:
// (i-1,j)); the first maximal source wins, as argmax does.  Scores that the
// reference keeps at NEG_INF (-1e30, summed like any other number) are
// reproduced bit for bit, so the path matches the reference's.
//
// Two launches:
//   viterbi_stripe_kernel   the stripe wavefront of stripe64.cuh, one thread per
//                           (row, state);
//   traceback_kernel        one CTA per pair walks the path back through tiles of
//                           backpointers staged in shared memory.
//
// What bounds the recursion is the FP64 unit (two lanes per SM and clock): N
// additions and N comparisons per state would take all of a step.  Each thread
// therefore screens its sources in float32 -- scores truncated from the float64
// values, with a bound on their distance from the exact ones -- and adds in
// float64 only the sources that can be the maximum, nearly always one: two
// float64 additions per state and cell instead of 2N operations, the same
// values and backpointers.  Cells without a reachable source, and scores
// outside the screen's range, take the plain float64 loop.  Measured on 24 pairs of
// 80-400 residues at 17 states: 34.2 ms for one CTA per pair sweeping the
// anti-diagonals with the dense float64 loop, 0.94 ms here.
#include "stripe64.cuh"

extern "C" __attribute__((visibility("hidden"))) void phmm_internal_set_error(const char *msg);

namespace vit {

using namespace s64;

// Backpointer of a state the envelope left out (hmm_beam.py:455-476 stores
// the triple (0, 0, S) there): the traceback jumps to the origin.
constexpr uint8_t BP_ORIGIN = 255;
constexpr uint8_t BP_STATE = 64;       // backpointers are slots; a state without one is BP_STATE + state
constexpr float FAR = 1.2676506e30f;   // 2^100: magnitudes above it are clamped in the screen
constexpr float LIVE = 1e27f;          // screened scores beyond it take the plain loop

struct Args {
    Desc d;
    const Meta *meta;
    const Item *items;
    int *ctl;   // claim counter, then one progress word per stripe
    const uint8_t *res;
    const double *lchi, *lM, *lI, *lD;
    int chi_pp, emit_pp;
    double *edge;
    uint8_t *tb;   // [cell][SB]: backpointer of every slot
    int *fin;      // [P] best terminal state
    double *ll;
    int32_t *status;
    const uint8_t *env;
};

// Bytes of a cell's backpointers (one per slot, in whole words).
__host__ __device__ inline int bp_stride(int ns) { return (ns + 3) & ~3; }

// float32 of v, truncated to 23 mantissa bits by integer operations (a
// conversion would run on the FP64 unit): within 2^-23 |v| of v; beyond 2^100
// clamped to -2^100 below and to +inf above; NaN becomes +inf.
__device__ __forceinline__ float screen32(double v) {
    const int hi = __double2hiint(v);
    const unsigned lo = (unsigned)__double2loint(v);
    const int a = hi & 0x7fffffff;
    const unsigned m = __funnelshift_l(lo, (unsigned)(a - (896 << 20)), 3);
    const float f = __uint_as_float((m & 0x7fffffffu) | ((unsigned)hi & 0x80000000u));
    if ((unsigned)(a - (897 << 20)) < (unsigned)((1123 - 897) << 20)) return f;
    if (a < (897 << 20)) return 0.f;
    const bool nan = a > 0x7ff00000 || (a == 0x7ff00000 && lo != 0u);
    return hi < 0 && !nan ? -FAR : __int_as_float(0x7f800000);
}

// L lanes per row, R rows per stripe; ENV: with an envelope.  A step's FP64 work
// is two additions for each of L x R threads, 16 clocks a warp; R is the most
// rows that keep it below the step's latency (loads, screen and barrier).
template <int L, int R, bool ENV>
__global__ void __launch_bounds__(L * R + 64, L * R <= 256 ? 2 : 1)
viterbi_stripe_kernel(const __grid_constant__ Args A) {
    constexpr int NT = L * R, Q4 = L / 4;
    constexpr int ZH = 4 * R * L, Z = ZH + HALO * L;   // values of the step ring, and with the row above
    extern __shared__ __align__(16) double smem[];
    double *lc = smem;                  // [L][L] exact transitions by source and destination slot
    double *V = lc + L * L;             // [4][R][L] values of the last steps, then [HALO][L] the row above
    double *O = V + Z;                  // [HALO][L] the last row, for the publisher
    float *V32 = (float *)(O + HALO * L);   // V, screened
    __shared__ Channel ch;
    __shared__ unsigned lmax_bits;
    const int tid = threadIdx.x;
    const Desc &d = A.d;
    const int N = d.N, ns = d.ns;
    if (tid == 0) {
        lmax_bits = 0u;
        ch.avail = ch.taken = 0;
        ch.step = -1;
    }
    const Item it = claim(A.ctl, A.items);      // (barrier)
    const int p = it.pair;
    const Meta m = A.meta[p];
    const int Lx = m.Lx, Ly = m.Ly;
    const double *lcg = A.lchi + (A.chi_pp ? (int64_t)p * N * N : 0);
    unsigned lmx = 0u;
    for (int idx = tid; idx < L * L; idx += NT + 64) {
        const int a = idx / L, b = idx % L;
        const double l = (a < ns && b < ns) ? lcg[d.state[a] * N + d.state[b]] : NEG;
        lc[idx] = l;
        if (fabs(l) < 1e29) lmx = max(lmx, __float_as_uint(fabsf(screen32(l))));
    }
    if (lmx) atomicMax(&lmax_bits, lmx);
    for (int idx = tid; idx < Z; idx += NT + 64) {
        V[idx] = NEG;
        V32[idx] = -FAR;
    }
    __syncthreads();
    if (it.stripe == 0 && tid == 0) V[0] = V32[0] = 0.0;   // the start, at the origin
    __syncthreads();
    const bool last = it.stripe == m.n_stripes - 1;
    int *prog = A.ctl + 1 + m.stripe0 + it.stripe;
    const int er = ns - 1;                      // doubles of an edge column
    if (tid >= NT) {                            // hand-off warps
        if (tid < NT + 32) {
            if (it.stripe > 0)
                load_edges(A.edge + m.edge_off + (int64_t)(it.stripe - 1) * (Ly + 1) * er, er, Ly, prog - 1, ch,
                           A.status + p, [&](int c, int k, double v) {
                               const int o = ZH + (c & (HALO - 1)) * L + k + 1;
                               V[o] = v;
                               V32[o] = screen32(v);
                           });
        } else if (!last) {
            publish_edges(A.edge + m.edge_off + (int64_t)it.stripe * (Ly + 1) * er, er, R, Ly, prog, ch,
                          [&](int c, int k) { return O[(c & (HALO - 1)) * L + k + 1]; });
        }
        return;
    }
    const int r = tid / L, q = tid % L;
    const float lmax = 1.0001f * __uint_as_float(lmax_bits);
    float lr[L];   // this slot's screened incoming transitions, by source slot
#pragma unroll
    for (int s = 0; s < L; ++s) lr[s] = screen32(lc[s * L + q]);

    const int i = it.stripe * R + r;
    const int k = q < ns ? d.state[q] : 0;
    const int st = q > 0 && q < ns ? d.type[k] : TS;
    const int rows = last ? Lx + 1 - it.stripe * R : R;
    const int T = Ly + rows;
    const bool row_in = r < rows && q < ns;
    // cells with a predecessor: columns jlo..Ly of a valid thread (the others keep the ring's NEG)
    const bool valid = row_in && (st == TI || ((st == TM || st == TD) && i > 0));
    const int jlo = st == TD ? 0 : 1;
    // the predecessor's record at step t: pbase + ((t + poff) & pmask) * pstr
    const bool above = st != TI;
    const bool halo = above && r == 0;
    const int pbase = halo ? ZH : (above ? r - 1 : r) * L;
    const int poff = halo ? (st == TM ? -1 : 0) : (st == TM ? -2 : -1);
    const int pmask = halo ? HALO - 1 : 3, pstr = halo ? L : R * L;
    const bool waits = it.stripe > 0 && r == 0;
    const uint8_t *x = A.res + m.x_off, *y = A.res + m.y_off;
    const int g = d.group[k];
    const int xa = (row_in && i > 0) ? min((int)x[i - 1], 20) : 0;
    const int64_t eg = (int64_t)(A.emit_pp ? p : 0) * d.G + g;
    const double *eb = st == TI ? A.lI + eg * 21 : st == TD ? A.lD + eg * 21 + xa : A.lM + eg * 441 + xa * 21;
    uint8_t *bp = A.tb + m.tab_off + ((int64_t)i * (Ly + 1) - r) * bp_stride(ns) + q;
    const int SB = bp_stride(ns);
    const uint8_t *env = ENV ? A.env + m.mask_off + (int64_t)i * (Ly + 1) - r : nullptr;
    const int epred = st == TI ? -1 : -(Ly + 1) - (st == TM ? 1 : 0);
    const bool edge_out = !last && r == R - 1 && q > 0 && q < ns;
    // characters and emissions one column ahead
    double e1 = valid && st == TD ? __ldg(eb) : 0.0;
    int c1 = valid && r == 0 && Ly > 0 ? min((int)y[0], 20) : 0;   // character of column j + 1
    int have = 0, taken = 0;
    for (int t = 0; t < T; ++t) {
        const int j = t - r;
        const double e = e1;
        if (valid && st != TD && j >= 0 && j < Ly) e1 = __ldg(eb + c1);
        if (valid && j >= -1 && j + 1 < Ly) c1 = min((int)__ldg(y + j + 1), 20);
        if (waits && have <= min(t, Ly)) have = wait_word(ch.avail, min(t, Ly) + 1);
        double v = NEG;
        if (valid && j >= jlo && j <= Ly) {
            const int o = pbase + ((t + poff) & pmask) * pstr;
            int best = BP_ORIGIN;
            // an envelope leaves out cells outside it and states whose predecessor cell is
            if (!ENV || (env[t] && env[t + epred])) {
                const float4 *P32 = (const float4 *)(V32 + o);
                const double *P64 = V + o;
                float mx = -2.f * FAR, mx2 = mx;
                float sc[L <= 32 ? L : 4];
#pragma unroll
                for (int s4 = 0; s4 < Q4; ++s4) {
                    if (L <= 8 || 4 * s4 < ns) {
                        const float4 f = P32[s4];
                        const float2 a = __fadd2_rn(make_float2(f.x, f.y), make_float2(lr[4 * s4], lr[4 * s4 + 1]));
                        const float2 b = __fadd2_rn(make_float2(f.z, f.w), make_float2(lr[4 * s4 + 2], lr[4 * s4 + 3]));
                        if constexpr (L <= 32) {
                            sc[4 * s4] = a.x; sc[4 * s4 + 1] = a.y; sc[4 * s4 + 2] = b.x; sc[4 * s4 + 3] = b.y;
                        }
                        mx = fmaxf(fmaxf(mx, a.x), a.y);
                        mx2 = fmaxf(fmaxf(mx2, b.x), b.y);
                    } else if constexpr (L <= 32) {
                        sc[4 * s4] = sc[4 * s4 + 1] = sc[4 * s4 + 2] = sc[4 * s4 + 3] = -2.f * FAR;
                    }
                }
                mx = fmaxf(mx, mx2);
                double bv;
                if (mx > -LIVE && mx < LIVE) {
                    // A screened score is within 2^-22 (|V| + |l|) of the exact one, and |V| <= |score| + lmax
                    // for the sources that matter, so every maximal source lies above this threshold.
                    const float thr = mx - 9.5367432e-07f * (fabsf(mx) + 2.f * lmax);
                    const float2 th = make_float2(-thr, -thr);
                    unsigned cand[(L + 31) / 32];
#pragma unroll
                    for (int w = 0; w < (L + 31) / 32; ++w) {
                        constexpr int QW = Q4 < 8 ? Q4 : 8;
                        unsigned below = 0u;    // sign bits of score - threshold, slot by slot
#pragma unroll
                        for (int z4 = QW - 1; z4 >= 0; --z4) {
                            const int s4 = 8 * w + z4;
                            float2 a, b;
                            if constexpr (L <= 32) {
                                a = make_float2(sc[4 * s4], sc[4 * s4 + 1]);
                                b = make_float2(sc[4 * s4 + 2], sc[4 * s4 + 3]);
                            } else {
                                const float4 f = P32[s4];
                                a = __fadd2_rn(make_float2(f.x, f.y), make_float2(lr[4 * s4], lr[4 * s4 + 1]));
                                b = __fadd2_rn(make_float2(f.z, f.w), make_float2(lr[4 * s4 + 2], lr[4 * s4 + 3]));
                            }
                            a = __fadd2_rn(a, th);
                            b = __fadd2_rn(b, th);
                            // four bits of their own (no chain through the other slots), then in place
                            unsigned n4 = __funnelshift_l(__float_as_uint(b.x), __float_as_uint(b.y) >> 31, 1);
                            n4 = __funnelshift_l(__float_as_uint(a.y), n4, 1);
                            n4 = __funnelshift_l(__float_as_uint(a.x), n4, 1);
                            below |= n4 << (4 * z4);
                        }
                        cand[w] = ~below & (L >= 32 ? 0xffffffffu : (1u << (L & 31)) - 1u);
                    }
                    int w0 = 0;
                    if (L > 32 && cand[0] == 0u) w0 = 1;
                    unsigned left = w0 ? cand[(L + 31) / 32 - 1] : cand[0];
                    best = 32 * w0 + __ffs(left) - 1;
                    bv = P64[best] + lc[best * L + q];
                    left &= left - 1;
                    for (;;) {                  // rarely more than one candidate
                        while (left) {
                            const int s = 32 * w0 + __ffs(left) - 1;
                            left &= left - 1;
                            const double c = P64[s] + lc[s * L + q];
                            if (c > bv) { bv = c; best = s; }
                        }
                        if (L <= 32 || w0) break;
                        w0 = 1;
                        left = cand[(L + 31) / 32 - 1];
                    }
                } else {                        // no reachable source, or beyond the screen: every state in order
                    int bs = 0;
                    bv = P64[0] + lc[q];
                    for (int s = 1; s < N; ++s) {
                        const int z = d.slot[s];
                        const double c = z >= 0 ? P64[z] + lc[z * L + q] : NEG + lcg[s * N + k];
                        if (c > bv) { bv = c; bs = s; }
                    }
                    best = d.slot[bs] >= 0 ? d.slot[bs] : BP_STATE + bs;
                }
                v = bv + e;
            }
            const int z = ((t & 3) * R + r) * L + q;
            V[z] = v;
            V32[z] = screen32(v);
            bp[(int64_t)t * SB] = (uint8_t)best;
        }
        if (edge_out && j >= 0 && j <= Ly) {
            if (taken + HALO <= j) taken = wait_word(ch.taken, j - HALO + 1);
            O[(j & (HALO - 1)) * L + q] = v;
        }
        if (t == 3 && tid == 0) { V[0] = NEG; V32[0] = -FAR; }   // the origin's cells are done with the start
        compute_barrier(NT);
        if (tid == 0) ch.step = t;
    }
    if (last && tid == 0) {
        const double *fv = V + (((T - 1) & 3) * R + rows - 1) * L;
        const double *le = lcg + d.e_idx;
        int best = 0;
        double bv = fv[0] + le[0];
        for (int s = 1; s < N; ++s) {
            const int z = d.slot[s];
            const double c = (z >= 0 ? fv[z] : NEG) + le[(int64_t)s * N];
            if (c > bv) { bv = c; best = s; }
        }
        A.ll[p] = bv;
        A.fin[p] = best;
        if (!(bv > -1e29)) atomicOr(A.status + p, PHMM_ST_ZERO_LL);
    }
}

// Backpointer tiles of TILE x TILE cells ending at the current cell; thread 0
// walks inside the tile (a shared-memory load a step instead of an L2 round
// trip), the CTA loads the next one and writes the steps out.
constexpr int TB_THREADS = 128;
constexpr int TILE = 16;

__global__ void __launch_bounds__(TB_THREADS)
traceback_kernel(const __grid_constant__ Args A, int32_t *__restrict__ path, int32_t *__restrict__ path_len) {
    extern __shared__ uint32_t tile[];          // [TILE][TILE * SB / 4]
    __shared__ int steps[2 * TILE][3];
    __shared__ int s_i, s_j, s_k, s_n, s_done;
    const int p = blockIdx.x, tid = threadIdx.x;
    const Desc &d = A.d;
    const Meta m = A.meta[p];
    const int Lx = m.Lx, Ly = m.Ly, SB = bp_stride(d.ns), W = TILE * SB / 4;
    int32_t *pp = path + m.path_off * 3;
    const bool failed = (A.status[p] & PHMM_ST_TIMEOUT) != 0;   // the table is incomplete: no path
    if (tid == 0) {
        s_i = Lx; s_j = Ly; s_k = A.fin[p];
        s_done = failed || (Lx == 0 && Ly == 0);
        if (failed) A.ll[p] = NEG;
    }
    __syncthreads();
    int n = 0;                                  // triples written
    while (!s_done && n < Lx + Ly) {
        const int ci = s_i, cj = s_j, i0 = max(0, ci - TILE + 1), j0 = max(0, cj - TILE + 1);
        const int ni = ci - i0 + 1, words = (cj - j0 + 1) * (SB / 4);
        const uint32_t *src = (const uint32_t *)(A.tb + m.tab_off);
        for (int idx = tid; idx < ni * words; idx += TB_THREADS) {
            const int a = idx / words, b = idx % words;
            tile[a * W + b] = __ldcg(src + ((int64_t)(i0 + a) * (Ly + 1) + j0) * (SB / 4) + b);
        }
        __syncthreads();
        if (tid == 0) {
            const uint8_t *tb = (const uint8_t *)tile;
            int a = ci, b = cj, k = s_k, c = 0;
            bool done = false;
            while (a >= i0 && b >= j0 && !done && n + c < Lx + Ly) {
                steps[c][0] = a; steps[c][1] = b; steps[c][2] = k;
                ++c;
                const int st = d.type[k], z = d.slot[k];
                // a state that does not emit kept the reference's zero pointers
                const int from = z > 0 ? tb[((a - i0) * W) * 4 + (b - j0) * SB + z] : 0;
                if (from == BP_ORIGIN) { done = true; break; }
                // a state with no predecessor cell here (S/E, or M/I/D on the lattice
                // edge): the walk ends at the origin
                if (st == TM && a > 0 && b > 0) { --a; --b; }
                else if (st == TI && b > 0) { --b; }
                else if (st == TD && a > 0) { --a; }
                else { done = true; break; }
                k = from < BP_STATE ? d.state[from] : from - BP_STATE;
                if (a == 0 && b == 0) done = true;
            }
            s_i = a; s_j = b; s_k = k; s_n = c;
            s_done = done;
        }
        __syncthreads();
        for (int idx = tid; idx < 3 * s_n; idx += TB_THREADS) pp[3 * n + idx] = steps[idx / 3][idx % 3];
        n += s_n;
        __syncthreads();
    }
    if (tid == 0) {
        pp[3 * n] = 0; pp[3 * n + 1] = 0; pp[3 * n + 2] = 0;   // the origin, in the start state
        path_len[p] = n + 1;
    }
    ++n;
    __syncthreads();
    for (int a = tid; a < n / 2; a += TB_THREADS)
        for (int c = 0; c < 3; ++c) {
            const int32_t u = pp[3 * a + c], w = pp[3 * (n - 1 - a) + c];
            pp[3 * a + c] = w;
            pp[3 * (n - 1 - a) + c] = u;
        }
}

struct Shape {
    int lanes, rows;
};
// Lanes and rows of a stripe by slots: 256 threads (512 above 16 slots, where a
// row takes 32 or 64 lanes), the most that keep two stripes on an SM at 96
// registers a thread.
inline Shape shape_of(int ns) {
    if (ns <= 4) return {4, 64};
    if (ns <= 8) return {8, 32};
    if (ns <= 16) return {16, 16};
    if (ns <= 32) return {32, 16};
    return {64, 8};
}

template <int L, int R>
cudaError_t launch(const Args &a, int items, cudaStream_t st) {
    const size_t cells = 4 * R * L + HALO * L;
    const size_t smem = sizeof(double) * ((size_t)L * L + cells + HALO * L) + sizeof(float) * cells;
    auto kernel = a.env ? viterbi_stripe_kernel<L, R, true> : viterbi_stripe_kernel<L, R, false>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    kernel<<<items, L * R + 64, smem, st>>>(a);
    return cudaGetLastError();
}

}  // namespace vit

static int vit_fail(int code, const char *msg) {
    phmm_internal_set_error(msg);
    return code;
}

static size_t vit_align(size_t v) { return (v + 255) & ~(size_t)255; }

struct VitLayout {
    s64::Layout lay;
    size_t o_ctl, o_fin, o_edge, o_tb, total;
};

static int vit_layout(const phmm_batch *b, int ns, VitLayout &L) {
    const vit::Shape sh = vit::shape_of(ns);
    if (!L.lay.build(b, sh.rows, ns - 1)) return vit_fail(PHMM_E_ARG, "phmm_viterbi: negative length");
    int64_t tb = 0, pth = 0;
    for (s64::Meta &m : L.lay.meta) {
        m.tab_off = tb;
        m.path_off = pth;
        tb += (int64_t)(m.Lx + 1) * (m.Ly + 1) * vit::bp_stride(ns);
        pth += m.Lx + m.Ly + 1;
    }
    L.o_ctl = vit_align(L.lay.head_bytes());
    L.o_fin = vit_align(L.o_ctl + L.lay.ctl_bytes());
    L.o_edge = vit_align(L.o_fin + sizeof(int) * L.lay.meta.size());
    L.o_tb = vit_align(L.o_edge + sizeof(double) * (size_t)L.lay.edge_doubles);
    L.total = vit_align(L.o_tb + (size_t)tb);
    return PHMM_OK;
}

static int vit_model(const phmm_model_desc *model, vit::Desc &d, bool &has_ends) {
    const int N = model->n_states, G = model->n_groups;
    if (!model->state_types || !model->state_group) return vit_fail(PHMM_E_ARG, "phmm_viterbi: bad model description or batch");
    if (N < 2 || N > vit::MAXN) return vit_fail(PHMM_E_ARG, "phmm_viterbi: n_states must be in 2..64");
    if (G < 1) return vit_fail(PHMM_E_ARG, "phmm_viterbi: n_groups must be positive");
    has_ends = s64::make_desc(model, d);
    return PHMM_OK;
}

extern "C" int phmm_viterbi_workspace_bytes(const phmm_model_desc *model, const phmm_batch *batch, size_t *bytes) {
    if (!model || !batch || !bytes) return vit_fail(PHMM_E_ARG, "phmm_viterbi_workspace_bytes: null argument");
    *bytes = 0;
    if (batch->n_pairs <= 0) return PHMM_OK;
    if (!batch->Lx_host || !batch->Ly_host || !batch->x_off_host || !batch->y_off_host)
        return vit_fail(PHMM_E_ARG, "phmm_viterbi: null host length or offset array");
    vit::Desc d;
    bool has_ends;
    int rc = vit_model(model, d, has_ends);
    if (rc) return rc;
    VitLayout L;
    rc = vit_layout(batch, d.ns, L);
    if (rc) return rc;
    *bytes = L.total;
    return PHMM_OK;
}

extern "C" int phmm_viterbi(const phmm_model_desc *model, const phmm_batch *batch, const double *log_chi,
                            const double *log_emit_M, const double *log_emit_I, const double *log_emit_D,
                            void *workspace, size_t workspace_bytes, double *ll_out, int32_t *path,
                            int32_t *path_len, int32_t *status_out, void *stream) {
    using namespace vit;
    if (!model || !model->state_types || !model->state_group || !batch)
        return vit_fail(PHMM_E_ARG, "phmm_viterbi: bad model description or batch");
    Args a;
    bool has_ends;
    int rc = vit_model(model, a.d, has_ends);
    if (rc) return rc;
    const int P = batch->n_pairs;
    if (P < 0) return vit_fail(PHMM_E_ARG, "phmm_viterbi: negative n_pairs");
    if (P == 0) return PHMM_OK;
    if (!batch->Lx_host || !batch->Ly_host || !batch->x_off_host || !batch->y_off_host || !batch->residues ||
        !log_chi || !log_emit_M || !log_emit_I || !log_emit_D || !workspace || !ll_out || !path || !path_len ||
        !status_out)
        return vit_fail(PHMM_E_ARG, "phmm_viterbi: null pointer");
    if ((uintptr_t)workspace & 255) return vit_fail(PHMM_E_ARG, "phmm_viterbi: workspace must be 256-byte aligned");
    if (!has_ends) return vit_fail(PHMM_E_ARG, "phmm_viterbi: state 0 must be S and one state E");
    VitLayout L;
    rc = vit_layout(batch, a.d.ns, L);
    if (rc) return rc;
    if (workspace_bytes < L.total) return vit_fail(PHMM_E_ARG, "phmm_viterbi: workspace too small");
    cudaStream_t st = (cudaStream_t)stream;
    char *ws = (char *)workspace;
    const std::vector<char> head = L.lay.head();
    cudaError_t e = cudaMemcpyAsync(ws, head.data(), head.size(), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(ws + L.o_ctl, 0, L.lay.ctl_bytes(), st);
    if (e == cudaSuccess) e = cudaMemsetAsync(status_out, 0, sizeof(int32_t) * P, st);
    if (e != cudaSuccess) return vit_fail(PHMM_E_CUDA, cudaGetErrorString(e));
    a.meta = (const Meta *)ws;
    a.items = (const Item *)(ws + sizeof(Meta) * P);
    a.ctl = (int *)(ws + L.o_ctl);
    a.res = batch->residues;
    a.lchi = log_chi;
    a.lM = log_emit_M;
    a.lI = log_emit_I;
    a.lD = log_emit_D;
    a.chi_pp = batch->chi_per_pair;
    a.emit_pp = batch->emit_per_pair;
    a.edge = (double *)(ws + L.o_edge);
    a.tb = (uint8_t *)(ws + L.o_tb);
    a.fin = (int *)(ws + L.o_fin);
    a.ll = ll_out;
    a.status = status_out;
    a.env = batch->cell_mask;
    const int items = (int)L.lay.items.size();
    switch (shape_of(a.d.ns).lanes) {
        case 4: e = launch<4, 64>(a, items, st); break;
        case 8: e = launch<8, 32>(a, items, st); break;
        case 16: e = launch<16, 16>(a, items, st); break;
        case 32: e = launch<32, 16>(a, items, st); break;
        default: e = launch<64, 8>(a, items, st); break;
    }
    if (e != cudaSuccess) return vit_fail(PHMM_E_CUDA, cudaGetErrorString(e));
    traceback_kernel<<<P, TB_THREADS, TILE * TILE * bp_stride(a.d.ns), st>>>(a, path, path_len);
    e = cudaGetLastError();
    if (e != cudaSuccess) return vit_fail(PHMM_E_CUDA, cudaGetErrorString(e));
    return PHMM_OK;
}
