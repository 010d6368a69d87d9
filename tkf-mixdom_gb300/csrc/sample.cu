// sample.cu -- batched stochastic forward traceback of the 2D pair HMM
// (dp/hmm.py:2043-2101 sample_traceback_2d).
//
// Launches:
//   linear_kernel      exponentials of the log transition and emission tables,
//                      once per table;
//   forward_stripe_kernel  the forward recursion on the stripe wavefront of
//                      stripe64.cuh, float64 in probability space: every cell
//                      normalised by the power of two of its largest state (exact)
//                      with the exponent carried beside it, so a state costs one
//                      multiply-add per source instead of the reference's
//                      float64 exponential.  The table F keeps each cell's
//                      normalised states; the log-likelihood is
//                      log(sum_s F[Lx][Ly][s] chi[s][E]) plus the exponent;
//   fwdlog_kernel      only for pairs the first two marked (a finite log table
//                      entry below -230 or above 230, a state below 2^-300 of its
//                      cell's largest, a likelihood of zero): the same table in
//                      log space with the reference's arithmetic, one CTA per
//                      pair: F[i][j][k] = logsumexp_s (F[pred(k)][s] +
//                      logchi[s][k]) + logemit_k, NEG_INF (-1e30) summed like any
//                      other number;
//   sample_kernel      one thread per (pair, sample) walks back from (Lx, Ly): the
//                      final state with probability proportional to
//                      P(F[Lx][Ly][s]) chi[s][E], then at each cell the
//                      predecessor cell fixed by the current state's type (M: i-1,
//                      j-1; I: j-1; D: i-1) and its state with probability
//                      proportional to P(F[pred][s]) chi[s][k], until (0, 0) -- a
//                      cell's exponent cancels; the path is written from (0, 0, S)
//                      on, as the reference returns it.
//
// Random numbers: a counter-based stream, no state between launches.  Draw n
// of sample s of pair p is u = top 53 bits of mix(mix(seed + K (p * 2^32 +
// s)) + K n) / 2^53, mix the SplitMix64 output function (Steele, Lea and
// Flood, "Fast splittable pseudorandom number generators", OOPSLA 2014) and K
// its golden-ratio increment.  A state is chosen as the first index whose
// running sum of weights exceeds u times the total, the inverse-CDF rule; the
// reference draws with jax.random.choice (other numbers, the same
// distribution).
//
// Measured on 16 pairs of 60-300 residues at 5 states, 32 samples each: forward
// 17.1 -> 0.46 ms (one CTA per pair with a float64 exponential per source before),
// walks 2.06 -> 0.28 ms (two exponentials per source and step, each path turned
// round by its own thread before).
#include "stripe64.cuh"

extern "C" __attribute__((visibility("hidden"))) void phmm_internal_set_error(const char *msg);

namespace smp {

using namespace s64;

constexpr int NT = 256;
constexpr int ST = 128;          // sampler threads per CTA
constexpr double SAFE = 230.0;   // |log| of the table entries the probability-space recursion takes
constexpr int LOW = -300;        // smallest exponent of a state below its cell's largest
constexpr int NOEXP = -(1 << 28);   // exponent of a cell without probability
constexpr unsigned long long GOLDEN = 0x9e3779b97f4a7c15ULL;

struct Args {
    Desc d;
    const Meta *meta;
    const Item *items;
    int *ctl;      // claim counter, then one progress word per stripe
    int *flag;     // [P + 1] pairs that take the log-space kernel; the last word: all of them
    const uint8_t *res;
    const double *lchi, *lM, *lI, *lD;   // log tables
    double *chi, *eM, *eI, *eD;          // the same, linear
    int chi_pp, emit_pp, P;
    double *edge;
    double *F;
    double *ll;
    int32_t *status;
};

__host__ __device__ inline unsigned long long mix64(unsigned long long z) {
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ULL;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebULL;
    return z ^ (z >> 31);
}

__device__ inline double uniform(unsigned long long stream, unsigned long long n) {
    return (double)(mix64(stream + GOLDEN * n) >> 11) * (1.0 / 9007199254740992.0);
}

// First double of a pair's normalised table (ns states a cell): inside the N
// states a cell of its log-space table, which the two share.
__device__ __forceinline__ double *pair_table(const Args &A, const Meta &m) { return A.F + m.tab_off; }

// blockIdx.x: table (pair, or 0 when shared); blockIdx.y: 0 transitions, 1 emissions.
__global__ void __launch_bounds__(NT)
linear_kernel(const __grid_constant__ Args A) {
    const int t = blockIdx.x, NN = A.d.N * A.d.N;
    const bool trans = blockIdx.y == 0;
    const int pp = trans ? A.chi_pp : A.emit_pp;
    if (t > 0 && !pp) return;
    bool bad = false;
    auto lin = [&](double l) {
        if (l <= -1e29) return 0.0;             // NEG_INF
        if (!(fabs(l) <= SAFE)) bad = true;
        return exp(l);
    };
    if (trans) {
        for (int i = threadIdx.x; i < NN; i += NT) A.chi[(int64_t)t * NN + i] = lin(A.lchi[(int64_t)t * NN + i]);
    } else {
        const int G = A.d.G;
        const int64_t oM = (int64_t)t * G * 441, o1 = (int64_t)t * G * 21;
        for (int i = threadIdx.x; i < G * 441; i += NT) A.eM[oM + i] = lin(A.lM[oM + i]);
        for (int i = threadIdx.x; i < G * 21; i += NT) {
            A.eI[o1 + i] = lin(A.lI[o1 + i]);
            A.eD[o1 + i] = lin(A.lD[o1 + i]);
        }
    }
    if (bad) A.flag[pp ? t : A.P] = 1;
}

// L lanes per row, R rows per stripe, DPT states per lane (slots q, q + L).
// FP64 work bounds a step (two lanes per SM and clock): ns - 1 multiply-adds
// for each of the row's states, so R is small, comparisons and powers of two are
// integer operations, and the transitions are read from shared memory (their
// loads cost an eighth of the multiply-adds).
template <int L, int R, int DPT>
__global__ void __launch_bounds__(L * R + 64)
forward_stripe_kernel(const __grid_constant__ Args A) {
    constexpr int NT = L * R, W = L * DPT;      // W: slots per row
    constexpr int ZH = 4 * R;                   // cells of the step ring; then HALO cells of the row above
    extern __shared__ __align__(16) double smem[];
    double *lc = smem;                          // [W][W] transitions by source and destination slot
    double *V = lc + W * W;                     // [ZH + HALO][W] normalised states
    double *O = V + (ZH + HALO) * W;            // [HALO][W] the last row, for the publisher: exponent, states
    __shared__ int VE[ZH + HALO];               // exponents of those cells
    __shared__ Channel ch;
    const int tid = threadIdx.x;
    const Desc &d = A.d;
    const int N = d.N, ns = d.ns;
    if (tid == 0) {
        ch.avail = ch.taken = 0;
        ch.step = -1;
    }
    const Item it = claim(A.ctl, A.items);      // (barrier)
    const int p = it.pair;
    const Meta m = A.meta[p];
    const int Lx = m.Lx, Ly = m.Ly;
    const double *chi = A.chi + (A.chi_pp ? (int64_t)p * N * N : 0);
    for (int idx = tid; idx < W * W; idx += NT + 64) {
        const int a = idx / W, b = idx % W;
        lc[idx] = (a < ns && b < ns) ? chi[d.state[a] * N + d.state[b]] : 0.0;
    }
    for (int idx = tid; idx < (ZH + HALO) * W; idx += NT + 64) V[idx] = 0.0;
    for (int idx = tid; idx < ZH + HALO; idx += NT + 64) VE[idx] = NOEXP;
    __syncthreads();
    const bool last = it.stripe == m.n_stripes - 1;
    int *prog = A.ctl + 1 + m.stripe0 + it.stripe;
    const int er = ns;                          // doubles of an edge column: the exponent and the states
    if (tid >= NT) {                            // hand-off warps
        if (tid < NT + 32) {
            if (it.stripe > 0)
                load_edges(A.edge + m.edge_off + (int64_t)(it.stripe - 1) * (Ly + 1) * er, er, Ly, prog - 1, ch,
                           A.status + p, [&](int c, int k, double v) {
                               const int z = ZH + (c & (HALO - 1));
                               if (k > 0) V[z * W + k] = v;
                               else VE[z] = (int)v;
                           });
        } else if (!last) {
            publish_edges(A.edge + m.edge_off + (int64_t)it.stripe * (Ly + 1) * er, er, R, Ly, prog, ch,
                          [&](int c, int k) { return O[(c & (HALO - 1)) * W + k]; });
        }
        return;
    }
    const int r = tid / L, q = tid % L;
    const int i = it.stripe * R + r;
    const int rows = last ? Lx + 1 - it.stripe * R : R;
    const int T = Ly + rows;
    const bool row_in = r < rows;
    const uint8_t *x = A.res + m.x_off, *y = A.res + m.y_off;
    const int xa = (row_in && i > 0) ? min((int)x[i - 1], 20) : 0;
    const int64_t ep = A.emit_pp ? p : 0;
    int jlo[DPT];                               // first column with a predecessor (past Ly: none)
    int pbase[DPT], poff[DPT], pmask[DPT], pstr[DPT];   // its cell at step t: pbase + ((t + poff) & pmask) * pstr
    int org[DPT];                               // column whose predecessor is the origin, or -1
    bool fixed[DPT];                            // emission independent of the column (deletions)
    const double *eb[DPT];
    double e1[DPT];
#pragma unroll
    for (int z = 0; z < DPT; ++z) {
        const int sl = q + z * L, k = sl < ns ? d.state[sl] : 0, g = d.group[k];
        const int st = sl > 0 && sl < ns ? d.type[k] : TS;
        const bool valid = row_in && (st == TI || ((st == TM || st == TD) && i > 0));
        const bool halo = st != TI && r == 0;
        jlo[z] = !valid ? Ly + 1 : st == TD ? 0 : 1;
        pbase[z] = halo ? ZH : st != TI ? r - 1 : r;
        poff[z] = halo ? (st == TM ? -1 : 0) : (st == TM ? -2 : -1);
        pmask[z] = halo ? HALO - 1 : 3;
        pstr[z] = halo ? 1 : R;
        org[z] = st == TI && i == 0 ? 1 : st == TM && i == 1 ? 1 : st == TD && i == 1 ? 0 : -1;
        fixed[z] = st == TD;
        eb[z] = st == TI ? A.eI + (ep * d.G + g) * 21 : st == TD ? A.eD + (ep * d.G + g) * 21 + xa
                                                                : A.eM + (ep * d.G + g) * 441 + xa * 21;
        e1[z] = valid && st == TD ? __ldg(eb[z]) : 0.0;
    }
    const bool waits = it.stripe > 0 && r == 0;
    double *out = pair_table(A, m) + ((int64_t)i * (Ly + 1) - r) * ns + q;
    const bool edge_out = !last && r == R - 1;
    int c1 = row_in && r == 0 && Ly > 0 ? min((int)y[0], 20) : 0;   // character of column j + 1
    int have = 0, taken = 0;
    bool odd = false;                           // a state left the range of the normalised table
    for (int t = 0; t < T; ++t) {
        const int j = t - r;
        double e[DPT];
#pragma unroll
        for (int z = 0; z < DPT; ++z) {
            e[z] = e1[z];
            if (jlo[z] == 1 && !fixed[z] && j >= 0 && j < Ly) e1[z] = __ldg(eb[z] + c1);
        }
        if (row_in && j >= -1 && j + 1 < Ly) c1 = min((int)__ldg(y + j + 1), 20);
        if (waits && have <= min(t, Ly)) have = wait_word(ch.avail, min(t, Ly) + 1);
        const bool act = row_in && j >= 0 && j <= Ly;
        double v[DPT];
        int ex[DPT], top = NOEXP;               // exponents: of the value, of the row's largest
#pragma unroll
        for (int z = 0; z < DPT; ++z) {
            const int sl = q + z * L;
            v[z] = 0.0;
            ex[z] = NOEXP;
            if (act && j >= jlo[z]) {
                const int cell = pbase[z] + ((t + poff[z]) & pmask[z]) * pstr[z];
                const double *pv = V + cell * W;
                double a0 = pv[1 % W] * lc[(1 % W) * W + sl], a1 = 0.0;
#pragma unroll
                for (int s = 2; s < W; ++s) {
                    if (W <= 8 || s < ns) {
                        if (W <= 8 || (s & 1)) a0 = fma(pv[s], lc[s * W + sl], a0);
                        else a1 = s == 2 ? pv[s] * lc[s * W + sl] : fma(pv[s], lc[s * W + sl], a1);
                    }
                }
                if (W > 8) a0 += a1;
                if (j == org[z]) a0 = fma(pv[0], lc[sl], a0);   // the start is a source beside the origin only
                v[z] = a0 * e[z];
                const int hi = __double2hiint(v[z]);
                if (hi > 0) ex[z] = (hi >> 20) - 1022 + VE[cell];
                if ((hi & 0x7fffffff) >= 0x7e300000) odd = true;   // not a number, or beyond 1e300
            } else if (act && i == 0 && j == 0 && sl == 0) {
                v[z] = 1.0;
                ex[z] = 1;
            }
            top = max(top, ex[z]);
        }
#pragma unroll
        for (int o = L / 2; o > 0; o >>= 1) top = max(top, __shfl_xor_sync(0xffffffffu, top, o, L));
        if (act) {
            const int cell = (t & 3) * R + r;
            if (edge_out && taken + HALO <= j) taken = wait_word(ch.taken, j - HALO + 1);
#pragma unroll
            for (int z = 0; z < DPT; ++z) {
                const int sl = q + z * L;
                if (ex[z] > NOEXP) {            // exact: a power of two
                    const int rel = ex[z] - top, hi = __double2hiint(v[z]);
                    if (rel < LOW) odd = true;
                    v[z] = rel < LOW ? 0.0 : __hiloint2double((hi & 0xfffff) | ((rel + 1022) << 20), __double2loint(v[z]));
                }
                V[cell * W + sl] = v[z];
                if (sl < ns) out[(int64_t)t * ns + z * L] = v[z];
                if (edge_out && sl > 0) O[(j & (HALO - 1)) * W + sl] = v[z];
            }
            if (q == 0) {
                VE[cell] = top;
                if (edge_out) O[(j & (HALO - 1)) * W] = (double)top;
            }
        }
        compute_barrier(NT);
        if (tid == 0) ch.step = t;
    }
    if (odd) A.flag[p] = 1;
    if (last && tid == 0) {
        const int cell = ((T - 1) & 3) * R + rows - 1;
        const double *fv = V + cell * W;
        double sum = 0.0;
        for (int s = 0; s < ns; ++s) sum += fv[s] * chi[d.state[s] * N + d.e_idx];
        const bool ok = sum > 0.0;
        A.ll[p] = ok ? log(sum) + 0.69314718055994530942 * (double)VE[cell] : NEG;
        if (!ok) A.flag[p] = 1;
    }
}

__global__ void __launch_bounds__(NT)
fwdlog_kernel(const __grid_constant__ Args A) {
    extern __shared__ double lchi[];   // [N][N]
    const int p = blockIdx.x, tid = threadIdx.x;
    if (!(A.flag[p] | A.flag[A.P])) return;
    const Meta m = A.meta[p];
    const Desc &d = A.d;
    const uint8_t *res = A.res;
    const int N = d.N, G = d.G, emit_pp = A.emit_pp;
    const double *lM = A.lM, *lI = A.lI, *lD = A.lD;
    const double *lc = A.lchi + (A.chi_pp ? (int64_t)p * N * N : 0);
    for (int idx = tid; idx < N * N; idx += NT) lchi[idx] = lc[idx];
    const double *eM = lM + (emit_pp ? (int64_t)p * G * 441 : 0);
    const double *eI = lI + (emit_pp ? (int64_t)p * G * 21 : 0);
    const double *eD = lD + (emit_pp ? (int64_t)p * G * 21 : 0);
    const int Lx = m.Lx, Ly = m.Ly;
    double *Fp = pair_table(A, m);
    __syncthreads();
    for (int dd = 0; dd <= Lx + Ly; ++dd) {
        const int i_lo = max(0, dd - Ly), i_hi = min(dd, Lx);
        const int ncell = i_hi - i_lo + 1;
        for (int item = tid; item < ncell * N; item += NT) {
            const int i = i_lo + item / N, k = item % N, j = dd - i;
            double *out = Fp + ((int64_t)i * (Ly + 1) + j) * N + k;
            if (dd == 0) {
                *out = k == 0 ? 0.0 : NEG;
                continue;
            }
            const int st = d.type[k];
            const double *pred = nullptr;
            if (st == TM && i > 0 && j > 0) pred = Fp + ((int64_t)(i - 1) * (Ly + 1) + j - 1) * N;
            else if (st == TI && j > 0) pred = Fp + ((int64_t)i * (Ly + 1) + j - 1) * N;
            else if (st == TD && i > 0) pred = Fp + ((int64_t)(i - 1) * (Ly + 1) + j) * N;
            if (!pred) {
                *out = NEG;
                continue;
            }
            double mx = pred[0] + lchi[k];
            for (int s = 1; s < N; ++s) mx = fmax(mx, pred[s] + lchi[s * N + k]);
            double sum = 0.0;
            for (int s = 0; s < N; ++s) sum += exp(pred[s] + lchi[s * N + k] - mx);
            const int xa = i > 0 ? min((int)res[m.x_off + i - 1], 20) : 0;
            const int yb = j > 0 ? min((int)res[m.y_off + j - 1], 20) : 0;
            const int g = d.group[k];
            double e;
            if (st == TM) e = eM[g * 441 + xa * 21 + yb];
            else if (st == TI) e = eI[g * 21 + yb];
            else e = eD[g * 21 + xa];
            *out = mx + log(sum) + e;
        }
        __syncthreads();
    }
    if (tid == 0) {
        const double *last = Fp + ((int64_t)Lx * (Ly + 1) + Ly) * N;
        double mx = last[0] + lchi[d.e_idx];
        for (int s = 1; s < N; ++s) mx = fmax(mx, last[s] + lchi[s * N + d.e_idx]);
        double sum = 0.0;
        for (int s = 0; s < N; ++s) sum += exp(last[s] + lchi[s * N + d.e_idx] - mx);
        const double ll = mx + log(sum);
        A.ll[p] = ll;
        if (!(ll > -1e29)) atomicOr(A.status + p, PHMM_ST_ZERO_LL);
    }
}

// Log-space draw of a marked pair: the state of the cell whose table entry is
// f, before a state reached over the transitions lc (stride N), with
// probability proportional to exp(f[s] + lc[s N]).
__device__ __noinline__ int draw_log(const double *f, const double *lc, int N, double u) {
    double mx = f[0] + lc[0];
    for (int s = 1; s < N; ++s) mx = fmax(mx, f[s] + lc[s * N]);
    double tot = 0.0;
    for (int s = 0; s < N; ++s) tot += exp(f[s] + lc[s * N] - mx);
    const double target = u * tot;
    double cum = 0.0;
    for (int s = 0; s < N; ++s) {
        cum += exp(f[s] + lc[s * N] - mx);
        if (cum > target) return s;
    }
    return N - 1;
}

// W: bound of the slots of a cell (its weights stay in registers).
template <int W>
__global__ void __launch_bounds__(ST)
sample_kernel(const __grid_constant__ Args A, int n_samples, unsigned long long seed, int32_t *__restrict__ paths,
              int32_t *__restrict__ path_len) {
    extern __shared__ double chs[];   // [N][W] linear transitions by destination state and source slot
    __shared__ int lens[ST];
    const Desc &d = A.d;
    const int p = blockIdx.x, tid = threadIdx.x, smp0 = blockIdx.y * ST, smp = smp0 + tid;
    const Meta m = A.meta[p];
    const int N = d.N, ns = d.ns, Lx = m.Lx, Ly = m.Ly;
    const bool logs = (A.flag[p] | A.flag[A.P]) != 0;   // the pair's table holds logs
    const bool failed = (A.status[p] & PHMM_ST_TIMEOUT) != 0;
    const double *lc = A.lchi + (A.chi_pp ? (int64_t)p * N * N : 0);
    const double *ch = A.chi + (A.chi_pp ? (int64_t)p * N * N : 0);
    for (int idx = tid; idx < N * W; idx += ST) chs[idx] = idx % W < ns ? ch[d.state[idx % W] * N + idx / W] : 0.0;
    __syncthreads();
    const double *Fp = pair_table(A, m);
    const int slot = Lx + Ly + 1;
    int32_t *base = paths + 3 * m.path_off;
    if (smp < n_samples) {
        int32_t *pp = base + 3 * (int64_t)smp * slot;
        const unsigned long long stream = mix64(seed + GOLDEN * (((unsigned long long)p << 32) | (unsigned)smp));
        unsigned long long n = 0;
        // the state of `cell` before which the walk is in state `to`
        auto pick = [&](int64_t cell, int to) {
            const double u = uniform(stream, n++);
            if (logs) return draw_log(Fp + cell * N, lc + to, N, u);
            const double *f = Fp + cell * ns, *c = chs + to * W;
            double v[W], tot = 0.0;
#pragma unroll
            for (int s = 0; s < W; ++s) v[s] = s < ns ? f[s] : 0.0;
#pragma unroll
            for (int s = 0; s < W; ++s) {
                v[s] *= c[s];
                tot += v[s];
            }
            const double target = u * tot;
            double cum = 0.0;
            int got = -1;
#pragma unroll
            for (int s = 0; s < W; ++s) {
                cum += v[s];
                if (got < 0 && cum > target) got = s;
            }
            return got < 0 ? N - 1 : (int)d.state[got];
        };
        int ci = failed ? 0 : Lx, cj = failed ? 0 : Ly, len = 0, ck = 0;
        if (!failed) ck = pick((int64_t)Lx * (Ly + 1) + Ly, d.e_idx);
        while ((ci > 0 || cj > 0) && len < Lx + Ly) {
            pp[3 * len] = ci; pp[3 * len + 1] = cj; pp[3 * len + 2] = ck;
            ++len;
            const int st = d.type[ck];
            int pi_, pj_;
            if (st == TM && ci > 0 && cj > 0) { pi_ = ci - 1; pj_ = cj - 1; }
            else if (st == TI && cj > 0) { pi_ = ci; pj_ = cj - 1; }
            else if (st == TD && ci > 0) { pi_ = ci - 1; pj_ = cj; }
            else break;
            ck = pick((int64_t)pi_ * (Ly + 1) + pj_, ck);
            ci = pi_;
            cj = pj_;
        }
        pp[3 * len] = 0; pp[3 * len + 1] = 0; pp[3 * len + 2] = 0;   // the origin, in the start state
        ++len;
        lens[tid] = len;
        path_len[(int64_t)p * n_samples + smp] = len;
    }
    if (failed && smp0 == 0 && tid == 0) A.ll[p] = NEG;
    __syncthreads();
    // the warps turn the paths round
    for (int s = tid >> 5; s < ST && smp0 + s < n_samples; s += ST / 32) {
        int32_t *pp = base + 3 * (int64_t)(smp0 + s) * slot;
        const int len = lens[s];
        for (int a = tid & 31; a < len / 2; a += 32)
            for (int c = 0; c < 3; ++c) {
                const int32_t u = pp[3 * a + c], w = pp[3 * (len - 1 - a) + c];
                pp[3 * a + c] = w;
                pp[3 * (len - 1 - a) + c] = u;
            }
    }
}

struct Shape {
    int lanes, rows;
};
// Lanes and rows of a stripe by slots: 128 threads (256 above 16 slots), few rows so
// that the FP64 work of a step, R x lanes x slots / 2 clocks, stays near its latency.
inline Shape shape_of(int ns) {
    if (ns <= 4) return {4, 32};
    if (ns <= 8) return {8, 16};
    if (ns <= 16) return {16, 8};
    return {32, 8};
}

template <int L, int R, int DPT>
cudaError_t launch(const Args &a, int items, cudaStream_t st) {
    constexpr int W = L * DPT;
    const size_t smem = sizeof(double) * ((size_t)W * W + (4 * R + 2 * HALO) * W);
    cudaError_t e = cudaFuncSetAttribute(forward_stripe_kernel<L, R, DPT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    forward_stripe_kernel<L, R, DPT><<<items, L * R + 64, smem, st>>>(a);
    return cudaGetLastError();
}

}  // namespace smp

static int smp_fail(int code, const char *msg) {
    phmm_internal_set_error(msg);
    return code;
}

static size_t smp_align(size_t v) { return (v + 255) & ~(size_t)255; }

struct SmpLayout {
    s64::Layout lay;
    size_t o_ctl, ctl_bytes, o_lin, o_edge, o_F, total;
};

// doubles of the linear tables of the batch
static size_t smp_linear(const phmm_batch *b, int N, int G, size_t *n_chi) {
    const size_t P = (size_t)b->n_pairs;
    *n_chi = (b->chi_per_pair ? P : 1) * N * N;
    return *n_chi + (b->emit_per_pair ? P : 1) * G * (441 + 42);
}

static int smp_layout(const phmm_batch *b, const smp::Desc &d, int n_samples, SmpLayout &L) {
    if (!L.lay.build(b, smp::shape_of(d.ns).rows, d.ns)) return smp_fail(PHMM_E_ARG, "phmm_sample_paths: negative length");
    int64_t f = 0, pth = 0;
    for (s64::Meta &m : L.lay.meta) {
        m.tab_off = f;
        m.path_off = pth;
        f += (int64_t)(m.Lx + 1) * (m.Ly + 1) * d.N;
        pth += (int64_t)n_samples * (m.Lx + m.Ly + 1);
    }
    size_t n_chi;
    L.o_ctl = smp_align(L.lay.head_bytes());
    L.ctl_bytes = L.lay.ctl_bytes() + sizeof(int) * (L.lay.meta.size() + 1);   // with the flags
    L.o_lin = smp_align(L.o_ctl + L.ctl_bytes);
    L.o_edge = smp_align(L.o_lin + sizeof(double) * smp_linear(b, d.N, d.G, &n_chi));
    L.o_F = smp_align(L.o_edge + sizeof(double) * (size_t)L.lay.edge_doubles);
    L.total = smp_align(L.o_F + sizeof(double) * (size_t)f);
    return PHMM_OK;
}

// The checks of a model that come before the batch's; has_ends: state 0 is S and some state E.
static int smp_model(const phmm_model_desc *model, smp::Desc &d, bool &has_ends) {
    if (!model->state_types || !model->state_group)
        return smp_fail(PHMM_E_ARG, "phmm_sample_paths: bad model description or batch");
    if (model->n_states < 2 || model->n_states > smp::MAXN)
        return smp_fail(PHMM_E_ARG, "phmm_sample_paths: n_states must be in 2..64");
    if (model->n_groups < 1) return smp_fail(PHMM_E_ARG, "phmm_sample_paths: n_groups must be positive");
    has_ends = s64::make_desc(model, d);
    return PHMM_OK;
}

extern "C" int phmm_sample_workspace_bytes(const phmm_model_desc *model, const phmm_batch *batch, size_t *bytes) {
    if (!model || !batch || !bytes) return smp_fail(PHMM_E_ARG, "phmm_sample_workspace_bytes: null argument");
    *bytes = 0;
    if (batch->n_pairs <= 0) return PHMM_OK;
    if (!batch->Lx_host || !batch->Ly_host || !batch->x_off_host || !batch->y_off_host)
        return smp_fail(PHMM_E_ARG, "phmm_sample_paths: null host length or offset array");
    smp::Desc d;
    bool has_ends;
    int rc = smp_model(model, d, has_ends);
    if (rc) return rc;
    SmpLayout L;
    rc = smp_layout(batch, d, 0, L);
    if (rc) return rc;
    *bytes = L.total;
    return PHMM_OK;
}

extern "C" int phmm_sample_paths(const phmm_model_desc *model, const phmm_batch *batch, const double *log_chi,
                                 const double *log_emit_M, const double *log_emit_I, const double *log_emit_D,
                                 int32_t n_samples, uint64_t seed, void *workspace, size_t workspace_bytes,
                                 double *ll_out, int32_t *paths, int32_t *path_len, int32_t *status_out,
                                 void *stream) {
    using namespace smp;
    if (!model || !model->state_types || !model->state_group || !batch)
        return smp_fail(PHMM_E_ARG, "phmm_sample_paths: bad model description or batch");
    Args a;
    bool has_ends;
    int rc = smp_model(model, a.d, has_ends);
    if (rc) return rc;
    const int N = model->n_states, G = model->n_groups, P = batch->n_pairs;
    if (P < 0 || n_samples < 0) return smp_fail(PHMM_E_ARG, "phmm_sample_paths: negative n_pairs or n_samples");
    if (P == 0) return PHMM_OK;
    if (n_samples > 65535 * ST)
        return smp_fail(PHMM_E_ARG, "phmm_sample_paths: at most 8388480 samples per pair in one call");
    if (!batch->Lx_host || !batch->Ly_host || !batch->x_off_host || !batch->y_off_host || !batch->residues ||
        !log_chi || !log_emit_M || !log_emit_I || !log_emit_D || !workspace || !ll_out || !status_out ||
        (n_samples > 0 && (!paths || !path_len)))
        return smp_fail(PHMM_E_ARG, "phmm_sample_paths: null pointer");
    if ((uintptr_t)workspace & 255)
        return smp_fail(PHMM_E_ARG, "phmm_sample_paths: workspace must be 256-byte aligned");
    if (!has_ends) return smp_fail(PHMM_E_ARG, "phmm_sample_paths: state 0 must be S and one state E");
    SmpLayout L;
    rc = smp_layout(batch, a.d, n_samples, L);
    if (rc) return rc;
    if (workspace_bytes < L.total) return smp_fail(PHMM_E_ARG, "phmm_sample_paths: workspace too small");
    cudaStream_t st = (cudaStream_t)stream;
    char *ws = (char *)workspace;
    const std::vector<char> head = L.lay.head();
    cudaError_t e = cudaMemcpyAsync(ws, head.data(), head.size(), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(ws + L.o_ctl, 0, L.ctl_bytes, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(status_out, 0, sizeof(int32_t) * P, st);
    if (e != cudaSuccess) return smp_fail(PHMM_E_CUDA, cudaGetErrorString(e));
    size_t n_chi;
    smp_linear(batch, N, G, &n_chi);
    const size_t n_emit = (size_t)(batch->emit_per_pair ? P : 1) * G;
    a.meta = (const Meta *)ws;
    a.items = (const Item *)(ws + sizeof(Meta) * P);
    a.ctl = (int *)(ws + L.o_ctl);
    a.flag = a.ctl + L.lay.ctl_bytes() / sizeof(int);
    a.res = batch->residues;
    a.lchi = log_chi;
    a.lM = log_emit_M;
    a.lI = log_emit_I;
    a.lD = log_emit_D;
    a.chi = (double *)(ws + L.o_lin);
    a.eM = a.chi + n_chi;
    a.eI = a.eM + n_emit * 441;
    a.eD = a.eI + n_emit * 21;
    a.chi_pp = batch->chi_per_pair;
    a.emit_pp = batch->emit_per_pair;
    a.P = P;
    a.edge = (double *)(ws + L.o_edge);
    a.F = (double *)(ws + L.o_F);
    a.ll = ll_out;
    a.status = status_out;
    const bool per_pair = a.chi_pp || a.emit_pp;
    linear_kernel<<<dim3(per_pair ? P : 1, 2), NT, 0, st>>>(a);
    const int items = (int)L.lay.items.size();
    switch (a.d.ns <= 32 ? shape_of(a.d.ns).lanes : 64) {
        case 4: e = launch<4, 32, 1>(a, items, st); break;
        case 8: e = launch<8, 16, 1>(a, items, st); break;
        case 16: e = launch<16, 8, 1>(a, items, st); break;
        case 32: e = launch<32, 8, 1>(a, items, st); break;
        default: e = launch<32, 8, 2>(a, items, st); break;
    }
    if (e != cudaSuccess) return smp_fail(PHMM_E_CUDA, cudaGetErrorString(e));
    const size_t smem = sizeof(double) * N * N;
    e = cudaFuncSetAttribute(fwdlog_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return smp_fail(PHMM_E_CUDA, cudaGetErrorString(e));
    fwdlog_kernel<<<P, NT, smem, st>>>(a);
    if (n_samples > 0) {
        dim3 grid(P, (n_samples + ST - 1) / ST);
        const int W = a.d.ns <= 4 ? 4 : a.d.ns <= 16 ? 16 : 64;
        auto kernel = W == 4 ? sample_kernel<4> : W == 16 ? sample_kernel<16> : sample_kernel<64>;
        kernel<<<grid, ST, sizeof(double) * N * W, st>>>(a, n_samples, (unsigned long long)seed, paths, path_len);
    }
    e = cudaGetLastError();
    if (e != cudaSuccess) return smp_fail(PHMM_E_CUDA, cudaGetErrorString(e));
    return PHMM_OK;
}
