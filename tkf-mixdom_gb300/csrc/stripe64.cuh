// stripe64.cuh -- shared parts of the float64 stripe wavefronts of the
// decoders (viterbi.cu, sample.cu).
//
// The lattice rows of a pair are cut into stripes of R rows, one CTA per stripe:
// L x R compute threads and two hand-off warps.  Lane q of a row owns one
// emitting state (slot q; slot 0 is the start state), and at step t row r works
// on column t - r, so the three predecessor cells of every cell are one or two
// steps old and sit in a ring of four shared-memory steps.  One barrier of the
// compute warps per step.  The last row of a stripe passes through a shared ring
// to the publisher warp, which writes it to an edge buffer in global memory and
// releases its progress; the loader warp of the stripe below brings the columns
// into a shared ring HALO deep.  The hand-off's fences and L2 round trips
// (1-2 us) thus cost the wavefront a few columns of lag per stripe and no step
// waits for them (done by the compute threads every four columns, a stripe's step
// took 1.33 us instead of 0.87 at 17 states, 1.34 instead of 0.62 in the sampler's
// forward at 5).
//
// What bounds a step then is one warp's chain of dependent instructions (about
// five clocks each; a lone 7-row stripe of the 5-state Viterbi takes 0.42 us a
// step, with its FP64 pipe 4 % busy), so the wavefront's time is the longest
// pair's steps, Ly + stripes x (R + lag).
//
// Stripes are claimed from an atomic counter in list order (longest pairs
// first, a pair's stripes top down).  A stripe waits only for the stripe claimed
// before it of the same pair, so the wait ends whatever the residency; it is
// bounded all the same (WAIT_POLLS), and a stripe that gives up marks the pair
// PHMM_ST_TIMEOUT and runs on without waiting.
#pragma once
#include "pairhmm.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <vector>

namespace s64 {

constexpr int MAXN = 64;
constexpr double NEG = -1e30;   // the reference's NEG_INF (dp/hmm.py:108)
constexpr int TS = 0, TM = 1, TI = 2, TD = 3, TE = 4;
constexpr int HALO = 16;                      // columns of the row above kept in shared memory
constexpr int PUBLISH = 4;                    // columns per release
constexpr int WAIT_POLLS = 40 * 1000 * 1000;  // about 5 s

struct Meta {
    int64_t x_off, y_off;
    int64_t tab_off;    // first byte (Viterbi) or double (sampler) of the pair's table
    int64_t edge_off;   // first double of the pair's edge rows
    int64_t path_off, mask_off;
    int32_t Lx, Ly, stripe0, n_stripes;
};

struct Item {
    int32_t pair, stripe;
};

// The state space: slot 0 the start, slots 1..ns-1 the M/I/D states in state
// order (a maximum's first state is then its first slot).
struct Desc {
    int N, G, e_idx, ns;
    int8_t type[MAXN], group[MAXN];   // by state
    int8_t state[MAXN], slot[MAXN];   // state of a slot; slot of a state or -1
};

inline bool make_desc(const phmm_model_desc *m, Desc &d) {
    std::memset(&d, 0, sizeof(d));
    d.N = m->n_states;
    d.G = m->n_groups;
    d.e_idx = -1;
    d.ns = 1;
    for (int s = 0; s < d.N; ++s) {
        d.type[s] = m->state_types[s];
        d.group[s] = (int8_t)std::max(0, std::min(d.G - 1, (int)m->state_group[s]));
        d.slot[s] = -1;
        if (d.type[s] == TE && d.e_idx < 0) d.e_idx = s;
        if (s > 0 && d.type[s] >= TM && d.type[s] <= TD) {
            d.slot[s] = (int8_t)d.ns;
            d.state[d.ns++] = (int8_t)s;
        }
    }
    d.slot[0] = 0;
    return d.type[0] == TS && d.e_idx >= 0;
}

// Per-pair offsets and the work list, uploaded in one copy; `rows` rows per
// stripe, `edge_rec` doubles per edge column.  tab_off and path_off are the caller's.
struct Layout {
    std::vector<Meta> meta;
    std::vector<Item> items;
    int64_t edge_doubles = 0;

    bool build(const phmm_batch *b, int rows, int edge_rec) {
        const int P = b->n_pairs;
        meta.resize(P);
        int64_t mk = 0;
        int st = 0;
        std::vector<int> order(P);
        for (int p = 0; p < P; ++p) {
            const int Lx = b->Lx_host[p], Ly = b->Ly_host[p];
            if (Lx < 0 || Ly < 0) return false;
            const int n = Lx / rows + 1;
            meta[p] = Meta{b->x_off_host[p], b->y_off_host[p], 0, edge_doubles, 0, mk, Lx, Ly, st, n};
            mk += (int64_t)(Lx + 1) * (Ly + 1);
            edge_doubles += (int64_t)(n - 1) * (Ly + 1) * edge_rec;
            st += n;
            order[p] = p;
        }
        std::stable_sort(order.begin(), order.end(), [&](int a, int c) {
            return (int64_t)meta[a].Lx + meta[a].Ly > (int64_t)meta[c].Lx + meta[c].Ly;
        });
        items.reserve(st);
        for (int p : order)
            for (int s = 0; s < meta[p].n_stripes; ++s) items.push_back(Item{p, s});
        return true;
    }
    size_t head_bytes() const { return sizeof(Meta) * meta.size() + sizeof(Item) * items.size(); }
    // claim counter and one progress word per stripe
    size_t ctl_bytes() const { return sizeof(int) * (1 + items.size()); }
    std::vector<char> head() const {
        std::vector<char> h(head_bytes());
        if (!meta.empty()) std::memcpy(h.data(), meta.data(), sizeof(Meta) * meta.size());
        if (!items.empty()) std::memcpy(h.data() + sizeof(Meta) * meta.size(), items.data(), sizeof(Item) * items.size());
        return h;
    }
};

__device__ __forceinline__ int ld_acquire(const int *p) {
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void st_release(int *p, int v) {
    asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Shared words between the compute and hand-off warps of a CTA: columns of the
// row above that are in the ring, the last step every compute thread has done,
// and columns of the last row that the publisher has taken.  Only shared memory
// passes through these words, in the order of the step's barrier, so the compute
// warps execute no fence.
struct Channel {
    volatile int avail, step, taken;
};

__device__ __forceinline__ void compute_barrier(int threads) { asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory"); }

// Waits until a channel word reaches `need` (it always does: the hand-off warps
// give up after WAIT_POLLS and then pass on whatever is there).
__device__ __forceinline__ int wait_word(const volatile int &word, int need) {
    int have = word;
    for (long long n = 0; have < need && n < 16LL * WAIT_POLLS; ++n) have = word;
    asm volatile("" ::: "memory");
    return have;
}

// The loader warp: columns 0..Ly of `er` doubles each, handed to put(column,
// index, value) once the stripe above has released them and the ring has room.
template <class Put>
__device__ __forceinline__ void load_edges(const double *edge, int er, int Ly, const int *above, Channel &ch,
                                           int32_t *status, Put put) {
    const int lane = threadIdx.x & 31;
    int c = 0, have = 0, polls = 0;
    while (c <= Ly) {
        // a step reads columns t and t - 1: those below the last done step are free
        const int room = min(__shfl_sync(0xffffffffu, ch.step, 0) + HALO, Ly + 1);
        if (have <= c) have = __shfl_sync(0xffffffffu, ld_acquire(above), 0);
        const int to = min(room, have);
        if (to > c) {
            for (int z = lane; z < (to - c) * er; z += 32) {
                const int col = c + z / er, k = z % er;
                put(col, k, __ldcg(edge + (int64_t)col * er + k));
            }
            __threadfence_block();
            __syncwarp();
            if (lane == 0) ch.avail = to;
            c = to;
            polls = 0;
        } else {
            __nanosleep(32);
            if (++polls >= WAIT_POLLS) {
                if (lane == 0) atomicOr(status, PHMM_ST_TIMEOUT);
                have = Ly + 1;
                polls = 0;
            }
        }
    }
}

// The publisher warp: writes the columns of the stripe's last row (row R - 1,
// column t - (R - 1) at step t; get(column, index) reads the shared ring) to the
// edge buffer and releases them.
template <class Get>
__device__ __forceinline__ void publish_edges(double *edge, int er, int R, int Ly, int *prog, Channel &ch, Get get) {
    const int lane = threadIdx.x & 31;
    int out = 0;
    for (long long n = 0; out <= Ly && n < 16LL * WAIT_POLLS; ++n) {
        const int done = min(__shfl_sync(0xffffffffu, ch.step, 0) - (R - 1) + 1, Ly + 1);
        if (done >= out + PUBLISH || (done > out && done == Ly + 1)) {
            for (int z = lane; z < (done - out) * er; z += 32) {
                const int col = out + z / er, k = z % er;
                __stcg(edge + (int64_t)col * er + k, get(col, k));
            }
            __syncwarp();
            if (lane == 0) {
                ch.taken = done;
                __threadfence();
                st_release(prog, done);
            }
            __syncwarp();
            out = done;
        } else {
            __nanosleep(32);
        }
    }
}

// Claims the CTA's stripe.
__device__ __forceinline__ Item claim(int *counter, const Item *items) {
    __shared__ int at;
    if (threadIdx.x == 0) at = atomicAdd(counter, 1);
    __syncthreads();
    return items[at];
}

}  // namespace s64
