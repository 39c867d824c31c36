// Culberson rounds (reference src/runner.c:139-152: p := color, recolor): the next coloring takes the old
// color classes in descending order and gives every vertex the smallest color that no neighbour of a
// larger old color has now.
//
// Adjacent vertices never share an old color, so the old colors alone say who precedes whom, and no
// predecessor lists are built: a round is
//
//   1. begin - word[u] = old color << 16 | 0: one 4-byte gather tells a neighbour both whether u
//              precedes it and u's new color once it has one (two 16-bit halves are enough: a greedy
//              coloring with k colors needs k (k - 1) directed edges, and M < 2^32);
//   2. sort  - vertices by degree tier, then by descending old color;
//   3. color - one persistent kernel.  Workers of three tiers take vertices in that order, each tier
//              from its own counter: a CTA per vertex above ROUND_MED_DEG neighbours, a warp up to it,
//              eight lanes up to ROUND_LIGHT_DEG.  A worker waits (bounded) on neighbours of larger old
//              color that have no new one yet.  The oldest unfinished vertex of all tiers is held by a
//              running worker and has all its predecessors done, so the kernel always progresses; a
//              CTA's role follows the order in which the CTAs start, so the first two cover all tiers.
//
// The rounds are queued without host synchronisation (the number of colors never grows, so the first
// round's bound on the key width holds for all), and can be captured.
//
// What bounds it: each round reads E once and gathers one word per edge.  On the 256^3 stencil (1.12 ms, 1.35 with the
// sort)
// the rows in class order cost 1.6 x their bytes in 64-byte pieces, and half the issue slots go by waiting
// for them; on the random geometric graph the L1 serves one gather per cycle (80 % of its peak).
// Measured per round with its sort (B200), lists of predecessors + class by class before -> this: 256^3 stencil
// 3.3 -> 1.35 ms, random geometric 2^23 1.9 -> 0.77 ms, R-MAT of 100,003 vertices 1.25 -> 0.25 ms (there a
// warp colored up to 32 large vertices of a class in turn).
#include <algorithm>

#include "gc_internal.h"

namespace {
using namespace gc;

constexpr unsigned int FULL = 0xffffffffu;
constexpr uint32_t ROUND_LIGHT_DEG = 64;   // eight lanes per vertex, colors in a 64-bit mask
constexpr uint32_t ROUND_MED_DEG = 1024;   // a warp per vertex
constexpr int ROUND_THREADS = 256;
constexpr int ROUND_MED_WARPS = 2;         // of a mixed CTA's warps, those on the middle tier while it lasts
constexpr uint32_t ROUND_MED_MANY = 48;    // middle vertices per CTA above which all its warps end up there
constexpr uint32_t ROUND_HUB_EVERY = 4;    // every fourth CTA takes the top tier while it lasts
constexpr uint32_t HUB_WORDS = 2048;       // bitmap of colors 1..65,536
constexpr uint32_t HUB_PEND = 2048;        // uncolored predecessors a CTA remembers
constexpr uint32_t MED_PEND = 64;          // the same for a warp (256: cliques of 600 0.98 -> 1.68 ms a round)
constexpr uint32_t MED_WINDOW = 1024;      // colors per pass of a warp over its list

// Work counters of a round, zeroed before it.
enum { RC_HUB = 0, RC_MED, RC_LIGHT, RC_CTA, RC_N_HUB, RC_N_MED, RC_WORDS = 8 };

__device__ __forceinline__ uint32_t tier_of(uint32_t d) { return d > ROUND_MED_DEG ? 2u : d > ROUND_LIGHT_DEG ? 1u : 0u; }

// Old colors from the coloring (first round) or from the last round's new colors; the sort keys, with
// the tier above key_bits when the graph has more than the light one, and the tiers' sizes.  In a captured pass the
// coloring before may have stopped: its colors are none, waits on them would run to their limit, and the pass is
// thrown away, so all vertices count as taken then.
template <typename T>
__global__ void __launch_bounds__(256) k_round_begin(const int *__restrict__ color, T *__restrict__ word,
                                                     const uint32_t *__restrict__ V, uint32_t N, int tiers, int key_bits,
                                                     uint32_t *__restrict__ key, uint32_t *__restrict__ ctr,
                                                     const DevState *st) {
    if (blockIdx.x == 0 && threadIdx.x == 0 && st->flow_stall) ctr[RC_HUB] = ctr[RC_MED] = ctr[RC_LIGHT] = N;
    constexpr int HALF = 4 * sizeof(T);  // bits of a color
    const uint32_t stride = gridDim.x * blockDim.x;
    uint32_t hubs = 0, meds = 0;
    for (uint32_t u = blockIdx.x * blockDim.x + threadIdx.x; u < N; u += stride) {
        const uint32_t old = color ? (uint32_t)color[u] : word[u] & ((1u << HALF) - 1u);
        word[u] = (T)(old << HALF);
        uint32_t t = 0;
        if (tiers) {
            t = tier_of(V[u + 1] - V[u]);
            hubs += t == 2u;
            meds += t == 1u;
        }
        key[u] = t << key_bits | old;
    }
    if (tiers) {
        hubs = __reduce_add_sync(FULL, hubs);
        meds = __reduce_add_sync(FULL, meds);
        if ((threadIdx.x & 31) == 0) {
            if (hubs) atomicAdd(ctr + RC_N_HUB, hubs);
            if (meds) atomicAdd(ctr + RC_N_MED, meds);
        }
    }
}

// The last round's words as colors and (old) keys.
template <typename T>
__global__ void k_round_end(const T *__restrict__ word, uint32_t N, int *__restrict__ color,
                            uint32_t *__restrict__ key) {
    for (uint32_t u = blockIdx.x * blockDim.x + threadIdx.x; u < N; u += gridDim.x * blockDim.x) {
        const uint32_t w = word[u];
        color[u] = (int)(w & ((1u << (4 * sizeof(T))) - 1u));
        key[u] = w >> (4 * sizeof(T));
    }
}

__global__ void k_max_color(const int *__restrict__ color, uint32_t N, DevState *st) {
    uint32_t m = 0;
    for (uint32_t u = blockIdx.x * blockDim.x + threadIdx.x; u < N; u += gridDim.x * blockDim.x)
        m = max(m, (uint32_t)max(color[u], 0));
    m = __reduce_max_sync(FULL, m);
    if ((threadIdx.x & 31) == 0 && m) atomicMax(&st->first_colors, m);
}

// A fruitless poll: true when the wait is over its limit or another one was.
__device__ __forceinline__ bool round_expired(unsigned int &spins, unsigned int limit, const DevState *st) {
    return ++spins > limit || ((spins & 255u) == 0 && ld_relaxed_u32(&st->err));
}

// Light tier: `batch` consecutive vertices of the order per grab, four at a time, eight lanes each.
// The batch's ids, CSR ranges and old colors come in three loads for all of them, and each step's
// neighbour ids are on their way while the step before is colored.  The four vertices of a step may
// depend on one another, so each stores its color as soon as it has it.
__device__ __forceinline__ void round_light(const uint32_t *__restrict__ order, uint32_t n, const uint32_t *__restrict__ V,
                                            const uint32_t *__restrict__ E, uint32_t *word, uint32_t *next,
                                            uint32_t batch, DevState *st, unsigned int limit) {
    constexpr int HALF = 4, LOADS = 2 * HALF;  // entries per lane; the second half only for lists above 32
    static_assert(8 * LOADS == ROUND_LIGHT_DEG, "a step covers a light vertex's list");
    const int lane = threadIdx.x & 31, q = lane & 7, grp = lane >> 3;
    for (;;) {
        uint32_t t0 = 0;
        if (lane == 0) t0 = atomicAdd(next, batch);
        t0 = __shfl_sync(FULL, t0, 0);
        if (t0 >= n) return;
        const uint32_t cnt = min(batch, n - t0);
        uint32_t u_l = 0, beg_l = 0, d_l = 0, old_l = 0;
        if ((uint32_t)lane < cnt) {
            u_l = order[t0 + lane];
            beg_l = V[u_l];
            d_l = V[u_l + 1] - beg_l;
            old_l = ld_relaxed_u32(word + u_l) >> 16;
        }
        uint32_t v[LOADS], d, dmax;
        auto ids = [&](int src) {
            const uint32_t beg = __shfl_sync(FULL, beg_l, src);
            d = __shfl_sync(FULL, d_l, src);
            dmax = __reduce_max_sync(FULL, d);
#pragma unroll
            for (int i = 0; i < HALF; i++) v[i] = 8u * i + q < d ? ld_stream(E + beg + 8 * i + q) : 0u;
            if (dmax > 8 * HALF) {
#pragma unroll
                for (int i = HALF; i < LOADS; i++) v[i] = 8u * i + q < d ? ld_stream(E + beg + 8 * i + q) : 0u;
            }
        };
        ids(grp);
        for (uint32_t j = 0; j < cnt; j += 4) {
            const uint32_t u = __shfl_sync(FULL, u_l, (int)j + grp), old = __shfl_sync(FULL, old_l, (int)j + grp);
            uint32_t id[LOADS], w[LOADS], wait = 0;  // wait, bit i: entry i is a predecessor without a color
            unsigned long long used = 0;
            const bool wide = dmax > 8 * HALF;
#pragma unroll
            for (int i = 0; i < HALF; i++) {  // (a stale word only costs a poll)
                id[i] = v[i];
                w[i] = 8u * i + q < d ? word[id[i]] : 0u;
            }
            if (wide) {
#pragma unroll
                for (int i = HALF; i < LOADS; i++) {
                    id[i] = v[i];
                    w[i] = 8u * i + q < d ? word[id[i]] : 0u;
                }
            }
            if (j + 4 < cnt) ids((int)j + 4 + grp);
            auto take = [&](int i) {
                if ((w[i] >> 16) > old) {  // a predecessor
                    const uint32_t c = w[i] & 0xffffu;
                    if (!c) wait |= 1u << i;
                    else if (c <= 64u) used |= 1ull << (c - 1u);
                }
            };
#pragma unroll
            for (int i = 0; i < HALF; i++) take(i);
            if (wide) {
#pragma unroll
                for (int i = HALF; i < LOADS; i++) take(i);
            }
            bool open = j + grp < cnt;  // this group's vertex has no color yet
            unsigned int spins = 0;
            for (;;) {
                const unsigned int waiting = __ballot_sync(FULL, wait != 0u);
                const bool done = open && !((waiting >> (8 * grp)) & 0xffu);
                if (__any_sync(FULL, done)) {
                    unsigned long long all = used;
#pragma unroll
                    for (int o = 1; o < 8; o <<= 1) all |= __shfl_xor_sync(FULL, all, o);
                    if (done) {
                        const uint32_t c = ~all ? (uint32_t)__ffsll((long long)~all) : 65u;
                        if (q == 0) st_relaxed_u32(word + u, old << 16 | c);
                        open = false;
                    }
                }
                if (!waiting) break;
                auto poll = [&](int i) {
                    if ((wait >> i) & 1u) {
                        const uint32_t c = ld_relaxed_u32(word + id[i]) & 0xffffu;
                        if (c) {
                            wait &= ~(1u << i);
                            if (c <= 64u) used |= 1ull << (c - 1u);
                        }
                    }
                };
#pragma unroll
                for (int i = 0; i < HALF; i++) poll(i);
                if (wide) {
#pragma unroll
                    for (int i = HALF; i < LOADS; i++) poll(i);
                }
                if (__any_sync(FULL, wait && round_expired(spins, limit, st))) {
                    if (lane == 0) raise_error(st, ERR_WAIT_EXPIRED, u);
                    return;
                }
            }
        }
    }
}

// Middle tier: one vertex per warp; colors in a bitmap of MED_WINDOW colors, uncolored predecessors
// remembered (beyond MED_PEND of them, waited for in place).
__device__ __forceinline__ void round_med(const uint32_t *__restrict__ order, uint32_t n, const uint32_t *__restrict__ V,
                                          const uint32_t *__restrict__ E, uint32_t *word, uint32_t *next, uint32_t *fb,
                                          uint32_t *pend, DevState *st, unsigned int limit) {
    constexpr int LOADS = 4;
    const int lane = threadIdx.x & 31;
    const unsigned int lt = (1u << lane) - 1u;
    for (;;) {
        uint32_t t = 0;
        if (lane == 0) t = atomicAdd(next, 1u);
        t = __shfl_sync(FULL, t, 0);
        if (t >= n) return;
        const uint32_t u = order[t], beg = V[u], d = V[u + 1] - beg, old = ld_relaxed_u32(word + u) >> 16;
        uint32_t c = 0;
        for (uint32_t first = 1; !c; first += MED_WINDOW) {
            fb[lane] = 0;
            __syncwarp();
            uint32_t np = 0;
            bool bad = false;
            auto mark = [&](uint32_t col) {
                const uint32_t x = col - first;
                if (x < MED_WINDOW) atomicOr(fb + (x >> 5), 1u << (x & 31u));
            };
            for (uint32_t j0 = 0; j0 < d; j0 += 32 * LOADS) {
                uint32_t v[LOADS], w[LOADS];
#pragma unroll
                for (int i = 0; i < LOADS; i++) v[i] = j0 + 32 * i + lane < d ? ld_stream(E + beg + j0 + 32 * i + lane) : 0u;
#pragma unroll
                for (int i = 0; i < LOADS; i++) w[i] = j0 + 32 * i + lane < d ? word[v[i]] : 0u;
#pragma unroll
                for (int i = 0; i < LOADS; i++) {
                    const bool pred = (w[i] >> 16) > old;
                    const uint32_t col = w[i] & 0xffffu;
                    if (pred && col) mark(col);
                    const unsigned int zero = __ballot_sync(FULL, pred && !col);
                    if (!zero) continue;
                    const uint32_t at = np + __popc(zero & lt);
                    if (pred && !col) {
                        if (at < MED_PEND) {
                            pend[at] = v[i];
                        } else {
                            unsigned int spins = 0;
                            uint32_t x;
                            while (!(x = ld_relaxed_u32(word + v[i]) & 0xffffu) && !bad) bad = round_expired(spins, limit, st);
                            if (!bad) mark(x);
                        }
                    }
                    np = min(MED_PEND, np + (uint32_t)__popc(zero));
                }
            }
            __syncwarp();
            for (uint32_t i = lane; i < np; i += 32) {
                unsigned int spins = 0;
                uint32_t x;
                while (!(x = ld_relaxed_u32(word + pend[i]) & 0xffffu) && !bad) bad = round_expired(spins, limit, st);
                if (!bad) mark(x);
            }
            if (__any_sync(FULL, bad)) {
                if (lane == 0) raise_error(st, ERR_WAIT_EXPIRED, u);
                return;
            }
            __syncwarp();
            const uint32_t open = ~fb[lane];
            const unsigned int has = __ballot_sync(FULL, open != 0u);
            if (has) {
                const int l = __ffs(has) - 1;
                c = first + 32u * l + (uint32_t)__ffs(__shfl_sync(FULL, open, l)) - 1u;
            }
            __syncwarp();
        }
        if (lane == 0) st_relaxed_u32(word + u, old << 16 | c);
        __syncwarp();
    }
}

// Top tier: one vertex per CTA; the bitmap covers every color.
__device__ __forceinline__ void round_hub(const uint32_t *__restrict__ order, uint32_t n, const uint32_t *__restrict__ V,
                                          const uint32_t *__restrict__ E, uint32_t *word, uint32_t *next, uint32_t *bm,
                                          uint32_t *pend, uint32_t *shared, DevState *st, unsigned int limit) {
    constexpr int LOADS = 4;
    for (;;) {
        if (threadIdx.x == 0) {
            shared[0] = atomicAdd(next, 1u);
            shared[1] = 0;           // pending predecessors
            shared[2] = 0xffffffffu; // smallest word with a free color
        }
        for (uint32_t i = threadIdx.x; i < HUB_WORDS; i += ROUND_THREADS) bm[i] = 0;
        __syncthreads();
        const uint32_t t = shared[0];
        if (t >= n) return;
        const uint32_t u = order[t], beg = V[u], d = V[u + 1] - beg, old = ld_relaxed_u32(word + u) >> 16;
        bool bad = false;
        auto mark = [&](uint32_t col) {
            const uint32_t x = col - 1u, b = 1u << (x & 31u);
            if (!(bm[x >> 5] & b)) atomicOr(bm + (x >> 5), b);  // (most colors come many times)
        };
        for (uint32_t j0 = 0; j0 < d; j0 += ROUND_THREADS * LOADS) {
            uint32_t v[LOADS], w[LOADS];
#pragma unroll
            for (int i = 0; i < LOADS; i++) {
                const uint32_t j = j0 + ROUND_THREADS * i + threadIdx.x;
                v[i] = j < d ? ld_stream(E + beg + j) : 0u;
            }
#pragma unroll
            for (int i = 0; i < LOADS; i++) w[i] = j0 + ROUND_THREADS * i + threadIdx.x < d ? word[v[i]] : 0u;
#pragma unroll
            for (int i = 0; i < LOADS; i++) {
                if ((w[i] >> 16) <= old) continue;
                uint32_t col = w[i] & 0xffffu;
                if (!col) {
                    const uint32_t at = atomicAdd(shared + 1, 1u);
                    if (at < HUB_PEND) {
                        pend[at] = v[i];
                        continue;
                    }
                    unsigned int spins = 0;
                    while (!(col = ld_relaxed_u32(word + v[i]) & 0xffffu) && !bad) bad = round_expired(spins, limit, st);
                }
                if (col) mark(col);
            }
        }
        __syncthreads();
        const uint32_t np = min(shared[1], HUB_PEND);
        for (uint32_t i = threadIdx.x; i < np; i += ROUND_THREADS) {
            unsigned int spins = 0;
            uint32_t col;
            while (!(col = ld_relaxed_u32(word + pend[i]) & 0xffffu) && !bad) bad = round_expired(spins, limit, st);
            if (col) mark(col);
        }
        if (__syncthreads_or(bad)) {
            if (threadIdx.x == 0) raise_error(st, ERR_WAIT_EXPIRED, u);
            return;
        }
        for (uint32_t i = threadIdx.x; i < HUB_WORDS; i += ROUND_THREADS)
            if (~bm[i]) {
                atomicMin(shared + 2, i);
                break;
            }
        __syncthreads();
        if (threadIdx.x == 0) {
            const uint32_t x = shared[2];  // (at most 65,535 colors are taken: a free one exists)
            st_relaxed_u32(word + u, old << 16 | (32u * x + (uint32_t)__ffs(~bm[x])));
        }
        __syncthreads();
    }
}

// Graphs of at most NARROW_DEG neighbours and NARROW_COLORS colors (meshes): the word is 16 bits wide
// (old color << 8 | new), and a predecessor's color sets its own bit of one 32-bit mask -- bit 0 when it
// has none yet, so that one reduction over the group's lanes gives both the free color and whether
// anything must be waited for.  Per entry that leaves a compare, a shift and an or: a round on the 256^3
// stencil took 1.16 ms in 32 registers (a full SM of warps) against 1.23 ms in the general kernel.
// With longer lists the extra entries cost more than that (random geometric, 2^23 vertices, at most 37
// neighbours: 0.69 ms here with eight entries per lane, 0.81 with the entries past 32 read in place, 0.65
// in the general kernel).
constexpr uint32_t NARROW_DEG = 32, NARROW_COLORS = 31;

__device__ __forceinline__ uint32_t ld_relaxed_u16(const uint16_t *p) {
    uint16_t v;
    asm volatile("ld.relaxed.gpu.global.u16 %0, [%1];" : "=h"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed_u16(uint16_t *p, uint32_t v) {
    asm volatile("st.relaxed.gpu.global.u16 [%0], %1;" ::"l"(p), "h"((uint16_t)v) : "memory");
}

__global__ void __launch_bounds__(ROUND_THREADS, 8)
    k_jp_round_narrow(const uint32_t *__restrict__ order, const uint32_t *__restrict__ V, const uint32_t *__restrict__ E,
                      uint32_t n, uint16_t *word, uint32_t *next, uint32_t batch, DevState *st, unsigned int limit) {
    constexpr int LOADS = NARROW_DEG / 8;  // entries per lane
    const int lane = threadIdx.x & 31, q = lane & 7, grp = lane >> 3;
    for (;;) {
        uint32_t t0 = 0;
        if (lane == 0) t0 = atomicAdd(next, batch);
        t0 = __shfl_sync(FULL, t0, 0);
        if (t0 >= n) return;
        const uint32_t cnt = min(batch, n - t0);
        uint32_t u_l = 0, beg_l = 0, d_l = 0, old_l = 0;
        if ((uint32_t)lane < cnt) {
            u_l = order[t0 + lane];
            beg_l = V[u_l];
            d_l = V[u_l + 1] - beg_l;
            old_l = ld_relaxed_u16(word + u_l) >> 8;
        }
        uint32_t v[LOADS];
        auto ids = [&](int src) {
            const uint32_t *row = E + __shfl_sync(FULL, beg_l, src) + q;
            const uint32_t d = __shfl_sync(FULL, d_l, src);
#pragma unroll
            for (int i = 0; i < LOADS; i++) v[i] = 8u * i + q < d ? ld_stream(row + 8 * i) : 0xffffffffu;
        };
        ids(grp);
        for (uint32_t j = 0; j < cnt; j += 4) {
            const int src = (int)j + grp;
            const uint32_t u = __shfl_sync(FULL, u_l, src), old = __shfl_sync(FULL, old_l, src);
            const uint32_t least = (old + 1u) << 8;  // words of predecessors are no smaller
            uint32_t id[LOADS], w[LOADS], used = 0;
#pragma unroll
            for (int i = 0; i < LOADS; i++) {  // (a stale word only costs a poll)
                id[i] = v[i];
                w[i] = id[i] != 0xffffffffu ? word[id[i]] : 0u;
            }
            if (j + 4 < cnt) ids(src + 4);
#pragma unroll
            for (int i = 0; i < LOADS; i++)
                if (w[i] >= least) used |= 1u << (w[i] & 31u);
            bool open = j + grp < cnt;  // this group's vertex has no color yet
            unsigned int spins = 0;
            for (;;) {
                uint32_t all = used;
#pragma unroll
                for (int o = 1; o < 8; o <<= 1) all |= __shfl_xor_sync(FULL, all, o);
                if (open && !(all & 1u)) {
                    if (q == 0) st_relaxed_u16(word + u, old << 8 | (uint32_t)(__ffs(~(all | 1u)) - 1));
                    open = false;
                }
                if (!__any_sync(FULL, open)) break;
                used &= ~1u;
#pragma unroll
                for (int i = 0; i < LOADS; i++)
                    if (w[i] >= least && !(w[i] & 31u)) {
                        w[i] = ld_relaxed_u16(word + id[i]);
                        used |= 1u << (w[i] & 31u);
                    }
                if (__any_sync(FULL, open && round_expired(spins, limit, st))) {
                    if (lane == 0) raise_error(st, ERR_WAIT_EXPIRED, u);
                    return;
                }
            }
        }
    }
}

// order: the top tier's vertices, the middle tier's, the light ones,
// each by descending old color.
template <bool TIERS>  // false: the light tier alone
__global__ void __launch_bounds__(ROUND_THREADS, 5) k_jp_round(const uint32_t *__restrict__ order,
                                                            const uint32_t *__restrict__ V,
                                                            const uint32_t *__restrict__ E, uint32_t N, uint32_t *word,
                                                            uint32_t *ctr, uint32_t batch, DevState *st,
                                                            unsigned int limit) {
    if (!TIERS) {
        round_light(order, N, V, E, word, ctr + RC_LIGHT, batch, st, limit);
        return;
    }
    static_assert(ROUND_THREADS / 32 * MED_PEND <= HUB_PEND && ROUND_THREADS <= HUB_WORDS, "the warps share the CTA's arrays");
    __shared__ uint32_t bm[TIERS ? HUB_WORDS : 1], pend[TIERS ? HUB_PEND : 1], shared[4];
    const uint32_t nh = ctr[RC_N_HUB], nm = ctr[RC_N_MED];
    if (threadIdx.x == 0) shared[3] = atomicAdd(ctr + RC_CTA, 1u);
    __syncthreads();
    if (shared[3] % ROUND_HUB_EVERY == 0) round_hub(order, nh, V, E, word, ctr + RC_HUB, bm, pend, shared, st, limit);
    __syncthreads();
    // the middle tier by some warps at once, and where it is large by the others too when there are no light vertices
    // left to take (a round, without / with: 500 complete bipartite graphs of 120 + 120 253 / 191 us, 8,000 cliques of
    // 120 1,597 / 977, Erdos-Renyi 50,000 x 200 236 / 203; but 30,000 rows of a band of 100 281 / 308)
    const int warp = threadIdx.x >> 5;
    const int passes = nm >= ROUND_MED_MANY * gridDim.x ? 3 : 2;
    for (int pass = warp < ROUND_MED_WARPS ? 0 : 1; pass < passes; pass++) {
        if (pass == 1) round_light(order + nh + nm, N - nh - nm, V, E, word, ctr + RC_LIGHT, batch, st, limit);
        else round_med(order + nh, nm, V, E, word, ctr + RC_MED, bm + 32 * warp, pend + MED_PEND * warp, st, limit);
    }
}

}  // namespace

bool gc_rounds_eligible(const gc_graph *g) {
    // colors fit 16 bits unless the graph could hold a clique of 65,536 vertices
    return g->ctx->jp_classes && g->colors_ours && (uint64_t)g->M < 65535ull * 65534ull;
}

gc_status gc_queue_max_color(gc_graph *g) {
    gc_ctx *ctx = g->ctx;
    if (g->N == 0) return GC_OK;
    k_max_color<<<std::min<uint32_t>((uint32_t)ctx->num_sms * 4, (g->N + 255) / 256), 256, 0, ctx->stream>>>(g->color, g->N, ctx->dstate);
    ctx->launches++;
    return gc_check_launch(ctx, "largest color");
}

gc_status gc_culberson_rounds(gc_graph *g, int rounds, uint32_t colors) {
    gc_ctx *ctx = g->ctx;
    gc_status s;
    const uint32_t N = g->N;
    if (N == 0 || rounds <= 0) return GC_OK;
    if ((s = gc_alloc(ctx, &g->pc, g->cap_N, "color words")) != GC_OK) return s;
    if ((s = gc_alloc(ctx, &g->order, g->cap_N, "class order")) != GC_OK) return s;
    if ((s = gc_alloc(ctx, &g->round_ctr, RC_WORDS, "round counters")) != GC_OK) return s;
    int key_bits = 0;
    while (std::min(colors, 65535u) >> key_bits) key_bits++;
    const int tiers = g->max_deg > ROUND_LIGHT_DEG ? 1 : 0;
    // vertices per grab: whole warps of them where there are enough to go round (the counter then costs
    // 0.02 ns a vertex); few where a vertex behind others in a grab would hold up its class
    const uint32_t batch = N >= (1u << 19) ? 32u : 8u;
    const bool narrow = g->max_deg <= NARROW_DEG && colors <= NARROW_COLORS;
    const int kind = tiers ? 2 : narrow ? 0 : 1;
    int &occ = ctx->round_blocks_per_sm[kind];
    if (!occ) {
        const void *f = kind == 2   ? (const void *)k_jp_round<true>
                        : kind == 1 ? (const void *)k_jp_round<false>
                                    : (const void *)k_jp_round_narrow;
        if ((s = gc_check_cuda(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, f, ROUND_THREADS, 0),
                               "occupancy")) != GC_OK)
            return s;
        if (occ < 1) occ = 1;
    }
    const uint32_t full = (uint32_t)ctx->num_sms * (uint32_t)occ;
    const uint32_t blocks = tiers ? full : std::max<uint32_t>(2u, std::min<uint32_t>(full, (N + 8 * batch - 1) / (8 * batch)));
    const uint32_t sweep = std::min<uint32_t>((uint32_t)ctx->num_sms * 8, (N + 255) / 256);
    uint16_t *word16 = reinterpret_cast<uint16_t *>(g->pc);
    for (int it = 0; it < rounds; it++) {
        if ((s = gc_check_cuda(ctx, cudaMemsetAsync(g->round_ctr, 0, 4 * RC_WORDS, ctx->stream), "round counters")) != GC_OK)
            return s;
        {
            ProfScope ps(ctx, "round_begin", ctx->stream);
            if (narrow)
                k_round_begin<uint16_t><<<sweep, 256, 0, ctx->stream>>>(it ? nullptr : g->color, word16, g->V, N, 0, key_bits,
                                                                        g->key, g->round_ctr, ctx->dstate);
            else
                k_round_begin<uint32_t><<<sweep, 256, 0, ctx->stream>>>(it ? nullptr : g->color, g->pc, g->V, N, tiers,
                                                                        key_bits, g->key, g->round_ctr, ctx->dstate);
            ctx->launches++;
        }
        if ((s = gc_sort_order_bits(g, key_bits + 2 * tiers, false, &ctx->dstate->ordered)) != GC_OK) return s;
        ProfScope ps(ctx, "jp_round", ctx->stream);
        if (kind == 2)
            k_jp_round<true><<<blocks, ROUND_THREADS, 0, ctx->stream>>>(g->order, g->V, g->E, N, g->pc, g->round_ctr, batch,
                                                                        ctx->dstate, ctx->spin_limit);
        else if (kind == 1)
            k_jp_round<false><<<blocks, ROUND_THREADS, 0, ctx->stream>>>(g->order, g->V, g->E, N, g->pc, g->round_ctr, batch,
                                                                         ctx->dstate, ctx->spin_limit);
        else
            k_jp_round_narrow<<<blocks, ROUND_THREADS, 0, ctx->stream>>>(g->order, g->V, g->E, N, word16,
                                                                         g->round_ctr + RC_LIGHT, batch, ctx->dstate,
                                                                         ctx->spin_limit);
        ctx->launches++;
        if ((s = gc_check_launch(ctx, "culberson round")) != GC_OK) return s;
    }
    if (narrow) k_round_end<uint16_t><<<sweep, 256, 0, ctx->stream>>>(word16, N, g->color, g->key);
    else k_round_end<uint32_t><<<sweep, 256, 0, ctx->stream>>>(g->pc, N, g->color, g->key);
    ctx->launches++;
    g->key_kind = 100;
    g->has_keys = true;
    g->has_colors = true;
    return gc_check_launch(ctx, "culberson colors");
}
