// Jones-Plassmann on graphs of small maximum degree, as a dataflow (reference src/coloring.c:223-330).
//
// Meshes, geometric and Erdos-Renyi graphs have short neighbour lists, and their priority DAG is often
// a wavefront: on a stencil the priority follows the vertex id, so the vertices that are ready at one
// time lie far apart in the priority order.  Kernels that hand vertices out in priority order (k_jp.cu)
// then see only the few ready ones inside their window.  Here a vertex is handed out when it is ready:
//
//   1. init - one pass over the edges.  Each vertex records which of its neighbours precede it, as a
//             bit mask, and how many do (rem, in its counter word).  Sources (no predecessor) take
//             color 1 and are queued.
//   2. flow - a warp takes a queued vertex u, one lane per neighbour.  It subtracts one from rem of
//             every successor.  It goes on with the first successor whose rem it took to zero and
//             queues the others, then reads the predecessors' colors and stores the smallest color
//             none of them has.
//
// rem counts predecessors that have STARTED, not those that are done: the subtractions go out before
// u's own color is known, so a successor's neighbour ids are fetched while u still waits.  A vertex
// therefore polls its predecessors' colors (all held by running warps); the color is itself the whole
// message, so no fences are needed.
//
// The queue is FLOW_QUEUES arrays, vertex v in array v mod FLOW_QUEUES, each with its own head and tail
// counter: a single counter serves an atomic every 0.7 ns, which alone would cost 10 ms for 16.8 M
// vertices.  The powers of two have 36 different remainders modulo 37, so the strides of a mesh spread over
// the arrays (modulo 31 they have five, and the 256^3 stencil took 10.5 ms first fit, now 5.1).  Where the sides are 2
// modulo 37 a whole wavefront has one remainder, which costs nothing that shows (first fit 112^3 / 113^3 1,410 / 1,421
// us, 149^3 / 150^3 2,076 / 2,099).  Hundreds of
// warps wait at an array's end, each for a slot of its own, so consecutive slots lie in different lines: side
// by side, their polls and stores met in a few lines (256^3 GNN4 9.0 -> 7.5 ms, Erdos-Renyi 400,000 GNN3 184 ->
// 134 us, 65,536 LF 96 -> 86).  Every vertex is either queued in its array once or gone on with once (the
// array's skip counter), so an array is done after as many vertices as it has, and warps take its slots in order: a slot below the
// tail always belongs to a running warp.  Arrays are served by the warps whose number (in the order in
// which the CTAs start) has that remainder: the first five CTAs that run serve them all, so the kernel
// advances whatever else occupies the GPU.
//
// A DAG that is narrow -- a band, a strip, a path, a caterpillar -- has its next vertices known long before:
// its hops cost 0.63 to 3 us here, 0.1 to 0.3 among tickets whose colors stay in one cluster's shared memory
// (k_jp_core).  So one CTA only counts what becomes ready, in windows of 120 us, and stops a coloring that it finds
// narrow (flow_watch); the tickets then color the graph, as many as fit in the cluster.  First fit, dataflow to
// the end / this: a path of 20,000 12.8 / 5.2 ms, 20,000 rows of a band matrix with 31 entries on either side 22.9
// / 2.4, a 5-point strip of 4 x 5,000 3.5 / 1.6, a path of 10,000 with 50 leaves each 23.6 / 2.9.
//
// A CSR that is not symmetric (a caller's mistake that the upload does not check) can leave vertices
// that never become ready.  Idle warps watch the counters; when none moves for a while they set
// DevState::flow_stall and every warp leaves.  The host then runs the ticket kernels, whose waits
// only follow each vertex's own list.
//
// What bounds it: on a wavefront the chain of hops.  A hop to the successor a warp goes on with takes 0.63 us
// (its counter's atomic, then its neighbour ids); one through a queue adds the tail's atomic, the slot's
// store and poll, so a slot holds where the list begins as well: fetched after the counter word, stencils
// took up to 15 % longer (256^3 GNN4 10.5 -> 9.0 ms, Erdos-Renyi 400,000 GNN3 229 -> 184 us).
// Elsewhere the vertices in flight (one per warp, 2 to 3 us each).
// Measured on a B200, coloring kernels of one job, tickets (sort, cluster core, streams, ticket kernel,
// leaves) -> dataflow: 256^3 stencil with cut-outs, GNN4 keys 272 -> 8.9 ms (the full grid 7.2, first fit 5.7), 97 x 61 x
// 113 stencil first fit 8.9 -> 1.1 ms, random geometric 2^23 GNN4 4.0 -> 2.6 ms, Erdos-Renyi 65,536 LF 0.36 -> 0.11 ms.
// Measured and not kept: eight lanes per vertex and four vertices per warp (hops of 3.3 us: the longer
// code path of a lane is on the chain), a separate 16-byte record (hops of 1.9 us), a slot taken
// before the color is stored, four slots taken at once under backlog; ready vertices handed to waiting
// warps of the same CTA through shared memory (97 x 61 x 113 first fit 1.1 -> 1.4 ms and more: the atomics
// of many vertices in one SM are slower); lists fetched into L2 when one predecessor is left to start
// (stencils 5 % faster, the others 1 to 5 % slower); fewer instructions per poll, that is more polls (97 x 61
// x 113 first fit 1.04 -> 1.31 ms), or sleeps between them (1.7 ms); arrays by a hash of the id (300,000 x 32
// 9 % slower).
#include <algorithm>

#include "gc_internal.h"

namespace {
using namespace gc;

constexpr uint32_t FLOW_QUEUES = 37;
constexpr uint32_t FLOW_MIN_CTAS = 5;  // a warp for every array
constexpr uint32_t FLOW_PAD = 32;  // words between counters: one 128-byte line each
constexpr uint32_t FLOW_CTA = 3 * FLOW_QUEUES * FLOW_PAD;  // the CTAs' start counter
constexpr uint32_t FLOW_SLOTS = FLOW_CTA + FLOW_PAD;       // first queue slot
constexpr int FLOW_THREADS = 256;
constexpr uint32_t FLOW_FEW_N = 1u << 18;

// A vertex's counter word: rem in bits 48..63, the degree in bits 32..47, the first CSR entry below.
// The subtraction that makes a successor ready so returns where its neighbour list is, and the list is
// on its way one load earlier.  rem is the top field: one subtraction too many (a self-loop, a CSR that
// is not symmetric) wraps there and leaves the others alone.  A vertex that thousands name one-sidedly would become
// ready a second time, take another's place in its array, and leave that one without a color: the subtraction
// that finds a multiple of FLOW_LEAF in rem stops the kernel long before.
constexpr unsigned long long FLOW_ONE = 1ull << 48;

// Leaves (every neighbour precedes them) make nobody ready.  In graphs whose longest lists are far above the mean
// -- trees, hubs with their leaves -- they are most of the vertices, and a warp that queues dozens of them per
// hop holds up the chain.  There the leaves stay out of the queues: rem starts at FLOW_LEAF + the predecessors,
// so it never says ready, and a pass after the flow colors them all (trees of 2^20 vertices, first fit, leaves
// queued / apart: arity 30 286 / 175 us, 60 338 / 199; a path of 5,000 with 100 leaves each 15,600 / 6,200).
constexpr uint32_t FLOW_LEAF = 0x4000u;
constexpr uint32_t FLOW_SKEW = 4;  // leaves apart where the largest degree is above this many times the mean
// W words of 32 mask bits per vertex (bit j of word w: neighbour 32 w + j precedes).
constexpr int FLOW_WIDE = 4;
template <int W>
struct FlowMask;
template <>
struct FlowMask<1> {
    using T = uint32_t;
    static __device__ __forceinline__ void get(T t, uint32_t *m) { m[0] = t; }
    static __device__ __forceinline__ T put(const uint32_t *m) { return m[0]; }
};
template <>
struct FlowMask<2> {
    using T = uint2;
    static __device__ __forceinline__ void get(T t, uint32_t *m) { m[0] = t.x, m[1] = t.y; }
    static __device__ __forceinline__ T put(const uint32_t *m) { return make_uint2(m[0], m[1]); }
};
template <>
struct FlowMask<4> {
    using T = uint4;
    static __device__ __forceinline__ void get(T t, uint32_t *m) { m[0] = t.x, m[1] = t.y, m[2] = t.z, m[3] = t.w; }
    static __device__ __forceinline__ T put(const uint32_t *m) { return make_uint4(m[0], m[1], m[2], m[3]); }
};

__device__ __forceinline__ uint32_t *flow_head(uint32_t *fq, uint32_t k) { return fq + k * FLOW_PAD; }
__device__ __forceinline__ uint32_t *flow_tail(uint32_t *fq, uint32_t k) { return fq + (FLOW_QUEUES + k) * FLOW_PAD; }
__device__ __forceinline__ uint32_t *flow_skip(uint32_t *fq, uint32_t k) { return fq + (2 * FLOW_QUEUES + k) * FLOW_PAD; }

__device__ __forceinline__ unsigned long long *flow_slots(uint32_t *fq) {
    return reinterpret_cast<unsigned long long *>(fq + FLOW_SLOTS);
}

// Slots that are filled one after the other lie in different lines, since as many warps poll them.
__device__ __forceinline__ uint32_t flow_place(uint32_t at) {
    return (at & ~1023u) | (at & 63u) << 4 | (at >> 6 & 15u);
}

// Queues vertex v, whose list begins at `beg`: slots hold v + 1 and beg, so that the zeroed buffer reads as
// empty and the list can be fetched along with the counter word.
__device__ __forceinline__ void flow_push(uint32_t *fq, uint32_t stride, uint32_t v, uint32_t beg) {
    const uint32_t k = v % FLOW_QUEUES;
    const uint32_t at = atomicAdd(flow_tail(fq, k), 1u);
    if (at < stride) st_relaxed_u64(flow_slots(fq) + (size_t)k * stride + flow_place(at), (unsigned long long)beg << 32 | (v + 1u));
}

// Four lanes per vertex, vertices in id order (records, CSR offsets and rows stream).
template <int W, bool LEAVES>
__global__ void __launch_bounds__(FLOW_THREADS) k_flow_init(const uint32_t *__restrict__ V, const uint32_t *__restrict__ E,
                                                            const uint32_t *__restrict__ key, uint32_t N,
                                                            unsigned long long *__restrict__ word,
                                                            typename FlowMask<W>::T *__restrict__ mask,
                                                            int *__restrict__ color,
                                                            uint32_t *__restrict__ fq, uint32_t stride) {
    constexpr int LOADS = 8;
    __shared__ uint32_t apart[LEAVES ? FLOW_QUEUES : 1];  // vertices that stay out of each array
    if (LEAVES) {
        if (threadIdx.x < FLOW_QUEUES) apart[threadIdx.x] = 0;
        __syncthreads();
    }
    const int lane = threadIdx.x & 31, q = lane & 3, qbase = lane & ~3;
    const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
    const uint64_t keep = l2_keep_policy();  // the keys (4N bytes) stay in L2 while E streams past
    for (uint32_t base = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 8; base < N; base += nwarps * 8) {
        const uint32_t u = base + (lane >> 2);
        const bool valid = u < N;
        const uint32_t beg = valid ? V[u] : 0u, d = valid ? V[u + 1] - beg : 0u;
        const uint32_t ku = valid ? key[u] : 0u;
        const uint32_t dmax = __reduce_max_sync(0xffffffffu, d);
        uint32_t m[W];
        uint32_t cnt = 0;
#pragma unroll
        for (int w = 0; w < W; w++) {
            m[w] = 0;
            if (32u * w >= dmax) continue;
            uint32_t v[LOADS], kv[LOADS];
#pragma unroll
            for (int k = 0; k < LOADS; k++) {
                const uint32_t i = 32 * w + 4 * k + q;
                v[k] = i < d ? ld_stream(E + beg + i) : 0u;
            }
#pragma unroll
            for (int k = 0; k < LOADS; k++) kv[k] = 32 * w + 4 * k + q < d ? ld_keep(key + v[k], keep) : 0u;
#pragma unroll
            for (int k = 0; k < LOADS; k++) {
                const bool pk = 32 * w + 4 * k + q < d && precedes(kv[k], v[k], ku, u);
                m[w] |= ((__ballot_sync(0xffffffffu, pk) >> qbase) & 0xfu) << (4 * k);
            }
            cnt += __popc(m[w]);
        }
        if (valid && q == 0) {
            const bool out = LEAVES && cnt == d;
            word[u] = (unsigned long long)(out && d ? cnt | FLOW_LEAF : cnt) << 48 | (unsigned long long)d << 32 | beg;
            mask[u] = FlowMask<W>::put(m);
            color[u] = cnt == 0 ? 1 : 0;
            if (out) atomicAdd(apart + u % FLOW_QUEUES, 1u);
            else if (cnt == 0) flow_push(fq, stride, u, beg);
        }
    }
    if (LEAVES) {
        __syncthreads();
        if (threadIdx.x < FLOW_QUEUES && apart[threadIdx.x]) atomicAdd(flow_skip(fq, threadIdx.x), apart[threadIdx.x]);
    }
}

// Vertices started or queued so far; every lane gets it.
__device__ __forceinline__ uint32_t flow_progress(uint32_t *fq, int lane) {
    uint32_t n = 0;
    for (uint32_t k = lane; k < FLOW_QUEUES; k += 32) n += ld_relaxed_u32(flow_tail(fq, k)) + ld_relaxed_u32(flow_skip(fq, k));
    return __reduce_add_sync(0xffffffffu, n);
}

// The watching CTA.  A coloring is narrow when in the first window fewer than FLOW_THIN vertices became ready for each
// look at the counters, or in a later one fewer than FLOW_FEW, while half of what was not ready at the start is
// still to come and would take four windows more.  A look is a trip to L2 (0.63 us on an idle GPU), as a hop is one or
// two, and beside other streams' work both get longer together: the clock would take a mesh there for narrow.  Windows
// begin when all CTAs run.  By tickets in the cluster, strips of 4 to 50 vertices' width run at 11 to 55 vertices a
// microsecond, bars of 4 x 4 to 16 x 16 at 8 to 23; wavefronts start narrow as well but have passed FLOW_THIN by the end
// of the first window (a mesh's corner: 50, a square 5-point grid 40), and a second window costs less than a wrong turn.
// To stop it, FLOW_VOID is added to the counters, so that no vertex becomes ready any more, and to the arrays' skip
// counters, so that nobody waits for one.  What has started runs to its end, since it only waits for what has started.
// (The warps that color know nothing of this: a look at a flag in their loops cost path and mesh 40 %.)
constexpr uint32_t FLOW_THIN = 10, FLOW_FEW = 19, FLOW_VOID = 0x2000u;  // (16 and 30 a microsecond)

__device__ void flow_watch(unsigned long long *word, uint32_t *fq, uint32_t N, uint32_t window, DevState *st, uint32_t check) {
    __shared__ bool stop;
    const int lane = threadIdx.x & 31;
    if (threadIdx.x < 32) {
        uint32_t looks = 0, same = 0, ready = 0, last = 0, left0 = 0;
        bool begun = false, first = true, narrow = false;
        for (;;) {
            const uint32_t flag = lane == 0 ? ld_relaxed_u32(&st->flow_stall) : 0u;
            const uint32_t ctas = begun ? gridDim.x : ld_relaxed_u32(fq + FLOW_CTA);
            const uint32_t now = flow_progress(fq, lane), left = N - min(now, N);
            if (left == 0 || __shfl_sync(0xffffffffu, flag, 0)) break;
            same = now == last ? same + 1u : 0u;
            last = now;
            if (same > check) break;
            if (!begun) {
                begun = ctas >= gridDim.x;
                ready = now;
                left0 = left;
            } else if (++looks == window) {
                const uint32_t got = now - ready;
                narrow = got < window * (first ? FLOW_THIN : FLOW_FEW) && left >= left0 / 2 && left >= 4ull * got;
                if (narrow) break;
                looks = 0;
                ready = now;
                first = false;
            }
        }
        if (lane == 0) {
            stop = narrow;
            if (narrow) st_relaxed_u32(&st->flow_stall, FLOW_NARROW);
        }
    }
    __syncthreads();
    if (!stop) return;
    for (uint32_t v = threadIdx.x; v < N; v += FLOW_THREADS) atomicAdd(word + v, (unsigned long long)FLOW_VOID << 48);
    __syncthreads();
    if (threadIdx.x < FLOW_QUEUES) atomicAdd(flow_skip(fq, threadIdx.x), N);
}

// One more fruitless poll of a warp: true when the warp must leave.  After `check` polls the warp
// compares the tails with their last sum; unchanged means that nothing moves.
struct FlowWait {
    uint32_t spins = 0, seen = 0xffffffffu;
    __device__ __forceinline__ bool give_up(uint32_t *fq, DevState *st, uint32_t check, int lane) {
        ++spins;
        if ((spins & 1023u) == 0 && __shfl_sync(0xffffffffu, lane == 0 ? ld_relaxed_u32(&st->flow_stall) : 0u, 0)) return true;
        if (spins <= check) return false;
        const uint32_t now = flow_progress(fq, lane);
        if (now == seen) {
            if (lane == 0) st_relaxed_u32(&st->flow_stall, FLOW_STUCK);
            return true;
        }
        seen = now;
        spins = 0;
        return false;
    }
};

template <int W>
__global__ void __launch_bounds__(FLOW_THREADS, W <= 2 ? 8 : 4) k_jp_flow(unsigned long long *word,
                                                          const typename FlowMask<W>::T *__restrict__ mask,
                                                          const uint32_t *__restrict__ E, uint32_t M, int *color, uint32_t *fq,
                                                          uint32_t N, uint32_t stride, DevState *st, uint32_t check,
                                                          uint32_t window) {
    constexpr unsigned int FULL = 0xffffffffu;
    __shared__ uint32_t cta_s;
    if (threadIdx.x == 0) cta_s = atomicAdd(fq + FLOW_CTA, 1u);
    __syncthreads();
    if (window && cta_s == FLOW_MIN_CTAS) {
        flow_watch(word, fq, N, window, st, check);
        return;
    }
    const int lane = threadIdx.x & 31;
    const uint32_t k = (cta_s * (FLOW_THREADS / 32) + (threadIdx.x >> 5)) % FLOW_QUEUES;
    const uint32_t nk = k < N ? (N - k + FLOW_QUEUES - 1) / FLOW_QUEUES : 0u;  // vertices of this array
    uint32_t *head = flow_head(fq, k), *skip = flow_skip(fq, k);
    const unsigned long long *slots = flow_slots(fq) + (size_t)k * stride;
    FlowWait fw;
    uint32_t u, d, v[W];  // the vertex, its degree, and this lane's neighbours (entries 32 w + lane)
    typename FlowMask<W>::T mt;
    auto fetch = [&](uint32_t lo, uint32_t hi) {  // from the vertex's counter word
        d = hi & 0xffffu;
#pragma unroll
        for (int w = 0; w < W; w++) v[w] = 32u * w + lane < d ? ld_stream(E + lo + 32 * w + lane) : 0u;
        mt = __ldg(mask + u);
    };
    for (;;) {
        // a queued vertex: take a slot and wait until it is filled, or can no longer be (vertices that a
        // warp went on with leave that many slots at the array's end unfilled)
        uint32_t slot = 0;
        unsigned long long u1 = 0;
        if (lane == 0) slot = atomicAdd(head, 1u);
        slot = __shfl_sync(FULL, slot, 0);
        if (slot >= nk) return;
        for (;;) {
            u1 = __shfl_sync(FULL, lane == 0 ? ld_relaxed_u64(slots + flow_place(slot)) : 0ull, 0);
            if (u1) break;
            if ((fw.spins & 7u) == 7u && slot + min(nk, __shfl_sync(FULL, lane == 0 ? ld_relaxed_u32(skip) : 0u, 0)) >= nk) return;
            if (fw.give_up(fq, st, check, lane)) return;
        }
        fw.spins = 0;
        u = (uint32_t)u1 - 1u;
        {   // the list's first 32 entries are fetched before its length is known
            const uint32_t lo = (uint32_t)(u1 >> 32);
            mt = __ldg(mask + u);
            v[0] = lane < M - lo ? ld_stream(E + lo + lane) : 0u;
            d = (uint32_t)(__ldcg(word + u) >> 32) & 0xffffu;
#pragma unroll
            for (int w = 1; w < W; w++) v[w] = 32u * w + lane < d ? ld_stream(E + lo + 32 * w + lane) : 0u;
        }
        for (;;) {  // u, then a successor that u made ready, and so on
            uint32_t m[W], wait = 0;  // wait, bit w: entry 32 w + lane is a predecessor without a color
            FlowMask<W>::get(mt, m);
            uint32_t got[W];             // predecessors' colors
            unsigned long long old[W];   // successors' counter words before this subtraction
            uint32_t keep[W];            // (v[] is refilled for the next vertex below)
#pragma unroll
            for (int w = 0; w < W; w++) {  // all in flight
                got[w] = 0;
                old[w] = 0;
                keep[w] = v[w];
                if (32u * w + lane < d) {
                    if ((m[w] >> lane) & 1u) {
                        wait |= 1u << w;
                        got[w] = (uint32_t)ld_relaxed(color + v[w]);
                    } else {
                        old[w] = atomicAdd(word + v[w], 0ull - FLOW_ONE);
                    }
                }
            }
            // the warp goes on with one ready successor (its list is on the way while u's color is made)
            // and queues the others
            const uint32_t self = u;
            bool more = false;
#pragma unroll
            for (int w = 0; w < W; w++) {
                const uint32_t left = (uint32_t)(old[w] >> 48);
                bool ready = left == 1u;
                const unsigned int rm = __ballot_sync(FULL, ready);
                if (rm) {
                    if (!more) {
                        more = true;
                        const int first = __ffs(rm) - 1;
                        u = __shfl_sync(FULL, keep[w], first);
                        const uint32_t lo = __shfl_sync(FULL, (uint32_t)old[w], first);
                        const uint32_t hi = __shfl_sync(FULL, (uint32_t)(old[w] >> 32), first);
                        fetch(lo, hi);
                        if (lane == first) {
                            ready = false;
                            atomicAdd(flow_skip(fq, u % FLOW_QUEUES), 1u);
                        }
                    }
                    if (ready) flow_push(fq, stride, keep[w], (uint32_t)old[w]);
                }
                if (left && left % FLOW_LEAF == 0) st_relaxed_u32(&st->flow_stall, FLOW_STUCK);
            }
            uint32_t used[W];
#pragma unroll
            for (int x = 0; x < W; x++) used[x] = 0;
            FlowWait cw;
            for (;;) {
#pragma unroll
                for (int w = 0; w < W; w++) {
                    if (((wait >> w) & 1u) && got[w]) {
                        wait &= ~(1u << w);
#pragma unroll
                        for (int x = 0; x < W; x++)
                            if (W == 1 || ((got[w] - 1u) >> 5) == (uint32_t)x) used[x] |= 1u << ((got[w] - 1u) & 31u);
                    }
                }
                if (!__any_sync(FULL, wait != 0u)) break;
                if (cw.give_up(fq, st, check, lane)) return;
#pragma unroll
                for (int w = 0; w < W; w++)
                    if ((wait >> w) & 1u) got[w] = (uint32_t)ld_relaxed(color + keep[w]);
            }
            int c = 0;
#pragma unroll
            for (int x = 0; x < W; x++) {
                const uint32_t all = __reduce_or_sync(FULL, used[x]);
                if (c == 0 && ~all) c = 32 * x + __ffs(~all);
            }
            if (lane == 0) st_relaxed(color + self, c);
            if (!more) break;
        }
    }
}

// The leaves: a warp looks through 32 vertices and colors four leaves at a time, eight lanes each.
template <int W>
__global__ void __launch_bounds__(FLOW_THREADS) k_flow_leaves(const unsigned long long *__restrict__ word,
                                                              const uint32_t *__restrict__ E, uint32_t N, int *color,
                                                              DevState *st) {
    constexpr unsigned int FULL = 0xffffffffu;
    constexpr int LOADS = 4;
    if (st->flow_stall) return;
    const int lane = threadIdx.x & 31, q = lane & 7;
    const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t base = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 32; base < N; base += nwarps * 32) {
        const unsigned long long mine = base + lane < N ? word[base + lane] : 0ull;
        unsigned int found = __ballot_sync(FULL, ((uint32_t)(mine >> 48) & ~127u) == FLOW_LEAF);
        while (found) {
            int src = -1;  // the leaf of this lane's group
            for (int k = 0; k < 4 && found; k++, found &= found - 1)
                if (k == lane >> 3) src = __ffs(found) - 1;
            const unsigned long long w0 = __shfl_sync(FULL, mine, max(src, 0));
            const uint32_t beg = (uint32_t)w0, d = src < 0 ? 0u : (uint32_t)(w0 >> 32) & 0xffffu;
            uint32_t used[W];
#pragma unroll
            for (int x = 0; x < W; x++) used[x] = 0;
            for (uint32_t j = q; j < d; j += 8 * LOADS) {
                uint32_t v[LOADS], c[LOADS];
#pragma unroll
                for (int k = 0; k < LOADS; k++) v[k] = j + 8 * k < d ? ld_stream(E + beg + j + 8 * k) : 0u;
#pragma unroll
                for (int k = 0; k < LOADS; k++) c[k] = j + 8 * k < d ? (uint32_t)color[v[k]] : 1u << 31;
#pragma unroll
                for (int k = 0; k < LOADS; k++) {
                    // (in a symmetric CSR a leaf's neighbours all have their colors)
                    if (c[k] == 0 && v[k] != base + src) st_relaxed_u32(&st->flow_stall, FLOW_STUCK);
#pragma unroll
                    for (int x = 0; x < W; x++)
                        if ((c[k] - 1u) >> 5 == (uint32_t)x) used[x] |= 1u << ((c[k] - 1u) & 31u);
                }
            }
            __syncwarp();
            int c = 0;
#pragma unroll
            for (int x = 0; x < W; x++) {
#pragma unroll
                for (int o = 1; o < 8; o <<= 1) used[x] |= __shfl_xor_sync(FULL, used[x], o);
                if (c == 0 && ~used[x]) c = 32 * x + __ffs(~used[x]);
            }
            if (src >= 0 && q == 0) color[base + src] = c;
        }
    }
}

template <int W>
gc_status flow_run(gc_graph *g, uint32_t stride) {
    gc_ctx *ctx = g->ctx;
    gc_status s;
    // counter words in the first half of the ticket records' buffer; masks in the second half (up to 8
    // bytes per vertex), else in the ticket streams' buffer
    unsigned long long *word = reinterpret_cast<unsigned long long *>(g->jprec);
    uint32_t *fq = g->sort_buf;
    using MaskT = typename FlowMask<W>::T;
    MaskT *mask = W <= 2 ? reinterpret_cast<MaskT *>(word + g->cap_N) : reinterpret_cast<MaskT *>(g->jpsplit);
    int &occ = ctx->flow_blocks_per_sm[W == FLOW_WIDE ? 2 : W - 1];
    if (!occ) {
        if ((s = gc_check_cuda(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_jp_flow<W>, FLOW_THREADS, 0),
                               "occupancy")) != GC_OK)
            return s;
        if (occ < 1) occ = 1;
    }
    if ((s = gc_check_cuda(ctx, cudaMemsetAsync(fq, 0, 4 * ((size_t)FLOW_SLOTS + 2 * (size_t)FLOW_QUEUES * stride),
                                                ctx->stream), "flow queues")) != GC_OK)
        return s;
    const uint32_t N = g->N;
    const bool leaves = (uint64_t)g->max_deg * N > (uint64_t)FLOW_SKEW * g->M;
    {
        ProfScope ps(ctx, "flow_init", ctx->stream);
        const uint32_t blocks = std::min<uint32_t>((uint32_t)ctx->num_sms * 8, (N + 63) / 64);
        (leaves ? k_flow_init<W, true> : k_flow_init<W, false>)<<<blocks, FLOW_THREADS, 0, ctx->stream>>>(
            g->V, g->E, g->key, N, word, mask, g->color, fq, stride);
    }
    {
        ProfScope ps(ctx, "jp_flow", ctx->stream);
        // at least FLOW_MIN_CTAS; a warp per four vertices at most; up to FLOW_FEW_N
        // vertices half of what fits, since the chains are then all there is and idle warps' polls slow them
        // (colorings with keys by degree, 8 / 4 per SM: Erdos-Renyi 65,536 130 / 126 us, random geometric 200,000 116 /
        // 126, 500,000 189 / 226, Erdos-Renyi 600,000 270 / 360)
        const int per_sm = std::min(occ, N <= FLOW_FEW_N ? std::max(1, ctx->flow_ctas_per_sm / 2) : ctx->flow_ctas_per_sm);
        const uint32_t most = (uint32_t)ctx->num_sms * (uint32_t)per_sm;
        // (a long path stays: one successor per hop is 0.63 us here, and past the cluster's tickets 0.73 there)
        const uint32_t window = g->max_deg <= 2 && N > (1u << 17) ? 0u : ctx->narrow_window;
        const uint32_t blocks = std::max<uint32_t>(FLOW_MIN_CTAS + 1, std::min<uint32_t>(most, (N + 31) / 32));
        k_jp_flow<W><<<blocks, FLOW_THREADS, 0, ctx->stream>>>(word, mask, g->E, g->M, g->color, fq, N, stride,
                                                               ctx->dstate, std::min(ctx->spin_limit, ctx->flow_limit),
                                                               window);
    }
    ctx->launches += 2;
    if (leaves) {
        ProfScope ps(ctx, "flow_leaves", ctx->stream);
        const uint32_t blocks = std::min<uint32_t>((uint32_t)ctx->num_sms * 8, (N + FLOW_THREADS - 1) / FLOW_THREADS);
        k_flow_leaves<W><<<blocks, FLOW_THREADS, 0, ctx->stream>>>(word, g->E, N, g->color, ctx->dstate);
        ctx->launches++;
    }
    return gc_check_launch(ctx, "jp flow");
}

}  // namespace

// Which graphs go by dataflow: a maximum degree below 64 always (whole calls, largest degree first, dataflow /
// tickets: Erdos-Renyi 200,000 x 16 167 / 281 us, 1 M x 24 545 / 1,038, 4 M x 16 1,607 / 3,459); below 128 up to
// FLOW_WIDE_MAX_N vertices, the largest size measured, since the wide kernel keeps half as many vertices in
// flight (250,000 x 40 363 / 397, 500,000 x 34 461 / 639, 1 M x 34 939 / 1,185), and not where the mean degree is
// below FLOW_WIDE_MEAN: there most vertices are a whole warp's work for a few entries (arity-100 tree of 2^20
// vertices, dataflow / tickets: random priorities 429 / 248, first fit 213 / 187).  Larger degrees would put long
// lists on the chain, and power-law graphs have their chains colored inside one cluster (k_jp_core).
// (The line is the whole graph's: one vertex of 200 neighbours sends a mesh to the tickets, 112^3 first fit 1.4 -> 6.8 ms
// by two streams.)
// Plain graphs only: the rule, the masks' width and the queues are one graph's.  And no nearly complete graphs: one
// chain, for the cluster.
constexpr uint32_t FLOW_WIDE_MAX_N = 1u << 20, FLOW_WIDE_MEAN = 4, FLOW_CLIQUE = 100;

bool gc_flow_eligible(const gc_graph *g) {
    const bool wide = g->N <= FLOW_WIDE_MAX_N && g->M / FLOW_WIDE_MEAN >= g->N;
    const uint32_t widest = wide ? 32u * FLOW_WIDE : 64u;
    if (g->N > FLOW_CLIQUE && gc_nearly_complete(g)) return false;
    return g->n_seg == 0 && g->N > 0 && g->max_deg < std::min(g->ctx->flow_max_deg, widest);
}

// Counters and slots (two words each).  They share the sort's scratch, so that a graph which the tickets color after
// all holds no more than they need.
size_t gc_flow_queue_words(uint32_t cap_N) {
    return 2 * ((size_t)cap_N + 1024 * FLOW_QUEUES) + FLOW_SLOTS;
}

gc_status gc_jp_flow(gc_graph *g) {
    gc_ctx *ctx = g->ctx;
    gc_status s;
    const bool wide = g->max_deg >= 64;
    const uint32_t stride = ((g->N + FLOW_QUEUES - 1) / FLOW_QUEUES + 1023u) & ~1023u;
    if ((s = gc_alloc(ctx, &g->jprec, g->cap_N, "vertex records")) != GC_OK) return s;
    if (wide && (s = gc_alloc(ctx, &g->jpsplit, g->cap_N, "vertex records")) != GC_OK) return s;
    if ((s = gc_sort_scratch(g)) != GC_OK) return s;
    return wide ? flow_run<FLOW_WIDE>(g, stride) : g->max_deg >= 32 ? flow_run<2>(g, stride) : flow_run<1>(g, stride);
}
