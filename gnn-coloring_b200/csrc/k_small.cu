// Small graphs: Jones-Plassmann, Culberson rounds and the color count of one graph in one CTA, out of shared
// memory (reference src/coloring.c:223-330).
//
// A graph of a few thousand vertices is all latency in the other kernels: a hop of a priority chain is an L2
// atomic and an L2 load (0.7 to 1.7 us in k_flow.cu), and a round takes three launches more.  Here the CSR
// (16-bit ids), the counters and the colors are in one SM's shared memory, and all rounds and the color
// count run in one launch that writes its result to the host's state.
//
// Level by level: q holds the vertices of a level (no uncolored predecessor is left), a barrier ends it.  A
// vertex's colored neighbours are exactly its predecessors: a successor waits for it, and two vertices of a
// level are not adjacent.  So one pass over its list collects the predecessors' colors and subtracts one from
// the counter of each uncolored neighbour; who takes one to zero puts that vertex into the next level.
// Eight lanes per vertex; 32 in levels of up to 32 vertices and for more than HEAVY neighbours, which are
// queued from the other end of q.
//
// That reading of "colored" needs a symmetric CSR: with one-sided entries a vertex could start before a
// predecessor, and its color would follow the warps' timing.  So the first counting pass also adds up a hash of
// every entry (u, v) that is the negative of (v, u)'s.  The sum of a symmetric CSR is zero; any other graph's is
// not (but for a chance of 2^-32), and the other kernels, which ask each entry who precedes, color it.
//
// What bounds it: a level's serial chain, about 1,400 cycles (barrier, queue, list, colors, two shared atomics),
// and in wide levels the SM's instruction rate.  Erdos-Renyi 1,000 x 16 first fit (36 levels): 71,000 cycles,
// 4,800 of them loading, 54,500 levels; the call 94 -> 53 us.  512 threads 59 us, 256 threads 65.  Eight lanes
// per vertex in the counting passes took 11,000 cycles each where one takes 6,000.
#include <algorithm>
#include <cstddef>

#include "gc_internal.h"

namespace {
using namespace gc;

constexpr int SMALL_THREADS = 1024;
constexpr uint32_t HEAVY = 96, LONG = 64;
// A coloring whose levels are mostly of SLIM vertices or fewer is a chain, 0.6 us a level here and 0.1 to 0.3 among
// tickets inside a cluster (k_jp_core).  So after SLIM_LEVELS of those, with half of the vertices to come, this kernel
// gives up (FLOW_NARROW): 3,000 vertices in a path 1.78 / 0.93 ms, 2,900 rows of a band with 15 entries on either side 1.72 /
// 0.57.  (One warp that colors such levels without barriers takes 0.42 us for each.)
constexpr uint32_t SLIM = 3, SLIM_LEVELS = 128;
constexpr size_t SMALL_BYTES = 226 * 1024;  // (a CTA may have 227 KB; the rest is static)
constexpr unsigned int FULL = 0xffffffffu;

__host__ __device__ inline uint32_t even(uint32_t n) { return (n + 1u) & ~1u; }

constexpr uint32_t HEAD = 8;

size_t small_bytes(uint32_t N, uint32_t M) { return 4ull * (HEAD + 2ull * N + 1) + 2ull * (3ull * even(N) + M); }

// Shared memory, as offsets from its base (so that every access is known to be a shared one).
extern __shared__ uint32_t sm[];
struct Small {
    uint32_t N, rem_, a_, b_, q_, ids_;  // rem_ in words, the others in half words
    __device__ __forceinline__ uint32_t &off(uint32_t i) const { return sm[HEAD + i]; }        // first entry of a list
    __device__ __forceinline__ uint32_t &rem(uint32_t i) const { return sm[rem_ + i]; }        // uncolored predecessors
    __device__ __forceinline__ uint16_t &half(uint32_t i) const { return reinterpret_cast<uint16_t *>(sm)[i]; }
    __device__ __forceinline__ uint16_t &a(uint32_t i) const { return half(a_ + i); }          // colors of this coloring
    __device__ __forceinline__ uint16_t &b(uint32_t i) const { return half(b_ + i); }          // and of the one before
    __device__ __forceinline__ uint16_t &q(uint32_t i) const { return half(q_ + i); }          // level queue
    __device__ __forceinline__ uint16_t &ids(uint32_t i) const { return half(ids_ + i); }      // neighbours
    __device__ __forceinline__ uint32_t &light(uint32_t i) const { return sm[i]; }  // vertices queued for the levels
    __device__ __forceinline__ uint32_t &heavy(uint32_t i) const { return sm[4 + i]; }  // l, l + 1, l + 2 (mod 3)
};

constexpr uint32_t BIG = 1u << 31;  // in rem: more than HEAVY neighbours

__device__ __forceinline__ void push(const Small &s, uint32_t v, bool big, uint32_t lbase, uint32_t hbase, uint32_t slot) {
    const uint32_t at = big ? hbase + atomicAdd(&s.heavy(slot), 1u) : lbase + atomicAdd(&s.light(slot), 1u);
    if (at < s.N) s.q(big ? s.N - 1 - at : at) = (uint16_t)v;
}

// Over all vertices with their entries: g(u, the sum of f(u, v), whether u has more than HEAVY).  One vertex
// per thread, since the SM's instruction rate is what bounds this; long lists by whole warps.
template <class F, class G>
__device__ __forceinline__ void for_vertices(const Small &s, F f, G g) {
    const int lane = threadIdx.x & 31;
    for (uint32_t base = threadIdx.x & ~31u; base < s.N; base += blockDim.x) {
        const uint32_t u = base + lane;
        const uint32_t beg = u < s.N ? s.off(u) : 0u, end = u < s.N ? s.off(u + 1) : 0u, d = end - beg;
        if (u < s.N && d <= LONG) {
            uint32_t sum = 0, j = beg;
            for (; j + 4 <= end; j += 4) {
                const uint32_t v0 = s.ids(j), v1 = s.ids(j + 1), v2 = s.ids(j + 2), v3 = s.ids(j + 3);
                sum += f(u, v0) + f(u, v1) + f(u, v2) + f(u, v3);
            }
            for (; j < end; j++) sum += f(u, s.ids(j));
            g(u, sum, false);
        }
        for (unsigned int m = __ballot_sync(FULL, d > LONG); m; m &= m - 1) {
            const int src = __ffs(m) - 1;
            const uint32_t x = base + src, xe = __shfl_sync(FULL, end, src), xd = __shfl_sync(FULL, d, src);
            uint32_t t = 0;
#pragma unroll 4
            for (uint32_t j = xe - xd + lane; j < xe; j += 32) t += f(x, s.ids(j));
            t = __reduce_add_sync(FULL, t);
            if (lane == 0) g(x, t, xd > HEAVY);
        }
    }
}

// Colors u by G lanes with UN entries in flight each (32 / G vertices per warp, all lanes take part; `valid`: this group
// has a vertex).
template <int G, int UN>
__device__ __forceinline__ void color_vertex(const Small &s, uint32_t u, bool valid, uint32_t lbase, uint32_t hbase,
                                             uint32_t slot) {
    const int gl = threadIdx.x & (G - 1);
    const uint32_t beg = valid ? s.off(u) : 0u, d = valid ? s.off(u + 1) - beg : 0u;
    auto group_or = [](uint32_t x) {
        if constexpr (G == 32) {
            return __reduce_or_sync(FULL, x);
        } else {
#pragma unroll
            for (int o = 1; o < G; o <<= 1) x |= __shfl_xor_sync(FULL, x, o);
            return x;
        }
    };
    uint32_t m = 0;  // colors 1..32
    for (uint32_t j = gl; j < d; j += UN * G) {
        uint32_t v[UN], c[UN], old[UN];
#pragma unroll
        for (int k = 0; k < UN; k++) v[k] = j + G * k < d ? s.ids(beg + j + G * k) : u;
#pragma unroll
        for (int k = 0; k < UN; k++) c[k] = s.a(v[k]);
#pragma unroll
        for (int k = 0; k < UN; k++) old[k] = c[k] == 0 && (k == 0 || j + G * k < d) ? atomicSub(&s.rem(v[k]), 1u) : 0u;
#pragma unroll
        for (int k = 0; k < UN; k++)
            if (c[k] - 1 < 32) m |= 1u << (c[k] - 1);
#pragma unroll
        for (int k = 0; k < UN; k++)
            if ((old[k] & ~BIG) == 1u) push(s, v[k], old[k] & BIG, lbase, hbase, slot);
    }
    __syncwarp();
    m = group_or(m);
    uint32_t c = ~m ? (uint32_t)__ffs(~m) : 0u;
    for (uint32_t w = 32; __any_sync(FULL, c == 0); w += 32) {  // colors w + 1 .. w + 32
        m = 0;
        for (uint32_t j = gl; j < d; j += G) {
            const uint32_t x = s.a(s.ids(beg + j)) - w - 1;
            if (x < 32) m |= 1u << x;
        }
        __syncwarp();
        m = group_or(m);
        if (c == 0 && ~m) c = w + (uint32_t)__ffs(~m);
    }
    if (valid && gl == 0) s.a(u) = (uint16_t)c;
}

// A hash of the entry (u, v), the negative of that of (v, u): the pair by multiplicative hashing (Knuth, The
// Art of Computer Programming 3, 6.4) twice, signed by its order.  A self-loop counts as symmetric.
__device__ __forceinline__ uint32_t entry_hash(uint32_t u, uint32_t v) {
    uint32_t h = (min(u, v) << 16 | max(u, v)) * 0x9e3779b9u;
    h = (h ^ h >> 15) * 0x9e3779b9u;
    h ^= h >> 16;
    return u < v ? h : u > v ? 0u - h : 0u;
}

__global__ void __launch_bounds__(SMALL_THREADS, 1) k_small(const uint32_t *__restrict__ V, const uint32_t *__restrict__ E,
                                                            uint32_t *key, uint32_t N, uint32_t M, int rounds, bool stats,
                                                            int *__restrict__ color, DevState *state) {
    __shared__ uint32_t invalid, top, sides;  // sides: the entries' hashes, zero for a symmetric CSR
    Small s;
    s.N = N;
    s.rem_ = HEAD + N + 1;
    s.a_ = 2 * (s.rem_ + N);
    s.b_ = s.a_ + even(N);
    s.q_ = s.b_ + even(N);
    s.ids_ = s.q_ + even(N);
    const uint32_t t = threadIdx.x, warp = t >> 5, lane = t & 31, nwarps = blockDim.x >> 5;
    uint32_t *ks = sm + s.rem_ + N;  // the first coloring's keys, until the colors take their place
    for (uint32_t i = t; i <= N; i += blockDim.x) s.off(i) = V[i];
    for (uint32_t i = t; i < N; i += blockDim.x) ks[i] = key[i];
    for (uint32_t i = t; i < M; i += 16 * blockDim.x) {
        uint32_t v[16];
#pragma unroll
        for (int k = 0; k < 16; k++) v[k] = i + k * blockDim.x < M ? ld_stream(E + i + k * blockDim.x) : 0u;
#pragma unroll
        for (int k = 0; k < 16; k++)
            if (i + k * blockDim.x < M) s.ids(i + k * blockDim.x) = (uint16_t)v[k];
    }
    if (t < 3) s.light(t) = s.heavy(t) = 0;
    if (t == 0) invalid = top = sides = 0;
    bool done = true;
    uint32_t hashes = 0, slim = 0;
    for (int it = 0; it <= rounds; it++) {
        __syncthreads();
        auto found = [&](uint32_t u, uint32_t cnt, bool big) {
            s.rem(u) = cnt | (big ? BIG : 0u);
            if (cnt == 0) push(s, u, big, 0, 0, 0);
        };
        if (it == 0) {
            for_vertices(s, [&](uint32_t u, uint32_t v) {
                hashes += entry_hash(u, v);
                return precedes(ks[v], v, ks[u], u) ? 1u : 0u;
            }, found);
            hashes = __reduce_add_sync(FULL, hashes);
            if (lane == 0) atomicAdd(&sides, hashes);
        } else for_vertices(s, [&](uint32_t u, uint32_t v) { return precedes(s.b(v), v, s.b(u), u) ? 1u : 0u; }, found);
        __syncthreads();
        if (sides) {
            done = false;
            break;
        }
        if (it == 0)
            for (uint32_t i = t; i < N; i += blockDim.x) ks[i] = 0;  // (both color arrays)
        uint32_t la = 0, ha = 0;
        for (uint32_t l = 0;; l = l == 2 ? 0 : l + 1) {
            __syncthreads();
            const uint32_t nl = s.light(l), nh = s.heavy(l), next = l == 2 ? 0 : l + 1;
            if (t == 0) s.light(l == 0 ? 2 : l - 1) = s.heavy(l == 0 ? 2 : l - 1) = 0;
            if (nl + nh == 0) break;
            if (it == 0 && nl + nh <= SLIM && ++slim > SLIM_LEVELS && la + ha < N / 2) break;
            const uint32_t per = nl > nwarps ? 4u : 1u, items = nh + (nl + per - 1) / per;
            const uint32_t lb = la + nl, hb = ha + nh;
            for (uint32_t i = warp; i < items; i += nwarps) {
                if (i < nh) {
                    color_vertex<32, 4>(s, s.q(N - 1 - (ha + i)), true, lb, hb, next);
                } else if (per == 1) {
                    color_vertex<32, 1>(s, s.q(la + i - nh), true, lb, hb, next);
                } else {
                    const uint32_t at = la + 4 * (i - nh) + (lane >> 3);
                    color_vertex<8, 2>(s, at < lb ? s.q(at) : 0u, at < lb, lb, hb, next);
                }
            }
            la = lb;
            ha = hb;
        }
        __syncthreads();
        if (t < 3) s.light(t) = s.heavy(t) = 0;
        done = la + ha == N;
        if (done) slim = 0;
        if (!done || it == rounds) break;
        const uint32_t x = s.a_;  // the next keys are these colors
        s.a_ = s.b_;
        s.b_ = x;
        for (uint32_t i = t; i < N; i += blockDim.x) s.a(i) = 0;
    }
    if (done) {
        uint32_t most = 0;
        for (uint32_t i = t; i < N; i += blockDim.x) {
            color[i] = s.a(i);
            if (rounds) key[i] = s.b(i);
            most = max(most, (uint32_t)s.a(i));
        }
        if (stats) {
            most = __reduce_max_sync(FULL, most);
            if (lane == 0) atomicMax(&top, most);
            for_vertices(s, [&](uint32_t u, uint32_t v) { return s.a(u) == s.a(v) ? 1u : 0u; },
                         [&](uint32_t, uint32_t bad, bool) { if (bad) invalid = 1u; });
        }
    }
    __syncthreads();
    if (t < sizeof(DevState) / 4)  // (the host's copy)
        reinterpret_cast<uint32_t *>(state)[t] = t == offsetof(DevState, max_color) / 4    ? top
                                                 : t == offsetof(DevState, invalid) / 4    ? invalid
                                                 : t == offsetof(DevState, flow_stall) / 4 ? (done ? 0u : slim > SLIM_LEVELS ? FLOW_NARROW : FLOW_STUCK)
                                                                                           : 0u;
}

}  // namespace

// Graphs whose CSR and working arrays fit one SM's shared memory, up to the sizes at which one SM's
// instruction rate costs more than the other kernels' latency.  Against the dataflow kernel that is a matter
// of vertices (calls with first fit or largest degree first, other kernels / this one: Erdos-Renyi 1,000 x 16
// 88 / 55 us, 2,000 x 16 90 / 71, 3,000 x 24 119 / 109, 4,000 x 12 79 / 87, 6,000 x 8 68 / 93; with two rounds
// 201 / 89, 208 / 120, 264 / 200, 210 / 168, 203 / 186), against the ticket kernels, whose graphs have long lists
// and many levels, one of entries (R-MAT 1,000 x 16, 12,000 entries 125 / 86, 1,000 x 32, 21,000 128 / 119, 1,400
// x 32, 28,000 124 / 145; with two rounds 274 / 164, 320 / 223, 312 / 278, 4,000 x 16, 52,000 371 / 447).  A quarter
// of all entries and more makes a chain of nearly all vertices, which the cluster takes faster from some hundred on
// (tickets / this: cliques of 64 139 / 73 us, of 120 160 / 188, of 140 174 / 243).
constexpr uint32_t SMALL_CLIQUE = 100;

bool gc_small_eligible(const gc_graph *g, int rounds) {
    if (g->n_seg || !g->N || small_bytes(g->N, g->M) > SMALL_BYTES) return false;
    const uint32_t most = g->ctx->small_max;
    if (most != GC_SMALL_AUTO) return g->N <= std::min<uint32_t>(most, 65535u);
    if (g->N > SMALL_CLIQUE && gc_nearly_complete(g)) return false;
    return gc_flow_eligible(g) ? g->N <= (rounds ? 6144u : 3072u) : g->M <= (rounds ? 36864u : 20480u);
}

gc_status gc_small_color(gc_graph *g, int rounds, bool stats) {
    gc_ctx *ctx = g->ctx;
    gc_status s;
    if (!ctx->small_ready) {
        if ((s = gc_check_cuda(ctx, cudaFuncSetAttribute(k_small, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMALL_BYTES),
                               "small graph smem")) != GC_OK)
            return s;
        ctx->small_ready = true;
    }
    {
        ProfScope ps(ctx, "jp_small", ctx->stream);
        k_small<<<1, SMALL_THREADS, small_bytes(g->N, g->M), ctx->stream>>>(g->V, g->E, g->key, g->N, g->M, rounds, stats,
                                                                           g->color, ctx->hstate);
        ctx->launches++;
    }
    if ((s = gc_check_launch(ctx, "small graph")) != GC_OK) return s;
    if ((s = gc_check_cuda(ctx, cudaStreamSynchronize(ctx->stream), "kernel execution")) != GC_OK) return s;
    if (ctx->hstate->flow_stall) return GC_OK;
    if (rounds) g->key_kind = 100;
    g->has_keys = g->has_colors = g->colors_ours = true;
    return GC_OK;
}
