// Integer priority heuristics on the device.
//
//   FF  key = N - u                      (reference src/first_fit.c:8-12)
//   LF  key = deg(u)                     (src/largest_degree_first.c:12-16)
//   LLF key = 32 - clz(deg), 0 if deg=0  (src/largest_degree_first.c:87-97)
//   SL / SLL  bucket peeling             (src/smallest_degree_last.c:155-246, :359-443)
//
// Keys are uint32; the coloring orders vertices by (key, id) descending, exactly like the
// reference's double comparisons on these integer-valued priorities.
#include <algorithm>

#include "gc_internal.h"

namespace {
using gc::ld_stream;

// FF in a segmented CSR: N - u with the graph's own N and local u, i.e. (end of u's graph) - u.
__global__ void k_simple_keys(const uint32_t *__restrict__ V, uint32_t N, int h, const uint32_t *__restrict__ voff,
                              uint32_t nseg, uint32_t *__restrict__ key) {
    for (uint32_t u = blockIdx.x * blockDim.x + threadIdx.x; u < N; u += gridDim.x * blockDim.x) {
        uint32_t k;
        if (h == GC_FF) {
            k = (nseg ? __ldg(voff + gc::seg_of(voff, nseg, u) + 1) : N) - u;
        } else {
            uint32_t d = V[u + 1] - V[u];
            k = (h == GC_LF) ? d : (d ? 32u - (uint32_t)__clz(d) : 0u);
        }
        key[u] = k;
    }
}

// ---- bucket peeling -----------------------------------------------------------------------------
//
// Round r removes every remaining vertex whose remaining degree is <= threshold (delta for SL,
// 2^delta for SLL), gives it key = delta, and takes one degree off each remaining neighbour per
// removed neighbour.  SL then sets delta = max(delta + 1, smallest remaining degree); SLL sets
// delta + 1.  Removal within a round depends only on the degrees at the round's start and the
// decrements commute, so the keys equal the reference's at any thread count.
//
// All rounds run in one cooperative kernel, a CTA of 1,024 threads per SM.  A power-law graph has hundreds
// of rounds, most of which remove a few vertices, so a round is bound by its latencies: a grid barrier (1.9
// us) and a few dependent loads.
//   - While the remaining vertices are more than the threads can keep (four each), a round is filter, barrier,
//     decrement, barrier: the filter scans a list of them and puts the removed ones on lists.
//   - After that every thread keeps its own vertices and their degrees in registers, and a round has one
//     barrier.  Round r counts neighbours down in array r mod 2, and in round r + 1 the owner of a vertex
//     takes what that array has lost since it last looked off the vertex's degree.  So nobody reads what
//     others are counting down, and a removed vertex's neighbours are counted down at once: lists of up to
//     PEEL_WARP_DEG by its warp, eight lanes each, longer ones by its CTA.
//   - The decrements go to every neighbour without asking whether it is still there (nothing reads a removed vertex's
//     degree again), so nothing waits for their results.  They do ask where most vertices of a graph with a mean
//     degree of PEEL_DENSE and more leave together: in the first round of a graph whose vertices are all kept, by
//     their lists' lengths, and after a round over lists that took three quarters of what there was, by the degrees,
//     which then say GONE.  SLL on Erdos-Renyi graphs of 300,000 x 200 and 1 M x 100: 578 and 851 us without asking,
//     404 and 575 so.
//   - SL tries delta + 1 first; only when that removes nothing does it look for the smallest remaining
//     degree (one more barrier).
//   - The barrier's counter and the round's count are one 64-bit word, polled by one thread per CTA: a scalar
//     that only atomics change, so whoever reads the last arrival reads the final count.
// Measured (B200), three launches per round queued in batches -> this: SL on R-MAT of 2^20 vertices and
// edge factor 16 (217 rounds) 8.2 -> 1.6 ms, on Erdos-Renyi 65,536 (16 rounds) 0.41 -> 0.09 ms.  With two
// barriers in every round and long lists shared by the grid: 1.9 and 0.10.  Rounds that remove thousands
// take longer (decrements of the same hubs, one at a time).  All removed vertices on lists: 2.2 ms; a whole
// warp for every kept one: 2.3 ms.
constexpr uint32_t GONE = 0xffffffffu;
constexpr uint32_t NO_DEGREE = 0xffffffffu;
constexpr int PEEL_THREADS = 1024;
constexpr int PEEL_ITEMS = 4;              // vertices a thread keeps
constexpr uint32_t PEEL_WARP_DEG = 64;
constexpr uint32_t PEEL_WIDE = 512;
constexpr uint32_t PEEL_MOST_MUL = 3, PEEL_MOST_DIV = 4, PEEL_DENSE = 32;
constexpr unsigned int PEEL_WAIT_LIMIT = 1u << 24;  // polls of one barrier

struct PeelSlot {
    unsigned long long word;  // arrivals at the filter's barrier; above bit 32 the removed vertices on the short
                              // list (or kept by their warps)
    unsigned int longs;       // removed vertices on the long list
    unsigned int packed;      // remaining vertices on the next list
};

struct PeelState {
    PeelSlot slot[3];      // round r in slot r mod 3, cleared a round ahead
    unsigned int pad0[20];
    unsigned int arrived;  // arrivals at the other barriers so far
    unsigned int pad1[31];
    unsigned int min_deg[3];  // smallest remaining degree, when a round needs it (slots as above)
    unsigned int min0;     // smallest degree of the graph
    unsigned int failed;   // a barrier wait expired
    unsigned int rounds;   // rounds run (written at the end)
};

__device__ __forceinline__ void red_release(unsigned int *p) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(p) : "memory");
}
__device__ __forceinline__ unsigned int ld_acquire(const unsigned int *p) {
    unsigned int v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void red_release_u64(unsigned long long *p) {
    asm volatile("red.release.gpu.global.add.u64 [%0], 1;" ::"l"(p) : "memory");
}
__device__ __forceinline__ bool peel_expired(PeelState *ps, unsigned int &spins) {
    return ++spins > PEEL_WAIT_LIMIT || ((spins & 255u) == 0 && gc::ld_relaxed_u32(&ps->failed));
}

// Grid barriers: every CTA's earlier writes are visible to all after them.  False when the wait expired
// (in some CTA).  One thread per CTA polls (thousands of warps asking one address would queue for
// microseconds).  The first kind arrives at a round's slot and returns its counts, which are complete when
// all CTAs have arrived, since each adds to them before it arrives; those of the lists are read on request.
struct PeelCounts {
    uint32_t removed, longs, packed;
};

template <bool LISTS>
__device__ __forceinline__ bool peel_slot_barrier(PeelState *ps, PeelSlot *slot, PeelCounts &got) {
    __shared__ uint4 got_s;
    __syncthreads();
    if (threadIdx.x == 0) {
        red_release_u64(&slot->word);
        unsigned int spins = 0, good = 1;
        unsigned long long v;
        while ((uint32_t)(v = gc::ld_relaxed_u64(&slot->word)) != gridDim.x)
            if (peel_expired(ps, spins)) {
                gc::st_relaxed_u32(&ps->failed, 1u);
                good = 0;
                break;
            }
        asm volatile("fence.acq_rel.gpu;" ::: "memory");
        got_s = make_uint4(good, (uint32_t)(v >> 32), LISTS ? gc::ld_relaxed_u32(&slot->longs) : 0u,
                           LISTS ? gc::ld_relaxed_u32(&slot->packed) : 0u);
    }
    __syncthreads();
    got = PeelCounts{got_s.y, got_s.z, got_s.w};
    return got_s.x != 0;
}
// `read`: a word to return in `value` (may be null).
__device__ __forceinline__ bool peel_barrier(PeelState *ps, unsigned int &target, const unsigned int *read, unsigned int &value) {
    __shared__ unsigned int ok, value_s;
    __syncthreads();
    if (threadIdx.x == 0) {
        target += gridDim.x;
        red_release(&ps->arrived);
        unsigned int spins = 0, good = 1;
        while ((int)(ld_acquire(&ps->arrived) - target) < 0)
            if (peel_expired(ps, spins)) {
                gc::st_relaxed_u32(&ps->failed, 1u);
                good = 0;
                break;
            }
        ok = good;
        if (read) value_s = gc::ld_relaxed_u32(read);
    }
    __syncthreads();
    if (read) value = value_s;
    return ok;
}

// One degree off the neighbours E[j], E[j + step], ... below end for which there(v) holds.
template <class F>
__device__ __forceinline__ void peel_neighbours(const uint32_t *__restrict__ E, uint32_t j, uint32_t end, uint32_t step,
                                                uint32_t *deg, F there) {
    for (; j < end && end - j > 3 * step; j += 4 * step) {
        const uint32_t a = ld_stream(E + j), b = ld_stream(E + j + step), c = ld_stream(E + j + 2 * step),
                       d = ld_stream(E + j + 3 * step);
        const bool ta = there(a), tb = there(b), tc = there(c), td = there(d);
        if (ta) atomicSub(deg + a, 1u);
        if (tb) atomicSub(deg + b, 1u);
        if (tc) atomicSub(deg + c, 1u);
        if (td) atomicSub(deg + d, 1u);
    }
    for (; j < end; j += step) {
        const uint32_t a = ld_stream(E + j);
        if (there(a)) atomicSub(deg + a, 1u);
        if (end - j <= step) break;
    }
}

__global__ void __launch_bounds__(PEEL_THREADS, 1) k_peel(const uint32_t *__restrict__ V, const uint32_t *__restrict__ E,
                                                         uint32_t N, int log_mode, uint32_t *deg, uint32_t *list0,
                                                         uint32_t *list1, uint32_t *removed, uint32_t *__restrict__ key,
                                                         PeelState *ps) {
    constexpr unsigned int FULL = 0xffffffffu;
    constexpr int ITEMS = PEEL_ITEMS;
    __shared__ unsigned int cta_min;
    __shared__ uint2 own[PEEL_THREADS / 32][32 * ITEMS];  // per warp: the lists it decrements
    __shared__ uint2 wide[PEEL_WIDE];                     // long lists that the CTA shares
    __shared__ unsigned int wide_n[2];                    // their number, by the round's parity
    const int lane = threadIdx.x & 31;
    const unsigned int lt = (1u << lane) - 1u;
    const uint32_t tid = blockIdx.x * PEEL_THREADS + threadIdx.x, threads = gridDim.x * PEEL_THREADS;
    unsigned int target = 0, value = 0;
    const bool dense = V[N] / PEEL_DENSE >= N;
    // the smallest of the threads' values, for all
    auto grid_min = [&](uint32_t v, unsigned int *at) {
        if (threadIdx.x == 0) cta_min = NO_DEGREE;
        __syncthreads();
        v = __reduce_min_sync(FULL, v);
        if (lane == 0 && v != NO_DEGREE) atomicMin(&cta_min, v);
        __syncthreads();
        if (threadIdx.x == 0 && cta_min != NO_DEGREE) atomicMin(at, cta_min);
        return peel_barrier(ps, target, at, value);
    };
    uint32_t low = NO_DEGREE;
    for (uint32_t u = tid; u < N; u += threads) {
        const uint32_t d = V[u + 1] - V[u];
        deg[u] = d;
        list0[u] = u;
        low = min(low, d);
    }
    if (!grid_min(low, &ps->min0)) return;
    uint32_t delta = value;
    if (log_mode) {
        delta = 0;
        while (delta < 32 && (1ull << delta) < (unsigned long long)value) delta++;
    }
    uint32_t alive = N, len = N, r = 0;
    uint32_t *cur = list0, *other = list1;
    uint32_t u[ITEMS], d[ITEMS], beg[ITEMS], end[ITEMS];
    PeelCounts got;
    bool done = false;
    auto round_end = [&]() {  // once the decrements are out; the slots of the round after next are free
        if (tid == 0) {
            ps->slot[(r + 2) % 3] = PeelSlot{0ull, 0u, 0u};
            ps->min_deg[(r + 2) % 3] = NO_DEGREE;
        }
        return peel_barrier(ps, target, nullptr, value);
    };
    auto threshold = [&]() { return !log_mode ? delta : delta < 32 ? 1u << delta : 0xffffffffu; };
    // The neighbours of n listed vertices (list[0], list[dir], ...), each shared by as many lanes as there are
    // for it: a power of two, at least `few`.
    auto decrement = [&](const uint32_t *list, int dir, uint32_t n, uint32_t few, bool ask) {
        const uint32_t most = threads / n;
        const uint32_t lanes = most <= few ? few : 1u << (31 - __clz(most)), groups = threads / lanes;
        if (tid < groups * lanes)
            for (uint32_t i = tid / lanes; i < n; i += groups) {
                const uint32_t x = __ldcg(list + (long long)dir * i);
                const uint32_t j = V[x] + (tid & (lanes - 1u)), e = V[x + 1];
                if (ask) peel_neighbours(E, j, e, lanes, deg, [&](uint32_t v) { return (int)__ldcg(deg + v) >= 0; });
                else peel_neighbours(E, j, e, lanes, deg, [](uint32_t) { return true; });
            }
    };
    // ---- the remaining vertices on a list
    for (bool pack = false; len > threads * ITEMS; r++) {
        PeelSlot *sl = &ps->slot[r % 3];
        const uint32_t thr = threshold();
        // short: at most 16 neighbours for each of the lanes a vertex is sure to get in the decrement (a
        // removed vertex has about as many neighbours as the threshold)
        const uint32_t few = thr <= 8 ? 4u : thr <= 32 ? 8u : 32u, long_deg = 16u * few;
        low = NO_DEGREE;
        for (uint32_t base = (tid & ~31u) * ITEMS; base < len; base += threads * ITEMS) {
#pragma unroll
            for (int k = 0; k < ITEMS; k++) {
                const uint32_t i = base + 32 * k + lane;
                u[k] = i < len ? __ldcg(cur + i) : GONE;
            }
#pragma unroll
            for (int k = 0; k < ITEMS; k++) d[k] = u[k] != GONE ? __ldcg(deg + u[k]) : 0u;
#pragma unroll
            for (int k = 0; k < ITEMS; k++) {  // (lists of the removed ones, all in flight)
                beg[k] = end[k] = 0;
                if (u[k] != GONE && d[k] <= thr) {
                    beg[k] = V[u[k]];
                    end[k] = V[u[k] + 1];
                    key[u[k]] = delta;
                    deg[u[k]] = GONE;
                    if (!pack) cur[base + 32 * k + lane] = GONE;
                }
            }
            uint32_t kept = 0, shorts = 0, longs = 0;
#pragma unroll
            for (int k = 0; k < ITEMS; k++) {
                const bool there = u[k] != GONE, rm = there && d[k] <= thr, is_long = end[k] - beg[k] > long_deg;
                if (there && !rm) low = min(low, d[k]);
                shorts += __popc(__ballot_sync(FULL, rm && !is_long));
                longs += __popc(__ballot_sync(FULL, is_long));
                if (pack) kept += __popc(__ballot_sync(FULL, there && !rm));
            }
            if (shorts | longs) {
                uint32_t at = 0;
                if (lane == 0 && shorts) at = (uint32_t)(atomicAdd(&sl->word, (unsigned long long)shorts << 32) >> 32);
                if (lane == 1 && longs) at = atomicAdd(&sl->longs, longs);
                uint32_t as = __shfl_sync(FULL, at, 0), al = __shfl_sync(FULL, at, 1);
#pragma unroll
                for (int k = 0; k < ITEMS; k++) {
                    const bool rm = u[k] != GONE && d[k] <= thr, is_long = end[k] - beg[k] > long_deg;
                    const unsigned int ms = __ballot_sync(FULL, rm && !is_long), ml = __ballot_sync(FULL, is_long);
                    if (rm && !is_long) removed[as + __popc(ms & lt)] = u[k];
                    if (is_long) removed[N - 1u - (al + __popc(ml & lt))] = u[k];
                    as += __popc(ms);
                    al += __popc(ml);
                }
            }
            if (pack && kept) {
                uint32_t at = 0;
                if (lane == 0) at = atomicAdd(&sl->packed, kept);
                at = __shfl_sync(FULL, at, 0);
#pragma unroll
                for (int k = 0; k < ITEMS; k++) {
                    const bool keep = u[k] != GONE && d[k] > thr;
                    const unsigned int mk = __ballot_sync(FULL, keep);
                    if (keep) other[at + __popc(mk & lt)] = u[k];
                    at += __popc(mk);
                }
            }
        }
        if (!peel_slot_barrier<true>(ps, sl, got)) return;
        const uint32_t ns = got.removed, nl = got.longs;
        if (pack) {
            len = got.packed;
            uint32_t *t = cur;
            cur = other;
            other = t;
        }
        const bool ask = dense && ns + nl >= alive / PEEL_MOST_DIV * PEEL_MOST_MUL;
        alive -= ns + nl;
        if (alive == 0) {
            done = true;
            break;
        }
        if (nl) decrement(removed + (N - 1u), -1, nl, PEEL_THREADS, ask);
        if (ns) decrement(removed, 1, ns, few, ask);
        pack = alive < len - len / 4 || alive <= threads * ITEMS;
        if (ns + nl == 0 && !log_mode) {  // nothing has this degree: the next threshold is the smallest left
            if (!grid_min(low, &ps->min_deg[r % 3])) return;
            delta = max(delta, value);
        } else {
            delta++;
        }
        if (!round_end()) return;
    }
    // ---- each thread keeps its vertices and their degrees (neighbouring list entries in different warps: the
    // list is close to id order, and vertices that leave together are often neighbours in it)
    uint32_t seen[ITEMS], seen_next[ITEMS];  // a kept vertex's counters when they were last read
    if (!done) {
        const uint32_t slot0 = (threadIdx.x >> 5) * gridDim.x + blockIdx.x, warps = threads >> 5;
        const uint32_t *past = (r & 1) ? deg : other, *next = (r & 1) ? other : deg;
#pragma unroll
        for (int k = 0; k < ITEMS; k++) {
            const uint32_t i = ((uint32_t)k * 32u + lane) * warps + slot0;
            u[k] = i < len ? __ldcg(cur + i) : GONE;
            beg[k] = end[k] = d[k] = seen[k] = seen_next[k] = 0;
            if (u[k] != GONE) {
                beg[k] = V[u[k]];
                end[k] = V[u[k] + 1];
                d[k] = __ldcg(deg + u[k]);
                seen[k] = __ldcg(past + u[k]);
                seen_next[k] = __ldcg(next + u[k]);
            }
        }
        if (threadIdx.x < 2) wide_n[threadIdx.x] = 0;
        if (!peel_barrier(ps, target, nullptr, value)) return;  // (nothing is counted down before all have read)
    }
    for (; !done; r++) {
        PeelSlot *sl = &ps->slot[r % 3];
        const uint32_t thr = threshold();
        const uint32_t *past = (r & 1) ? deg : other;
        uint32_t *count = (r & 1) ? other : deg;
        const bool ask = dense && r == 0;  // (every vertex still has all its neighbours)
        auto count_down = [&](uint2 list, uint32_t from, uint32_t step) {
            if (ask) peel_neighbours(E, list.x + from, list.y, step, count, [&](uint32_t v) { return V[v + 1] - V[v] > thr; });
            else peel_neighbours(E, list.x + from, list.y, step, count, [](uint32_t) { return true; });
        };
        low = NO_DEGREE;
        uint32_t rm = 0, cnt = 0, out_n = 0;  // rm, bit k: vertex k leaves and this warp counts its neighbours down
        uint32_t x[ITEMS];
#pragma unroll
        for (int k = 0; k < ITEMS; k++) x[k] = u[k] != GONE ? __ldcg(past + u[k]) : 0u;
#pragma unroll
        for (int k = 0; k < ITEMS; k++) {
            const bool there = u[k] != GONE;
            d[k] -= seen[k] - x[k];
            seen[k] = seen_next[k];
            seen_next[k] = x[k];
            const bool out = there && d[k] <= thr;
            if (out) {
                key[u[k]] = delta;
                u[k] = GONE;
                uint32_t at = PEEL_WIDE;
                if (end[k] - beg[k] > PEEL_WARP_DEG) at = atomicAdd(&wide_n[r & 1], 1u);
                if (at < PEEL_WIDE) wide[at] = make_uint2(beg[k], end[k]);
                else rm |= 1u << k;
            } else if (there) {
                low = min(low, d[k]);
            }
            out_n += __popc(__ballot_sync(FULL, out));
            cnt += __popc(__ballot_sync(FULL, (rm >> k) & 1u));
        }
        if (lane == 0 && out_n) atomicAdd(&sl->word, (unsigned long long)out_n << 32);
        if (cnt) {  // the warp's own: their lists packed, eight lanes each
            uint2 *mine = own[threadIdx.x >> 5];
            uint32_t at = 0;
#pragma unroll
            for (int k = 0; k < ITEMS; k++) {
                const bool here = (rm >> k) & 1u;
                const unsigned int mk = __ballot_sync(FULL, here);
                if (here) mine[at + __popc(mk & lt)] = make_uint2(beg[k], end[k]);
                at += __popc(mk);
            }
            __syncwarp();
            for (uint32_t i = lane >> 3; i < cnt; i += 4) count_down(mine[i], lane & 7, 8u);
            __syncwarp();
        }
        __syncthreads();
        if (const uint32_t n = min(wide_n[r & 1], PEEL_WIDE)) {  // the CTA's long lists, a power of two of lanes each
            const uint32_t most = PEEL_THREADS / n, lanes = most <= 32 ? 32u : 1u << (31 - __clz(most));
            for (uint32_t i = threadIdx.x / lanes; i < n; i += PEEL_THREADS / lanes)
                count_down(wide[i], threadIdx.x & (lanes - 1u), lanes);
        }
        if (threadIdx.x == 0) wide_n[(r + 1) & 1] = 0;
        if (tid == 0) {  // the next round's slot: every CTA has left the barrier of the round before last
            ps->slot[(r + 1) % 3] = PeelSlot{0ull, 0u, 0u};
            ps->min_deg[(r + 1) % 3] = NO_DEGREE;
        }
        if (!peel_slot_barrier<false>(ps, sl, got)) return;
        alive -= got.removed;
        if (alive == 0) {
            r++;
            break;
        }
        if (got.removed == 0 && !log_mode) {
            if (!grid_min(low, &ps->min_deg[r % 3])) return;
            delta = max(delta, value);
        } else {
            delta++;
        }
    }
    if (tid == 0) ps->rounds = r ? r : 1u;
}

}  // namespace

gc_status gc_priority_simple(gc_graph *g, gc_heuristic h) {
    gc_ctx *ctx = g->ctx;
    if (g->N == 0) return GC_OK;
    int grid = ctx->num_sms * 4;
    ProfScope ps(ctx, "priority_keys", ctx->stream);
    k_simple_keys<<<grid, 256, 0, ctx->stream>>>(g->V, g->N, (int)h, g->seg_voff, g->n_seg, g->key);
    ctx->launches++;
    return gc_check_launch(ctx, "priority keys");
}

gc_status gc_priority_peel(gc_graph *g, bool log_thresholds) {
    gc_ctx *ctx = g->ctx;
    gc_status s;
    const uint32_t N = g->N;
    if (N == 0) return GC_OK;
    if ((s = gc_alloc(ctx, &g->deg_rem, g->cap_N, "peel degrees")) != GC_OK) return s;
    if ((s = gc_alloc(ctx, &g->frontier, g->cap_N, "peel list")) != GC_OK) return s;
    if ((s = gc_alloc(ctx, &g->frontier2, g->cap_N, "peel list")) != GC_OK) return s;
    const size_t state_at = ((size_t)g->cap_N + 31) & ~(size_t)31;  // words: the state starts a 128-byte line
    if ((s = gc_alloc(ctx, &g->removed, state_at + sizeof(PeelState) / 4, "peel removed list")) != GC_OK) return s;
    // the round state sits behind the removed list
    PeelState *ps = reinterpret_cast<PeelState *>(g->removed + state_at);
    PeelState host{};
    host.min0 = NO_DEGREE;
    for (auto &m : host.min_deg) m = NO_DEGREE;
    if ((s = gc_check_cuda(ctx, cudaMemcpyAsync(ps, &host, sizeof(host), cudaMemcpyHostToDevice, ctx->stream),
                           "peel state")) != GC_OK)
        return s;
    {
        ProfScope prof(ctx, "peel", ctx->stream);
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
        // every SM; fewer for graphs of less than 256 vertices per CTA (the barriers get cheaper)
        cfg.gridDim = dim3(std::max<uint32_t>(1u, std::min<uint32_t>((uint32_t)ctx->num_sms, N / 256)));
        cfg.blockDim = dim3(PEEL_THREADS);
        cfg.stream = ctx->stream;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        const uint32_t *V = g->V, *E = g->E;
        if ((s = gc_check_cuda(ctx, cudaLaunchKernelEx(&cfg, k_peel, V, E, N, log_thresholds ? 1 : 0, g->deg_rem,
                                                       g->frontier, g->frontier2, g->removed, g->key, ps),
                               "peel")) != GC_OK)
            return s;
        ctx->launches++;
    }
    if ((s = gc_check_cuda(ctx, cudaMemcpyAsync(&host, ps, sizeof(host), cudaMemcpyDeviceToHost, ctx->stream),
                           "peel state")) != GC_OK)
        return s;
    if ((s = gc_check_cuda(ctx, cudaStreamSynchronize(ctx->stream), "peel rounds")) != GC_OK) return s;
    if (host.failed || !host.rounds) return gc_fail(ctx, GC_ERR_DEVICE, "peeling did not terminate");
    return GC_OK;
}
