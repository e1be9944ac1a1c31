// Incremental bucketed refinement (src/refine_incremental.cuh:7-361,
// src/refine.cu:52-142).  B200 layout:
//
// * the dense n x k affinity cache is u32 when the graph's total directed
//   edge weight fits 32 bits (halving the dominant HBM stream), else u64;
// * LP proposals append proposers to a list; the priority filter, the fused
//   cache+cut update and the commit then touch proposers/movers only;
// * list-driven kernels use a fixed grid with grid-stride loops so the host
//   never has to size a launch from a device count;
// * the rebalance moves, per (source part, gain bucket, section), vertices in
//   the order (gain per weight descending, vertex ascending).  The order is
//   needed inside one bucket per part only: buckets before the one that
//   crosses the part's quota are taken whole, later ones not at all, and the
//   crossing bucket is cut at a threshold found by a weighted radix selection,
//   so nothing is sorted and labels are bit-reproducible.
#pragma once

#include <cooperative_groups.h>

#include "gp_prim.cuh"
#include "gp_sclp.cuh"

namespace gp {

constexpr int kBalBuckets = 50, kBalSections = 16, kBalWidth = kBalBuckets * kBalSections;

struct RefineCounters {
    i64 proposers;
    i64 movers;
    long long delta;      // cut decrease of the last apply
    u64 directed_cut;
    i64 mover_degree;     // sum of the movers' degrees
    i64 big;              // movers of degree > kSplitDegree handed to apply_big_rows_kernel
    i64 big_degree;       // their degree sum
    i64 walked_degree;    // edges apply_cache_cut_kernel walked itself
    i64 hub_edges;        // edges of moving hubs walked by hub_apply_kernel
    i64 hub_chunks;       // their chunks
    i64 filter_degree;    // edges of the LP proposers below the hub degree (profiling only)
};

// Profiling only: the edges the priority filter walks (proposers' rows below
// the hub degree), into ctr->filter_degree.
template <typename O>
__global__ void filter_degree_kernel(const i32* __restrict__ list, const RefineCounters* ctr_in,
                                     const O* __restrict__ off, RefineCounters* ctr) {
    const i64 count = ctr_in->proposers;
    i64 sum = 0;
    for (i64 i = static_cast<i64>(blockIdx.x) * blockDim.x + threadIdx.x; i < count;
         i += static_cast<i64>(gridDim.x) * blockDim.x) {
        const i32 v = list[i];
        const i64 d = static_cast<i64>(off[v + 1]) - static_cast<i64>(off[v]);
        if (d <= kHubDegree) sum += d;
    }
    sum = warp_sum(sum);
    if ((threadIdx.x & 31) == 0 && sum)
        atomicAdd(reinterpret_cast<unsigned long long*>(&ctr->filter_degree), static_cast<unsigned long long>(sum));
}

// Per-vertex proposal record written by the LP pass: the priority filter
// gathers one 16-byte record per neighbour instead of three arrays.
struct alignas(16) PropRec {
    i32 label;
    i32 target;   // -1: no proposal
    i64 gain;
};

__device__ __forceinline__ void cache_add(u32* p, u64 v) { atomicAdd(p, static_cast<u32>(v)); }
__device__ __forceinline__ void cache_add(u64* p, u64 v) { atomic_add_u64(p, v); }

// Exact directed cut, one atomic per block (refine_cut_kernel,
// src/refine.cu:52-87).  A warp takes four consecutive rows at a time: rows of
// at most 32 entries are walked by 8 lanes each, longer ones (up to the hub
// degree) by the whole warp one after the other.  Bound by the label gathers;
// with a warp per row a mesh's rows of 4-7 entries left most lanes idle
// (grid of 10^6 vertices 128 -> 45 us, 320^3 grid 606 -> 378 us a launch).
template <typename O, typename W>
__global__ void __launch_bounds__(kThreads) cut_kernel(i64 n, const O* __restrict__ off, const i32* __restrict__ nbr,
                                                       const W* __restrict__ ew, const i32* __restrict__ labels,
                                                       u64* out) {
    __shared__ u64 sh[kWarps + 1];
    const int lane = threadIdx.x & 31, grp = lane >> 3, gl = lane & 7;
    u64 local = 0;
    const i64 warps_total = static_cast<i64>(gridDim.x) * kWarps;
    for (i64 q = static_cast<i64>(blockIdx.x) * kWarps + (threadIdx.x >> 5); q * 4 < n; q += warps_total) {
        const i64 v = q * 4 + grp;
        i64 b = 0, deg = 0;
        i32 s = 0;
        if (v < n) {
            b = static_cast<i64>(off[v]);
            deg = static_cast<i64>(off[v + 1]) - b;
            s = labels[v];
        }
        if (deg <= 32) {
            i32 u[4];
#pragma unroll
            for (int r = 0; r < 4; ++r) u[r] = gl + 8 * r < deg ? nbr[b + gl + 8 * r] : -1;
#pragma unroll
            for (int r = 0; r < 4; ++r)
                if (u[r] >= 0 && labels[u[r]] != s) local += static_cast<u64>(weight_at(ew, b + gl + 8 * r));
        }
        unsigned longs = __ballot_sync(0xffffffffu, gl == 0 && deg > 32 && deg <= kHubDegree);
        while (longs) {
            const int src = __ffs(longs) - 1;
            longs &= longs - 1;
            const i64 lb = __shfl_sync(0xffffffffu, b, src), ld = __shfl_sync(0xffffffffu, deg, src);
            const i32 ls = __shfl_sync(0xffffffffu, s, src);
            for (i64 e = lb + lane; e < lb + ld; e += 32)
                if (labels[nbr[e]] != ls) local += static_cast<u64>(weight_at(ew, e));
        }
    }
    local = block_sum(local, sh);
    if (threadIdx.x == 0 && local) atomic_add_u64(out, local);
}

// Sum of `w` over the lanes that share this lane's `key` (the lanes of
// `peers`), the same value in every lane of the group.
template <typename C>
__device__ __forceinline__ u64 group_sum(unsigned peers, u64 w) {
    if constexpr (sizeof(C) == 4) {
        return __reduce_add_sync(peers, static_cast<u32>(w));
    } else {
        u64 sum = 0;
#pragma unroll
        for (int s = 0; s < 32; ++s) {
            const u64 x = __shfl_sync(0xffffffffu, w, s);
            if (peers & (1u << s)) sum += x;
        }
        return sum;
    }
}

// group_sum of weights that usually are small: one 32-bit reduction when no
// lane's weight reaches 2^26 (32 of them then fit 32 bits).  All 32 lanes call it.
__device__ __forceinline__ u64 weight_group_sum(unsigned peers, u64 w) {
    if (__any_sync(0xffffffffu, (w >> 26) != 0)) return group_sum<u64>(peers, w);
    return __reduce_add_sync(peers, static_cast<u32>(w));
}

// One vertex's k cache entries into registers, with 16-byte loads when the
// row is 16-byte aligned (k a multiple of 4 for 32-bit entries, of 2 for
// 64-bit entries); entries past k are left untouched.
template <typename C>
__device__ __forceinline__ void load_row(const C* row, int k, C (&vals)[32]) {
    if constexpr (sizeof(C) == 4) {
        if ((k & 3) == 0) {
            const uint4* r4 = reinterpret_cast<const uint4*>(row);
#pragma unroll
            for (int q = 0; q < 8; ++q)
                if (4 * q < k) {
                    const uint4 x = r4[q];
                    vals[4 * q] = x.x; vals[4 * q + 1] = x.y; vals[4 * q + 2] = x.z; vals[4 * q + 3] = x.w;
                }
            return;
        }
    } else {
        if ((k & 1) == 0) {
            const ulonglong2* r2 = reinterpret_cast<const ulonglong2*>(row);
#pragma unroll
            for (int q = 0; q < 16; ++q)
                if (2 * q < k) {
                    const ulonglong2 x = r2[q];
                    vals[2 * q] = x.x; vals[2 * q + 1] = x.y;
                }
            return;
        }
    }
#pragma unroll
    for (int p = 0; p < 32; ++p)
        if (p < k) vals[p] = row[p];
}

// incremental_build_affinity (src/refine_incremental.cuh:7-25).  A warp
// takes four consecutive vertices: rows of at most 32 entries are walked by
// 8 lanes each (up to four steps, all four rows at once), longer rows (up to
// the hub degree) by the whole warp one after the other.  Each row is summed
// in a private accumulator in shared memory: with a 32-bit cache (every sum
// fits 32 bits) every lane adds its edge with a 32-bit shared atomic; with a
// 64-bit cache lanes holding the same part are grouped with __match_any_sync
// and only the group leader adds their sum (measured at RMAT-24: the 32-bit
// atomics take 26% less time than the match, 64-bit shared atomics 45% more).
// The four cache rows, consecutive in memory, are then stored by the whole
// warp in one coalesced pass.  Hub rows are left to the chunked kernel
// (zero_hub_rows_kernel clears them after this one).
// `rows`: one accumulator per warp of the block.  With CUT every lane's share
// of the rows' connections to other parts is returned: summed over all rows
// the directed cut, without a pass of its own over the edges.
template <bool CUT, typename O, typename W, typename C>
__device__ __forceinline__ u64 build_cache_rows(i64 n, const O* __restrict__ off, const i32* __restrict__ nbr,
                                                const W* __restrict__ ew, const i32* labels, int k, C* cache,
                                                u64 (*rows)[4][32]) {
    u64 cut = 0;
    u32 (*rows32)[4][32] = reinterpret_cast<u32 (*)[4][32]>(&rows[0][0][0]);   // C = u32: 32-bit accumulators
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, grp = lane >> 3, gl = lane & 7;
    const int block_warps = static_cast<int>(blockDim.x >> 5);
    const i64 warps_total = static_cast<i64>(gridDim.x) * block_warps;
    for (i64 q = static_cast<i64>(blockIdx.x) * block_warps + warp; q * 4 < n; q += warps_total) {
        const i64 v = q * 4 + grp;
        i64 b = 0, deg = 0;
        if (v < n) {
            b = static_cast<i64>(off[v]);
            deg = static_cast<i64>(off[v + 1]) - b;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if constexpr (sizeof(C) == 4) rows32[warp][grp][gl + 8 * j] = 0;
            else rows[warp][grp][gl + 8 * j] = 0;
        }
        __syncwarp();
        const bool short_row = deg <= 32;
        const unsigned steps = __reduce_max_sync(0xffffffffu, short_row ? static_cast<unsigned>((deg + 7) >> 3) : 0u);
        for (unsigned r = 0; r < steps; ++r) {
            const i64 e = static_cast<i64>(r) * 8 + gl;
            int p = -1;
            u64 w = 0;
            if (short_row && e < deg) {
                const i32 u = nbr[b + e];
                if (u != v) { p = labels[u]; w = static_cast<u64>(weight_at(ew, b + e)); }
            }
            if constexpr (sizeof(C) == 4) {
                if (p >= 0) atomicAdd(&rows32[warp][grp][p], static_cast<u32>(w));
            } else {
                const unsigned peers = __match_any_sync(0xffffffffu, p < 0 ? -1 - grp : grp * 32 + p);
                const u64 sum = group_sum<C>(peers, w);
                if (p >= 0 && lane == __ffs(peers) - 1) rows[warp][grp][p] += sum;
            }
            __syncwarp();
        }
        // rows of 33..kHubDegree entries, one at a time by the whole warp
        unsigned longs = __ballot_sync(0xffffffffu, gl == 0 && !short_row && deg <= kHubDegree);
        while (longs) {
            const int src = __ffs(longs) - 1;
            longs &= longs - 1;
            const int g = src >> 3;
            const i64 lb = __shfl_sync(0xffffffffu, b, src), ld = __shfl_sync(0xffffffffu, deg, src);
            const i64 lv = q * 4 + g;
            for (i64 base = 0; base < ld; base += 32) {
                const i64 e = base + lane;
                int p = -1;
                u64 w = 0;
                if (e < ld) {
                    const i32 u = nbr[lb + e];
                    if (u != lv) { p = labels[u]; w = static_cast<u64>(weight_at(ew, lb + e)); }
                }
                if constexpr (sizeof(C) == 4) {
                    if (p >= 0) atomicAdd(&rows32[warp][g][p], static_cast<u32>(w));
                } else {
                    const unsigned peers = __match_any_sync(0xffffffffu, p);
                    const u64 sum = group_sum<C>(peers, w);
                    if (p >= 0 && lane == __ffs(peers) - 1) rows[warp][g][p] += sum;
                }
                __syncwarp();
            }
        }
        // the four rows are consecutive in the cache: entries [4qk, 4qk + 4k)
        const i64 first = q * 4;
        const int nrows = static_cast<int>(n - first < 4 ? n - first : 4);
        const unsigned hub_rows = __ballot_sync(0xffffffffu, gl == 0 && deg > kHubDegree);
        C* dst = cache + first * k;
        const i32 own = CUT && v < n ? labels[v] : 0;
        for (int i0 = 0; i0 < nrows * k; i0 += 32) {
            const int i = i0 + lane;
            const int row = i / k;
            i32 part = 0;
            if constexpr (CUT) part = __shfl_sync(0xffffffffu, own, (row & 3) * 8);
            if (i < nrows * k && !(hub_rows & (1u << (row * 8)))) {
                C value;
                if constexpr (sizeof(C) == 4) value = static_cast<C>(rows32[warp][row][i - row * k]);
                else value = static_cast<C>(rows[warp][row][i - row * k]);
                dst[i] = value;
                if (CUT && i - row * k != part) cut += static_cast<u64>(value);
            }
        }
        __syncwarp();
    }
    return cut;
}

template <bool CUT, typename O, typename W, typename C>
__global__ void __launch_bounds__(kThreads) build_cache_kernel(i64 n, const O* __restrict__ off,
                                                               const i32* __restrict__ nbr, const W* __restrict__ ew,
                                                               const i32* __restrict__ labels, int k, C* cache,
                                                               u64* directed_cut) {
    __shared__ u64 rows[kWarps][4][32];
    u64 cut = build_cache_rows<CUT>(n, off, nbr, ew, labels, k, cache, rows);
    if constexpr (CUT) {
        cut = warp_sum(cut);
        if ((threadIdx.x & 31) == 0 && cut) atomic_add_u64(directed_cut, cut);
    }
}

// The hub rows' share of the directed cut, from their finished cache rows.
template <typename C>
__global__ void __launch_bounds__(kThreads) hub_cache_cut_kernel(i64 hubs, const i32* __restrict__ hub_list,
                                                                 const i32* __restrict__ labels, int k,
                                                                 const C* __restrict__ cache, u64* directed_cut) {
    u64 cut = 0;
    for (i64 i = static_cast<i64>(blockIdx.x) * kThreads + threadIdx.x; i < hubs * k; i += static_cast<i64>(gridDim.x) * kThreads) {
        const i64 h = i / k;
        const int p = static_cast<int>(i - h * k);
        const i64 v = hub_list[h];
        if (p != labels[v]) cut += static_cast<u64>(cache[v * k + p]);
    }
    cut = warp_sum(cut);
    if ((threadIdx.x & 31) == 0 && cut) atomic_add_u64(directed_cut, cut);
}

// The LP filter of refine_incremental.cuh:332-333, from the level's maximum
// edge weight (nullptr: unit weights).
__device__ __forceinline__ double lp_filter(const u64* max_edge_weight) {
    return !max_edge_weight || *max_edge_weight <= 1 ? 0.25 : 0.75;
}

// incremental_lp_proposals (src/refine_incremental.cuh:27-46) for one vertex;
// true when it proposes.
template <typename C>
__device__ __forceinline__ bool lp_choice(i64 v, const C* cache, const i32* labels, int k, double filter,
                                          unsigned char* locks, i32* targets, i64* gains, PropRec* props) {
    i32 target = -1;
    i64 g = INT64_MIN;
    const i32 s = labels[v];
    if (locks[v]) {
        locks[v] = 0;
    } else {
        C vals[32];
        load_row(cache + v * k, k, vals);
        u64 best = 0, current = 0;
        int t = -1;
#pragma unroll
        for (int p = 0; p < 32; ++p) {
            if (p >= k) break;
            const u64 c = static_cast<u64>(vals[p]);
            if (p == s) current = c;
            else if (c > best) { best = c; t = p; }
        }
        if (t >= 0 &&
            (best >= current || current - best < static_cast<u64>(filter * static_cast<double>(current)))) {
            g = best >= current ? static_cast<i64>(best - current) : -static_cast<i64>(current - best);
            target = t;
        }
    }
    targets[v] = target;
    gains[v] = g;
    props[v] = {s, target, g};
    return target >= 0;
}

// Proposers are appended to `list`.
template <typename C>
__global__ void lp_proposals_kernel(i64 n, const C* __restrict__ cache, const i32* __restrict__ labels, int k,
                                    const u64* __restrict__ max_edge_weight, unsigned char* locks, i32* targets,
                                    i64* gains, PropRec* props, i32* list, RefineCounters* ctr) {
    const i64 v = static_cast<i64>(blockIdx.x) * blockDim.x + threadIdx.x;
    const bool propose = v < n && lp_choice(v, cache, labels, k, lp_filter(max_edge_weight), locks, targets, gains, props);
    const u64 slot = warp_append(propose, reinterpret_cast<u64*>(&ctr->proposers));
    if (propose) list[slot] = static_cast<i32>(v);
}

// incremental_priority_filter (src/refine_incremental.cuh:48-67); movers are
// appended to `movers` and flagged.
// A warp takes up to 32 proposers and walks their edges together; each
// row's correction is summed in shared memory (hub rows: chunked kernel).
template <typename O, typename W>
__device__ __forceinline__ void priority_filter(const i32* list, i64 count, const O* __restrict__ off,
                                                const i32* __restrict__ nbr, const W* __restrict__ ew,
                                                const PropRec* props, unsigned char* flags, i32* movers,
                                                RefineCounters* ctr, long long (*corr_sh)[32]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int block_warps = static_cast<int>(blockDim.x >> 5);
    const i64 warps = static_cast<i64>(gridDim.x) * block_warps;
    const int G = rows_per_warp(count, warps);
    for (i64 i0 = (static_cast<i64>(blockIdx.x) * block_warps + warp) * G; i0 < count; i0 += warps * G) {
        const i64 i = i0 + lane;
        const bool has = lane < G && i < count;
        const i32 v = has ? list[i] : 0;
        const i64 b = has ? static_cast<i64>(off[v]) : 0;
        const i64 deg = has ? static_cast<i64>(off[v + 1]) - b : 0;
        const bool hub = deg > kHubDegree;
        const PropRec me = has ? props[v] : PropRec{0, -1, 0};
        corr_sh[warp][lane] = 0;
        __syncwarp();
        warp_edge_walk(b, hub ? 0 : deg, [&](bool valid, int owner, i64 e) {
            const i32 ov = __shfl_sync(0xffffffffu, v, owner);
            const i32 s = __shfl_sync(0xffffffffu, me.label, owner);
            const i32 t = __shfl_sync(0xffffffffu, me.target, owner);
            const i64 g = __shfl_sync(0xffffffffu, me.gain, owner);
            long long c = 0;
            if (valid) {
                const i32 u = nbr[e];
                if (u != ov) {
                    const PropRec o = props[u];
                    if (o.target >= 0 && (o.gain > g || (o.gain == g && u < ov))) {
                        const auto w = static_cast<long long>(weight_at(ew, e));
                        c = w * ((o.target == t) - (o.target == s) - (o.label == t) + (o.label == s));
                    }
                }
            }
            const long long run = warp_run_sum(c, owner);
            const int next = __shfl_down_sync(0xffffffffu, owner, 1);
            if ((lane == 31 || next != owner) && run != 0) corr_sh[warp][owner] += run;
            __syncwarp();
        });
        const bool move = has && !hub && me.gain + corr_sh[warp][lane] >= 0;
        const u64 slot = warp_append(move, reinterpret_cast<u64*>(&ctr->movers));
        if (move) {
            flags[v] = 1;
            movers[slot] = v;
        }
        const i64 moved_degree = warp_sum(move ? deg : i64{0});
        if (lane == 0 && moved_degree)
            atomicAdd(reinterpret_cast<unsigned long long*>(&ctr->mover_degree),
                      static_cast<unsigned long long>(moved_degree));
        __syncwarp();
    }
}

template <typename O, typename W>
__global__ void __launch_bounds__(kThreads) priority_filter_kernel(
    const i32* __restrict__ list, const RefineCounters* ctr_in, const O* __restrict__ off,
    const i32* __restrict__ nbr, const W* __restrict__ ew, const PropRec* __restrict__ props, unsigned char* flags,
    i32* movers, RefineCounters* ctr) {
    __shared__ long long corr_sh[kWarps][32];
    priority_filter(list, ctr_in->proposers, off, nbr, ew, props, flags, movers, ctr, corr_sh);
}

// incremental_update_cache_and_cut (src/refine_incremental.cuh:69-95) for
// one edge of mover v (label s, target t): the neighbour's cache row loses w
// at s and gains it at t; the cut change is counted once per undirected edge
// (the neighbour is not a mover, or has the larger id).
//
// Here over the edges [b, e1) of mover v, thread `tid` of `nthreads`
// taking every nthreads-th edge, kApplyBatch of them per step: the batch's
// neighbour ids are loaded first, then their flags and labels, then the cache
// updates issued, so a thread keeps kApplyBatch independent gather chains in
// flight instead of one.  Integer sums, so the result does not depend on the
// order.
constexpr int kApplyBatch = 4;

template <typename W, typename C>
__device__ __forceinline__ long long apply_edges_batched(i32 v, i32 s, i32 t, i64 b, i64 e1, int tid, int nthreads,
                                                         const i32* __restrict__ nbr, const W* __restrict__ ew,
                                                         const i32* __restrict__ labels,
                                                         const i32* __restrict__ targets,
                                                         const unsigned char* __restrict__ flags, int k, C* cache) {
    long long gain = 0;
    const i64 step = static_cast<i64>(nthreads);
    for (i64 e0 = b + tid; e0 < e1; e0 += kApplyBatch * step) {
        i32 u[kApplyBatch];
#pragma unroll
        for (int j = 0; j < kApplyBatch; ++j) {
            const i64 e = e0 + j * step;
            u[j] = e < e1 ? nbr[e] : v;   // past the row: treated as a self loop, skipped
        }
        bool fu[kApplyBatch];
        i32 lu[kApplyBatch];
#pragma unroll
        for (int j = 0; j < kApplyBatch; ++j) {
            fu[j] = false;
            lu[j] = 0;
            if (u[j] != v) {
                fu[j] = flags[u[j]] != 0;
                lu[j] = labels[u[j]];
            }
        }
#pragma unroll
        for (int j = 0; j < kApplyBatch; ++j) {
            if (u[j] == v) continue;
            const u64 w = static_cast<u64>(weight_at(ew, e0 + j * step));
            cache_add(&cache[static_cast<i64>(u[j]) * k + s], 0ULL - w);
            cache_add(&cache[static_cast<i64>(u[j]) * k + t], w);
            if (fu[j] && u[j] < v) continue;
            const i32 nn = fu[j] ? targets[u[j]] : lu[j];
            gain += static_cast<long long>(w) * ((s != lu[j]) - (t != nn));
        }
    }
    return gain;
}

// The same update over the edges of up to 32 movers, one per lane (v, s, t, first
// edge `begin`, `deg` edges; deg 0 for no mover), walked as warp_edge_walk
// walks them but kApplyBatch 32-edge steps at a time: each lane resolves its
// kApplyBatch positions (owning lane, edge) and loads their neighbour ids,
// then their flags and labels, before any cache update.
template <typename W, typename C>
__device__ __forceinline__ long long warp_apply_rows(i32 v, i32 s, i32 t, i64 begin, i64 deg,
                                                     const i32* __restrict__ nbr, const W* __restrict__ ew,
                                                     const i32* labels, const i32* targets,
                                                     const unsigned char* flags, int k, C* cache) {
    const int lane = threadIdx.x & 31;
    const i64 inc = warp_inclusive_sum(deg);
    const i64 pre = inc - deg;
    const i64 total = __shfl_sync(0xffffffffu, inc, 31);
    long long gain = 0;
    for (i64 base = 0; base < total; base += kApplyBatch * 32) {
        i32 ov[kApplyBatch], os[kApplyBatch], ot[kApplyBatch], u[kApplyBatch];
        i64 e[kApplyBatch];
#pragma unroll
        for (int j = 0; j < kApplyBatch; ++j) {
            const i64 q = base + j * 32 + lane;
            int lo = 0;
#pragma unroll
            for (int step = 16; step; step >>= 1) {
                const i64 probe = __shfl_sync(0xffffffffu, pre, lo + step);
                if (probe <= q) lo += step;
            }
            const i64 my_pre = __shfl_sync(0xffffffffu, pre, lo);
            const i64 my_begin = __shfl_sync(0xffffffffu, begin, lo);
            ov[j] = __shfl_sync(0xffffffffu, v, lo);
            os[j] = __shfl_sync(0xffffffffu, s, lo);
            ot[j] = __shfl_sync(0xffffffffu, t, lo);
            e[j] = my_begin + (q - my_pre);
            u[j] = q < total ? nbr[e[j]] : ov[j];   // past the last edge: treated as a self loop, skipped
        }
        bool fu[kApplyBatch];
        i32 lu[kApplyBatch];
#pragma unroll
        for (int j = 0; j < kApplyBatch; ++j) {
            fu[j] = false;
            lu[j] = 0;
            if (u[j] != ov[j]) {
                fu[j] = flags[u[j]] != 0;
                lu[j] = labels[u[j]];
            }
        }
#pragma unroll
        for (int j = 0; j < kApplyBatch; ++j) {
            if (u[j] == ov[j]) continue;
            const u64 w = static_cast<u64>(weight_at(ew, e[j]));
            cache_add(&cache[static_cast<i64>(u[j]) * k + os[j]], 0ULL - w);
            cache_add(&cache[static_cast<i64>(u[j]) * k + ot[j]], w);
            if (fu[j] && u[j] < ov[j]) continue;
            const i32 nn = fu[j] ? targets[u[j]] : lu[j];
            gain += static_cast<long long>(w) * ((os[j] != lu[j]) - (ot[j] != nn));
        }
    }
    return gain;
}

// Movers of degree above this are walked by a whole block
// (apply_big_rows_kernel): one warp would take deg/32 dependent steps, and the
// launch would wait for that one warp.
constexpr i64 kSplitDegree = 256;

template <typename O, typename W, typename C>
__global__ void __launch_bounds__(kThreads) apply_cache_cut_kernel(
    const i32* __restrict__ movers, const RefineCounters* ctr_in, const O* __restrict__ off,
    const i32* __restrict__ nbr, const W* __restrict__ ew, const i32* __restrict__ labels,
    const i32* __restrict__ targets, const unsigned char* __restrict__ flags, int k, C* cache, RefineCounters* ctr,
    i32* __restrict__ big) {
    // A warp takes up to 32 movers and walks their edges together (rows above
    // kSplitDegree: block kernel; hub rows: chunked kernel).  The cut delta is
    // summed per warp and added with one atomic per warp, so warps never wait
    // for each other.
    const int lane = threadIdx.x & 31;
    const i64 count = ctr_in->movers;
    const i64 warps = static_cast<i64>(gridDim.x) * kWarps;
    const int G = rows_per_warp(count, warps);
    long long gain = 0;
    for (i64 i0 = (static_cast<i64>(blockIdx.x) * kWarps + (threadIdx.x >> 5)) * G; i0 < count; i0 += warps * G) {
        const i64 i = i0 + lane;
        const bool has = lane < G && i < count;
        const i32 v = has ? movers[i] : 0;
        const i64 b = has ? static_cast<i64>(off[v]) : 0;
        i64 deg = has ? static_cast<i64>(off[v + 1]) - b : 0;
        const bool split = deg > kSplitDegree && deg <= kHubDegree;
        const u64 slot = warp_append(split, reinterpret_cast<u64*>(&ctr->big));
        if (split) big[slot] = v;
        const i64 big_degree = warp_sum(split ? deg : i64{0});
        if (lane == 0 && big_degree)
            atomicAdd(reinterpret_cast<unsigned long long*>(&ctr->big_degree), static_cast<unsigned long long>(big_degree));
        if (deg > kSplitDegree) deg = 0;
        const i64 walked = warp_sum(deg);
        if (lane == 0 && walked)
            atomicAdd(reinterpret_cast<unsigned long long*>(&ctr->walked_degree), static_cast<unsigned long long>(walked));
        const i32 s = has ? labels[v] : 0, t = has ? targets[v] : 0;
        gain += warp_apply_rows(v, s, t, b, deg, nbr, ew, labels, targets, flags, k, cache);
    }
    gain = warp_sum(gain);
    if (lane == 0 && gain) atomicAdd(reinterpret_cast<unsigned long long*>(&ctr->delta), static_cast<unsigned long long>(gain));
}

// The movers set aside by apply_cache_cut_kernel (kSplitDegree < degree <=
// kHubDegree), one block per row over a grid-stride loop.
template <typename O, typename W, typename C>
__global__ void __launch_bounds__(kThreads) apply_big_rows_kernel(
    const i32* __restrict__ big, const RefineCounters* ctr_in, const O* __restrict__ off,
    const i32* __restrict__ nbr, const W* __restrict__ ew, const i32* __restrict__ labels,
    const i32* __restrict__ targets, const unsigned char* __restrict__ flags, int k, C* cache, RefineCounters* ctr) {
    __shared__ long long sh[kWarps + 1];
    const i64 count = ctr_in->big;
    long long gain = 0;
    for (i64 r = blockIdx.x; r < count; r += gridDim.x) {
        const i32 v = big[r];
        const i32 s = labels[v], t = targets[v];
        gain += apply_edges_batched(v, s, t, static_cast<i64>(off[v]), static_cast<i64>(off[v + 1]),
                                    static_cast<int>(threadIdx.x), kThreads, nbr, ew, labels, targets, flags, k,
                                    cache);
    }
    gain = block_sum(gain, sh);
    if (threadIdx.x == 0 && gain)
        atomicAdd(reinterpret_cast<unsigned long long*>(&ctr->delta), static_cast<unsigned long long>(gain));
}

// incremental_commit (src/refine_incremental.cuh:97-109); also clears the
// mover flag so that `flags` is all-zero outside an apply.  All movers hit the
// same k part weights, and after an LP round or a rebalance most lanes of a
// warp share a part, so the changes are summed per warp and part, then per
// block in shared memory, before one global atomic per block and part.
template <typename W>
__device__ __forceinline__ void commit_moves(const i32* movers, i64 count, i32* labels, const i32* targets,
                                             const W* __restrict__ vw, u64* pw, unsigned char* locks,
                                             unsigned char* flags, bool lp, unsigned long long* delta) {
    if (static_cast<i64>(blockIdx.x) * blockDim.x >= count) return;   // uniform over the block
    if (threadIdx.x < 32) delta[threadIdx.x] = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    for (i64 base = static_cast<i64>(blockIdx.x) * blockDim.x; base < count; base += static_cast<i64>(gridDim.x) * blockDim.x) {
        const i64 i = base + threadIdx.x;
        i32 s = -1, t = -1;
        u64 w = 0;
        if (i < count) {
            const i32 v = movers[i];
            s = labels[v];
            t = targets[v];
            w = static_cast<u64>(weight_at(vw, v));
            labels[v] = t;
            if (lp) locks[v] = 1;
            flags[v] = 0;
        }
        const unsigned from = __match_any_sync(0xffffffffu, s), to = __match_any_sync(0xffffffffu, t);
        const u64 out = vw ? weight_group_sum(from, w) : static_cast<u64>(__popc(from));
        const u64 in = vw ? weight_group_sum(to, w) : static_cast<u64>(__popc(to));
        if (s >= 0 && lane == __ffs(from) - 1) atomicAdd(&delta[s], 0ULL - out);
        if (t >= 0 && lane == __ffs(to) - 1) atomicAdd(&delta[t], static_cast<unsigned long long>(in));
    }
    __syncthreads();
    if (threadIdx.x < 32 && delta[threadIdx.x]) atomic_add_u64(&pw[threadIdx.x], delta[threadIdx.x]);
}

template <typename W>
__global__ void commit_kernel(const i32* __restrict__ movers, const RefineCounters* ctr_in,
                              i32* labels, const i32* __restrict__ targets, const W* __restrict__ vw, u64* pw,
                              unsigned char* locks, unsigned char* flags, int lp) {
    __shared__ unsigned long long delta[32];
    commit_moves(movers, ctr_in->movers, labels, targets, vw, pw, locks, flags, lp != 0, delta);
}

// Rebalance gain bucket (refine_incremental.cuh:167-171) restated with host
// thresholds 1.5^j: for g < 0, 25 + the smallest j with -g <= 1.5^j,
// clamped to [2, 49].
struct BucketThresholds { double t[48]; };   // j = -23 .. 24

__device__ __forceinline__ int gain_bucket(double g, const BucketThresholds& th) {
    if (g > 0) return 0;
    if (g == 0) return 1;
    const double a = -g;
    if (a <= th.t[0]) return 2;
    int lo = 1, hi = 47;   // smallest index in [1,47] with a <= t[idx], else 48
    if (a > th.t[47]) return 49;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (a <= th.t[mid]) hi = mid; else lo = mid + 1;
    }
    return 25 + (lo - 23);
}

// Weight sums per bucket gathered by one block in shared memory and added to
// the global counts once at its end.  The candidates of a large part crowd
// into a few buckets (the interior of a grid part has one gain: 16 buckets),
// so a global atomic per warp and bucket would queue at a few addresses.
// A key that finds its few slots taken goes to the global count directly.
struct BucketTable {
    static constexpr int kSlots = 512, kProbes = 4;
    int key[kSlots];
    u64 sum[kSlots];
    __device__ void clear() {
        for (int i = threadIdx.x; i < kSlots; i += blockDim.x) { key[i] = -1; sum[i] = 0; }
    }
    // All 32 lanes of a warp call it; b < 0 means no item.
    __device__ void add(int b, u64 w, bool unit, u64* counts) {
        const unsigned peers = __match_any_sync(0xffffffffu, b);
        const u64 total = unit ? static_cast<u64>(__popc(peers)) : weight_group_sum(peers, w);
        if (b < 0 || (threadIdx.x & 31) != __ffs(peers) - 1) return;
        int slot = static_cast<int>(mix32(static_cast<u32>(b)) % kSlots);
        for (int probe = 0; probe < kProbes; ++probe) {
            const int found = atomicCAS(&key[slot], -1, b);
            if (found == -1 || found == b) {
                atomic_add_u64(&sum[slot], total);
                return;
            }
            slot = (slot + 1) % kSlots;
        }
        atomic_add_u64(&counts[b], total);
    }
    __device__ void flush(u64* counts) {
        for (int i = threadIdx.x; i < kSlots; i += blockDim.x)
            if (key[i] >= 0) atomic_add_u64(&counts[key[i]], sum[i]);
    }
};

// One rebalance candidate (incremental_rebalance_proposals,
// src/refine_incremental.cuh:111-165): the destination with slack that it is
// best connected to (ties: more slack), a zero-connection vertex spread over
// the parts with slack by a hashed ticket; returns the vertex's bucket (source
// part, gain-per-weight bucket, hashed section) or -1.
template <typename C, typename W>
__device__ __forceinline__ int rebalance_choice(i64 v, const C* cache, const i32* labels, const W* __restrict__ vw,
                                                int k, const u64* spw, u64 cap, const BucketThresholds& th,
                                                i32* targets, u64& w) {
    const i32 s = labels[v];
    if (spw[s] <= cap) return -1;
    w = static_cast<u64>(weight_at(vw, v));
    C vals[32];
    load_row(cache + v * k, k, vals);
    int best = -1;
    u64 best_conn = 0, best_slack = 0, current = 0;
#pragma unroll
    for (int p = 0; p < 32; ++p) {
        if (p >= k) break;
        const u64 value = static_cast<u64>(vals[p]);
        if (p == s) { current = value; continue; }
        const u64 pp = spw[p];
        if (pp >= cap || w > cap - pp) continue;
        const u64 slack = cap - pp;
        if (best < 0 || value > best_conn || (value == best_conn && slack > best_slack)) {
            best = p; best_conn = value; best_slack = slack;
        }
    }
    if (best >= 0 && best_conn == 0) {
        u64 total_slack = 0;
        for (int p = 0; p < k; ++p) {
            const u64 pp = spw[p];
            if (p != s && pp < cap && w <= cap - pp)
                total_slack = UINT64_MAX - total_slack < cap - pp ? UINT64_MAX : total_slack + cap - pp;
        }
        u64 ticket = static_cast<u64>(mix32(static_cast<u32>(v))) % total_slack;
        for (int p = 0; p < k; ++p) {
            const u64 pp = spw[p];
            if (p == s || pp >= cap || w > cap - pp) continue;
            const u64 slack = cap - pp;
            if (ticket < slack) { best = p; break; }
            ticket -= slack;
        }
    }
    if (best < 0) return -1;
    const double gain = best_conn >= current ? static_cast<double>(best_conn - current)
                                             : -static_cast<double>(current - best_conn);
    targets[v] = best;
    return s * kBalWidth + gain_bucket(gain / static_cast<double>(w), th) * kBalSections +
           static_cast<int>(mix32(static_cast<u32>(v)) % kBalSections);
}

// Order of vertex v inside its bucket: gain per weight descending as an
// ascending integer (v itself breaks ties).  The gain is that of the chosen
// destination, whose connection rebalance_choice compared: a destination taken
// by ticket has connection 0 there as here.
template <typename C, typename W>
__device__ __forceinline__ u64 bucket_order(i64 v, i32 s, i32 t, const C* cache, const W* __restrict__ vw, int k) {
    const u64 current = static_cast<u64>(cache[v * k + s]), conn = static_cast<u64>(cache[v * k + t]);
    const double gain = conn >= current ? static_cast<double>(conn - current) : -static_cast<double>(current - conn);
    double g = gain / static_cast<double>(static_cast<u64>(weight_at(vw, v)));
    if (g == 0.0) g = 0.0;   // -0 and +0 tie
    const u64 b = static_cast<u64>(__double_as_longlong(g));
    const u64 ord = (b & 0x8000000000000000ULL) ? ~b : (b | 0x8000000000000000ULL);
    return ~ord;
}

// The list of items whose bucket crosses its part's quota, and per part the
// crossing bucket (kBalWidth: none) with the quota left for it.
struct CrossItem {
    u64 key;   // bucket_order
    i32 i;     // candidate index
    i32 v;     // vertex
};

struct CrossParts {
    u64 left[32];
    int bucket[32];
    u32 count;      // items in the list
    u32 pad;
};

// The rebalance kernels run over list[0, n), or over list[0, *count) when
// `count` is given (the candidate count left on the device, no round trip);
// their grid-stride loops keep whole warps together for the warp collectives.
__device__ __forceinline__ i64 list_length(i64 n, const i64* count) { return count ? *count : n; }

// Vertices of the parts above capacity, in any order: the only rebalance
// candidates, and a superset of them for the whole rebalance (destinations
// never exceed the capacity, so no part becomes overloaded and vertices only
// leave).
// Each block appends the vertices of 2048 consecutive ids at once: one atomic
// per tile, and the cache rows of neighbouring list entries stay close.
constexpr int kCollectItems = 8;
constexpr int kCollectTile = kThreads * kCollectItems;

__global__ void __launch_bounds__(kThreads) collect_overloaded_kernel(i64 n, const i32* __restrict__ labels, int k,
                                                                      const u64* __restrict__ pw, u64 cap, i32* list,
                                                                      i64* count) {
    __shared__ u32 over;
    __shared__ int warp_base[kWarps];
    __shared__ i64 tile_base;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp == 0) {
        const u32 m = __ballot_sync(0xffffffffu, lane < k && pw[lane] > cap);
        if (lane == 0) over = m;
    }
    __syncthreads();
    const u32 parts = over;
    for (i64 base = static_cast<i64>(blockIdx.x) * kCollectTile; base < n; base += static_cast<i64>(gridDim.x) * kCollectTile) {
        unsigned took[kCollectItems];
        int mine = 0;
        const i64 v0 = base + warp * 32 * kCollectItems + lane;
#pragma unroll
        for (int j = 0; j < kCollectItems; ++j) {
            const i64 v = v0 + j * 32;
            took[j] = __ballot_sync(0xffffffffu, v < n && ((parts >> labels[v]) & 1u));
            mine += __popc(took[j]);
        }
        if (lane == 0) warp_base[warp] = mine;
        __syncthreads();
        if (threadIdx.x == 0) {
            int sum = 0;
            for (int w = 0; w < kWarps; ++w) { const int c = warp_base[w]; warp_base[w] = sum; sum += c; }
            tile_base = sum ? static_cast<i64>(atomic_add_u64(reinterpret_cast<u64*>(count), static_cast<u64>(sum))) : 0;
        }
        __syncthreads();
        i64 at = tile_base + warp_base[warp];
#pragma unroll
        for (int j = 0; j < kCollectItems; ++j) {
            if ((took[j] >> lane) & 1u) list[at + __popc(took[j] & lanemask_lt())] = static_cast<i32>(v0 + j * 32);
            at += __popc(took[j]);
        }
        __syncthreads();   // warp_base and tile_base are free again
    }
}

// Choices of the candidates and the weight of every source bucket
// (balance_source_histogram, src/refine_incremental.cuh:167-186); part weights
// are staged in shared memory.
template <typename C, typename W>
__device__ __forceinline__ void rebalance_proposals(i64 n, const i32* list, const C* cache, const i32* labels,
                                                    const W* __restrict__ vw, int k, const u64* pw, u64 cap,
                                                    const BucketThresholds& th, i32* targets, i32* bucket, u64* counts,
                                                    u64* spw, BucketTable& table) {
    if (static_cast<i64>(blockIdx.x) * blockDim.x >= n) return;
    if (threadIdx.x < 32) spw[threadIdx.x] = static_cast<int>(threadIdx.x) < k ? pw[threadIdx.x] : ~0ULL;
    table.clear();
    __syncthreads();
    for (i64 base = static_cast<i64>(blockIdx.x) * blockDim.x; base < n; base += static_cast<i64>(gridDim.x) * blockDim.x) {
        const i64 i = base + threadIdx.x;
        u64 w = 0;
        int b = -1;
        if (i < n) {
            b = rebalance_choice(static_cast<i64>(list[i]), cache, labels, vw, k, spw, cap, th, targets, w);
            bucket[i] = b;
        }
        table.add(b, w, vw == nullptr, counts);
    }
    __syncthreads();
    table.flush(counts);
}

template <typename C, typename W>
__global__ void rebalance_proposals_kernel(i64 n, const i64* count, const i32* __restrict__ list,
                                           const C* __restrict__ cache, const i32* __restrict__ labels,
                                           const W* __restrict__ vw, int k, const u64* __restrict__ pw, u64 cap,
                                           BucketThresholds th, i32* targets, i32* bucket, u64* counts) {
    __shared__ u64 spw[32];
    __shared__ BucketTable table;
    rebalance_proposals(list_length(n, count), list, cache, labels, vw, k, pw, cap, th, targets, bucket, counts, spw,
                        table);
}

constexpr int kSelectThreads = 1024;
static_assert(kBalWidth <= 2 * 512, "at most two buckets of a part per thread of a 512-thread block");

// Exclusive block-wide sum for blocks of 512 or 1024 threads; `shared` needs
// 32 entries.
__device__ __forceinline__ u64 select_exclusive_sum(u64 v, u64* shared) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const u64 inc = warp_inclusive_sum(v);
    __syncthreads();
    if (lane == 31) shared[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        const u64 s = lane < static_cast<int>(blockDim.x >> 5) ? shared[lane] : 0;
        const u64 si = warp_inclusive_sum(s);
        shared[lane] = si - s;
    }
    __syncthreads();
    return shared[warp] + inc - v;
}

// Finds the bucket that crosses part p's quota among its kBalWidth bucket
// weights, which are left zero for the next pass (balance_scan_buckets,
// src/refine_incremental.cuh:188-202).  The quota is used up before a bucket's
// end: an item is taken while the weight before it is below the quota
// (SOURCES), or while the weight up to its own end is within it
// (!SOURCES).  A block of 512 or 1024 threads.
template <bool SOURCES>
__device__ void cross_bucket(int p, u64 quota, u64* counts, CrossParts* cross, u64* shared) {
    // two neighbouring buckets per thread
    const int b = 2 * static_cast<int>(threadIdx.x);
    u64 w[2] = {0, 0};
    if (b < kBalWidth) {
        ulonglong2* c = reinterpret_cast<ulonglong2*>(counts + p * kBalWidth + b);
        const ulonglong2 x = *c;
        *c = make_ulonglong2(0, 0);
        w[0] = x.x; w[1] = x.y;
    }
    if (b == 0) cross->bucket[p] = kBalWidth;
    u64 before = select_exclusive_sum(w[0] + w[1], shared);
    if (b < kBalWidth) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const bool crosses = SOURCES ? before < quota && before + w[j] >= quota
                                         : before <= quota && before + w[j] > quota;
            if (crosses) {
                cross->bucket[p] = b + j;
                cross->left[p] = quota - before;
            }
            before += w[j];
        }
    }
    __syncthreads();
}

struct SelectShared {
    u64 scan[32];
    u64 hist[256];
    u32 members[256];
    u64 key_and, key_or;
    u32 v_and, v_or;
    u64 left;              // quota left for the items that match the threshold
    u32 count, few;
    int digit;
    static constexpr u32 kItems = 2048;
    u64 key[kItems];
    i32 v[kItems];
    i32 i[kItems];
    static constexpr u32 kFew = 128;
    u64 few_key[kFew], few_w[kFew];
    u32 few_v[kFew];
};

// The items of part p's crossing bucket that are taken: their order's
// longest prefix within the quota.  A threshold is built from the high end of
// (key, v), eight varying bits a step: the weights of the items that match it
// so far are summed by digit, and the digit that crosses what is left of the
// quota extends it.  Bits in which the items agree cost no step, and once at
// most kFew items match they are ranked directly, 4 or 8 lanes an item (a
// step costs a microsecond of barriers, so most lists finish after one or
// two).  Lists of up to kItems items are staged in shared memory.
// f(item index, v, taken) is called for every item of the part.  A block of
// 512 or 1024 threads.
template <bool SOURCES, typename W, typename F>
__device__ void resolve_bucket(int p, const CrossParts* cross, const CrossItem* items,
                               const unsigned char* item_part, const W* __restrict__ vw, SelectShared& sh, F f) {
    const u32 total = cross->count;
    if (cross->bucket[p] == kBalWidth) return;   // uniform over the block
    const int lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        sh.count = sh.few = 0;
        sh.key_and = ~0ULL; sh.key_or = 0; sh.v_and = ~0u; sh.v_or = 0;
        sh.left = cross->left[p];
    }
    __syncthreads();
    u64 ka = ~0ULL, ko = 0;
    u32 va = ~0u, vo = 0;
    for (u32 j = threadIdx.x; j < total; j += static_cast<u32>(blockDim.x)) {
        if (item_part[j] != p) continue;
        const CrossItem x = items[j];
        ka &= x.key; ko |= x.key;
        va &= static_cast<u32>(x.v); vo |= static_cast<u32>(x.v);
        const u32 at = atomicAdd(&sh.count, 1u);
        if (at < SelectShared::kItems) { sh.key[at] = x.key; sh.v[at] = x.v; sh.i[at] = x.i; }
    }
    __syncthreads();
    const u32 count = sh.count;
    if (count == 0) return;
    const bool staged = count <= SelectShared::kItems;
    auto for_items = [&](auto g) {
        if (staged) {
            for (u32 j = threadIdx.x; j < count; j += static_cast<u32>(blockDim.x)) g(sh.key[j], sh.v[j], sh.i[j]);
        } else {
            for (u32 j = threadIdx.x; j < total; j += static_cast<u32>(blockDim.x))
                if (item_part[j] == p) { const CrossItem x = items[j]; g(x.key, x.v, x.i); }
        }
    };
    u64 hi_key = 0, key_above = 0;   // the threshold's bits so far
    u32 hi_v = 0, v_above = 0;
    auto matches = [&](u64 key, u32 v) { return (key & key_above) == hi_key && (v & v_above) == hi_v; };
    u32 matching = count;
    if (matching > SelectShared::kFew) {
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            ka &= __shfl_xor_sync(0xffffffffu, ka, o);
            ko |= __shfl_xor_sync(0xffffffffu, ko, o);
            va &= __shfl_xor_sync(0xffffffffu, va, o);
            vo |= __shfl_xor_sync(0xffffffffu, vo, o);
        }
        if (lane == 0) {
            atomicAnd(reinterpret_cast<unsigned long long*>(&sh.key_and), static_cast<unsigned long long>(ka));
            atomicOr(reinterpret_cast<unsigned long long*>(&sh.key_or), static_cast<unsigned long long>(ko));
            atomicAnd(&sh.v_and, va);
            atomicOr(&sh.v_or, vo);
        }
        __syncthreads();
        // one step: the digit of the matching items at which the quota is crossed
        auto step = [&](auto digit) {
            if (threadIdx.x < 256) { sh.hist[threadIdx.x] = 0; sh.members[threadIdx.x] = 0; }
            if (threadIdx.x == 0) sh.digit = 255;
            __syncthreads();
            for_items([&](u64 key, i32 v, i32) {
                if (!matches(key, static_cast<u32>(v))) return;
                const u32 dg = digit(key, static_cast<u32>(v));
                atomicAdd(&sh.members[dg], 1u);
                if (vw) atomic_add_u64(&sh.hist[dg], static_cast<u64>(vw[v]));
            });
            __syncthreads();
            u64 w = 0;
            if (threadIdx.x < 256) w = vw ? sh.hist[threadIdx.x] : static_cast<u64>(sh.members[threadIdx.x]);
            const u64 before = select_exclusive_sum(w, sh.scan);
            const u64 left = sh.left;
            __syncthreads();
            const bool crosses = SOURCES ? before < left && before + w >= left : before <= left && before + w > left;
            if (crosses && threadIdx.x < 256) {
                sh.digit = static_cast<int>(threadIdx.x);
                sh.left = left - before;
            }
            __syncthreads();
            const u32 dg = static_cast<u32>(sh.digit);
            matching = sh.members[dg];
            __syncthreads();   // the counts may be cleared again
            return dg;
        };
        u64 key_vary = sh.key_and ^ sh.key_or;
        hi_key = sh.key_and;
        key_above = ~key_vary;            // bits in which the items agree match from the start
        while (key_vary && matching > SelectShared::kFew) {
            const int top = 63 - __clzll(static_cast<long long>(key_vary));
            const int shift = top > 7 ? top - 7 : 0;
            const u64 field = 0xffULL >> (7 - (top - shift));
            const u32 dg = step([&](u64 key, u32) { return static_cast<u32>((key >> shift) & field); });
            key_above |= field << shift;
            hi_key = (hi_key & ~(field << shift)) | (static_cast<u64>(dg) << shift);
            key_vary &= ~(~0ULL << shift);
        }
        u32 v_vary = 0;
        if (matching > SelectShared::kFew) {
            v_vary = sh.v_and ^ sh.v_or;
            hi_v = sh.v_and;
            v_above = ~v_vary;
        }
        while (v_vary && matching > SelectShared::kFew) {
            const int top = 31 - __clz(static_cast<int>(v_vary));
            const int shift = top > 7 ? top - 7 : 0;
            const u32 field = 0xffu >> (7 - (top - shift));
            const u32 dg = step([&](u64, u32 v) { return (v >> shift) & field; });
            v_above |= field << shift;
            hi_v = (hi_v & ~(field << shift)) | (dg << shift);
            v_vary &= ~(~0u << shift);
        }
    }
    // rank the few that still match
    for_items([&](u64 key, i32 v, i32) {
        if (!matches(key, static_cast<u32>(v))) return;
        const u32 at = atomicAdd(&sh.few, 1u);
        if (at >= SelectShared::kFew) return;   // cannot happen: vertices differ
        sh.few_key[at] = key;
        sh.few_v[at] = static_cast<u32>(v);
        sh.few_w[at] = static_cast<u64>(weight_at(vw, v));
    });
    __syncthreads();
    {
        const u32 few = min(sh.few, SelectShared::kFew), lanes = blockDim.x / SelectShared::kFew;
        const u32 at = threadIdx.x / lanes;
        u64 key = 0, before = 0;
        u32 v = 0;
        if (at < few) {
            key = sh.few_key[at];
            v = sh.few_v[at];
            for (u32 j = threadIdx.x % lanes; j < few; j += lanes)
                if (sh.few_key[j] < key || (sh.few_key[j] == key && sh.few_v[j] < v)) before += sh.few_w[j];
        }
        for (int o = static_cast<int>(lanes) >> 1; o; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
        const u64 left = sh.left;
        const bool taken = at < few && (SOURCES ? before < left : before <= left && sh.few_w[at] <= left - before);
        __syncthreads();
        if (at < few && threadIdx.x % lanes == 0) sh.few_w[at] = taken ? 1 : 0;   // the weights are used up
    }
    __syncthreads();
    const u32 few = min(sh.few, SelectShared::kFew);
    for_items([&](u64 key, i32 v, i32 i) {
        const u32 uv = static_cast<u32>(v);
        bool taken;
        if (matches(key, uv)) {
            taken = false;
            for (u32 j = 0; j < few; ++j)
                if (sh.few_v[j] == uv) { taken = sh.few_w[j] != 0; break; }
        } else {
            // above the threshold's bits: ahead of every matching item or behind them
            const u64 a = key & key_above;
            taken = a < hi_key || (a == hi_key && (uv & v_above) < hi_v);
        }
        f(i, v, taken);
    });
    __syncthreads();
}

// One block per part: the crossing bucket of every overloaded part's
// excess; also clears the counters that the rest of the iteration adds to.
__global__ void __launch_bounds__(kSelectThreads) cross_sources_kernel(const u64* __restrict__ pw, u64 cap, u64* counts,
                                                                       CrossParts* cross, RefineCounters* ctr) {
    __shared__ u64 shared[32];
    const int p = blockIdx.x;
    if (p == 0 && threadIdx.x == 0) { *ctr = RefineCounters{}; cross->count = 0; }
    const u64 load = pw[p];
    cross_bucket<true>(p, load > cap ? load - cap : 0, counts, cross, shared);
}

// Appends the lanes' crossing items.  All 32 lanes call it.
template <typename C, typename W>
__device__ __forceinline__ void append_crossing(bool take, i64 i, i64 v, int part, const C* cache, const i32* labels,
                                                const i32* targets, const W* __restrict__ vw, int k,
                                                CrossParts* cross, CrossItem* items, unsigned char* item_part) {
    const unsigned m = __ballot_sync(0xffffffffu, take);
    if (!m) return;
    const int lane = threadIdx.x & 31, leader = __ffs(m) - 1;
    u32 base = 0;
    if (lane == leader) base = atomicAdd(&cross->count, static_cast<u32>(__popc(m)));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (!take) return;
    const u32 at = base + __popc(m & lanemask_lt());
    items[at] = {bucket_order(v, labels[v], targets[v], cache, vw, k), static_cast<i32>(i), static_cast<i32>(v)};
    item_part[at] = static_cast<unsigned char>(part);
}

// balance_select_sources (src/refine_incremental.cuh:204-217): candidates in
// buckets before their part's crossing bucket leave it and are counted in
// their destination's buckets; those in it are listed for the selection.
template <typename C, typename W>
__device__ __forceinline__ void select_sources(i64 n, const i32* list, i32* bucket, const C* cache, const i32* labels,
                                               const i32* targets, const W* __restrict__ vw, int k, u64* counts,
                                               CrossParts* cross, CrossItem* items, unsigned char* item_part,
                                               int* crossing, BucketTable& table) {
    if (static_cast<i64>(blockIdx.x) * blockDim.x >= n) return;
    if (static_cast<int>(threadIdx.x) < k) crossing[threadIdx.x] = cross->bucket[threadIdx.x];
    table.clear();
    __syncthreads();
    for (i64 base = static_cast<i64>(blockIdx.x) * blockDim.x; base < n; base += static_cast<i64>(gridDim.x) * blockDim.x) {
        const i64 i = base + threadIdx.x;
        int d = -1, s = 0;
        i64 v = 0;
        bool listed = false;
        const int b = i < n ? bucket[i] : -1;
        if (b >= 0) {
            s = b / kBalWidth;
            const int lb = b - s * kBalWidth;
            if (lb <= crossing[s]) {
                v = list[i];
                d = targets[v] * kBalWidth + lb;
                listed = lb == crossing[s];
            }
            bucket[i] = d;
        }
        const bool now = d >= 0 && !listed;
        table.add(now ? d : -1, now ? static_cast<u64>(weight_at(vw, v)) : 0, vw == nullptr, counts);
        append_crossing(listed, i, v, s, cache, labels, targets, vw, k, cross, items, item_part);
    }
    __syncthreads();
    table.flush(counts);
}

template <typename C, typename W>
__global__ void select_sources_kernel(i64 n, const i64* count, const i32* __restrict__ list, i32* bucket,
                                      const C* __restrict__ cache, const i32* __restrict__ labels,
                                      const i32* __restrict__ targets, const W* __restrict__ vw, int k, u64* counts,
                                      CrossParts* cross, CrossItem* items, unsigned char* item_part) {
    __shared__ int crossing[32];
    __shared__ BucketTable table;
    select_sources(list_length(n, count), list, bucket, cache, labels, targets, vw, k, counts, cross, items, item_part,
                   crossing, table);
}

constexpr int kSelectCluster = 8;

// One thread-block cluster between the two marking passes: the source
// selections (a block per part in turn), then, once every taken item is
// counted, the destinations' crossing buckets.  The cluster barrier stands
// where two launches stood.
template <typename W>
__global__ void __cluster_dims__(kSelectCluster, 1, 1) __launch_bounds__(kSelectThreads) resolve_sources_kernel(
    int k, const u64* __restrict__ pw, u64 cap, i32* bucket, const W* __restrict__ vw, u64* counts,
    CrossParts* sources, CrossParts* dests, const CrossItem* items, const unsigned char* item_part) {
    __shared__ SelectShared sh;
    const int rank = static_cast<int>(blockIdx.x);
    for (int p = rank; p < k; p += kSelectCluster)
        resolve_bucket<true>(p, sources, items, item_part, vw, sh, [&](i32 i, i32 v, bool taken) {
            if (taken) atomic_add_u64(&counts[bucket[i]], static_cast<u64>(weight_at(vw, v)));
            else bucket[i] = -1;
        });
    cooperative_groups::this_cluster().sync();
    if (rank == 0 && threadIdx.x == 0) dests->count = 0;
    for (int p = rank; p < k; p += kSelectCluster) {
        const u64 load = pw[p];
        cross_bucket<false>(p, load < cap ? cap - load : 0, counts, dests, sh.scan);
    }
}

// balance_select_destinations (src/refine_incremental.cuh:219-232): the
// candidates left whose destination bucket lies before the crossing bucket
// of the destination's slack move.
template <typename C, typename W>
__device__ __forceinline__ void select_destinations(i64 n, const i32* list, const i32* bucket, const C* cache,
                                                    const i32* labels, const i32* targets, const W* __restrict__ vw,
                                                    int k, CrossParts* cross, CrossItem* items,
                                                    unsigned char* item_part, unsigned char* flags, i32* movers,
                                                    RefineCounters* ctr, int* crossing) {
    if (static_cast<i64>(blockIdx.x) * blockDim.x >= n) return;
    if (static_cast<int>(threadIdx.x) < k) crossing[threadIdx.x] = cross->bucket[threadIdx.x];
    __syncthreads();
    for (i64 base = static_cast<i64>(blockIdx.x) * blockDim.x; base < n; base += static_cast<i64>(gridDim.x) * blockDim.x) {
        const i64 i = base + threadIdx.x;
        bool move = false, listed = false;
        int p = 0;
        i64 v = 0;
        const int b = i < n ? bucket[i] : -1;
        if (b >= 0) {
            v = list[i];
            p = b / kBalWidth;
            const int lb = b - p * kBalWidth;
            move = lb < crossing[p];
            listed = lb == crossing[p];
        }
        const u64 slot = warp_append(move, reinterpret_cast<u64*>(&ctr->movers));
        if (move) {
            flags[v] = 1;
            movers[slot] = static_cast<i32>(v);
        }
        append_crossing(listed, i, v, p, cache, labels, targets, vw, k, cross, items, item_part);
    }
}

template <typename C, typename W>
__global__ void select_destinations_kernel(i64 n, const i64* count, const i32* __restrict__ list,
                                           const i32* __restrict__ bucket, const C* __restrict__ cache,
                                           const i32* __restrict__ labels, const i32* __restrict__ targets,
                                           const W* __restrict__ vw, int k, CrossParts* cross, CrossItem* items,
                                           unsigned char* item_part, unsigned char* flags, i32* movers,
                                           RefineCounters* ctr) {
    __shared__ int crossing[32];
    select_destinations(list_length(n, count), list, bucket, cache, labels, targets, vw, k, cross, items, item_part,
                        flags, movers, ctr, crossing);
}

// One block per part: the movers of its destination crossing bucket.
template <typename W>
__global__ void __launch_bounds__(kSelectThreads) resolve_destinations_kernel(
    const W* __restrict__ vw, const CrossParts* cross, const CrossItem* items, const unsigned char* item_part,
    unsigned char* flags, i32* movers, RefineCounters* ctr) {
    __shared__ SelectShared sh;
    resolve_bucket<false>(static_cast<int>(blockIdx.x), cross, items, item_part, vw, sh, [&](i32, i32 v, bool taken) {
        if (!taken) return;
        flags[v] = 1;
        movers[atomic_add_u64(reinterpret_cast<u64*>(&ctr->movers), 1)] = v;
    });
}

__global__ void project_kernel(i64 n, const i32* map, const i32* coarse, i32* fine) {
    const i64 v = static_cast<i64>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (v < n) fine[v] = coarse[map[v]];
}

template <typename W>
__global__ void max_weight_kernel(i64 m, const W* ew, u64* out) {
    u64 mx = 0;
    for (i64 i = static_cast<i64>(blockIdx.x) * blockDim.x + threadIdx.x; i < m; i += static_cast<i64>(gridDim.x) * blockDim.x)
        mx = static_cast<u64>(ew[i]) > mx ? static_cast<u64>(ew[i]) : mx;
    mx = warp_max(mx);
    if ((threadIdx.x & 31) == 0 && mx) atomic_max_u64(out, mx);
}

}  // namespace gp
