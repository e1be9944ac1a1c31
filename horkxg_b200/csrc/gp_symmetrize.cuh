// Symmetrise and deduplicate a CSR on the GPU, with the semantics of the
// reference's external-memory tool (graph_untils/csr_symmetrize.cpp:277-538):
// every entry (v, u) with u != v stands for the undirected edge {u, v}; self
// loops are dropped and counted; the output holds both directions of every
// distinct edge, rows ascending by neighbour.
//
// The reference sorts (min, max) keys in disk runs, merges them, counts
// degrees and sorts again for the reverse direction.  Graphs of up to 2^22
// vertices are symmetrised row by row with the contraction's row sorts (see
// symmetrize_rows); above, and for generated graphs, the whole job is one
// device radix sort: each entry writes its two directed keys
// (v << b | u) and (u << b | v), b = bits of the vertex range, into slots 2e
// and 2e + 1 (a self loop writes two all-ones sentinels, which sort last);
// after the sort equal neighbours are adjacent, a flag-and-scan compaction
// keeps the first of each run, and the rows' lengths come from warp-
// aggregated counts of the sources.
#pragma once

#include "gp_contract.cuh"
#include "gp_prim.cuh"

namespace gp {

constexpr u64 kSymSentinel = ~0ULL;

// One warp per row: the two directed keys of every entry.
template <typename O>
__global__ void __launch_bounds__(kThreads) sym_keys_kernel(i64 n, const O* __restrict__ off,
                                                            const i32* __restrict__ nbr, int bits, u64* keys,
                                                            u64* self_loops) {
    const int lane = threadIdx.x & 31;
    const i64 warps_total = static_cast<i64>(gridDim.x) * kWarps;
    u64 loops = 0;
    for (i64 v = static_cast<i64>(blockIdx.x) * kWarps + (threadIdx.x >> 5); v < n; v += warps_total) {
        const i64 b = off[v], end = off[v + 1];
        for (i64 e = b + lane; e < end; e += 32) {
            const u64 u = static_cast<u64>(nbr[e]);
            if (u == static_cast<u64>(v)) {
                keys[2 * e] = kSymSentinel;
                keys[2 * e + 1] = kSymSentinel;
                ++loops;
            } else {
                keys[2 * e] = (static_cast<u64>(v) << bits) | u;
                keys[2 * e + 1] = (u << bits) | static_cast<u64>(v);
            }
        }
    }
    loops = warp_sum(loops);
    if (lane == 0 && loops) atomicAdd(reinterpret_cast<unsigned long long*>(self_loops), loops);
}

// R-MAT pairs generated on the device, drawn exactly as the host generator
// of this package draws them (horkxg_b200/csrc/gen.cpp, build_rmat): pair i,
// level l takes the uniform double of splitmix64(stream ^ splitmix64(64 i +
// l)) and descends into quadrant a | b | c | d; vertex ids then go through the
// seeded permutation `perm`.  Each pair writes its two directed keys (or two
// sentinels for a self loop), as sym_keys_kernel does for a CSR entry.
// splitmix64 is the published 64-bit mixer of Steele, Lea and Flood.
__host__ __device__ __forceinline__ u64 splitmix64(u64 x) {
    x += 0x9e3779b97f4a7c15ULL;
    x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ULL;
    x = (x ^ (x >> 27)) * 0x94d049bb133111ebULL;
    return x ^ (x >> 31);
}

__global__ void rmat_keys_kernel(i64 pairs, int scale, double a, double ab, double abc, u64 stream,
                                 const u32* __restrict__ perm, int bits, u64* keys) {
    for (i64 i = static_cast<i64>(blockIdx.x) * blockDim.x + threadIdx.x; i < pairs;
         i += static_cast<i64>(gridDim.x) * blockDim.x) {
        u32 s = 0, d = 0;
        for (int level = 0; level < scale; ++level) {
            const u64 x = splitmix64(stream ^ splitmix64(static_cast<u64>(i) * 64 + static_cast<u64>(level)));
            const double r = static_cast<double>(x >> 11) * (1.0 / 9007199254740992.0);
            s = (s << 1) | (r >= ab ? 1u : 0u);
            d = (d << 1) | (((r >= a && r < ab) || r >= abc) ? 1u : 0u);
        }
        const u64 ps = perm[s], pd = perm[d];
        keys[2 * i] = ps == pd ? kSymSentinel : (ps << bits) | pd;
        keys[2 * i + 1] = ps == pd ? kSymSentinel : (pd << bits) | ps;
    }
}

// Position of the first sentinel among sorted keys (= the count of keys
// that are not sentinels), into *first (preset to the key count).
__global__ void sym_first_sentinel_kernel(i64 count, const u64* __restrict__ keys, i64* first) {
    for (i64 i = static_cast<i64>(blockIdx.x) * blockDim.x + threadIdx.x; i < count;
         i += static_cast<i64>(gridDim.x) * blockDim.x)
        if (keys[i] == kSymSentinel && (i == 0 || keys[i - 1] != kSymSentinel)) *first = i;
}

// First key of each run among the `valid` sorted keys.
struct SymHead {
    const u64* keys;
    i64 valid;
    __device__ i64 operator()(i64 i) const { return i < valid && (i == 0 || keys[i] != keys[i - 1]) ? 1 : 0; }
};

// Writes the neighbour of every run head at its rank and counts the row
// lengths (keys sorted by source, so a warp's heads mostly share a source:
// one atomic per source and warp).
template <typename N>
__global__ void sym_compact_kernel(i64 valid, const u64* __restrict__ keys, const i64* __restrict__ rank, int bits,
                                   N* out_nbr, i64* degree) {
    const i64 stride = static_cast<i64>(gridDim.x) * blockDim.x;
    const i64 end = (valid + 31) / 32 * 32;   // whole warps, for the match below
    for (i64 i = static_cast<i64>(blockIdx.x) * blockDim.x + threadIdx.x; i < end; i += stride) {
        const bool head = i < valid && (i == 0 || keys[i] != keys[i - 1]);
        const u64 key = i < valid ? keys[i] : 0;
        const i64 src = head ? static_cast<i64>(key >> bits) : -1;
        if (head) out_nbr[rank[i]] = static_cast<N>(key & ((1ULL << bits) - 1));
        const unsigned peers = __match_any_sync(0xffffffffu, src);
        if (head && (threadIdx.x & 31) == __ffs(peers) - 1)
            atomicAdd(reinterpret_cast<unsigned long long*>(&degree[src]), static_cast<unsigned long long>(__popc(peers)));
    }
}

// ---------------------------------------------------------------------------
// Row by row.  A block takes a tile of consecutive entries, so hub rows are
// spread like any others; an entry's row is found by bisection among the rows
// of the tile.
// ---------------------------------------------------------------------------
constexpr int kSymItems = 8;
constexpr i64 kSymTile = kThreads * kSymItems;

// Last row r in [lo, hi] with off[r] <= e.
template <typename O>
__device__ __forceinline__ i64 row_of_entry(const O* __restrict__ off, i64 lo, i64 hi, i64 e) {
    while (lo < hi) {
        const i64 mid = (lo + hi + 1) >> 1;
        if (static_cast<i64>(off[mid]) <= e) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// f(entry, row) for the block's tile.
template <typename O, typename F>
__device__ __forceinline__ void for_tile_entries(i64 n, i64 m, const O* __restrict__ off, F f) {
    __shared__ i64 range[2];
    const i64 begin = static_cast<i64>(blockIdx.x) * kSymTile;
    const i64 end = begin + kSymTile < m ? begin + kSymTile : m;
    if (begin >= end) return;   // uniform over the block
    if (threadIdx.x < 2) range[threadIdx.x] = row_of_entry(off, 0, n - 1, threadIdx.x ? end - 1 : begin);
    __syncthreads();
    const i64 lo = range[0], hi = range[1];
#pragma unroll 2
    for (i64 e = begin + threadIdx.x; e < end; e += kThreads) f(e, row_of_entry(off, lo, hi, e));
}

// Arrivals of reversed entries per vertex; place[e] is entry e's number among
// its target's.
template <typename O>
__global__ void __launch_bounds__(kThreads) sym_count_kernel(i64 n, i64 m, const O* __restrict__ off,
                                                             const i32* __restrict__ nbr, u32* arrivals, u32* place,
                                                             u64* self_loops) {
    u64 loops = 0;
    for_tile_entries(n, m, off, [&](i64 e, i64 v) {
        const i32 u = nbr[e];
        if (u == v) ++loops;
        else place[e] = atomicAdd(&arrivals[u], 1u);
    });
    loops = warp_sum(loops);
    if ((threadIdx.x & 31) == 0 && loops) atomic_add_u64(self_loops, loops);
}

// Entries of a vertex's row before deduplication: its own, then the arrivals.
template <typename O>
struct SymRowTotal {
    const O* off;
    const u32* arrivals;
    i64 n;
    __device__ i64 operator()(i64 v) const {
        return v < n ? static_cast<i64>(off[v + 1]) - static_cast<i64>(off[v]) + arrivals[v] : 0;
    }
};

// Self loops become the sentinel n.
template <typename O>
__global__ void __launch_bounds__(kThreads) sym_scatter_kernel(i64 n, i64 m, const O* __restrict__ off,
                                                               const i32* __restrict__ nbr,
                                                               const u32* __restrict__ place,
                                                               const i64* __restrict__ temp_off, u32* __restrict__ tgt) {
    for_tile_entries(n, m, off, [&](i64 e, i64 v) {
        const i32 u = nbr[e];
        tgt[temp_off[v] + (e - static_cast<i64>(off[v]))] = u == v ? static_cast<u32>(n) : static_cast<u32>(u);
        if (u != v)
            tgt[temp_off[u] + (static_cast<i64>(off[u + 1]) - static_cast<i64>(off[u])) + place[e]] = static_cast<u32>(v);
    });
}

// The unique neighbours of the rows sorted in place, a warp per 32 rows.
template <typename N>
__global__ void __launch_bounds__(kThreads) sym_copy_rows_kernel(i64 rows, const i64* __restrict__ temp_off,
                                                                 const i64* __restrict__ off,
                                                                 const u32* __restrict__ tgt, N* __restrict__ nbr) {
    const int lane = threadIdx.x & 31;
    const i64 r0 = ((static_cast<i64>(blockIdx.x) * kThreads + threadIdx.x) >> 5) * 32;
    if (r0 >= rows) return;
    const i64 r = r0 + lane;
    i64 to = 0, len = 0, from = 0;
    if (r < rows) {
        to = off[r];
        len = off[r + 1] - to;
        from = temp_off[r];
        if (temp_off[r + 1] - from > seg_smem_capacity<u32>()) len = 0;   // sym_copy_big_rows_kernel
    }
    warp_edge_walk(from, len, [&](bool valid, int owner, i64 i) {
        const i64 shift = __shfl_sync(0xffffffffu, to - from, owner);
        if (valid) nbr[i + shift] = static_cast<N>(tgt[i]);
    });
}

template <typename N>
__global__ void __launch_bounds__(kThreads) sym_copy_big_rows_kernel(const i32* __restrict__ list,
                                                                     const i64* __restrict__ alt_off,
                                                                     const i64* __restrict__ off,
                                                                     const u32* __restrict__ keys, N* __restrict__ nbr) {
    const i32 r = list[blockIdx.x];
    const i64 to = off[r], len = off[r + 1] - to, from = alt_off[blockIdx.x];
    for (i64 i = threadIdx.x; i < len; i += kThreads) nbr[to + i] = static_cast<N>(keys[from + i]);
}

}  // namespace gp
