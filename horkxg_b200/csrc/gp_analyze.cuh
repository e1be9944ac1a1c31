// Partition analysis on the GPU: the per-part figures of the reference's CPU
// analyzer (graph_untils/analyze_partition.cpp:425-499) from the original CSR
// and a label array -- vertex counts, internal directed entries, outgoing and
// incoming cut entries, each also summed by edge weight.  The summary figures
// (imbalances, deviations, local cuts) follow on the host from these.
//
// Every entry (v, u) adds one to the counter of (u's part, whether v's part is
// the same): one shared-memory addition an entry.  The rest follows at the
// end: an entry's source part needs no count of its own, since the outgoing
// entries of a part are its row lengths less its internal entries.
//
// Layout of the 7 x parts counters: vertices, internal, outgoing, incoming,
// weighted internal, weighted outgoing, weighted incoming.
//
// Bound by the gather of one label per entry from L2.  A warp walks 32 rows
// at once, so short rows leave no lane idle.  RMAT-22 (128 M entries, k = 32):
// rows 1.69 -> 0.78 ms, hubs 0.32 -> 0.20 ms against a warp per vertex with
// matched 64-bit additions.
#pragma once

#include "gp_prim.cuh"
#include "gp_hub.cuh"

namespace gp {

constexpr int kAnalyzeMaxParts = 1024;
constexpr int kAnalyzeFields = 7;

// Shared counters of one block: per part the entries arriving from other
// parts and from inside, the row lengths, the vertices, and the same by weight.
struct AnalyzeShared {
    u32* entries;      // [2 part + inside]
    u64* weights;      // [2 part + inside], weighted graphs
    u64* row_weight;   // outgoing and internal by source, weighted graphs
    u64* row_length;
    u32* vertices;
};

__host__ __device__ inline size_t analyze_smem(int parts, bool weighted) {
    return static_cast<size_t>(parts) * (2 * sizeof(u32) + sizeof(u64) + sizeof(u32) + 4 +
                                         (weighted ? 3 * sizeof(u64) : 0));
}

__device__ __forceinline__ AnalyzeShared analyze_shared(unsigned char* raw, int parts, bool weighted) {
    AnalyzeShared s;
    s.row_length = reinterpret_cast<u64*>(raw);
    s.weights = s.row_length + parts;
    s.row_weight = s.weights + (weighted ? 2 * parts : 0);
    s.entries = reinterpret_cast<u32*>(s.row_weight + (weighted ? parts : 0));
    s.vertices = s.entries + 2 * parts;
    for (int i = threadIdx.x; i < parts; i += kThreads) {
        s.row_length[i] = 0;
        s.vertices[i] = s.entries[2 * i] = s.entries[2 * i + 1] = 0;
        if (weighted) s.weights[2 * i] = s.weights[2 * i + 1] = s.row_weight[i] = 0;
    }
    __syncthreads();
    return s;
}

// Walk steps whose label gathers are in flight together: RMAT-22's rows (k = 32)
// take 0.49 ms (2.2 TB/s) instead of 0.78 ms with one.
constexpr int kAnalyzeBatch = 4;

// One entry from source part `sp` to a neighbour of part `q`; false when that
// label is out of range.
template <typename W>
__device__ __forceinline__ bool analyze_entry(i64 e, int q, int sp, const W* __restrict__ ew, int parts,
                                              const AnalyzeShared& s) {
    if (q < 0 || q >= parts) return false;
    const int slot = 2 * q + (q == sp ? 1 : 0);
    atomicAdd(&s.entries[slot], 1u);
    if (ew) {
        const u64 w = static_cast<u64>(ew[e]);
        atomic_add_u64(&s.weights[slot], w);
        atomic_add_u64(&s.row_weight[sp], w);
    }
    return true;
}

__device__ __forceinline__ void analyze_flush(const AnalyzeShared& s, int parts, bool weighted, u64* out) {
    __syncthreads();
    for (int p = threadIdx.x; p < parts; p += kThreads) {
        const u64 in = s.entries[2 * p], inside = s.entries[2 * p + 1];
        if (s.vertices[p]) atomic_add_u64(&out[p], s.vertices[p]);
        if (inside) atomic_add_u64(&out[parts + p], inside);
        // modulo 2^64: another block may hold this part's internal entries
        if (s.row_length[p] != inside) atomic_add_u64(&out[2 * parts + p], s.row_length[p] - inside);
        if (in) atomic_add_u64(&out[3 * parts + p], in);
        const u64 win = weighted ? s.weights[2 * p] : in, winside = weighted ? s.weights[2 * p + 1] : inside;
        const u64 wrow = weighted ? s.row_weight[p] : s.row_length[p];
        if (winside) atomic_add_u64(&out[4 * parts + p], winside);
        if (wrow != winside) atomic_add_u64(&out[5 * parts + p], wrow - winside);
        if (win) atomic_add_u64(&out[6 * parts + p], win);
    }
}

// 32 rows per warp and step, of at most kHubDegree entries (hub rows are
// walked by analyze_hub_kernel); every vertex is counted here.
template <typename O, typename W>
__global__ void __launch_bounds__(kThreads) analyze_rows_kernel(i64 n, const O* __restrict__ off,
                                                                const i32* __restrict__ nbr, const W* __restrict__ ew,
                                                                const i32* __restrict__ labels, int parts, u64* out,
                                                                u32* err) {
    extern __shared__ __align__(16) unsigned char raw[];
    const AnalyzeShared s = analyze_shared(raw, parts, ew != nullptr);
    const int lane = threadIdx.x & 31;
    bool bad = false;
    const i64 warps = static_cast<i64>(gridDim.x) * kWarps;
    for (i64 v0 = (static_cast<i64>(blockIdx.x) * kWarps + (threadIdx.x >> 5)) * 32; v0 < n; v0 += warps * 32) {
        const i64 v = v0 + lane;
        int sp = -1;
        i64 b = 0, deg = 0;
        if (v < n) {
            sp = labels[v];
            if (sp < 0 || sp >= parts) {
                bad = true;
                sp = -1;
            } else {
                b = static_cast<i64>(off[v]);
                deg = static_cast<i64>(off[v + 1]) - b;
                if (deg > kHubDegree) deg = 0;
                atomicAdd(&s.vertices[sp], 1u);
                if (deg) atomic_add_u64(&s.row_length[sp], static_cast<u64>(deg));
            }
        }
        // warp_edge_walk kAnalyzeBatch steps at a time: the batch's neighbours
        // are loaded, then their labels, before any counter is touched
        const i64 inc = warp_inclusive_sum(deg);
        const i64 pre = inc - deg;
        const i64 total = __shfl_sync(0xffffffffu, inc, 31);
        for (i64 base = 0; base < total; base += kAnalyzeBatch * 32) {
            int from[kAnalyzeBatch], q[kAnalyzeBatch];
            i32 u[kAnalyzeBatch];
            i64 e[kAnalyzeBatch];
#pragma unroll
            for (int j = 0; j < kAnalyzeBatch; ++j) {
                const i64 at = base + j * 32 + lane;
                int lo = 0;
#pragma unroll
                for (int step = 16; step; step >>= 1) {
                    const i64 probe = __shfl_sync(0xffffffffu, pre, lo + step);
                    if (probe <= at) lo += step;
                }
                const i64 my_pre = __shfl_sync(0xffffffffu, pre, lo);
                e[j] = __shfl_sync(0xffffffffu, b, lo) + (at - my_pre);
                from[j] = __shfl_sync(0xffffffffu, sp, lo);
                u[j] = at < total ? nbr[e[j]] : -1;
            }
#pragma unroll
            for (int j = 0; j < kAnalyzeBatch; ++j) q[j] = u[j] >= 0 ? labels[u[j]] : -1;
#pragma unroll
            for (int j = 0; j < kAnalyzeBatch; ++j) {
                if (u[j] < 0) continue;
                if (!analyze_entry(e[j], q[j], from[j], ew, parts, s)) bad = true;
            }
        }
    }
    if (bad) set_error(err, kErrBadInput);
    analyze_flush(s, parts, ew != nullptr, out);
}

// Hub rows, 2048-entry chunks in a grid-stride loop.  Vertex counts are not
// touched (analyze_rows_kernel counted every vertex).
template <typename W>
__global__ void __launch_bounds__(kThreads) analyze_hub_kernel(i64 count, const Chunk* __restrict__ chunks,
                                                               const i32* __restrict__ nbr, const W* __restrict__ ew,
                                                               const i32* __restrict__ labels, int parts, u64* out,
                                                               u32* err) {
    extern __shared__ __align__(16) unsigned char raw[];
    const AnalyzeShared s = analyze_shared(raw, parts, ew != nullptr);
    bool bad = false;
    for (i64 c = blockIdx.x; c < count; c += gridDim.x) {
        const Chunk ch = chunks[c];
        const int sp = labels[ch.v];
        if (sp < 0 || sp >= parts) {
            bad = true;
            continue;
        }
        if (threadIdx.x == 0) atomic_add_u64(&s.row_length[sp], static_cast<u64>(ch.end - ch.begin));
        for (i64 e = ch.begin + threadIdx.x; e < ch.end; e += kThreads)
            if (!analyze_entry(e, labels[nbr[e]], sp, ew, parts, s)) bad = true;
    }
    if (bad) set_error(err, kErrBadInput);
    analyze_flush(s, parts, ew != nullptr, out);
}

}  // namespace gp
