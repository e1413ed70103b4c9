// CUDA-core kernels: SpMM and SDDMM for V = 1/2/4/8 in fp32 or fp16 (fp32 accumulate), and the masked row
// softmax.  These are the `cudaSpmm` / `cudaSddmm` family of the reference (src/cuda_spmm.cu,
// src/cuda_sddmm.cu) including the fp32 SpMM the reference leaves as a stub (src/cuda_spmm.cu:328-338).
//
// Design: no shared memory and no intra-CTA cooperation.  Each thread (SpMM) or 8-lane group (SDDMM) owns an
// independent piece of output, dense operands are read with 16-byte loads that coalesce across neighbouring
// threads, and the per-nonzero index / value-vector loads are warp-uniform broadcasts served by L1.
#pragma once
#include "common.cuh"

namespace vs {

constexpr int kCcThreads = 128;

// ---- SpMM ---------------------------------------------------------------------------------------------------
// Work item = (vector-row in row_indices order, kChunks 16-byte chunks of the dense width, 32 chunks apart so that
// the lanes of a warp still read consecutive chunks).  The thread keeps V x E x kChunks fp32 accumulators (E = elements
// per 16 bytes) and walks the row's nonzero vectors four at a time so that four independent gathers of B are in
// flight.  With two or four chunks per thread the warp-uniform loads of an entry (column index, value vector) feed
// that many times the FMAs; it needs the dense width to be a multiple of 32 kChunks chunks.
//
// kSlabs: wide fp32 products go slab by slab: the warps of an SM take the same columns, so that a row of B serves several of them from L1.  A kernel of
// its own: the choice inside this one cost the narrow products up to 8 % (fp16 operands, V = 1, 3 x (452 x 4237 x 72), 94.5 %: 51.9 -> 55.4 us).
constexpr int kSlabColumns = 4096;
template <typename TIn, typename TOut, int V, int kChunks, bool kSlabs>
__device__ __forceinline__ void spmm_cc_item(const SpmmParams &p, int b, int64_t item, int few = 0) {   // few > 0: only rows of 1 .. few - 1 entries
    constexpr int E = Chunk<TIn>::kElems;
    constexpr int U = kChunks == 1 ? 4 : (kChunks == 2 ? 2 : 1);
    const int chunks = p.N / (E * kChunks);            // items per vector-row
    int order, piece;
    if constexpr (kSlabs) {   // chunks is a multiple of 32
        const int64_t w = item / 32;
        order = (int)(w % p.m_vec);
        piece = (int)(w / p.m_vec) * 32 + (int)(item % 32);
    } else {
        order = (int)(item / chunks);
        piece = (int)(item - (int64_t)order * chunks);
    }
    // kChunks > 1: warp-sized groups of items take chunks 32 kChunks g + lane, + 32 + lane, ...
    const int chunk = kChunks == 1 ? piece : (piece / 32) * (32 * kChunks) + (piece % 32);
    const int row = __ldg(p.row_indices + order);

    const TIn *values = static_cast<const TIn *>(p.values) + (int64_t)b * p.stride_values;
    const TIn *rhs = static_cast<const TIn *>(p.rhs) + (int64_t)b * p.stride_rhs + (int64_t)chunk * E;
    TOut *out = static_cast<TOut *>(p.out) + (int64_t)b * p.stride_out + (int64_t)chunk * E;

    float acc[kChunks][V][E];
#pragma unroll
    for (int q = 0; q < kChunks; ++q)
#pragma unroll
        for (int v = 0; v < V; ++v)
#pragma unroll
            for (int e = 0; e < E; ++e) acc[q][v][e] = 0.f;

    int j = __ldg(p.row_offsets + row);
    const int end = __ldg(p.row_offsets + row + 1);
    if (few > 0 && (end <= j || end - j >= few)) return;

    for (; j + U <= end; j += U) {
        int col[U];
        float a[U][V];
        Chunk<TIn> bt[U][kChunks];
#pragma unroll
        for (int u = 0; u < U; ++u) col[u] = __ldg(p.col_indices + j + u);
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int q = 0; q < kChunks; ++q) bt[u][q].load(rhs + (int64_t)col[u] * p.N + q * 32 * E);
#pragma unroll
        for (int u = 0; u < U; ++u) VecLoad<TIn, V>::load(values + (int64_t)(j + u) * V, a[u]);
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int q = 0; q < kChunks; ++q)
#pragma unroll
                for (int v = 0; v < V; ++v)
#pragma unroll
                    for (int e = 0; e < E; ++e) acc[q][v][e] = fmaf(a[u][v], bt[u][q].f[e], acc[q][v][e]);
    }
    for (; j < end; ++j) {
        const int col = __ldg(p.col_indices + j);
        float a[V];
        Chunk<TIn> bt[kChunks];
#pragma unroll
        for (int q = 0; q < kChunks; ++q) bt[q].load(rhs + (int64_t)col * p.N + q * 32 * E);
        VecLoad<TIn, V>::load(values + (int64_t)j * V, a);
#pragma unroll
        for (int q = 0; q < kChunks; ++q)
#pragma unroll
            for (int v = 0; v < V; ++v)
#pragma unroll
                for (int e = 0; e < E; ++e) acc[q][v][e] = fmaf(a[v], bt[q].f[e], acc[q][v][e]);
    }

#pragma unroll
    for (int q = 0; q < kChunks; ++q)
#pragma unroll
        for (int v = 0; v < V; ++v) store_chunk(out + ((int64_t)row * V + v) * p.N + q * 32 * E, acc[q][v]);
}

template <typename TIn, typename TOut, int V, int kChunks, bool kSlabs = false>
__global__ void __launch_bounds__(kCcThreads) spmm_cc_kernel(const SpmmParams p) {
    const int64_t item = (int64_t)blockIdx.x * kCcThreads + threadIdx.x;
    if (item < (int64_t)p.m_vec * (p.N / (Chunk<TIn>::kElems * kChunks))) spmm_cc_item<TIn, TOut, V, kChunks, kSlabs>(p, blockIdx.y, item);
}

// The same work enqueued behind a densifying kernel that usually has taken the call: returns at once unless the plan
// header says otherwise, and walks its items in strides, because a grid of one thread per item takes longer to start and
// return than the rest of a small call.  fp32: rows of fewer than `few` entries it computes even then.
template <typename TIn, typename TOut, int V, int kChunks = 1, bool kSlabs = false>
__global__ void __launch_bounds__(kCcThreads) spmm_cc_standby_kernel(const SpmmParams p, const int32_t *plan_hdr, int plan_checks, int few) {
    pdl_launch_dependents();
    pdl_wait();
    bool stands, some = false;
    if constexpr (sizeof(TIn) == 4) stands = plan_split_stands(plan_hdr, plan_checks, some);
    else stands = plan_dense_stands(plan_hdr, plan_checks);
    if (stands && !some) return;
    const int64_t per = (int64_t)p.m_vec * (p.N / (Chunk<TIn>::kElems * kChunks)), total = per * p.batch;
    for (int64_t i = (int64_t)blockIdx.x * kCcThreads + threadIdx.x; i < total; i += (int64_t)gridDim.x * kCcThreads)
        spmm_cc_item<TIn, TOut, V, kChunks, kSlabs>(p, (int)(i / per), i % per, sizeof(TIn) == 4 && stands ? few : 0);
}

// The same sums for products that leave most of the GPU idle, where the threads above wait for one trip of gathers after another (72 x 205 x 48,
// V = 8, 55 %: 41 us for 90 entries in a row, 8 here; what is left is one warp's latency, ~45 cycles an entry).  A warp takes a vector-row and 32 x kBytes bytes of its columns: the indices and values of 32 entries
// come with one load per lane, 32 ahead, and are passed round through shared memory; the rows of B of kAhead entries are on their way while those of
// the kAhead before are multiplied.  kBytes = 4 spreads a narrow product over four times the warps.  Entries in list order, as above: the same bits.
constexpr int kFewThreads = 128, kFewWarps = kFewThreads / 32;
template <typename T, int kBytes> struct Piece;   // kBytes of T as they lie in memory, widened on use
template <> struct Piece<float, 16> {
    static constexpr int kElems = 4;
    float4 raw;
    __device__ __forceinline__ void load(const float *p) { asm volatile("ld.global.nc.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(raw.x), "=f"(raw.y), "=f"(raw.z), "=f"(raw.w) : "l"(p)); }
    __device__ __forceinline__ void widen(float (&f)[4]) const { f[0] = raw.x; f[1] = raw.y; f[2] = raw.z; f[3] = raw.w; }
};
template <> struct Piece<float, 4> {
    static constexpr int kElems = 1;
    float raw;
    __device__ __forceinline__ void load(const float *p) { raw = __ldg(p); }
    __device__ __forceinline__ void widen(float (&f)[1]) const { f[0] = raw; }
};
template <> struct Piece<__half, 16> {
    static constexpr int kElems = 8;
    uint4 raw;
    __device__ __forceinline__ void load(const __half *p) { asm volatile("ld.global.nc.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(raw.x), "=r"(raw.y), "=r"(raw.z), "=r"(raw.w) : "l"(p)); }
    __device__ __forceinline__ void widen(float (&f)[8]) const {
        const __half2 *h = reinterpret_cast<const __half2 *>(&raw);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 t = __half22float2(h[i]);
            f[2 * i] = t.x;
            f[2 * i + 1] = t.y;
        }
    }
};
template <> struct Piece<__half, 4> {
    static constexpr int kElems = 2;
    __half2 raw;
    __device__ __forceinline__ void load(const __half *p) { raw = __ldg(reinterpret_cast<const __half2 *>(p)); }
    __device__ __forceinline__ void widen(float (&f)[2]) const {
        const float2 t = __half22float2(raw);
        f[0] = t.x;
        f[1] = t.y;
    }
};
template <typename TIn, typename TOut, int V, int kBytes>
__global__ void __launch_bounds__(kFewThreads) spmm_cc_few_kernel(const SpmmParams p, int pieces) {
    using B = Piece<TIn, kBytes>;
    constexpr int E = B::kElems, kAhead = kBytes == 4 ? 16 : 8;
    __shared__ __align__(16) float s_val[kFewWarps][2][32][V];
    __shared__ int s_col[kFewWarps][2][32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t item = (int64_t)blockIdx.x * kFewWarps + warp;
    if (item >= (int64_t)p.m_vec * pieces) return;
    const int row = __ldg(p.row_indices + (int)(item / pieces)), b = blockIdx.y;
    const int n = ((int)(item % pieces) * 32 + lane) * E;
    const bool stored = n < p.N;   // lanes past the last column take part with the columns of the first lane
    const TIn *values = static_cast<const TIn *>(p.values) + (int64_t)b * p.stride_values;
    const TIn *rhs = static_cast<const TIn *>(p.rhs) + (int64_t)b * p.stride_rhs + (stored ? n : (int)(item % pieces) * 32 * E);

    int j = __ldg(p.row_offsets + row);
    const int end = __ldg(p.row_offsets + row + 1);
    int col = 0;
    float val[V];
    auto fetch = [&](int at) {   // the lane's entry of the 32 from `at`; past the end the last one again, whose row of B is read and not used
        const int from = min(at + lane, end - 1);
        col = __ldg(p.col_indices + from);
        VecLoad<TIn, V>::load(values + (int64_t)from * V, val);
    };
    auto stage = [&](int place) {
        s_col[warp][place][lane] = col;
#pragma unroll
        for (int v = 0; v < V; ++v) s_val[warp][place][lane][v] = val[v];
    };
    float acc[V][E];
#pragma unroll
    for (int v = 0; v < V; ++v)
#pragma unroll
        for (int e = 0; e < E; ++e) acc[v][e] = 0.f;
    B x[2][kAhead];
    // kAhead entries from the u0-th of the 32 in `place`; unconditional, a load under a condition is waited for at once
    auto request = [&](B (&to)[kAhead], int place, int u0) {
#pragma unroll
        for (int u = 0; u < kAhead; ++u) to[u].load(rhs + (int64_t)s_col[warp][place][u0 + u] * p.N);
    };
    auto multiply = [&](const B (&from)[kAhead], int place, int u0, int count) {
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            if (u0 + u < count) {
                float a[V], f[E];
                from[u].widen(f);
#pragma unroll
                for (int v = 0; v < V; ++v) a[v] = s_val[warp][place][u0 + u][v];
#pragma unroll
                for (int v = 0; v < V; ++v)
#pragma unroll
                    for (int e = 0; e < E; ++e) acc[v][e] = fmaf(a[v], f[e], acc[v][e]);
            }
        }
    };
    if (j < end) {
        fetch(j);
        stage(0);
        __syncwarp();
        fetch(j + 32);
        request(x[0], 0, 0);
    }
    for (int place = 0; j < end; j += 32, place ^= 1) {
        const int count = end - j;   // of the entries from here on
        stage(place ^ 1);
        __syncwarp();
        fetch(j + 64);
#pragma unroll
        for (int u0 = 0; u0 < 32; u0 += kAhead) {
            const int i = u0 / kAhead & 1;
            if (u0 + kAhead < 32) request(x[i ^ 1], place, u0 + kAhead);
            else request(x[i ^ 1], place ^ 1, 0);
            multiply(x[i], place, u0, count);
        }
        __syncwarp();
    }
    if (!stored) return;
    TOut *out = static_cast<TOut *>(p.out) + (int64_t)b * p.stride_out + n;
#pragma unroll
    for (int v = 0; v < V; ++v) {
        TOut *to = out + ((int64_t)row * V + v) * p.N;
        if constexpr (E >= 4) {
            store_chunk(to, acc[v]);
        } else {
#pragma unroll
            for (int e = 0; e < E; ++e) store_scalar(to + e, acc[v][e]);
        }
    }
}

// ---- SDDMM --------------------------------------------------------------------------------------------------
// Eight lanes share one mask entry j: lane g takes the 16-byte chunks g, g+8, ... of the contraction, keeps V
// partial sums (one per real row of the vector), and the eight partials are folded with three xor-shuffles.
// The vector-row of entry j is found by bisection in row_offsets, so the grid is exactly nnz_vec entries and
// no thread block is launched for empty parts of the mask.
template <typename TIn, typename TOut, int V>
__global__ void __launch_bounds__(kCcThreads) sddmm_cc_kernel(const SddmmParams p) {
    constexpr int E = Chunk<TIn>::kElems;
    constexpr int L = 8;
    const int g = threadIdx.x & (L - 1);
    const int64_t entry = ((int64_t)blockIdx.x * kCcThreads + threadIdx.x) / L;
    const bool valid = entry < p.nnz_vec;
    const int j = valid ? (int)entry : 0;
    const int b = blockIdx.y;

    int lo = 0, hi = p.m_vec;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(p.row_offsets + mid) <= j) lo = mid; else hi = mid;
    }
    const int i = lo;
    const int col = __ldg(p.col_indices + j);

    const TIn *lhs = static_cast<const TIn *>(p.lhs) + (int64_t)b * p.stride_lhs + (int64_t)i * V * p.k;
    const TIn *rhs = static_cast<const TIn *>(p.rhs) + (int64_t)b * p.stride_rhs + (int64_t)col * p.k;
    TOut *out = static_cast<TOut *>(p.out) + (int64_t)b * p.stride_out + (int64_t)j * V;

    float acc[V];
#pragma unroll
    for (int v = 0; v < V; ++v) acc[v] = 0.f;

    const int chunks = p.k / E;
    for (int c = g; c < chunks; c += L) {
        Chunk<TIn> r;
        r.load(rhs + c * E);
#pragma unroll
        for (int v = 0; v < V; ++v) {
            Chunk<TIn> l;
            l.load(lhs + (int64_t)v * p.k + c * E);
#pragma unroll
            for (int e = 0; e < E; ++e) acc[v] = fmaf(l.f[e], r.f[e], acc[v]);
        }
    }
#pragma unroll
    for (int off = L / 2; off > 0; off >>= 1)
#pragma unroll
        for (int v = 0; v < V; ++v) acc[v] += __shfl_xor_sync(0xffffffffu, acc[v], off);

    if (valid && g == 0) {
        if constexpr (V >= 4) {
            store_chunk(out, acc);
        } else {
#pragma unroll
            for (int v = 0; v < V; ++v) store_scalar(out + v, acc[v]);
        }
    }
}

// The same product with the V rows of lhs kept in registers: L lanes (8, 16 or 32) share one VECTOR-ROW, lane g holds
// the 16-byte chunk g of each of its V lhs rows (contraction lengths of up to L chunks), and the group walks the
// vector-row's mask entries: per entry one 16-byte load of the rhs row per lane, V x E FMAs and a folding reduction
// over the L lanes (each step halves the values a lane still carries: 9 shuffles for V = 8, L = 32, where a plain
// butterfly needs 40), after which lane g holds the sum of real row g >> log2(L / V).  Against the kernel above,
// which re-reads the V lhs rows for every entry, this moves a ninth of the bytes through L1.
//
// Entries do not depend on one another, so where the vector-rows are few `pieces` groups share one (185 x 714, k = 72, V = 8, 77 %, fp32 results: 24 CTAs,
// each with chains of 170 to 400 entries, 48 us; fp32 results of 158 x 4311, k = 160, V = 4, 94 %: 60 us with one group each,
// 10 with shared ones, 1570 x 3412, k = 48, V = 1, 91 %: 33 and 13).
template <typename TIn, typename TOut, int V, int L>
__global__ void __launch_bounds__(kCcThreads) sddmm_cc_row_kernel(const SddmmParams p, int pieces) {
    constexpr int E = Chunk<TIn>::kElems;
    static_assert(L >= 8 && L <= 32 && V <= L, "group size");
    const int g = threadIdx.x & (L - 1);
    const int64_t group = ((int64_t)blockIdx.x * kCcThreads + threadIdx.x) / L;
    const bool live = group < (int64_t)p.m_vec * pieces;
    const int row = live ? __ldg(p.row_indices + (int)(group / pieces)) : 0, piece = (int)(group % pieces);
    const int b = blockIdx.y;
    const int chunks = p.k / E;
    const bool mine = g < chunks;   // lanes past the contraction length contribute zeros

    const TIn *lhs = static_cast<const TIn *>(p.lhs) + (int64_t)b * p.stride_lhs + (int64_t)row * V * p.k + g * E;
    const TIn *rhs = static_cast<const TIn *>(p.rhs) + (int64_t)b * p.stride_rhs + g * E;
    TOut *out = static_cast<TOut *>(p.out) + (int64_t)b * p.stride_out;

    float l[V][E];
#pragma unroll
    for (int v = 0; v < V; ++v) {
        if (live && mine) {
            Chunk<TIn> c;
            c.load(lhs + (int64_t)v * p.k);
#pragma unroll
            for (int e = 0; e < E; ++e) l[v][e] = c.f[e];
        } else {
#pragma unroll
            for (int e = 0; e < E; ++e) l[v][e] = 0.f;
        }
    }
    int j = live ? min(max(__ldg(p.row_offsets + row), 0), p.nnz_vec) : 0;
    int end = live ? min(max(__ldg(p.row_offsets + row + 1), j), p.nnz_vec) : 0;
    const int share = (end - j + pieces - 1) / pieces;
    j = min(j + piece * share, end);
    end = min(j + share, end);
    // the groups of a warp walk rows of different lengths: the loop runs to the longest, shorter rows idle.  Four
    // entries per trip, so that four gathers of rhs are in flight; the column indices of a trip are loaded one trip ahead.
    constexpr int U = 4;
    int trips = (end - j + U - 1) / U;
#pragma unroll
    for (int d = 16; d >= L; d >>= 1) trips = max(trips, __shfl_xor_sync(0xffffffffu, trips, d));
    int col[U];
#pragma unroll
    for (int u = 0; u < U; ++u) col[u] = j + u < end ? __ldg(p.col_indices + j + u) : 0;
    for (int it = 0; it < trips; ++it, j += U) {
        Chunk<TIn> r[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (j + u < end && mine) {
                r[u].load(rhs + (int64_t)col[u] * p.k);
            } else {
#pragma unroll
                for (int e = 0; e < E; ++e) r[u].f[e] = 0.f;
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) col[u] = j + U + u < end ? __ldg(p.col_indices + j + U + u) : 0;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            float acc[V];
#pragma unroll
            for (int v = 0; v < V; ++v) {
                acc[v] = 0.f;
#pragma unroll
                for (int e = 0; e < E; ++e) acc[v] = fmaf(l[v][e], r[u].f[e], acc[v]);
            }
            // folding reduction over the L lanes of the group
            int n = V;
#pragma unroll
            for (int d = L / 2; d >= 1; d >>= 1) {
                if (n > 1) {
                    const bool upper = (g & d) != 0;
#pragma unroll
                    for (int i = 0; i < V / 2; ++i) {
                        if (i < n / 2) {
                            const float send = upper ? acc[i] : acc[i + n / 2];
                            const float keep = upper ? acc[i + n / 2] : acc[i];
                            acc[i] = keep + __shfl_xor_sync(0xffffffffu, send, d);
                        }
                    }
                    n >>= 1;
                } else {
                    acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], d);
                }
            }
            // lane g now holds the sum of real row g / (L / V) of the vector-row; the first lane of each run stores it
            if (j + u < end && (g & (L / V - 1)) == 0) store_scalar(out + (int64_t)(j + u) * V + g / (L / V), acc[0]);
        }
    }
}

// ---- masked row softmax -----------------------------------------------------------------------------------
// One warp per vector-row: lanes stride over the row's entries, each entry carrying the V real rows, so the V
// softmaxes of a vector-row run side by side on contiguous vector loads.  fp32 arithmetic.  Rows of up to
// 32 * kCache entries are read from memory ONCE: each lane keeps its entries' raw words in registers across the
// max, sum and normalise steps (2 passes over HBM instead of 4).  Longer rows take three passes over a row that
// stays in L1/L2.  probs may alias scores.
template <typename T, int V> struct EntryWords {  // one entry = V values of T = kWords 32-bit words
    static constexpr int kBytes = V * (int)sizeof(T);
    static constexpr int kWords = kBytes >= 4 ? kBytes / 4 : 1;
    static constexpr bool kVector = kBytes >= 4;
    __device__ __forceinline__ static void load(const T *p, uint32_t (&w)[kWords]) {
        if constexpr (kBytes == 4) {
            w[0] = __ldg(reinterpret_cast<const uint32_t *>(p));
        } else if constexpr (kBytes == 8) {
            const uint2 v = __ldg(reinterpret_cast<const uint2 *>(p));
            w[0] = v.x; w[1] = v.y;
        } else {
#pragma unroll
            for (int q = 0; q < kBytes / 16; ++q) {
                const uint4 v = __ldg(reinterpret_cast<const uint4 *>(p) + q);
                w[4 * q] = v.x; w[4 * q + 1] = v.y; w[4 * q + 2] = v.z; w[4 * q + 3] = v.w;
            }
        }
    }
    __device__ __forceinline__ static void unpack(const uint32_t (&w)[kWords], float (&f)[V]) {
        if constexpr (sizeof(T) == 4) {
#pragma unroll
            for (int v = 0; v < V; ++v) f[v] = __uint_as_float(w[v]);
        } else {
#pragma unroll
            for (int q = 0; q < V / 2; ++q) {
                const float2 t = __half22float2(*reinterpret_cast<const __half2 *>(&w[q]));
                f[2 * q] = t.x; f[2 * q + 1] = t.y;
            }
        }
    }
    __device__ __forceinline__ static void pack(const float (&f)[V], uint32_t (&w)[kWords]) {
        if constexpr (sizeof(T) == 4) {
#pragma unroll
            for (int v = 0; v < V; ++v) w[v] = __float_as_uint(f[v]);
        } else {
#pragma unroll
            for (int q = 0; q < V / 2; ++q) {
                const __half2 h = __floats2half2_rn(f[2 * q], f[2 * q + 1]);
                w[q] = *reinterpret_cast<const uint32_t *>(&h);
            }
        }
    }
    __device__ __forceinline__ static void store(T *p, const float (&f)[V]) {
        uint32_t w[kWords];
        pack(f, w);
        store_words(p, w);
    }
    __device__ __forceinline__ static void store_words(T *p, const uint32_t (&w)[kWords]) {
        if constexpr (kBytes == 4) {
            *reinterpret_cast<uint32_t *>(p) = w[0];
        } else if constexpr (kBytes == 8) {
            *reinterpret_cast<uint2 *>(p) = make_uint2(w[0], w[1]);
        } else {
#pragma unroll
            for (int q = 0; q < kBytes / 16; ++q)
                reinterpret_cast<uint4 *>(p)[q] = make_uint4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
        }
    }
};

template <typename T, int V>
__global__ void __launch_bounds__(kCcThreads) softmax_cvse_kernel(const SoftmaxParams p) {
    using EW = EntryWords<T, V>;
    constexpr int kCache = EW::kVector ? (64 / EW::kWords > 16 ? 16 : 64 / EW::kWords) : 0;   // entries per lane
    const int warp = (blockIdx.x * kCcThreads + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (warp >= p.m_vec) return;
    const int b = blockIdx.y;
    const T *s = static_cast<const T *>(p.scores) + (int64_t)b * p.stride;
    T *o = static_cast<T *>(p.probs) + (int64_t)b * p.stride;
    const int beg = __ldg(p.row_offsets + warp), end = __ldg(p.row_offsets + warp + 1);
    if (beg == end) return;

    float mx[V], sum[V];
#pragma unroll
    for (int v = 0; v < V; ++v) { mx[v] = -INFINITY; sum[v] = 0.f; }

    if constexpr (kCache > 0) {
        if (end - beg <= 32 * kCache) {
            uint32_t cache[kCache][EW::kWords];
            // fp16 scores with a non-negative scale: the row maxima are taken on the packed halves (the maximum
            // commutes with the scaling) and only the V results are widened; conversions are what this kernel
            // spends its time on
            constexpr bool kPacked = sizeof(T) == 2 && V >= 2;
            const bool packed_max = kPacked && p.scale >= 0.0f;
            if (packed_max) {
                uint32_t m2[EW::kWords];
                const __half2 lowest = __floats2half2_rn(-INFINITY, -INFINITY);
#pragma unroll
                for (int q = 0; q < EW::kWords; ++q) m2[q] = *reinterpret_cast<const uint32_t *>(&lowest);
#pragma unroll
                for (int c = 0; c < kCache; ++c) {
                    const int j = beg + lane + 32 * c;
                    if (j < end) {
                        EW::load(s + (int64_t)j * V, cache[c]);
#pragma unroll
                        for (int q = 0; q < EW::kWords; ++q) {
                            const __half2 h = __hmax2(*reinterpret_cast<const __half2 *>(&m2[q]), *reinterpret_cast<const __half2 *>(&cache[c][q]));
                            m2[q] = *reinterpret_cast<const uint32_t *>(&h);
                        }
                    }
                }
#pragma unroll
                for (int off = 16; off > 0; off >>= 1)
#pragma unroll
                    for (int q = 0; q < EW::kWords; ++q) {
                        const uint32_t other = __shfl_xor_sync(0xffffffffu, m2[q], off);
                        const __half2 h = __hmax2(*reinterpret_cast<const __half2 *>(&m2[q]), *reinterpret_cast<const __half2 *>(&other));
                        m2[q] = *reinterpret_cast<const uint32_t *>(&h);
                    }
                if constexpr (kPacked) {
                    float f[V];
                    EW::unpack(m2, f);
#pragma unroll
                    for (int v = 0; v < V; ++v) mx[v] = p.scale * f[v];
                }
            } else {
#pragma unroll
                for (int c = 0; c < kCache; ++c) {
                    const int j = beg + lane + 32 * c;
                    if (j < end) {
                        EW::load(s + (int64_t)j * V, cache[c]);
                        float f[V];
                        EW::unpack(cache[c], f);
#pragma unroll
                        for (int v = 0; v < V; ++v) mx[v] = fmaxf(mx[v], p.scale * f[v]);
                    }
                }
#pragma unroll
                for (int off = 16; off > 0; off >>= 1)
#pragma unroll
                    for (int v = 0; v < V; ++v) mx[v] = fmaxf(mx[v], __shfl_xor_sync(0xffffffffu, mx[v], off));
            }
            // exponentials are computed once (exp2 of a pre-scaled argument), kept in the cache in the element
            // type, and scaled by 1 / sum on the way out
            const float sl2 = p.scale * 1.4426950408889634f;
            float ml2[V];
#pragma unroll
            for (int v = 0; v < V; ++v) ml2[v] = mx[v] * 1.4426950408889634f;
#pragma unroll
            for (int c = 0; c < kCache; ++c) {
                if (beg + lane + 32 * c < end) {
                    float f[V];
                    EW::unpack(cache[c], f);
#pragma unroll
                    for (int v = 0; v < V; ++v) {
                        f[v] = exp2f(fmaf(f[v], sl2, -ml2[v]));
                        sum[v] += f[v];
                    }
                    EW::pack(f, cache[c]);
                }
            }
#pragma unroll
            for (int off = 16; off > 0; off >>= 1)
#pragma unroll
                for (int v = 0; v < V; ++v) sum[v] += __shfl_xor_sync(0xffffffffu, sum[v], off);
            float inv[V];
#pragma unroll
            for (int v = 0; v < V; ++v) inv[v] = 1.0f / sum[v];
            if constexpr (kPacked) {
                // the cached exponentials are already fp16: scale them there (two more roundings of 2^-11,
                // well inside the stated tolerance) instead of widening and narrowing every value again
                uint32_t inv2[EW::kWords];
                EW::pack(inv, inv2);
#pragma unroll
                for (int c = 0; c < kCache; ++c) {
                    const int j = beg + lane + 32 * c;
                    if (j < end) {
#pragma unroll
                        for (int q = 0; q < EW::kWords; ++q) {
                            const __half2 h = __hmul2(*reinterpret_cast<const __half2 *>(&cache[c][q]), *reinterpret_cast<const __half2 *>(&inv2[q]));
                            cache[c][q] = *reinterpret_cast<const uint32_t *>(&h);
                        }
                        EW::store_words(o + (int64_t)j * V, cache[c]);
                    }
                }
            } else {
#pragma unroll
                for (int c = 0; c < kCache; ++c) {
                    const int j = beg + lane + 32 * c;
                    if (j < end) {
                        float f[V];
                        EW::unpack(cache[c], f);
#pragma unroll
                        for (int v = 0; v < V; ++v) f[v] *= inv[v];
                        EW::store(o + (int64_t)j * V, f);
                    }
                }
            }
            return;
        }
    }

    for (int j = beg + lane; j < end; j += 32) {
#pragma unroll
        for (int v = 0; v < V; ++v) mx[v] = fmaxf(mx[v], p.scale * load_scalar(s + (int64_t)j * V + v));
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
#pragma unroll
        for (int v = 0; v < V; ++v) mx[v] = fmaxf(mx[v], __shfl_xor_sync(0xffffffffu, mx[v], off));
    for (int j = beg + lane; j < end; j += 32) {
#pragma unroll
        for (int v = 0; v < V; ++v) sum[v] += expf(p.scale * load_scalar(s + (int64_t)j * V + v) - mx[v]);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
#pragma unroll
        for (int v = 0; v < V; ++v) sum[v] += __shfl_xor_sync(0xffffffffu, sum[v], off);
    for (int j = beg + lane; j < end; j += 32) {
#pragma unroll
        for (int v = 0; v < V; ++v) {
            const float x = expf(p.scale * load_scalar(s + (int64_t)j * V + v) - mx[v]) / sum[v];
            store_scalar(o + (int64_t)j * V + v, x);
        }
    }
}

// Backward of the masked row softmax: for every real row r = i*V+v, over the entries j of vector-row i,
//   grad_scores[j*V+v] = scale * probs[j*V+v] * (grad_probs[j*V+v] - sum_j probs[j*V+v] * grad_probs[j*V+v]).
// (The forward kernel applies `scale` to the scores inside, so the gradient with respect to the scores it was
// given carries the factor.)  One warp per vector-row; rows that fit the lanes' registers are read once, longer ones
// twice (the second pass comes from L1/L2); fp32 sums; grad_scores may be grad_probs.  The reference has no softmax (README.md:76 points to an external
// repository for the attention layer).
struct SoftmaxBackwardParams {
    int m_vec;
    const int32_t *row_offsets;
    const void *probs;
    const void *grad_probs;
    void *grad_scores;
    int64_t stride;  // in elements, between batch entries
    float scale;
};

template <typename T, int V>
__global__ void __launch_bounds__(kCcThreads) softmax_cvse_backward_kernel(const SoftmaxBackwardParams p) {
    using EW = EntryWords<T, V>;
    const int warp = (blockIdx.x * kCcThreads + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (warp >= p.m_vec) return;
    const int64_t at = (int64_t)blockIdx.y * p.stride;
    const T *pr = static_cast<const T *>(p.probs) + at;
    const T *gp = static_cast<const T *>(p.grad_probs) + at;
    T *gs = static_cast<T *>(p.grad_scores) + at;
    const int beg = __ldg(p.row_offsets + warp), end = __ldg(p.row_offsets + warp + 1);
    float dot[V];
#pragma unroll
    for (int v = 0; v < V; ++v) dot[v] = 0.f;
    // Rows of up to 32 * kCache entries (config 5: 410) are read once: every lane keeps its entries of both arrays
    // in registers between the two passes, with all of its loads in flight together.
    constexpr int kCache = EW::kVector ? (52 / EW::kWords > 16 ? 16 : 52 / EW::kWords) : 0;
    if constexpr (kCache > 0) {
        if (end - beg <= 32 * kCache) {
            uint32_t cp[kCache][EW::kWords], cg[kCache][EW::kWords];
#pragma unroll
            for (int c = 0; c < kCache; ++c) {
                const int j = beg + lane + 32 * c;
                if (j < end) {
                    EW::load(pr + (int64_t)j * V, cp[c]);
                    EW::load(gp + (int64_t)j * V, cg[c]);
                }
            }
#pragma unroll
            for (int c = 0; c < kCache; ++c) {
                if (beg + lane + 32 * c < end) {
                    float a[V], g[V];
                    EW::unpack(cp[c], a);
                    EW::unpack(cg[c], g);
#pragma unroll
                    for (int v = 0; v < V; ++v) dot[v] = fmaf(a[v], g[v], dot[v]);
                }
            }
#pragma unroll
            for (int off = 16; off > 0; off >>= 1)
#pragma unroll
                for (int v = 0; v < V; ++v) dot[v] += __shfl_xor_sync(0xffffffffu, dot[v], off);
#pragma unroll
            for (int c = 0; c < kCache; ++c) {
                const int j = beg + lane + 32 * c;
                if (j < end) {
                    float a[V], g[V], o[V];
                    EW::unpack(cp[c], a);
                    EW::unpack(cg[c], g);
#pragma unroll
                    for (int v = 0; v < V; ++v) o[v] = p.scale * a[v] * (g[v] - dot[v]);
                    EW::store(gs + (int64_t)j * V, o);
                }
            }
            return;
        }
    }
    for (int j = beg + lane; j < end; j += 32) {
        float a[V], g[V];
        if constexpr (EW::kVector) {
            uint32_t wa[EW::kWords], wg[EW::kWords];
            EW::load(pr + (int64_t)j * V, wa);
            EW::load(gp + (int64_t)j * V, wg);
            EW::unpack(wa, a);
            EW::unpack(wg, g);
        } else {
            a[0] = (float)pr[j];
            g[0] = (float)gp[j];
        }
#pragma unroll
        for (int v = 0; v < V; ++v) dot[v] = fmaf(a[v], g[v], dot[v]);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
#pragma unroll
        for (int v = 0; v < V; ++v) dot[v] += __shfl_xor_sync(0xffffffffu, dot[v], off);
    __syncwarp();   // in-place use: every lane has read the row before any lane overwrites its part
    for (int j = beg + lane; j < end; j += 32) {
        float a[V], g[V], o[V];
        if constexpr (EW::kVector) {
            uint32_t wa[EW::kWords], wg[EW::kWords];
            EW::load(pr + (int64_t)j * V, wa);
            EW::load(gp + (int64_t)j * V, wg);
            EW::unpack(wa, a);
            EW::unpack(wg, g);
        } else {
            a[0] = (float)pr[j];
            g[0] = (float)gp[j];
        }
#pragma unroll
        for (int v = 0; v < V; ++v) o[v] = p.scale * a[v] * (g[v] - dot[v]);
        if constexpr (EW::kVector) {
            EW::store(gs + (int64_t)j * V, o);
        } else {
            gs[j] = (T)o[0];
        }
    }
}

// fp32 FMA throughput probe: every thread runs 8 independent chains of `iters` fused multiply-adds on registers;
// the result is stored so that nothing is optimised away.  2 * 8 * iters flops per thread, no memory traffic.
// The denominator for kernels that are bound by fp32 FMA issue (the fp32 CUDA-core SpMM).
__global__ void __launch_bounds__(256) fp32_fma_probe_kernel(int iters, float seed, float *sink) {
    float a[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) a[j] = seed + (float)(threadIdx.x + j);
    const float m = 1.0f - seed * 1e-7f, c = seed * 1e-7f;
    for (int i = 0; i < iters; ++i) {
#pragma unroll
        for (int j = 0; j < 8; ++j) a[j] = fmaf(a[j], m, c);
    }
    float s = 0.0f;
#pragma unroll
    for (int j = 0; j < 8; ++j) s += a[j];
    if (s == 12345.678f && sink) sink[0] = s;   // keeps the chains alive; `sink` may be null
}

}  // namespace vs
