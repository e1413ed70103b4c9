// Tensor-core SpMM for small problems in ONE kernel: the `wmmaSpmm` entry point of the reference
// (src/wmma_spmm.cu:388-409) where a call is too short for a plan.  Same formulation as spmm_dense.cuh — multiply
// zero-filled tiles of A — without the plan kernel in front of it and (mostly) without a stand-by kernel behind it:
//
//     C[128 rows x 64 cols] = A_dense[128 x K] * B[K x 64]          one CTA per tile, 128 columns of A at a time
//
// What bounds it.  One product of 2048 x 512 x 256 is a microsecond of work; the plan, the multiplying kernel and the
// gather kernel that returns at once took 15.4 us on the GPU, nearly all of it launches and dependent loads; this kernel
// takes 6.9 us (64 x 64 x 256: 11.2 -> 3.5).  Its chain is row offsets -> columns and values -> scatter -> MMA -> store, once,
// and after the first chunk ~0.55 us per chunk: filling it (an MMA of 64 columns takes as long as one of 128, ~61 cycles).  128 x 64 tiles and two CTAs per SM because
// at these sizes the number of CTAs is what is short; a larger problem re-reads A once per 64 columns and goes to the
// pair kernel instead.
//
// How a CTA finds its entries without a plan.  Each of eight fill warps owns 16 rows of the tile (16 / V vector-rows)
// and walks their entries in windows, one being scattered and the next one on its way: the entries below the chunk's last
// column are scattered, a window that is used up makes room for the next.  That needs columns that ascend strictly
// within a vector-row, which is checked on every entry.  A row that does not (unsorted, or a column named twice), and a row with
// a non-finite sum (0 x Inf of the densified tile, see spmm_dense.cuh), is computed again by the same CTA from the
// CVSE arrays on CUDA cores, entry by entry as the reference does.
//
// The K order of the MMAs is the one of the other densifying kernels (16 columns of A at a time, ascending), so that a product whose
// columns ascend has the same bits whichever of them multiplies it, where a tile is not shared (kSplit); a row computed entry by entry has those of spmm_cc_kernel.
//
// kSplit: a cluster of up to eight CTAs shares the tile, each with a part of A's columns, where few tiles have many chunks to walk (80 rows x 4023 columns x
// 320, V = 8, 52 %: 32 chunks on 5 CTAs, 37 us; on 40 CTAs 13.8, a share of four chunks, its search and the sums of the others).  Each takes a run of chunks.  A group of lanes finds the first entry of its vector-row in each part by a search
// that assumes ascending columns; the parts cover the row whatever its order.  Columns which do not ascend are found out all the same: a lane compares every
// entry that it looks at with the one before it, and it either looks at all of its entries or stops at a column past the end of its part, where an
// ascending row has none.  The parts' sums meet in shared memory, in order, a share of the rows in each CTA.
//
// Roles (320 threads): warps 0-7 fill, then epilogue (TMEM lanes 32 (w % 4) .., columns 32 (w / 4) ..); warp 8 the MMA-issuing
// thread; warp 9 the thread that loads B by TMA.  Rings: 2 chunks of A (32 KiB each), 3 of B (16 KiB each).  Every
// wait is bounded.
#pragma once
#include <cuda.h>

#include <climits>

#include "common.cuh"
#include "spmm_dense.cuh"
#include "tc_ptx.cuh"

namespace vs {
namespace directspmm {

using densespmm::scatter_vector;
using densespmm::ValueVec;
using densespmm::wait_or_abort;

constexpr int kTileM = 128;
constexpr int kTileN = 64;
constexpr int kChunkK = 128;                              // columns of A per chunk: two 64-column MMA operands
constexpr int kFillWarps = 8;
constexpr int kWarpRows = kTileM / kFillWarps;            // 16
constexpr int kMmaWarp = kFillWarps;
constexpr int kLoadWarp = kMmaWarp + 1;
constexpr int kThreads = (kLoadWarp + 1) * 32;            // 320
constexpr int kABuffers = 2, kBBuffers = 3;
constexpr int kABlockBytes = kTileM * 64 * 2;             // 16 KiB: 128 rows x 64 columns
constexpr int kAChunkBytes = 2 * kABlockBytes;
constexpr int kBBlockBytes = 64 * kTileN * 2;             // 8 KiB: 64 rows of B x 64 columns
constexpr int kBChunkBytes = 2 * kBBlockBytes;
constexpr int kTmemCols = 64;
constexpr int kPartPitch = kTileN + 4;                   // of a part's sums, fp32, in the place of the chunks of A
constexpr int kMaxSplit = 8;                              // CTAs that share a tile
static_assert(kTileM * kPartPitch * 4 <= kABuffers * kAChunkBytes && kTileM / kMaxSplit % 8 == 0, "a part's sums; whole vector-rows in a share");

struct Smem {   // offsets from the 1024-byte aligned base
    static constexpr int kA = 0;
    static constexpr int kB = kA + kABuffers * kAChunkBytes;
    // one pair of barriers per chunk in flight (chunk c: pair c % kBBuffers): `full` collects the fill warps, the loader
    // and the bytes of B, `done` the commit of the MMA-issuing thread, which pays ~100 cycles for each commit and wait
    static constexpr int kBarFull = kB + kBBuffers * kBChunkBytes;
    static constexpr int kBarDone = kBarFull + kBBuffers * 8;
    static constexpr int kTmemHolder = kBarDone + kBBuffers * 8;
    static constexpr int kAbort = kTmemHolder + 8;
    static constexpr int kRedo = kAbort + 8;              // vector-rows of the tile to be computed entry by entry, a bit each
    static constexpr int kTotal = kRedo + 2 * (kTileM / 8);
};
constexpr int kSmemBytes = Smem::kTotal;   // the dynamic segment is 1024-byte aligned (nothing static lies ahead of it)
static_assert(2 * (kSmemBytes + 1024) <= 228 * 1024, "two CTAs per SM");

// Vector-rows of one tile (a bit each in `which`) from the CVSE arrays on CUDA cores, fp32 sums in list order (the sums of
// spmm_cc_kernel, bit for bit).  kLanes lanes share a vector-row, each with E columns of the tile.  They fetch the indices and
// values of kLanes entries at a time, one each and a batch ahead, and pass them round; the rows of B of kAhead entries are in
// flight together.  What bounds it: the latency of a gather, on the few SMs that the call's tiles occupy.  512 x 1024 x 256, V = 2, 90 %
// sparse, every row with a column named twice: one entry at a time 84 us beside the 14 of the product, eight in flight 30, passed round 27.
template <typename TOut, int V>
__device__ __noinline__ void rows_by_entries(const SpmmParams &p, int b, int row0, int rows, int n0, const uint32_t *which) {
    constexpr int E = V >= 4 ? 4 : 8, kWords = E / 2;
    constexpr int kLanes = kTileN / E, kWarpVecRows = 32 / kLanes;
    constexpr int kAhead = V >= 4 ? 16 : 8;
    constexpr int kValueWords = V >= 2 ? V / 2 : 1;
    const __half *values = static_cast<const __half *>(p.values) + (int64_t)b * p.stride_values;
    TOut *out = static_cast<TOut *>(p.out) + (int64_t)b * p.stride_out;
    const int lane = threadIdx.x & 31, l = lane % kLanes;
    const int n = n0 + E * l;
    const bool stored = n < p.N;   // lanes past the last column take part with the columns of the first lane
    const __half *rhs = static_cast<const __half *>(p.rhs) + (int64_t)b * p.stride_rhs + (stored ? n : n0);
    for (int base = (threadIdx.x >> 5) * kWarpVecRows; base < rows; base += kThreads / 32 * kWarpVecRows) {
        const int i = base + lane / kLanes, r = row0 + i;
        const bool live = i < rows && (which[i >> 5] >> (i & 31) & 1u);
        if (!__any_sync(0xffffffffu, live)) continue;
        int j = live ? __ldg(p.row_offsets + r) : 0;
        const int end = live ? __ldg(p.row_offsets + r + 1) : 0;
        float acc[V][E];
#pragma unroll
        for (int v = 0; v < V; ++v)
#pragma unroll
            for (int e = 0; e < E; ++e) acc[v][e] = 0.f;
        int col;
        uint32_t val[kValueWords];
        auto look_up = [&](int at) {   // a column outside the matrix counts as no entry: column -1
            col = at < end ? __ldg(p.col_indices + at) : -1;
            if ((unsigned)col >= (unsigned)p.K) col = -1;
            ValueVec<V> a;
            a.raw = typename ValueVec<V>::Raw{};
            if (col >= 0) a.load(values + (int64_t)at * V);
            if constexpr (V == 8) {
                val[0] = a.raw.x; val[1] = a.raw.y; val[2] = a.raw.z; val[3] = a.raw.w;
            } else if constexpr (V == 4) {
                val[0] = a.raw.x; val[1] = a.raw.y;
            } else {
                val[0] = a.raw;
            }
        };
        look_up(j + l);
        while (__any_sync(0xffffffffu, j < end)) {
            const int batch_col = col;
            uint32_t batch_val[kValueWords];
#pragma unroll
            for (int w = 0; w < kValueWords; ++w) batch_val[w] = val[w];
            j += kLanes;
            look_up(j + l);
#pragma unroll
            for (int u0 = 0; u0 < kLanes; u0 += kAhead) {
                uint32_t x[kAhead][kWords];
                int c[kAhead];
#pragma unroll
                for (int u = 0; u < kAhead; ++u) {   // no entry: a row of zeros, whose values are zeros too
                    c[u] = __shfl_sync(0xffffffffu, batch_col, u0 + u, kLanes);
                    const __half *from = rhs + (int64_t)max(c[u], 0) * p.N;
                    if constexpr (E == 8) {
                        const uint4 q = __ldg(reinterpret_cast<const uint4 *>(from));
                        x[u][0] = q.x; x[u][1] = q.y; x[u][2] = q.z; x[u][3] = q.w;
                    } else {
                        const uint2 q = __ldg(reinterpret_cast<const uint2 *>(from));
                        x[u][0] = q.x; x[u][1] = q.y;
                    }
                }
#pragma unroll
                for (int u = 0; u < kAhead; ++u) {
                    uint32_t av[kValueWords];
                    float value[V];
#pragma unroll
                    for (int w = 0; w < kValueWords; ++w) {
                        av[w] = __shfl_sync(0xffffffffu, batch_val[w], u0 + u, kLanes);
                        const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&av[w]));
                        value[2 * w] = f.x;
                        if constexpr (V >= 2) value[2 * w + 1] = f.y;
                    }
#pragma unroll
                    for (int w = 0; w < kWords; ++w) {
                        if (c[u] < 0) x[u][w] = 0;
                        const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&x[u][w]));
#pragma unroll
                        for (int v = 0; v < V; ++v) {
                            acc[v][2 * w] = fmaf(value[v], f.x, acc[v][2 * w]);
                            acc[v][2 * w + 1] = fmaf(value[v], f.y, acc[v][2 * w + 1]);
                        }
                    }
                }
            }
        }
        if (live && stored)
#pragma unroll
            for (int v = 0; v < V; ++v) store_chunk(out + ((int64_t)r * V + v) * p.N + n, acc[v]);
    }
}

// map_b: the dense operand as {N, K, batch}, box {64, 64, 1}, 128-byte swizzle, zero fill outside.
// verdict: null when the densified product is the cheaper one whatever the number of nonzeros; otherwise the
// kernel compares the costs the plan kernel compares (dense_cost for its `stages`, gather_per_row, gather_per_entry), writes
// the answer there for the kernel enqueued behind this one, and returns at once when that kernel is to take the call.
template <typename TOut, int V, bool kSplit>
__global__ void __launch_bounds__(kThreads, 2)
spmm_direct_kernel(const __grid_constant__ SpmmParams p, const __grid_constant__ CUtensorMap map_b, int m_tiles, int n_tiles, float dense_cost,
                   float dense_per_entry, float gather_per_row, float gather_per_entry, int32_t *verdict, uint32_t *status) {
    constexpr int kRows = kWarpRows / V;                   // vector-rows per fill warp
    constexpr int kGroup = 32 / kRows;                     // lanes per vector-row
    constexpr int kWindow = kRows < 8 ? kRows : 8;         // entries per lane and window: 32 per vector-row (V = 1: 16)
    extern __shared__ __align__(1024) uint8_t sm[];
    const uint32_t base = tc::smem_u32(sm);
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    volatile int *abort_flag = reinterpret_cast<volatile int *>(sm + Smem::kAbort);
    uint32_t *redo_rows = reinterpret_cast<uint32_t *>(sm + Smem::kRedo), *own_redo = redo_rows + kTileM / 32;   // split: of this CTA's part of the columns; of its share of the rows
    const uint32_t bar_full = base + Smem::kBarFull, bar_done = base + Smem::kBarDone;

    pdl_launch_dependents();
    if (t == 0) {
        for (int s = 0; s < kBBuffers; ++s) {
            tc::mbar_init(bar_full + 8 * s, kFillWarps + 1);
            tc::mbar_init(bar_done + 8 * s, 1);
        }
        *abort_flag = 0;
        tc::fence_mbar_init();
    }
    if (t < 2 * (kTileM / 32)) redo_rows[t] = 0;
    if (warp == kMmaWarp) {
        tc::tmem_alloc(base + Smem::kTmemHolder, kTmemCols);
        tc::tmem_relinquish();
    }
    tc::tc_fence_before_sync();
    __syncthreads();
    tc::tc_fence_after_sync();
    const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t *>(sm + Smem::kTmemHolder);
    pdl_wait();   // the set-up above may run beside the call ahead; everything below reads or writes the caller's memory

    bool mine = true;
    if (verdict) {
        const float nnz = (float)__ldg(p.row_offsets + p.m_vec);
        mine = dense_cost + dense_per_entry * nnz < (float)p.m_vec * gather_per_row + gather_per_entry * nnz;
        if (blockIdx.x == 0 && t == 0) plan_publish(verdict, mine);
    }
    const int parts = kSplit ? (int)tc::cluster_nctarank() : 1, part = kSplit ? (int)tc::cluster_ctarank() : 0;
    const unsigned tile = blockIdx.x / (unsigned)parts;
    const int mt = (int)(tile % (unsigned)m_tiles);
    const unsigned rest = tile / (unsigned)m_tiles;
    const int n0 = (int)(rest % (unsigned)n_tiles) * kTileN, b = (int)(rest / (unsigned)n_tiles);
    // this CTA's chunks: `chunk0` .. + chunks - 1
    const int all_chunks = (p.K + kChunkK - 1) / kChunkK, chunk0 = kSplit ? part * all_chunks / parts : 0;
    const int chunks = mine ? (kSplit ? (part + 1) * all_chunks / parts - chunk0 : all_chunks) : 0;
    bool bad = false;

    if (warp < kFillWarps) {
        // =========================== fill ================================================================
        // kGroup lanes share a vector-row: lane g of the group takes its entries g, g + kGroup, ..., kWindow of them at a time
        // (`cols`, `vals`: window 0 is being scattered, window 1 is on its way; `left`: the columns in front of those of
        // window 1).  Lanes move on by themselves, without a shuffle.
        const int row = mt * (kTileM / V) + warp * kRows + lane / kGroup;
        int next = 0, begin = 0, end = 0;
        if (mine && row < p.m_vec) {
            begin = __ldg(p.row_offsets + row);
            end = __ldg(p.row_offsets + row + 1);
        }
        const int first = begin;   // of the vector-row
        if constexpr (kSplit) {
            // the first entry with a column of at least `bound`, for both ends of the part: every round cuts the range to one of kGroup + 1 pieces
            auto search = [&](int bound) {
                int lo = begin, hi = end;   // the answer lies in lo .. hi
                while (__any_sync(0xffffffffu, lo < hi)) {
                    const int at = lo + (int)((int64_t)(hi - lo) * (lane % kGroup) / kGroup);   // lane 0 of the group: lo itself
                    const bool below = lo < hi && __ldg(p.col_indices + at) < bound;
                    const uint32_t votes = __ballot_sync(0xffffffffu, below) >> (lane / kGroup * kGroup) & (uint32_t)((1ull << kGroup) - 1ull);
                    const int n = __popc(votes);   // ascending: the lanes below are the first n
                    const int new_lo = n ? lo + (int)((int64_t)(hi - lo) * (n - 1) / kGroup) + 1 : lo;
                    const int new_hi = n < kGroup ? lo + (int)((int64_t)(hi - lo) * n / kGroup) : hi;
                    if (lo < hi) {
                        lo = n ? new_lo : lo;
                        hi = max(new_hi, lo);
                    }
                }
                return lo;
            };
            const int from = part > 0 ? search(chunk0 * kChunkK) : begin, to = part + 1 < parts ? search((chunk0 + chunks) * kChunkK) : end;
            bad |= from > to;
            begin = from;
            end = max(from, to);
        }
        next = begin + lane % kGroup;
        const __half *values = static_cast<const __half *>(p.values) + (int64_t)b * p.stride_values;
        int cols[2][kWindow], left[kWindow];
        ValueVec<V> vals[2][kWindow];
        auto load_window = [&]() {   // window 1; columns past the end of the row lie beyond every chunk
#pragma unroll
            for (int e = 0; e < kWindow; ++e) {
                const int j = next + e * kGroup;
                cols[1][e] = INT_MAX;
                left[e] = INT_MIN;
                if (j < end) {
                    cols[1][e] = __ldg(p.col_indices + j);
                    if (j > first) left[e] = __ldg(p.col_indices + j - 1);
                    vals[1][e].load(values + (int64_t)j * V);
                }
            }
            next += kWindow * kGroup;
        };
        auto shift_window = [&]() {   // columns that do not ascend strictly: not a matrix for this kernel
#pragma unroll
            for (int e = 0; e < kWindow; ++e) {
                bad |= left[e] >= cols[1][e];
                cols[0][e] = cols[1][e];
                vals[0][e] = vals[1][e];
            }
        };
        load_window();
        shift_window();
        load_window();
        bool ok_run = true;
        for (int c = 0; c < chunks; ++c) {
            uint8_t *a = sm + Smem::kA + (c % kABuffers) * kAChunkBytes;
            if (c >= kABuffers) {   // the chunk that used this buffer before must have been multiplied
                const int prev = c - kABuffers;
                ok_run = __all_sync(0xffffffffu, wait_or_abort<0>(bar_done + 8 * (prev % kBBuffers), (prev / kBBuffers) & 1, abort_flag));
                if (!ok_run) break;   // warp-uniform
            }
            // the warp's 16 rows are two 16-byte pieces of every column's 128 bytes
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const uint32_t k = lane + 32 * (q & 1), piece = 2 * (warp & 3) + ((q >> 1) & 1);
                *reinterpret_cast<uint4 *>(a + (q >> 2) * kABlockBytes + (warp >> 2) * 8192 + (k >> 3) * 1024 + (k & 7u) * 128 +
                                           ((piece ^ (k & 7u)) << 4)) = make_uint4(0, 0, 0, 0);
            }
            __syncwarp();
            const int k0 = (chunk0 + c) * kChunkK, k1 = min(k0 + kChunkK, p.K);
            auto scatter = [&]() {
#pragma unroll
                for (int e = 0; e < kWindow; ++e)
                    if (cols[0][e] >= k0 && cols[0][e] < k1) {
                        const uint32_t k = (uint32_t)(cols[0][e] - k0);
                        scatter_vector<V, false>(a + (k >> 6) * kABlockBytes, ((uint32_t)(warp * kRows + lane / kGroup) << 6) | (k & 63u), vals[0][e].raw);
                    }
            };
            scatter();
            bool used_up = false;
            while (cols[0][kWindow - 1] < k1) {   // the whole window lies in this chunk
                if (used_up) load_window();       // dense rows: more than two windows in one chunk
                used_up = true;
                shift_window();
                scatter();
            }
            tc::fence_proxy_async();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(bar_full + 8 * (c % kBBuffers));
            if (used_up) load_window();   // behind the fence, which waits for outstanding loads as well as for stores
        }
        // A column at or past the end of this CTA's part: beyond the matrix, or of a row that does not ascend.  What stands behind it in the lane's list was
        // not looked at.
        const int part_end = min((chunk0 + chunks) * kChunkK, p.K);
#pragma unroll
        for (int e = 0; e < kWindow; ++e) bad |= cols[0][e] != INT_MAX && cols[0][e] >= part_end;
        const int fill_row = warp * kRows + lane / kGroup;
        if (bad) atomicOr(redo_rows + (fill_row >> 5), 1u << (fill_row & 31));

        // =========================== epilogue ============================================================
        if (chunks > 0)   // the last chunk multiplied is the accumulator complete
            ok_run = __all_sync(0xffffffffu, ok_run && wait_or_abort<0>(bar_done + 8 * ((chunks - 1) % kBBuffers), ((chunks - 1) / kBBuffers) & 1, abort_flag));
        if (ok_run && chunks > 0) {
            tc::tc_fence_after_sync();
            const int quarter = warp & 3, half = warp >> 2;
            uint32_t r[32];
            tc::tmem_ld_x32(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(half * 32), r);
            if constexpr (kSplit) {   // every MMA of this CTA is done: the chunks of A are read no more
                float *sums = reinterpret_cast<float *>(sm + Smem::kA) + (quarter * 32 + lane) * kPartPitch + half * 32;
#pragma unroll
                for (int q = 0; q < 8; ++q) reinterpret_cast<uint4 *>(sums)[q] = make_uint4(r[4 * q], r[4 * q + 1], r[4 * q + 2], r[4 * q + 3]);
            }
            const int m = mt * kTileM + quarter * 32 + lane, n = n0 + half * 32;
            if (!kSplit && m < p.m_vec * V) {
                TOut *out = static_cast<TOut *>(p.out) + (int64_t)b * p.stride_out + (int64_t)m * p.N + n;
                float probe = 0.0f;   // x * 0 is NaN for a sum that is not finite
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    if (n + 8 * q >= p.N) continue;
                    float f[8];
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        f[e] = __uint_as_float(r[8 * q + e]);
                        probe = fmaf(f[e], 0.0f, probe);
                    }
                    store_chunk(out + 8 * q, f);
                }
                const int row = (quarter * 32 + lane) / V;
                if (probe != 0.0f) atomicOr(redo_rows + (row >> 5), 1u << (row & 31));
                bad |= probe != 0.0f;
            }
        }
    } else if (warp == kMmaWarp) {
        if (lane == 0) {
            const uint32_t hi = tc::smem_desc_hi(1024, (uint32_t)tc::kSwizzle128B);
            const uint32_t a_lo0 = tc::smem_desc_lo(base + Smem::kA, 8192), b_lo0 = tc::smem_desc_lo(base + Smem::kB, kBBlockBytes);
            const uint32_t idesc = tc::make_idesc_f16(kTileM, kTileN, 1, 1);   // both operands MN-major
            for (int c = 0; c < chunks; ++c) {
                const int ab = c % kABuffers, bb = c % kBBuffers;
                if (!wait_or_abort<0>(bar_full + 8 * bb, (c / kBBuffers) & 1, abort_flag)) break;
                tc::tc_fence_after_sync();
                const int k_left = p.K - (chunk0 + c) * kChunkK;
                const uint32_t a_lo = a_lo0 + ab * (kAChunkBytes >> 4), b_lo = b_lo0 + bb * (kBChunkBytes >> 4);
#pragma unroll
                for (int kk = 0; kk < kChunkK / 16; ++kk)
                    if (k_left > 16 * kk)
                        tc::mma_f16_ss(tmem_base, tc::desc64(a_lo + (kk >> 2) * (kABlockBytes >> 4) + 128 * (kk & 3), hi),
                                       tc::desc64(b_lo + (kk >> 2) * (kBBlockBytes >> 4) + 128 * (kk & 3), hi), idesc, (c > 0 || kk > 0) ? 1u : 0u);
                tc::mma_commit(bar_done + 8 * bb);
            }
        }
    } else {
        if (lane == 0) {
            for (int c = 0; c < chunks; ++c) {
                const int bb = c % kBBuffers;
                if (c >= kBBuffers && !wait_or_abort<0>(bar_done + 8 * bb, ((c / kBBuffers) - 1) & 1, abort_flag)) break;
                const int boxes = p.K - (chunk0 + c) * kChunkK > 64 ? 2 : 1;
                tc::mbar_expect_tx(bar_full + 8 * bb, (uint32_t)boxes * kBBlockBytes);
                for (int s = 0; s < boxes; ++s)
                    tc::tma_load_3d(base + Smem::kB + bb * kBChunkBytes + s * kBBlockBytes, &map_b, bar_full + 8 * bb, n0, (chunk0 + c) * kChunkK + 64 * s, b);
            }
        }
        __syncwarp();
    }

    // ---- teardown, and the tiles that have to be computed entry by entry -----------------------------------
    tc::tc_fence_before_sync();
    if constexpr (kSplit) {
        // all parts' sums, and their rows to be computed anew, lie in shared memory: this CTA adds up its share of the rows
        tc::cluster_sync();
        const int share = kTileM / parts, row0 = part * share;
        uint32_t theirs = 0;
        if (t < kTileM / 32)
            for (int r = 0; r < parts; ++r) theirs |= tc::ld_remote_u32(tc::map_to_cta(base + Smem::kRedo + 4 * t, r));
        const bool failed = *abort_flag != 0;
        if (mine && !failed) {
            TOut *out = static_cast<TOut *>(p.out) + (int64_t)b * p.stride_out;
            for (int i = t; i < share * (kTileN / 8); i += kThreads) {
                const int row = row0 + i / (kTileN / 8), c = i % (kTileN / 8) * 8, m = mt * kTileM + row;
                if (m >= p.m_vec * V || n0 + c >= p.N) continue;
                float f[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) f[e] = 0.0f;
                for (int r = 0; r < parts; ++r) {
                    const uint32_t from = tc::map_to_cta(base + Smem::kA + (row * kPartPitch + c) * 4, r);
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        const float4 x = tc::ld_remote_f32x4(from + 16 * q);
                        f[4 * q] += x.x; f[4 * q + 1] += x.y; f[4 * q + 2] += x.z; f[4 * q + 3] += x.w;
                    }
                }
                float probe = 0.0f;
#pragma unroll
                for (int e = 0; e < 8; ++e) probe = fmaf(f[e], 0.0f, probe);
                store_chunk(out + (int64_t)m * p.N + n0 + c, f);
                if (probe != 0.0f) {
                    atomicOr(own_redo + (row / V >> 5), 1u << (row / V & 31));
                    bad = true;
                }
            }
        }
        // of the vector-rows found out by any part, those of this CTA's share
        if (t < kTileM / 32) {
            uint32_t share_bits = 0;
            for (int x = 0; x < 32; ++x) {
                const int vr = 32 * t + x;
                if (vr * V >= row0 && vr * V < row0 + share) share_bits |= 1u << x;
            }
            theirs &= share_bits;
            if (theirs) atomicOr(own_redo + t, theirs);
            bad |= theirs != 0u;
        }
        if (!mine) bad = false;
        tc::cluster_sync();   // nobody reads the others' shared memory any more
    }
    const int redo = __syncthreads_or(bad ? 1 : 0);
    if (*abort_flag) {   // a bounded wait ran out: copies that may still be in flight get time to land
        for (int i = 0; i < 64; ++i) __nanosleep(1000);
        if (t == 0) atomicOr(status, densespmm::kStatusTimeout);
        __syncthreads();
    }
    if (warp == kMmaWarp) tc::tmem_dealloc(tmem_base, kTmemCols);
    if (redo) {
        const int row0 = mt * (kTileM / V);
        rows_by_entries<TOut, V>(p, b, row0, min(kTileM / V, p.m_vec - row0), n0, kSplit ? own_redo : redo_rows);
    }
}

}  // namespace directspmm
}  // namespace vs
