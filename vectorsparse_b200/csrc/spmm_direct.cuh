// Tensor-core SpMM for small problems in ONE kernel: the `wmmaSpmm` entry point of the reference
// (src/wmma_spmm.cu:388-409) where a call is too short for a plan.  Same formulation as spmm_dense.cuh — multiply
// zero-filled tiles of A — without the plan kernel in front of it and (mostly) without a stand-by kernel behind it:
//
//     C[128 rows x 64 cols] = A_dense[128 x K] * B[K x 64]          one CTA per tile, 128 columns of A at a time
//
// What bounds it.  One product of 2048 x 512 x 256 is a microsecond of work; the plan, the multiplying kernel and the
// gather kernel that returns at once took 15.4 us on the GPU, nearly all of it launches and dependent loads; this kernel
// takes 6.5 us (64 x 64 x 256: 11.2 -> 2.7).  Its chain is row offsets -> columns and values -> scatter -> MMA -> store, once,
// and after the first chunk ~0.55 us per chunk: filling it (an MMA of 64 columns takes as long as one of 128, ~61 cycles).  128 x 64 tiles and two CTAs per SM because
// at these sizes the number of CTAs is what is short; a larger problem re-reads A once per 64 columns and goes to the
// pair kernel instead.
//
// How a CTA finds its entries without a plan.  Each of eight fill warps owns 16 rows of the tile (16 / V vector-rows)
// and walks their entries in windows, one being scattered and the next one on its way: the entries below the chunk's last
// column are scattered, a window that is used up makes room for the next.  That needs columns that ascend strictly
// within a vector-row, which is checked on every entry.  A tile with a row that does not (unsorted, or a column named twice), and a tile with
// a non-finite sum (0 x Inf of the densified tile, see spmm_dense.cuh), is computed again by the same CTA from the
// CVSE arrays on CUDA cores, entry by entry as the reference does.
//
// The K order of the MMAs is the one of the other densifying kernels (16 columns of A at a time, ascending), so that a
// product has the same bits whichever of them multiplies it.
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

struct Smem {   // offsets from the 1024-byte aligned base
    static constexpr int kA = 0;
    static constexpr int kB = kA + kABuffers * kAChunkBytes;
    // one pair of barriers per chunk in flight (chunk c: pair c % kBBuffers): `full` collects the fill warps, the loader
    // and the bytes of B, `done` the commit of the MMA-issuing thread, which pays ~100 cycles for each commit and wait
    static constexpr int kBarFull = kB + kBBuffers * kBChunkBytes;
    static constexpr int kBarDone = kBarFull + kBBuffers * 8;
    static constexpr int kTmemHolder = kBarDone + kBBuffers * 8;
    static constexpr int kAbort = kTmemHolder + 8;
    static constexpr int kTotal = kAbort + 8;
};
constexpr int kSmemBytes = Smem::kTotal;   // the dynamic segment is 1024-byte aligned (nothing static lies ahead of it)
static_assert(2 * (kSmemBytes + 1024) <= 228 * 1024, "two CTAs per SM");

// One tile from the CVSE arrays on CUDA cores: a thread per (vector-row, 8 columns), fp32 sums in list order.
template <typename TOut, int V>
__device__ __noinline__ void tile_by_entries(const SpmmParams &p, int b, int row0, int rows, int n0) {
    const __half *values = static_cast<const __half *>(p.values) + (int64_t)b * p.stride_values;
    const __half *rhs = static_cast<const __half *>(p.rhs) + (int64_t)b * p.stride_rhs;
    TOut *out = static_cast<TOut *>(p.out) + (int64_t)b * p.stride_out;
    const int chunks = min(kTileN, p.N - n0) / 8;
    for (int item = threadIdx.x; item < rows * chunks; item += kThreads) {
        const int r = row0 + item / chunks, n = n0 + 8 * (item % chunks);
        float acc[V][8];
#pragma unroll
        for (int v = 0; v < V; ++v)
#pragma unroll
            for (int e = 0; e < 8; ++e) acc[v][e] = 0.f;
        for (int j = __ldg(p.row_offsets + r), end = __ldg(p.row_offsets + r + 1); j < end; ++j) {
            const int c = __ldg(p.col_indices + j);
            if ((unsigned)c >= (unsigned)p.K) continue;
            float a[V];
            VecLoad<__half, V>::load(values + (int64_t)j * V, a);
            Chunk<__half> x;
            x.load(rhs + (int64_t)c * p.N + n);
#pragma unroll
            for (int v = 0; v < V; ++v)
#pragma unroll
                for (int e = 0; e < 8; ++e) acc[v][e] = fmaf(a[v], x.f[e], acc[v][e]);
        }
#pragma unroll
        for (int v = 0; v < V; ++v) store_chunk(out + ((int64_t)r * V + v) * p.N + n, acc[v]);
    }
}

// map_b: the dense operand as {N, K, batch}, box {64, 64, 1}, 128-byte swizzle, zero fill outside.
// verdict: null when the densified product is the cheaper one whatever the number of nonzeros; otherwise the
// kernel compares the costs the plan kernel compares (dense_cost for its `stages`, gather_per_row, gather_per_entry), writes
// the answer there for the kernel enqueued behind this one, and returns at once when that kernel is to take the call.
template <typename TOut, int V>
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
        if (blockIdx.x == 0 && t == 0) *verdict = mine ? 1 : 0;
    }
    const int mt = (int)(blockIdx.x % (unsigned)m_tiles);
    const unsigned rest = blockIdx.x / (unsigned)m_tiles;
    const int n0 = (int)(rest % (unsigned)n_tiles) * kTileN, b = (int)(rest / (unsigned)n_tiles);
    const int chunks = mine ? (p.K + kChunkK - 1) / kChunkK : 0;
    bool bad = false;

    if (warp < kFillWarps) {
        // =========================== fill ================================================================
        // kGroup lanes share a vector-row: lane g of the group takes its entries g, g + kGroup, ..., kWindow of them at a time
        // (`cols`, `vals`: window 0 is being scattered, window 1 is on its way; `left`: the columns in front of those of
        // window 1).  Lanes move on by themselves, without a shuffle.
        const int row = mt * (kTileM / V) + warp * kRows + lane / kGroup;
        int next = 0, begin = 0, end = 0;
        if (row < p.m_vec) {
            begin = __ldg(p.row_offsets + row);
            end = __ldg(p.row_offsets + row + 1);
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
                    if (j > begin) left[e] = __ldg(p.col_indices + j - 1);
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
            const int k0 = c * kChunkK, k1 = min(k0 + kChunkK, p.K);
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
        if (mine)
#pragma unroll
            for (int e = 0; e < kWindow; ++e) bad |= cols[0][e] != INT_MAX && cols[0][e] >= p.K;   // columns beyond the matrix

        // =========================== epilogue ============================================================
        if (chunks > 0)   // the last chunk multiplied is the accumulator complete
            ok_run = __all_sync(0xffffffffu, ok_run && wait_or_abort<0>(bar_done + 8 * ((chunks - 1) % kBBuffers), ((chunks - 1) / kBBuffers) & 1, abort_flag));
        if (ok_run && chunks > 0) {
            tc::tc_fence_after_sync();
            const int quarter = warp & 3, half = warp >> 2;
            uint32_t r[32];
            tc::tmem_ld_x32(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(half * 32), r);
            const int m = mt * kTileM + quarter * 32 + lane, n = n0 + half * 32;
            if (m < p.m_vec * V) {
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
                const int k_left = p.K - c * kChunkK;
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
                const int boxes = p.K - c * kChunkK > 64 ? 2 : 1;
                tc::mbar_expect_tx(bar_full + 8 * bb, (uint32_t)boxes * kBBlockBytes);
                for (int s = 0; s < boxes; ++s)
                    tc::tma_load_3d(base + Smem::kB + bb * kBChunkBytes + s * kBBlockBytes, &map_b, bar_full + 8 * bb, n0, c * kChunkK + 64 * s, b);
            }
        }
        __syncwarp();
    }

    // ---- teardown, and the tiles that have to be computed entry by entry -----------------------------------
    tc::tc_fence_before_sync();
    const int redo = __syncthreads_or(bad ? 1 : 0);
    if (*abort_flag) {   // a bounded wait ran out: copies that may still be in flight get time to land
        for (int i = 0; i < 64; ++i) __nanosleep(1000);
        if (t == 0) atomicOr(status, densespmm::kStatusTimeout);
        __syncthreads();
    }
    if (warp == kMmaWarp) tc::tmem_dealloc(tmem_base, kTmemCols);
    if (redo) {
        const int row0 = mt * (kTileM / V);
        tile_by_entries<TOut, V>(p, b, row0, min(kTileM / V, p.m_vec - row0), n0);
    }
}

}  // namespace directspmm
}  // namespace vs
