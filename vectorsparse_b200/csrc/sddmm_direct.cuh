// Tensor-core SDDMM for small problems in ONE kernel: the `wmmaSddmm` entry point of the reference
// (src/wmma_sddmm.cu:3175-3202) where a call is too short for a plan.  Dense tiles sampled at the mask, as in
// sddmm_pair.cuh, without the plan kernel in front of the multiplying kernel and the twin kernel behind it:
//
//     D[128 rows of lhs x tn mask columns] = lhs[128 x k] . rhs[tn x k]^T          one CTA per tile, tn = 128 or 64
//
// What bounds it.  One sampled product of 512 x 2048 x 256 is a microsecond of work; plan, multiplying kernel and twin
// kernel took 17 us on the GPU, nearly all of it launches and dependent loads; this kernel takes 6.0 us (64 x 64 x 64: 7.1 ->
// 2.5).  Here everything hangs on two short
// chains that run side by side: TMA -> MMA -> tensor memory -> shared memory, and row offsets -> mask columns.
//
// Sampling.  The vector-rows of a tile are neighbours, so their mask entries are ONE contiguous range.  Every thread
// of those warps looks at entries t, t + 256, ... of it, keeps those whose column lies in the tile (the other column tiles of the same
// rows look at the range again: it is a few thousand words, from L2) and finds the vector-row by bisection in the tile's
// offsets in shared memory.  The first kAhead of its entries are looked up before the product is there.  The product
// is laid out in shared memory by column, rows contiguous, so that the V outputs of an entry are one vector.  Any
// order of columns and any repetition is right, and nothing outside the mask is stored.
//
// The contraction order is the one of the other tensor-core SDDMM kernels (16 elements at a time, ascending): the
// same bits whichever of them multiplies.
//
// Roles (320 threads): warps 0-7 look entries up, move the accumulator out and sample; warp 8 the thread that loads by TMA;
// warp 9 the MMA-issuing thread.  Ring of three stages of 64 contraction elements; two CTAs per SM.
#pragma once
#include <cuda.h>

#include "common.cuh"
#include "sddmm_dense.cuh"
#include "spmm_dense.cuh"
#include "tc_ptx.cuh"

namespace vs {
namespace directsddmm {

using densespmm::wait_or_abort;

constexpr int kTileM = 128, kMaxTileN = 128, kBlockK = 64;
constexpr int kSampleThreads = 256;
constexpr int kLoadWarp = kSampleThreads / 32, kMmaWarp = kLoadWarp + 1;
constexpr int kThreads = (kMmaWarp + 1) * 32;             // 320
constexpr int kStages = 3;
constexpr int kLhsBytes = kTileM * kBlockK * 2;           // 16 KiB
constexpr int kStageBytes = kLhsBytes + kMaxTileN * kBlockK * 2;
constexpr int kPitch = kTileM + 4;                        // floats between columns of the laid-out product: 16-byte aligned, 4 banks on
constexpr int kAhead = 8;                                 // entries per thread looked up while the product is being computed
constexpr int kTmemCols = 128;

struct Smem {   // offsets from the 1024-byte aligned base
    static constexpr int kStage = 0;                      // the ring; once everything is multiplied, the product
    static constexpr int kOffsets = kStages * kStageBytes;
    static constexpr int kBarFull = kOffsets + (kTileM + 4) * 4;
    static constexpr int kBarEmpty = kBarFull + kStages * 8;
    static constexpr int kBarAcc = kBarEmpty + kStages * 8;
    static constexpr int kTmemHolder = kBarAcc + 8;
    static constexpr int kAbort = kTmemHolder + 8;
    static constexpr int kTotal = kAbort + 8;
};
constexpr int kSmemBytes = Smem::kTotal;
static_assert(kPitch * kMaxTileN * 4 <= kStages * kStageBytes, "the product overlays the ring");
static_assert(2 * (kSmemBytes + 1024) <= 228 * 1024, "two CTAs per SM");

// Barrier of the eight sampling warps.
__device__ __forceinline__ void sample_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(kSampleThreads) : "memory"); }

// map_lhs: {k, rows of lhs, batch}, box {64, 128, 1}; map_rhs: {k, n, batch}, box {64, tn, 1}; K-major, 128-byte swizzle,
// zero fill outside (contraction lengths that are no multiple of 64 included).
template <typename TOut, int V>
__global__ void __launch_bounds__(kThreads, 2)
sddmm_direct_kernel(const SddmmParams p, const __grid_constant__ CUtensorMap map_lhs, const __grid_constant__ CUtensorMap map_rhs,
                    int tn, int m_tiles, int n_tiles, uint32_t *status) {
    constexpr int kVecRows = kTileM / V;
    extern __shared__ __align__(1024) uint8_t sm[];
    const uint32_t base = tc::smem_u32(sm);
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    volatile int *abort_flag = reinterpret_cast<volatile int *>(sm + Smem::kAbort);
    int *offs = reinterpret_cast<int *>(sm + Smem::kOffsets);
    float *prod = reinterpret_cast<float *>(sm + Smem::kStage);
    const uint32_t bar_full = base + Smem::kBarFull, bar_empty = base + Smem::kBarEmpty, bar_acc = base + Smem::kBarAcc;

    pdl_launch_dependents();
    if (t == 0) {
        for (int s = 0; s < kStages; ++s) {
            tc::mbar_init(bar_full + 8 * s, 1);
            tc::mbar_init(bar_empty + 8 * s, 1);
        }
        tc::mbar_init(bar_acc, 1);
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
    pdl_wait();   // the set-up above may run beside the call ahead

    const int mt = (int)(blockIdx.x % (unsigned)m_tiles);
    const unsigned rest = blockIdx.x / (unsigned)m_tiles;
    const int c0 = (int)(rest % (unsigned)n_tiles) * tn, b = (int)(rest / (unsigned)n_tiles);
    const int k_blocks = (p.k + kBlockK - 1) / kBlockK;

    if (warp == kLoadWarp) {
        if (lane == 0) {
            for (int g = 0; g < k_blocks; ++g) {
                const int s = g % kStages;
                if (g >= kStages && !wait_or_abort<0>(bar_empty + 8 * s, ((g / kStages) - 1) & 1, abort_flag)) break;
                tc::mbar_expect_tx(bar_full + 8 * s, (uint32_t)(kLhsBytes + tn * kBlockK * 2));
                tc::tma_load_3d(base + Smem::kStage + s * kStageBytes, &map_lhs, bar_full + 8 * s, g * kBlockK, mt * kTileM, b);
                tc::tma_load_3d(base + Smem::kStage + s * kStageBytes + kLhsBytes, &map_rhs, bar_full + 8 * s, g * kBlockK, c0, b);
            }
        }
    } else if (warp == kMmaWarp) {
        if (lane == 0) {
            const uint32_t hi = tc::smem_desc_hi(1024, (uint32_t)tc::kSwizzle128B);
            const uint32_t idesc = tc::make_idesc_f16(kTileM, tn, 0, 0);   // both operands K-major
            bool ok_run = true;
            for (int g = 0; g < k_blocks; ++g) {
                const int s = g % kStages;
                ok_run = wait_or_abort<0>(bar_full + 8 * s, (g / kStages) & 1, abort_flag);
                if (!ok_run) break;
                tc::tc_fence_after_sync();
                const uint32_t a_lo = tc::smem_desc_lo(base + Smem::kStage + s * kStageBytes, 16);
                const uint32_t b_lo = tc::smem_desc_lo(base + Smem::kStage + s * kStageBytes + kLhsBytes, 16);
                const int k_left = p.k - g * kBlockK;
#pragma unroll
                for (int kk = 0; kk < kBlockK / 16; ++kk)
                    if (k_left > 16 * kk)
                        tc::mma_f16_ss(tmem_base, tc::desc64(a_lo + 2 * kk, hi), tc::desc64(b_lo + 2 * kk, hi), idesc, (g > 0 || kk > 0) ? 1u : 0u);
                tc::mma_commit(bar_empty + 8 * s);
            }
            if (ok_run) tc::mma_commit(bar_acc);
        }
    } else {
        // the tile's range of mask entries (the caller's count bounds what may be written)
        const int vr0 = mt * kVecRows, rows = min(kVecRows, p.m_vec - vr0);
        for (int i = t; i <= rows; i += kSampleThreads) offs[i] = min(max(__ldg(p.row_offsets + vr0 + i), 0), p.nnz_vec);
        sample_barrier();
        const int j0 = offs[0], j1 = max(offs[rows], j0);
        auto place_of = [&](int j, int c) -> int {   // row within the tile * 128 + column within the tile, or -1
            if ((unsigned)(c - c0) >= (unsigned)tn || c >= p.n) return -1;
            int lo = 0, hi = rows;
            while (hi - lo > 1) {
                const int mid = (lo + hi) >> 1;
                if (offs[mid] <= j) lo = mid; else hi = mid;
            }
            return (lo << 7) | (c - c0);
        };
        int place[kAhead];
        auto look_up = [&](int jb) {   // entries jb, + 256, ...: their loads fly together
#pragma unroll
            for (int u = 0; u < kAhead; ++u) place[u] = jb + u * kSampleThreads < j1 ? __ldg(p.col_indices + jb + u * kSampleThreads) : -1;
#pragma unroll
            for (int u = 0; u < kAhead; ++u) place[u] = place_of(jb + u * kSampleThreads, place[u]);
        };
        look_up(j0 + t);

        const bool ok_run = __all_sync(0xffffffffu, wait_or_abort<0>(bar_acc, 0, abort_flag));
        if (ok_run) {
            tc::tc_fence_after_sync();
            // lane = row of the tile: a column's 128 rows are contiguous, so the lanes of a store hit different banks
            const int quarter = warp & 3, half = warp >> 2;
            for (int c = half * (tn / 2); c < (half + 1) * (tn / 2); c += 32) {
                uint32_t r[32];
                tc::tmem_ld_x32(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)c, r);
#pragma unroll
                for (int e = 0; e < 32; ++e) prod[(c + e) * kPitch + quarter * 32 + lane] = __uint_as_float(r[e]);
            }
        }
        sample_barrier();
        if (*abort_flag == 0) {
            TOut *out = static_cast<TOut *>(p.out) + (int64_t)b * p.stride_out;
            auto emit = [&](int j, int at) {
                const float *src = prod + (at & 127) * kPitch + (at >> 7) * V;
                TOut *dst = out + (int64_t)j * V;
                if constexpr (V >= 4) {
                    float f[V];
#pragma unroll
                    for (int q = 0; q < V / 4; ++q) {
                        const float4 x = *reinterpret_cast<const float4 *>(src + 4 * q);
                        f[4 * q] = x.x; f[4 * q + 1] = x.y; f[4 * q + 2] = x.z; f[4 * q + 3] = x.w;
                    }
                    store_chunk(dst, f);
                } else if constexpr (V == 2 && sizeof(TOut) == 2) {
                    *reinterpret_cast<__half2 *>(dst) = __floats2half2_rn(src[0], src[1]);
                } else if constexpr (V == 2) {
                    *reinterpret_cast<float2 *>(dst) = make_float2(src[0], src[1]);
                } else {
                    store_scalar(dst, src[0]);
                }
            };
#pragma unroll
            for (int u = 0; u < kAhead; ++u)
                if (place[u] >= 0) emit(j0 + t + u * kSampleThreads, place[u]);
            for (int jb = j0 + t + kAhead * kSampleThreads; jb < j1; jb += kAhead * kSampleThreads) {
                look_up(jb);
#pragma unroll
                for (int u = 0; u < kAhead; ++u)
                    if (place[u] >= 0) emit(jb + u * kSampleThreads, place[u]);
            }
        }
    }
    tc::tc_fence_before_sync();
    __syncthreads();
    if (*abort_flag) {   // a bounded wait ran out: copies that may still be in flight get time to land
        for (int i = 0; i < 64; ++i) __nanosleep(1000);
        if (t == 0) atomicOr(status, densesddmm::kStatusTimeout);
        __syncthreads();
    }
    if (warp == kMmaWarp) tc::tmem_dealloc(tmem_base, kTmemCols);
}

}  // namespace directsddmm
}  // namespace vs
