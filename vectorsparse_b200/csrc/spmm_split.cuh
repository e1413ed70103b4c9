// fp32 SpMM on the tensor cores: the `cudaSpmm` float entry point (a stub in the reference, src/cuda_spmm.cu:328-338) for large
// products that are not too sparse.
//
// An fp32 number is the exact sum of three bf16 numbers (8 + 8 + 8 significant bits): x = x1 + x2 + x3 (the decomposition of Henry, Tang and
// Heinecke, "Leveraging the bfloat16 Artificial Intelligence Datatype For Higher-Precision Computations", 2019).  Of the nine products of
// two such sums the six largest are kept,
//     a b = a1 b1 + (a1 b2 + a2 b1) + (a1 b3 + a2 b2 + a3 b1) + dropped,
// each exact in the tensor core's fp32.  |x2| <= 2^-8 |x| and |x3| <= 2^-17 |x|, so |dropped| = |a2 b3 + a3 b2 + a3 b3| is at most a little above
// 2^-24 |a b|, half an ulp of the product.  The sums lose as much: the tensor core truncates at every addition.  So the small products of a block
// of 64 columns are added first and the large ones last, and the block's sum is then taken out of tensor memory and added, rounded to nearest, to sums in
// registers: an output sees four truncations per 64 columns, each of that block's partial sum.
//
// Against the CUDA-core kernel's chain of one rounding per entry that is the nearer one where many entries share a block and the farther one where few
// do.  Error of a row of L entries against 64 bits (2-norm over 256 columns, operands U(-1,1), CUDA cores / this one, times 1e-8): K = 64: L = 4 4.0 / 5.2, 8 5.4 / 5.4,
// 24 8.9 / 5.9; K = 512: L = 8 5.4 / 6.7, 16 7.4 / 7.3, 64 14 / 7.9, 512 41 / 9.1; K = 4096: L = 16 7.4 / 8.6, 32 10.4 / 10.7, 48 12.5 / 11.9, 512 41 / 16.
// All operands positive, or all near 1, it takes up to 24 resp. 48 entries to draw level.  So rows of fewer than few_entries(K) entries are computed
// anew by the CUDA-core kernel behind the product, and matrices whose rows are that short on average do not come here.
//
// spmm_split_prepare writes A, zeros included, and B as three bf16 matrices each (scratch of 6 bytes per element), in the order in which
// the tiles are read: a tile of a row-major matrix is 128-byte pieces kilobytes apart, and waiting for those took longer than multiplying
// (4096 x 4096 x 256: a product of 114 us, now 70).  The product is
// a dense one in pairs of CTAs (tcgen05 cta_group::2) with the tiles and the protocol of spmm_pair.cuh: per stage of 64 columns six
// times four 256 x 256 x 16 MMAs.  What it cannot do as well as the CUDA-core kernel, that kernel does behind it, from a
// verdict: rows with few entries, and all of matrices too sparse, a column named twice in a vector-row, and numbers whose parts or products would leave the range of
// normal fp32: non-finite results, inputs below 2^-100, results below 2^-96.
//
// Bound by the tensor pipe: 6 x the dense flops.
#pragma once
#include <cuda.h>
#include "common.cuh"
#include "densify.cuh"
#include "spmm_pair.cuh"
#include "tc_ptx.cuh"

namespace vs {
namespace splitspmm {

using pairspmm::abort_pair;
using pairspmm::wait_or_abort;
using pairspmm::Walk;

constexpr int kTileM = 256, kMaxTileN = 256, kCtaRows = 128, kBlockK = 64, kParts = 3;
constexpr int kPartBytes = 128 * kBlockK * 2;                  // 16 KiB: 128 rows of A or columns of B of one part
// Operands of a stage (64 columns of A): 96 KiB for 256-column items, 72 KiB for 128-column ones, two resp. three of them in flight.
template <int kTn> struct Stage {
    static constexpr int kBytes = kParts * (kPartBytes + kTn / 2 * kBlockK * 2), kCount = kTn == 256 ? 2 : 3;
};
constexpr int kMaxStages = 3, kOperandBytes = 3 * Stage<128>::kBytes;
static_assert(2 * Stage<256>::kBytes <= kOperandBytes, "operand slots");
constexpr int kEpiWarps = 8, kLoadWarp = 8, kMmaWarp = 9, kThreads = 320;
constexpr int kStoreCols = 8, kBoxBytes = 32 * kStoreCols * 4;   // 1 KiB of staging per epilogue warp: once per item, and the operands need the room
// One entry per block of 64 columns and some, at least 24: 1.2 to 2 times those where the two draw level.
inline int few_entries(int K) { return K / kBlockK + 16 > 24 ? K / kBlockK + 16 : 24; }
constexpr uint32_t kTinyResult = (127u - 96u) << 23;

struct Smem {
    static constexpr int kOperands = 0;
    static constexpr int kStaging = kOperandBytes;
    static constexpr int kBarFull = kStaging + kEpiWarps * kBoxBytes;
    static constexpr int kBarDone = kBarFull + kMaxStages * 8;
    static constexpr int kBarAccEmpty = kBarDone + kMaxStages * 8;
    static constexpr int kTmemHolder = kBarAccEmpty + 2 * 8;
    static constexpr int kAbort = kTmemHolder + 8;
    static constexpr int kTotal = kAbort + 8;
};
constexpr int kSmemBytes = Smem::kTotal + 1024;
static_assert(kSmemBytes <= 227 * 1024, "shared memory budget");

// ---- preparation ------------------------------------------------------------------------------------------
using densify::kPrepThreads;

struct PrepParams {
    int batch_a, batch_b;       // problems with values / a dense operand of their own
    int Kp, Np;                 // K and N rounded up to 64
    int64_t min_vectors;        // nonzero vectors from which the split product is the quicker one
    uint16_t *a;                // bf16 [batch][M / 128, rounded up][Kp / 64][part][128 rows][64 columns]
    uint16_t *b;                // bf16 [batch][Kp / 64][Np / 64][part][64 rows][64 columns]
    int few;                    // vector-rows of 1 .. few - 1 entries are the CUDA-core kernel's; 0: none are
    int32_t *verdict;           // plan header (common.cuh); words 4 ..: one per CTA of this kernel, kPlanLeft if it met what the product cannot do,
                                // kPlanFew if it met a vector-row with few entries
};

template <int V> __global__ void __launch_bounds__(kPrepThreads) spmm_split_prepare(const SpmmParams p, const PrepParams q) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ __align__(16) densify::Shared<float> sh;
    const int t = threadIdx.x;
    const int64_t vectors = (int64_t)__ldg(p.row_offsets + p.m_vec) - __ldg(p.row_offsets);
    const bool taken = vectors >= q.min_vectors;
    if (blockIdx.x == 0 && t == 0) plan_publish(q.verdict, taken);
    if (!taken) return;
    bool found = false;
    bool bad = densify::lay_out_rows<float, V, kParts>(p, q.batch_a, q.Kp, q.a, sh, q.few, found);
    const int k_blocks = q.Kp / kBlockK;
    const int chunks = q.Np / 8;
    const int64_t total = (int64_t)q.batch_b * q.Kp * chunks;
    for (int64_t i = (int64_t)blockIdx.x * kPrepThreads + t; i < total; i += (int64_t)gridDim.x * kPrepThreads) {
        const int c = (int)(i % chunks) * 8;
        const int64_t r = i / chunks;
        const int k = (int)(r % q.Kp), b = (int)(r / q.Kp);
        const float *src = static_cast<const float *>(p.rhs) + (int64_t)b * p.stride_rhs + (int64_t)k * p.N + c;
        float x[8];
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 lo = k < p.K && c < p.N ? __ldg(reinterpret_cast<const float4 *>(src)) : zero, hi = k < p.K && c + 4 < p.N ? __ldg(reinterpret_cast<const float4 *>(src) + 1) : zero;
        x[0] = lo.x; x[1] = lo.y; x[2] = lo.z; x[3] = lo.w; x[4] = hi.x; x[5] = hi.y; x[6] = hi.z; x[7] = hi.w;
        uint4 part[kParts];
        bad |= densify::split8(x, part);
#pragma unroll
        for (int s = 0; s < kParts; ++s) {
            const int64_t tile = (((int64_t)b * k_blocks + k / kBlockK) * (q.Np / 64) + c / 64) * kParts + s;
            *reinterpret_cast<uint4 *>(q.b + tile * (kBlockK * 64) + (k % kBlockK) * 64 + c % 64) = part[s];
        }
    }
    const int any = __syncthreads_or(bad), some = __syncthreads_or(found);
    if (t == 0) q.verdict[4 + blockIdx.x] = (any ? kPlanLeft : 0) | (some ? kPlanFew : 0);
}

// ---- product ----------------------------------------------------------------------------------------------
// map_a: the tiles of A as {64 columns, 128 rows, parts, tiles}, box {64, 128, 3, 1}; map_b: those of B as {64 columns, 64 rows, parts,
// tiles}, box {64, 64, 3, kTn / 128}: a CTA's operands of a stage are two copies.  map_out: {N, M, batch} fp32, box {8, 32, 1}; what lies
// outside is not written.  Rows and columns past the matrix are multiplied with whatever the scratch holds there, zeros within the
// last 64 columns and rows of K, and go nowhere.  kTn: columns per work item, 256 or 128.  No multicast anywhere.
template <int kTn>
__global__ void __launch_bounds__(kThreads, 1)
spmm_split_kernel(const SpmmParams p, int V, const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                  const __grid_constant__ CUtensorMap map_out, int batch_a, int batch_b, int m_tiles, int n_tiles, int k_blocks, int row_tiles, int slabs,
                  uint32_t *status, const int32_t *verdict, int checks, int32_t *redo) {
    // No pdl_launch_dependents(): CTAs of the kernel behind that became resident beside this one's would keep the division of the SM's memory that its
    // operands need, and have hardly any L1 where the call comes down to them (4096 x 4096 x 8192, V = 1, 80 %, one operand below 2^-100: 7216 us, so
    // 5666, the CUDA-core kernel alone 4730; a call that does not 0.4 to 0.8 us less).
    pdl_wait();
    const bool chosen = plan_split_chosen(verdict, checks);
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = tc::smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;   // the same offset in both CTAs
    uint8_t *sm = smem_raw + (base - raw);
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const uint32_t rank = tc::cluster_ctarank(), peer = rank ^ 1u;
    const uint32_t pair = tc::cluster_id_x(), pairs = tc::cluster_count_x();
    volatile int *abort_flag = reinterpret_cast<volatile int *>(sm + Smem::kAbort);
    const uint32_t abort_addr = base + Smem::kAbort;
    const uint32_t bar_full = base + Smem::kBarFull, bar_done = base + Smem::kBarDone, bar_acc_empty = base + Smem::kBarAccEmpty;
    constexpr int kStages = Stage<kTn>::kCount, kStageBytes = Stage<kTn>::kBytes, kHalfCols = kTn / 2;   // columns of B each CTA holds

    if (t == 0) {
        for (int s = 0; s < kStages; ++s) {
            tc::mbar_init(bar_full + 8 * s, 1);                     // first CTA: its loader's arrival + the bytes of both CTAs
            tc::mbar_init(bar_done + 8 * s, 1);                     // both: "stage multiplied": its operands are free, its accumulator complete
        }
        for (int s = 0; s < 2; ++s) {
            tc::mbar_init(bar_acc_empty + 8 * s, 2 * kEpiWarps);   // first CTA: read out by every epilogue warp of both
        }
        *abort_flag = 0;
        tc::fence_mbar_init();
    }
    if (warp == kMmaWarp) {
        tc::tmem_alloc_pair(base + Smem::kTmemHolder, 2 * kMaxTileN);
        tc::tmem_relinquish_pair();
    }
    tc::tc_fence_before_sync();
    tc::cluster_sync();
    tc::tc_fence_after_sync();
    const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t *>(sm + Smem::kTmemHolder);

    const int64_t total_items = chosen ? (int64_t)p.batch * n_tiles * m_tiles : 0;
    const uint32_t my_items = (total_items > pair) ? (uint32_t)((total_items - pair + pairs - 1) / pairs) : 0u;
    const uint32_t total_stages = my_items * (uint32_t)k_blocks;
    const int m_rows = p.m_vec * V;

    // stage g of the pair uses operand slot g % kStages and accumulator g % 2
    if (warp == kLoadWarp) {
        if (lane == 0) {
            bool ok_run = true;
            const uint32_t full_first = tc::map_to_cta(bar_full, 0);
            Walk walk;
            walk.init(pair, pairs, 0u, total_stages, m_tiles, n_tiles, k_blocks);
            for (uint32_t g = 0; g < total_stages && ok_run; ++g, walk.advance(1)) {
                const uint32_t slot = g % kStages;
                if (g >= (uint32_t)kStages)
                    ok_run = wait_or_abort<0>(bar_done + 8 * slot, (g / kStages - 1) & 1u, abort_flag, abort_addr, peer);
                if (!ok_run) break;
                const uint32_t bar = full_first + 8 * slot, a_dst = base + Smem::kOperands + slot * kStageBytes, b_dst = a_dst + kParts * kPartBytes;
                const int za = ((batch_a == 1 ? 0 : walk.b) * row_tiles + 2 * walk.mt + (int)rank) * k_blocks + walk.kb;
                const int zb = ((batch_b == 1 ? 0 : walk.b) * k_blocks + walk.kb) * slabs + ((walk.nt * kTn + (int)rank * kHalfCols) >> 6);
                if (rank == 0) tc::mbar_expect_tx(bar_full + 8 * slot, 2u * kStageBytes);
                tc::tma_load_4d_pair(a_dst, &map_a, bar, 0, 0, 0, za);
                tc::tma_load_4d_pair(b_dst, &map_b, bar, 0, 0, 0, zb);
            }
            // no signal addressed to this CTA may arrive after it has gone
            const uint32_t tail0 = total_stages > (uint32_t)kStages ? total_stages - kStages : 0u;
            for (uint32_t g = tail0; g < total_stages && ok_run; ++g)
                ok_run = wait_or_abort<0>(bar_done + 8 * (g % kStages), (g / kStages) & 1u, abort_flag, abort_addr, peer);
        }
    } else if (warp == kMmaWarp) {
        if (lane == 0 && rank == 0) {
            const uint32_t a_lo0 = tc::smem_desc_lo(base + Smem::kOperands, 16);                                  // K-major, 8-row groups 1 KiB apart
            const uint32_t b_lo0 = tc::smem_desc_lo(base + Smem::kOperands + kParts * kPartBytes, kParts * kPartBytes / 2);   // 64-column slabs, three parts of 8 KiB each
            const uint32_t hi = tc::smem_desc_hi(1024, (uint32_t)tc::kSwizzle128B);
            const uint32_t idesc = tc::make_idesc_f16(kTileM, kTn, 0, 1) | (1u << 7) | (1u << 10);             // both operands bf16
            const int steps_last = ((p.K - 1) & (kBlockK - 1)) / 16 + 1;
            bool ok_run = true;
            uint32_t g = 0;
            for (uint32_t i = 0; i < my_items && ok_run; ++i) {
                for (int kb = 0; kb < k_blocks; ++kb, ++g) {
                    const uint32_t slot = g % kStages, buf = g & 1u;
                    ok_run = wait_or_abort<0>(bar_acc_empty + 8 * buf, (g >> 1) & 1u, abort_flag, abort_addr, peer) &&
                             wait_or_abort<0>(bar_full + 8 * slot, (g / kStages) & 1u, abort_flag, abort_addr, peer);
                    if (!ok_run) break;
                    tc::tc_fence_after_sync();
                    const uint32_t d = tmem_base + buf * kMaxTileN;
                    const uint32_t a_lo = a_lo0 + slot * (kStageBytes >> 4), b_lo = b_lo0 + slot * (kStageBytes >> 4);
                    const int steps = kb + 1 < k_blocks ? kBlockK / 16 : steps_last;
                    // parts of A and B, smallest products first
                    constexpr int kA[6] = {2, 0, 1, 1, 0, 0}, kB[6] = {0, 2, 1, 0, 1, 0};
                    auto product = [&](int s, int kk) {   // 16 columns of A: 32 bytes on in A, 2 KiB in B
                        tc::mma_f16_ss_pair(d, tc::desc64(a_lo + kA[s] * (kPartBytes >> 4) + 2 * kk, hi),
                                            tc::desc64(b_lo + kB[s] * (kPartBytes >> 5) + 128 * kk, hi), idesc, (s | kk) ? 1u : 0u);
                    };
                    if (steps == kBlockK / 16) {   // written out: a loop issues them more slowly than 128 columns of B multiply
#pragma unroll
                        for (int s = 0; s < 6; ++s)
#pragma unroll
                            for (int kk = 0; kk < kBlockK / 16; ++kk) product(s, kk);
                    } else {
#pragma unroll
                        for (int s = 0; s < 6; ++s)
                            for (int kk = 0; kk < steps; ++kk) product(s, kk);
                    }
                    tc::mma_commit_pair_both(bar_done + 8 * slot);
                }
            }
        }
    } else {
        // epilogue warp (quarter, half): rows 32 quarter .. + 31 of the CTA's 128, kHalfCols columns from kHalfCols half
        const int quarter = warp & 3, half = warp >> 2;
        uint8_t *stg = sm + Smem::kStaging + warp * kBoxBytes;
        const uint32_t stg_u32 = base + Smem::kStaging + warp * kBoxBytes;
        const uint32_t lane_taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(half * kHalfCols);
        const uint32_t empty_first = tc::map_to_cta(bar_acc_empty, 0);
        tc::tc_fence_before_sync();
        if (lane == 0)
            for (int s = 0; s < 2; ++s) tc::mbar_arrive_remote(empty_first + 8 * s);   // both buffers start out free
        Walk walk;
        walk.init(pair, pairs, 0u, my_items, m_tiles, n_tiles, 1);
        bool ok_run = true, bad = false;
        uint32_t g = 0;
        for (uint32_t i = 0; i < my_items && ok_run; ++i, walk.advance(1)) {
            float acc[kHalfCols];
#pragma unroll
            for (int e = 0; e < kHalfCols; ++e) acc[e] = 0.f;
            for (int kb = 0; kb < k_blocks; ++kb, ++g) {
                const uint32_t buf = g & 1u, slot = g % kStages;
                ok_run = __all_sync(0xffffffffu, wait_or_abort<0>(bar_done + 8 * slot, (g / kStages) & 1u, abort_flag, abort_addr, peer));
                if (!ok_run) break;
                tc::tc_fence_after_sync();
#pragma unroll
                for (int c = 0; c < kHalfCols; c += 16) {
                    uint32_t r[16];
                    tc::tmem_ld_x16(lane_taddr + buf * kMaxTileN + (uint32_t)c, r);
#pragma unroll
                    for (int e = 0; e < 16; ++e) acc[c + e] += __uint_as_float(r[e]);
                }
                tc::tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) tc::mbar_arrive_remote(empty_first + 8 * buf);   // one per warp: 512 a stage were slower than its products
            }
            if (!ok_run) break;
            const int row0 = walk.mt * kTileM + (int)rank * kCtaRows + quarter * 32, col0 = walk.nt * kTn + half * kHalfCols;
            if (row0 < m_rows) {   // warp-uniform
#pragma unroll
                for (int c = 0; c < kHalfCols; c += kStoreCols) {
                    if (col0 + c < p.N) {
                        if (row0 + lane < m_rows) {
#pragma unroll
                            for (int e = 0; e < kStoreCols; ++e) {   // columns past the matrix hold zeros
                                const uint32_t bits = __float_as_uint(acc[c + e]) & 0x7fffffffu;
                                bad |= bits >= 0x7f800000u || bits - 1u < kTinyResult - 1u;
                            }
                        }
                        if (lane == 0) tc::bulk_wait_group_read<0>();
                        __syncwarp();
                        float4 *row = reinterpret_cast<float4 *>(stg + lane * (kStoreCols * 4));
                        row[0] = make_float4(acc[c], acc[c + 1], acc[c + 2], acc[c + 3]);
                        row[1] = make_float4(acc[c + 4], acc[c + 5], acc[c + 6], acc[c + 7]);
                        tc::fence_proxy_async();
                        __syncwarp();
                        if (lane == 0) {
                            tc::tma_store_3d(&map_out, stg_u32, col0 + c, row0, walk.b);
                            tc::bulk_commit_group();
                        }
                    }
                }
            }
        }
        if (lane == 0) tc::bulk_wait_group<0>();
        if (__any_sync(0xffffffffu, bad) && lane == 0) atomicExch(redo, 1);
    }

    tc::tc_fence_before_sync();
    __syncthreads();
    if (*abort_flag) {
        for (int i = 0; i < 64; ++i) __nanosleep(1000);   // copies that may still be in flight
        if (t == 0) atomicOr(status, densespmm::kStatusTimeout);
    }
    tc::cluster_sync();   // neither CTA's shared or tensor memory goes away while the other half of an MMA may use it
    if (warp == kMmaWarp) tc::tmem_dealloc_pair(tmem_base, 2 * kMaxTileN);
}

}  // namespace splitspmm
}  // namespace vs
