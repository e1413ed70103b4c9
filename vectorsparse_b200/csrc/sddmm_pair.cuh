// Tensor-core SDDMM on dense tiles sampled at the mask, computed by PAIRS of CTAs (a cluster of two SMs, tcgen05
// cta_group::2): the `wmmaSddmm` entry point of the reference (src/wmma_sddmm.cu:3175-3202).  Same formulation as
// sddmm_dense.cuh next to this file; what changes is the tile, its orientation and the way it is sampled:
//
//     D^T[256 mask columns x 256 rows of lhs] += rhs[256 x 64] . lhs[256 x 64]^T        per 64 contraction elements
//
// is ONE stream of 256 x 256 x 16 MMAs issued by one thread of the pair's first CTA.  CTA r of the pair loads rows
// 128 r .. of the rhs tile (its half of the M operand) and rows 128 r .. of the lhs tile (its half of the N operand)
// with its own plain TMA tile loads (no multicast), and receives mask columns 128 r .. of the product in its own
// tensor memory: lane = mask column, tensor-memory column = row of lhs.  Against the single-CTA kernel (256 x 128
// tiles, 128 x 128 x 16 MMAs) every SM reads 2/3 of the operand bytes per output from L2 and half as much from
// shared memory per flop, which is what that kernel is bound by.
//
// Sampling.  The V rows of a vector-row are V CONSECUTIVE tensor-memory columns, so after a 32-column load lane c
// holds, for each of the 32 / V vector-rows the load covers, exactly the V outputs of mask entry (vector-row, c) in
// the order they have in memory: a lane that has such an entry writes them with one vector store.  Whether it has,
// and which entry index j it is, comes from the mask as bits that the plan kernel lays out: per (vector-row, 32 columns) a word
// with a bit for each column it names and the index of the first of them.  A warp samples 32 neighbouring columns, so a word
// serves all its lanes, and j is that index plus the set bits below the lane's.  (Before, a lane looked up a word per (32 vector-rows, column)
// and then the index of each entry in a list ordered by column, which the plan had to make: 160 -> 156 us at 256 x (2048 x 512), k = 256, V = 8,
// 90 % sparse; 146 x (1008 x 1361), k = 128, V = 4 82 -> 78.)  Finding the entries ahead of the accumulator and without branches counts: by shuffles
// between the stores 88 us in the latter, with a branch for each 100, from shared memory 94.  No shared-memory boxes, no dynamic register indexing, nothing
// outside the mask is ever stored, so non-finite products elsewhere in the tile cannot leak.  A bit holds
// one entry: when the same column appears twice in a vector-row the plan kernel says so and a fix-up kernel copies
// the written entry's outputs to its twins (their values are equal by definition).
//
// Operand traffic.  With both operands streamed every SM takes 32 KiB from L2 per 540 cycles of tensor work.  When the
// rhs of one batch entry fits eight of the CTA's fourteen 16 KiB operand slots (n / 256 x k / 64 <= 8 tiles per CTA) it
// stays in shared memory instead: a pair then takes a contiguous run of work items (batch entry, row tile, column
// tile; column tiles fastest), a tile of rhs is loaded when a batch entry first needs it and is reused by every row
// tile of lhs, and only lhs streams through the remaining slots (0.64 GB instead of 1.07 GB from L2 per call at
// lhs 2048 x 256, rhs 512 x 256, 256 batch entries).  Otherwise both operands stream through rings of seven slots and
// the pairs interleave (items pair, pair + pairs, ...), so that neighbours read the same tiles at the same time.
// Measured on B200 at that shape (ms per call; the single-CTA kernel: 0.174): both modes 0.134-0.139.  With the loads
// switched off (timing experiment) 0.129 -> 0.094 and the SM clock rises from ~1.5-1.7 to 1.97 GHz: the part runs this
// kernel at its power cap, and a good part of what the loads "cost" is clock.  Handing the accumulator back early
// changes nothing.  What did not help: asking tiles into L2 two items ahead, by TMA prefetches from the loader (13 %
// slower) or by plain prefetch instructions from a warp of its own (no change); rings of 4, 6 or 7 stages (within
// 2 %); 128-row lhs tiles shared by two column tiles, which halves the bytes per stage but needs twice the MMA
// instructions (0.154); reading a warp's 64 accumulator columns with one wait instead of two (0.141-0.145, spills).
//
// Organisation per CTA (both CTAs of a pair run the same roles on their own halves):
//   warps 0-15  sampling epilogue: warp (quarter, part) owns accumulator lanes 32 quarter .. (32 mask columns) and
//               tensor-memory columns 64 part .. + 63 (64 rows of lhs); words are fetched one work item ahead
//   warp 16     one thread issuing the CTA's loads.  They are cta_group::2 loads: the tile lands in the issuing CTA, the
//               bytes are counted on the FIRST CTA's barrier, which that CTA's loader arms with the bytes of both
//   warp 17     first CTA: the MMA-issuing thread of the pair (idle in the second); its commits arrive on the barriers of
//               both CTAs at once, so that no thread has to forward anything
// Every wait is bounded; a wait that runs out raises the abort flag of both CTAs, all roles fall through, a status
// bit is set, both CTAs meet at the final cluster barrier and tensor memory is freed.
#pragma once
#include <cuda.h>

#include "common.cuh"
#include "sddmm_dense.cuh"
#include "spmm_pair.cuh"
#include "tc_ptx.cuh"

namespace vs {
namespace pairsddmm {

using densesddmm::kBlockK;
using densesddmm::kStatusTimeout;
using pairspmm::abort_pair;
using pairspmm::wait_or_abort;

constexpr int kTile = 256;                                // mask columns and rows of lhs per work item: 128 + 128 per pair
constexpr int kCtaRows = 128;
constexpr int kSlots = 14;                                // operand slots of 16 KiB per CTA
constexpr int kMaxResident = 8;                           // of them, at most this many hold a resident rhs
constexpr int kEpiWarps = 16;                             // TMEM lane quarter = warp % 4, 64 tensor-memory columns = warp / 4
constexpr int kLoadWarp = kEpiWarps;
constexpr int kMmaWarp = kLoadWarp + 1;
constexpr int kThreads = (kMmaWarp + 1) * 32;             // 576
constexpr int kOperandBytes = kCtaRows * kBlockK * 2;     // 16 KiB: 128 rows of either operand, 64 contraction elements
constexpr int kTmemCols = 2 * kTile;                      // two accumulator buffers
constexpr int kPlanWarps = 8, kPlanThreads = 32 * kPlanWarps;
constexpr int kTwinThreads = 1024;
constexpr int kMaxPlanColumns = 8192;                     // mask widths the plan kernel holds in shared memory
constexpr int kSleepLoad = 32, kSleepMma = 0, kSleepEpilogue = 32;

struct Smem {  // offsets from the 1024-byte aligned base; identical in both CTAs of a pair
    static constexpr int kOperands = 0;                   // kSlots slots: the ring of lhs tiles first, the rhs tiles behind it
    static constexpr int kBarFull = kOperands + kSlots * kOperandBytes;
    static constexpr int kBarDone = kBarFull + kSlots * 8;
    static constexpr int kBarAccFull = kBarDone + kSlots * 8;
    static constexpr int kBarAccEmpty = kBarAccFull + 2 * 8;
    static constexpr int kTmemHolder = kBarAccEmpty + 2 * 8;
    static constexpr int kAbort = kTmemHolder + 8;
    static constexpr int kTotal = kAbort + 8;
};
constexpr int kSmemBytes = Smem::kTotal;   // the dynamic segment is 1024-byte aligned (nothing static lies ahead of it)
static_assert(kSmemBytes <= 227 * 1024, "shared memory budget");

// The work items of one pair, as (batch entry, row tile of lhs, column tile of the mask).  With a resident rhs: a
// contiguous run of items, column tiles fastest, so that the pair stays with one batch entry as long as it can.
// Otherwise items pair, pair + pairs, ... with row tiles fastest, so that neighbouring pairs read the same rhs tile
// at the same time.  Walked with carries instead of divisions.
struct ItemWalk {
    int x0, x1, b, r0, r1, s0, s1, s2;
    bool nt_fast;
    __device__ __forceinline__ void init(int64_t w, int64_t stride, int m_tiles, int n_tiles, bool nt_fast_) {
        nt_fast = nt_fast_;
        r0 = nt_fast ? n_tiles : m_tiles;
        r1 = nt_fast ? m_tiles : n_tiles;
        x0 = (int)(w % r0);
        const int64_t q = w / r0;
        x1 = (int)(q % r1);
        b = (int)(q / r1);
        s0 = (int)(stride % r0);
        const int64_t sq = stride / r0;
        s1 = (int)(sq % r1);
        s2 = (int)(sq / r1);
    }
    __device__ __forceinline__ void next() {
        x0 += s0; x1 += s1; b += s2;
        if (x0 >= r0) { x0 -= r0; ++x1; }
        if (x1 >= r1) { x1 -= r1; ++b; }
    }
    __device__ __forceinline__ int mt() const { return nt_fast ? x1 : x0; }
    __device__ __forceinline__ int nt() const { return nt_fast ? x0 : x1; }
};

// ---- plan -------------------------------------------------------------------------------------------------
// The mask as bits: words[row * ceil(n / 32) + w] = (a bit per column 32 w .. 32 w + 31 that the vector-row names, the index of the first such
// entry).  Where a vector-row's columns ascend, entry number r of the row is its r-th set bit, and that is all; the others (columns in another
// order, named twice, or outside [0, n), which are dropped: their outputs are not written) have bit 31 of the index set, and the entry
// itself stands in `order` at that index.  twins[CTA] is set where a vector-row names a column twice (only one of the two reaches `order`).
//
// kShare warps take a vector-row together, so the plan takes the whole GPU.  The form before, a CTA per 32 vector-rows that ordered their entries by
// column, took 1.1 ns an entry of such a block: 80 us for 824 vector-rows of 1920 entries, 62 for 267 of 1520 skewed ones; now 10.5 and 6.4, of which 4 are a
// launch by itself.  Lanes that first put the bits of a word together, by shuffles or by a match, take longer than atomics that wait for each other.
template <int kShare>
__global__ void __launch_bounds__(kPlanThreads)
sddmm_cell_plan_kernel(const int32_t *__restrict__ row_offsets, const int32_t *__restrict__ col_indices, int m_vec, int n, int nnz_vec,
                       uint2 *__restrict__ words, int32_t *__restrict__ order, int32_t *__restrict__ twins) {
    static_assert(kShare == 1 || kShare == kPlanWarps, "a warp or the CTA");
    extern __shared__ uint32_t plan_sh[];   // per vector-row: bits, then positions
    __shared__ int warp_sum[kPlanWarps];
    pdl_launch_dependents();   // the multiplying kernel may set itself up while the plan is made
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, n_words = (n + 31) / 32;
    const int w0 = kShare == 1 ? 0 : warp, slot = kShare == 1 ? warp : 0;
    uint32_t *bits = plan_sh + slot * 2 * n_words, *first = bits + n_words;
    auto sync = [&]() {
        if constexpr (kShare == 1) __syncwarp();
        else __syncthreads();
    };
    pdl_wait();
    bool twin = false;
    for (int row = blockIdx.x * (kPlanWarps / kShare) + slot; row < m_vec; row += gridDim.x * (kPlanWarps / kShare)) {
        // the scratch holds nnz_vec entries (the caller's count): offsets that claim more are cut there
        const int beg = min(max(__ldg(row_offsets + row), 0), nnz_vec), end = min(max(__ldg(row_offsets + row + 1), beg), nnz_vec);
        for (int w = w0 * 32 + lane; w < n_words; w += 32 * kShare) bits[w] = 0u;
        sync();
        constexpr int kAhead = kShare == 1 ? 8 : 4;   // entries per lane whose loads fly together
        bool plain = true;
        for (int j0 = beg + w0 * 32 * kAhead; j0 < end; j0 += 32 * kAhead * kShare) {
            int c[kAhead], before = j0 > beg ? __ldg(col_indices + j0 - 1) : -1;
#pragma unroll
            for (int u = 0; u < kAhead; ++u) c[u] = __ldg(col_indices + min(j0 + 32 * u + lane, end - 1));
#pragma unroll
            for (int u = 0; u < kAhead; ++u) {
                int left = __shfl_up_sync(0xffffffffu, c[u], 1);
                if (lane == 0) left = before;
                before = __shfl_sync(0xffffffffu, c[u], 31);
                if (j0 + 32 * u + lane < end) {
                    plain = plain && c[u] > left && c[u] < n;
                    if ((unsigned)c[u] < (unsigned)n) atomicOr(bits + (c[u] >> 5), 1u << (c[u] & 31));
                }
            }
        }
        if constexpr (kShare == 1) {
            plain = __all_sync(0xffffffffu, plain);
            __syncwarp();
        } else {
            plain = __syncthreads_and(plain);
        }
        int run = beg;
        for (int x0 = 0; x0 < n_words; x0 += 32 * kShare) {
            const int w = x0 + w0 * 32 + lane;
            const uint32_t mine = w < n_words ? bits[w] : 0u;
            int sum = __popc(mine);
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int up = __shfl_up_sync(0xffffffffu, sum, d);
                if (lane >= d) sum += up;
            }
            int ahead = 0, total = __shfl_sync(0xffffffffu, sum, 31);
            if constexpr (kShare > 1) {
                if (lane == 0) warp_sum[warp] = total;
                __syncthreads();
                total = 0;
#pragma unroll
                for (int x = 0; x < kShare; ++x) {
                    if (x == warp) ahead = total;
                    total += warp_sum[x];
                }
                __syncthreads();
            }
            if (w < n_words) {
                const uint32_t at = (uint32_t)(run + ahead + sum - __popc(mine));
                words[(int64_t)row * n_words + w] = make_uint2(mine, plain ? at : at | 0x80000000u);
                first[w] = at;
            }
            run += total;
        }
        sync();
        if (!plain) {   // the same for all that share the row
            int named = 0;   // entries with a column of the matrix; more than set bits where one is named twice
            for (int j = beg + lane; j < end; j += 32) {
                const int c = __ldg(col_indices + j);
                if ((unsigned)c >= (unsigned)n) continue;
                ++named;
                if (w0 == 0) order[first[c >> 5] + __popc(bits[c >> 5] & ((1u << (c & 31)) - 1u))] = j;   // of twins one stays
            }
            twin = twin || (int)__reduce_add_sync(0xffffffffu, named) != run - beg;
        }
        sync();
    }
    twin = __syncthreads_or(twin);
    if (threadIdx.x == 0) twins[blockIdx.x] = twin;
}

// Runs behind the multiplying kernel; does nothing unless the plan kernel met a column twice in one vector-row.
// Entry j whose place in `order` holds another entry j' is a twin of j': same vector-row, same column, same outputs.
template <typename TOut, int V>
__global__ void __launch_bounds__(kTwinThreads)
sddmm_twin_kernel(const SddmmParams p, const uint2 *__restrict__ words, const int32_t *__restrict__ order, const int32_t *__restrict__ twins, int plan_ctas) {
    pdl_wait();
    int any = 0;
    for (int i = threadIdx.x; i < plan_ctas; i += kTwinThreads) any |= twins[i];
    if (__syncthreads_or(any) == 0) return;
    const int n_words = (p.n + 31) / 32;
    for (int64_t j = (int64_t)blockIdx.x * kTwinThreads + threadIdx.x; j < p.nnz_vec; j += (int64_t)gridDim.x * kTwinThreads) {
        const int c = __ldg(p.col_indices + j);
        if ((unsigned)c >= (unsigned)p.n) continue;
        int lo = 0, hi = p.m_vec;
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (__ldg(p.row_offsets + mid) <= j) lo = mid; else hi = mid;
        }
        const uint2 word = __ldg(words + (int64_t)lo * n_words + (c >> 5));
        // an entry behind the last row's (the caller may count more than the offsets do) need not be in the row found: `order` names none there
        if (!(word.y >> 31) || !(word.x >> (c & 31) & 1u)) continue;
        const int other = __ldg(order + (word.y & 0x7fffffffu) + __popc(word.x & ((1u << (c & 31)) - 1u)));
        if (other == j) continue;
        for (int b = 0; b < p.batch; ++b) {
            TOut *out = static_cast<TOut *>(p.out) + (int64_t)b * p.stride_out;
            for (int v = 0; v < V; ++v) out[(int64_t)j * V + v] = out[(int64_t)other * V + v];
        }
    }
}

// map_lhs: {k, rows of lhs, batch}, map_rhs: {k, n, batch}; both box {64, 128, 1}, K-major with the 128-byte swizzle
// and zero fill outside.  words / order: see sddmm_cell_plan_kernel.
// resident: keep the rhs tiles of the current batch entry in shared memory (the host checks that they fit).
template <typename TOut, int V>
__global__ void __launch_bounds__(kThreads, 1)
sddmm_pair_kernel(const SddmmParams p, const __grid_constant__ CUtensorMap map_lhs, const __grid_constant__ CUtensorMap map_rhs,
                  const uint2 *__restrict__ words, const int32_t *__restrict__ order, int m_tiles, int n_tiles,
                  int resident, uint32_t *status) {
    extern __shared__ __align__(1024) uint8_t sm[];
    const uint32_t base = tc::smem_u32(sm);   // the same offset in both CTAs

    const int t = threadIdx.x;
    const int warp = t >> 5;
    const int lane = t & 31;
    const uint32_t rank = tc::cluster_ctarank();   // 0: the CTA that issues the MMAs
    const uint32_t peer = rank ^ 1u;
    const uint32_t pair = tc::cluster_id_x(), pairs = tc::cluster_count_x();
    volatile int *abort_flag = reinterpret_cast<volatile int *>(sm + Smem::kAbort);
    const uint32_t abort_addr = base + Smem::kAbort;
    const uint32_t bar_full = base + Smem::kBarFull;
    const uint32_t bar_done = base + Smem::kBarDone;
    const uint32_t bar_acc_full = base + Smem::kBarAccFull;
    const uint32_t bar_acc_empty = base + Smem::kBarAccEmpty;

    if (t == 0) {
        for (int s = 0; s < kSlots; ++s) {
            tc::mbar_init(bar_full + 8 * s, 1);   // first CTA only: its loader's arrival + the bytes of BOTH CTAs' tiles
            tc::mbar_init(bar_done + 8 * s, 1);   // a commit of the MMA-issuing thread, which arrives in both CTAs
        }
        for (int s = 0; s < 2; ++s) {
            tc::mbar_init(bar_acc_full + 8 * s, 1);
            tc::mbar_init(bar_acc_empty + 8 * s, 2 * kEpiWarps);   // one lane per epilogue warp of both CTAs; first CTA only
        }
        *abort_flag = 0;
        tc::fence_mbar_init();
    }
    if (warp == kMmaWarp) {
        tc::tmem_alloc_pair(base + Smem::kTmemHolder, kTmemCols);
        tc::tmem_relinquish_pair();
    }
    tc::fence_proxy_async();
    tc::tc_fence_before_sync();
    tc::cluster_sync();   // barriers and flags of BOTH CTAs exist before anything crosses between them
    tc::tc_fence_after_sync();
    const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t *>(sm + Smem::kTmemHolder);

    pdl_launch_dependents();
    pdl_wait();   // the set-up above may have run beside the plan kernel; its words are read from here on
    const int k_blocks = (p.k + kBlockK - 1) / kBlockK;   // the last one may be filled up with zeros by TMA
    const int64_t total_items = (int64_t)p.batch * n_tiles * m_tiles;
    // this pair's items: a contiguous run with a resident rhs, every pairs-th item otherwise
    const int64_t item0 = resident ? total_items * pair / pairs : (int64_t)pair;
    const int64_t item_stride = resident ? 1 : (int64_t)pairs;
    const uint32_t my_items = resident ? (uint32_t)(total_items * (pair + 1) / pairs - item0)
                                       : (total_items > pair ? (uint32_t)((total_items - pair + pairs - 1) / pairs) : 0u);
    const uint32_t total_stages = my_items * (uint32_t)k_blocks;
    // Stage g = (item g / k_blocks, contraction block g % k_blocks).  Its lhs tile goes through ring slot g % ring; its
    // rhs tile sits in slot ring + nt * k_blocks + kb when rhs is resident, in slot ring + g % ring otherwise.
    const uint32_t ring = resident ? (uint32_t)(kSlots - n_tiles * k_blocks) : (uint32_t)(kSlots / 2);
    const uint32_t rhs_slots = base + Smem::kOperands + ring * kOperandBytes;

    if (warp == kLoadWarp) {
        // =========================== loader ==============================================================
        if (lane == 0) {
            bool ok_run = true;
            const uint32_t full_first = tc::map_to_cta(bar_full, 0);
            ItemWalk walk;
            walk.init(item0, item_stride, m_tiles, n_tiles, resident != 0);
            int res_b = -1;                       // the batch entry whose rhs tiles are in the resident slots
            uint32_t valid = 0;                   // which of them have been loaded for it
            uint32_t last_use[kMaxResident];      // the last stage that read each resident slot
#pragma unroll
            for (int i = 0; i < kMaxResident; ++i) last_use[i] = 0u;
            uint32_t used = 0;
            uint32_t g = 0;
            for (uint32_t i = 0; i < my_items && ok_run; ++i, walk.next()) {
                for (int kb = 0; kb < k_blocks && ok_run; ++kb, ++g) {
                    const uint32_t slot = g % ring;
                    if (g >= ring)   // the stage that used this ring slot before must have been multiplied
                        ok_run = wait_or_abort<kSleepLoad>(bar_done + 8 * slot, ((g - ring) / ring) & 1u, abort_flag, abort_addr, peer);
                    if (!ok_run) break;
                    bool need_rhs = true;
                    uint32_t rs = slot;
                    if (resident) {
                        if (walk.b != res_b) { res_b = walk.b; valid = 0u; }
                        rs = (uint32_t)(walk.nt() * k_blocks + kb);
                        need_rhs = ((valid >> rs) & 1u) == 0u;
                        if (need_rhs) {
                            // the previous batch entry's tile in this slot: its last reader may be one of the stages
                            // the ring wait above does not cover yet
                            const uint32_t old = last_use[rs];
                            if (((used >> rs) & 1u) && old + ring > g)
                                ok_run = wait_or_abort<kSleepLoad>(bar_done + 8 * (old % ring), (old / ring) & 1u, abort_flag, abort_addr, peer);
                            if (!ok_run) break;
                            valid |= 1u << rs;
                        }
                        last_use[rs] = g;
                        used |= 1u << rs;
                    }
                    // both CTAs load the same amounts and count them on the FIRST CTA's barrier, which its loader arms
                    const uint32_t bar = full_first + 8 * slot;
                    if (rank == 0) tc::mbar_expect_tx(bar_full + 8 * slot, (uint32_t)((need_rhs ? 4 : 2) * kOperandBytes));
                    tc::tma_load_3d_pair(base + Smem::kOperands + slot * kOperandBytes, &map_lhs, bar, kb * kBlockK,
                                         walk.mt() * kTile + (int)rank * kCtaRows, walk.b);
                    if (need_rhs)
                        tc::tma_load_3d_pair(rhs_slots + rs * kOperandBytes, &map_rhs, bar, kb * kBlockK,
                                             walk.nt() * kTile + (int)rank * kCtaRows, walk.b);
                }
            }
            // the last "multiplied" signals addressed to this CTA must not arrive after it has gone
            const uint32_t tail0 = total_stages > ring ? total_stages - ring : 0u;
            for (uint32_t q = tail0; q < total_stages && ok_run; ++q)
                ok_run = wait_or_abort<kSleepLoad>(bar_done + 8 * (q % ring), (q / ring) & 1u, abort_flag, abort_addr, peer);
        }
    } else if (warp == kMmaWarp) {
        if (lane == 0 && rank == 0) {
            // =========================== MMA issuer of the pair ==========================================
            const uint32_t a_lo0 = tc::smem_desc_lo(rhs_slots, 16);                       // M operand: rows of rhs
            const uint32_t b_lo0 = tc::smem_desc_lo(base + Smem::kOperands, 16);          // N operand: rows of lhs
            const uint32_t hi = tc::smem_desc_hi(1024, (uint32_t)tc::kSwizzle128B);       // K-major: 8-row groups 1 KiB apart
            const uint32_t idesc = tc::make_idesc_f16(kTile, kTile, 0, 0);                // both operands K-major
            uint32_t slot = 0, parity = 0;
            bool ok_run = true;
            ItemWalk walk;
            walk.init(item0, item_stride, m_tiles, n_tiles, resident != 0);
            for (uint32_t i = 0; i < my_items && ok_run; ++i, walk.next()) {
                const uint32_t buf = i & 1u;
                ok_run = wait_or_abort<kSleepMma>(bar_acc_empty + 8 * buf, (i >> 1) & 1u, abort_flag, abort_addr, peer);
                if (!ok_run) break;
                tc::tc_fence_after_sync();
                const uint32_t d = tmem_base + buf * kTile;
                for (int kb = 0; kb < k_blocks; ++kb) {
                    ok_run = wait_or_abort<kSleepMma>(bar_full + 8 * slot, parity, abort_flag, abort_addr, peer);
                    if (!ok_run) break;
                    // no tensor-core fence per stage: the operands were written by TMA, whose completion the barrier carries
                    const uint32_t rs = resident ? (uint32_t)(walk.nt() * k_blocks + kb) : slot;
                    const uint32_t a_lo = a_lo0 + rs * (kOperandBytes >> 4), b_lo = b_lo0 + slot * (kOperandBytes >> 4);
#pragma unroll
                    for (int kk = 0; kk < kBlockK / 16; ++kk)   // 16 contraction elements = 32 bytes along a row
                        tc::mma_f16_ss_pair(d, tc::desc64(a_lo + 2 * kk, hi), tc::desc64(b_lo + 2 * kk, hi), idesc,
                                            (kb > 0 || kk > 0) ? 1u : 0u);
                    tc::mma_commit_pair_both(bar_done + 8 * slot);      // "stage multiplied", to both CTAs' loaders
                    if (++slot == ring) { slot = 0; parity ^= 1u; }
                }
                if (ok_run) tc::mma_commit_pair_both(bar_acc_full + 8 * buf);   // "accumulator complete", to both CTAs' epilogues
            }
        }
    } else {
        // =========================== sampling epilogue ===================================================
        // This lane's mask column is nt * 256 + 128 rank + 32 quarter + lane; the warp's 64 tensor-memory columns are
        // rows 64 part .. + 63 of the lhs tile = 64 / V vector-rows, read by two 32-column loads of 32 / V vector-rows
        // each.  The warp's 32 mask columns are ONE word of each of those vector-rows: a lane fetches the word of vector-row `lane`
        // (at V = 1 of `lane` + 32 too), an item ahead, and they are passed round when they are sampled.
        constexpr int kPerLoad = 32 / V;                 // vector-rows per 32-column load
        constexpr int kHeld = 2 * kPerLoad > 32 ? 2 : 1; // words a lane holds
        constexpr bool kAheadEntries = 2 * kPerLoad <= 16;   // the entries are found before the accumulator is waited for; at V <= 2 there are too many to hold
        constexpr int kElems = 16 / (int)sizeof(TOut);   // outputs per 16-byte store
        const int quarter = warp & 3, part = warp >> 2;
        const uint32_t lane_taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(part * 64);
        const uint32_t acc_empty_first = tc::map_to_cta(bar_acc_empty, 0);
        if (lane == 0) {
            tc::mbar_arrive_remote(acc_empty_first);        // both accumulator buffers start out free
            tc::mbar_arrive_remote(acc_empty_first + 8);
        }
        const int n_words = (p.n + 31) / 32;
        auto words_of = [&](const ItemWalk &w, bool valid, uint2 (&held)[kHeld]) {
            const int cw = (w.nt() * kTile + (int)rank * kCtaRows) / 32 + quarter;
            const int vr = (w.mt() * kTile + part * 64) / V + lane;   // first vector-row this warp samples + lane
#pragma unroll
            for (int i = 0; i < kHeld; ++i)
                held[i] = valid && cw < n_words && lane < 2 * kPerLoad && vr + 32 * i < p.m_vec ? __ldg(words + (int64_t)(vr + 32 * i) * n_words + cw) : make_uint2(0u, 0u);
        };
        ItemWalk walk, ahead;   // `walk`: the item being sampled; `ahead`: one item further on
        walk.init(item0, item_stride, m_tiles, n_tiles, resident != 0);
        ahead = walk;
        uint2 held[kHeld], next[kHeld];
        words_of(ahead, my_items > 0, held);
        bool ok_run = true;
        for (uint32_t i = 0; i < my_items && ok_run; ++i, walk.next()) {
            const uint32_t buf = i & 1u;
            ahead.next();
            words_of(ahead, i + 1 < my_items, next);
            // entries named in `order`: rare, and the same for the whole warp
            bool listed = false;
#pragma unroll
            for (int x = 0; x < kHeld; ++x) listed = listed || __any_sync(0xffffffffu, held[x].y >> 31);
            auto entry_of = [&](uint32_t bits, uint32_t first) -> int {   // the lane's entry in a word, or -1; no branches, which the lanes would take one by one
                const int j = (int)((first & 0x7fffffffu) + __popc(bits & ((1u << lane) - 1u)));
                return bits >> lane & 1u ? j : -1;
            };
            int ent[kAheadEntries ? 2 * kPerLoad : 1];
            if constexpr (kAheadEntries) {
#pragma unroll
                for (int b = 0; b < 2 * kPerLoad; ++b) ent[b] = entry_of(__shfl_sync(0xffffffffu, held[0].x, b), __shfl_sync(0xffffffffu, held[0].y, b));
                if (listed) {
#pragma unroll
                    for (int b = 0; b < 2 * kPerLoad; ++b)
                        if (__shfl_sync(0xffffffffu, held[0].y, b) >> 31 && ent[b] >= 0) ent[b] = __ldg(order + ent[b]);
                }
            }
            ok_run = __all_sync(0xffffffffu, wait_or_abort<kSleepEpilogue>(bar_acc_full + 8 * buf, (i >> 1) & 1u, abort_flag, abort_addr, peer));
            if (!ok_run) break;
            tc::tc_fence_after_sync();
            TOut *out = static_cast<TOut *>(p.out) + (int64_t)walk.b * p.stride_out;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint2 half = held[kHeld == 2 ? h : 0];
                const int row0 = kHeld == 2 ? 0 : h * kPerLoad;   // the lane that holds the half's first word
                if (!__any_sync(0xffffffffu, half.x != 0u && lane >= row0 && lane < row0 + kPerLoad)) continue;   // no entry in these 32 rows
                uint32_t r[32];
                tc::tmem_ld_x32(lane_taddr + buf * kTile + (uint32_t)(h * 32), r);
#pragma unroll
                for (int b = 0; b < kPerLoad; ++b) {
                    int j;
                    if constexpr (kAheadEntries) j = ent[h * kPerLoad + b];
                    else j = entry_of(__shfl_sync(0xffffffffu, half.x, row0 + b), __shfl_sync(0xffffffffu, half.y, row0 + b));
                    if (!kAheadEntries && listed && __shfl_sync(0xffffffffu, half.y, row0 + b) >> 31 && j >= 0) j = __ldg(order + j);
                    if (j < 0) continue;
                    TOut *dst = out + (int64_t)j * V;
                    if constexpr (sizeof(TOut) == 2) {
                        if constexpr (V == 8) {
                            uint4 o;
                            __half2 *hh = reinterpret_cast<__half2 *>(&o);
#pragma unroll
                            for (int e = 0; e < 4; ++e)
                                hh[e] = __floats2half2_rn(__uint_as_float(r[b * V + 2 * e]), __uint_as_float(r[b * V + 2 * e + 1]));
                            *reinterpret_cast<uint4 *>(dst) = o;
                        } else if constexpr (V == 4) {
                            uint2 o;
                            __half2 *hh = reinterpret_cast<__half2 *>(&o);
                            hh[0] = __floats2half2_rn(__uint_as_float(r[b * V]), __uint_as_float(r[b * V + 1]));
                            hh[1] = __floats2half2_rn(__uint_as_float(r[b * V + 2]), __uint_as_float(r[b * V + 3]));
                            *reinterpret_cast<uint2 *>(dst) = o;
                        } else if constexpr (V == 2) {
                            *reinterpret_cast<__half2 *>(dst) = __floats2half2_rn(__uint_as_float(r[b * V]), __uint_as_float(r[b * V + 1]));
                        } else {
                            *dst = __float2half_rn(__uint_as_float(r[b]));
                        }
                    } else {
                        if constexpr (V >= 4) {
#pragma unroll
                            for (int e = 0; e < V / kElems; ++e)
                                reinterpret_cast<uint4 *>(dst)[e] = make_uint4(r[b * V + 4 * e], r[b * V + 4 * e + 1], r[b * V + 4 * e + 2], r[b * V + 4 * e + 3]);
                        } else if constexpr (V == 2) {
                            *reinterpret_cast<uint2 *>(dst) = make_uint2(r[b * V], r[b * V + 1]);
                        } else {
                            *reinterpret_cast<uint32_t *>(dst) = r[b];
                        }
                    }
                }
            }
            tc::tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive_remote(acc_empty_first + 8 * buf);   // sampled: the buffer is free for the pair
#pragma unroll
            for (int x = 0; x < kHeld; ++x) held[x] = next[x];
        }
    }

    // ---- teardown ---------------------------------------------------------------------------------------
    tc::tc_fence_before_sync();
    __syncthreads();
    if (*abort_flag) {
        for (int i = 0; i < 64; ++i) __nanosleep(1000);   // copies that may still be in flight
        if (t == 0) atomicOr(status, kStatusTimeout);
    }
    tc::cluster_sync();   // neither CTA's shared or tensor memory goes away while the other half of an MMA may use it
    if (warp == kMmaWarp) tc::tmem_dealloc_pair(tmem_base, kTmemCols);
}

}  // namespace pairsddmm
}  // namespace vs
