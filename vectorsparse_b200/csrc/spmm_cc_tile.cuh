// fp32 SpMM on CUDA cores from staged tiles of the dense operand, V = 1/2/4/8, for grids of about one CTA per SM.
//
// spmm_cc_kernel gives a thread up to 16 dense columns, so a product of a few hundred vector-rows leaves it a few warps
// per SM, each of them waiting for one gather of B from L2 after another (512 x 512 x 512, V = 1, 50 % sparse: 53 us for 2 us of
// multiply-adds).  Here a CTA owns 16 vector-rows, one per warp, and a slab of 128 dense columns, four per lane, and
// walks the columns of the sparse matrix in tiles of 128: one TMA copy brings 128 rows of the slab into a ring of three
// 64 KB stages, and the warps take the rows of B that their entries name from shared memory, where they wait tens of
// cycles and not hundreds.  The entries themselves are loaded 32 at a time, one batch ahead.  Two multiply-adds go out
// per instruction (fma.rn.f32x2).  A CTA with few entries (`direct`) gathers its rows of B itself, eight in flight,
// instead of streaming a slab that it would hardly read.  What bounds it: shared-memory bandwidth (16 bytes per lane
// feed 4 V multiply-adds) at V = 1 and 2, issue at V = 4 and 8.
//
// B200, us, spmm_cc_kernel -> this one, 50 / 90 / 98 % sparse: 512 x 512 x 512 at V = 1 53 -> 17 / 20 -> 8.4 / 8.4 -> 6.3, at V = 8
// 70 -> 33 / 21 -> 12.5 / 8.4 -> 6.8; 1024 x 1024 x 1024 at V = 4 142 -> 41 / 38 -> 15 / 13.5 -> 8.4.  More vector-rows per warp, for
// larger products, 4096 x 4096 x 1024 at V = 4, 80 / 90 / 95 % sparse: 248 / 161 / 124 us with two of them, 325 / 230 / 189 with four,
// against 297 / 161 / 90, so spmm_cc_kernel keeps those (and spmm_split.cuh the denser ones).
//
// Entries are taken in the order of col_indices, so every sum is formed in the order, and with the roundings, of
// spmm_cc_kernel.  Entries whose tile has gone by (columns that are not ascending) are gathered from global memory when
// their turn comes.
#pragma once
#include <cuda.h>

#include "common.cuh"
#include "tc_ptx.cuh"

namespace vs {
namespace cctile {

constexpr int kWarps = 16;
constexpr int kThreads = 32 * kWarps;
constexpr int kStages = 3;
constexpr int kCols = 128;                      // dense columns of a slab
constexpr int kTile = 128;                      // columns of the sparse matrix per stage
constexpr int kRowBytes = 4 * kCols;
constexpr int kStageBytes = kTile * kRowBytes;
constexpr int kNone = 0x7fffffff;               // the column of a lane without an entry
constexpr uint32_t kStatusTimeout = 256u;       // bit raised in the status word when a bounded wait ran out

template <int V> struct Layout {
    static constexpr int kEntryBytes = 32 * 4 * (1 + V);        // a warp's staged entries: offsets, then values
    static constexpr int kBars = kStages * kStageBytes + kWarps * kEntryBytes;
    static constexpr int kSmemBytes = kBars + 2 * kStages * 8 + 16 + 128;   // + the CTA's entries, alignment of the ring
    static_assert(kSmemBytes <= 232448, "shared memory of one CTA");
};

__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(uint64_t x, float &lo, float &hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(x)); }
__device__ __forceinline__ void fma2(uint64_t &acc, uint64_t a, uint64_t b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
template <int V>
__global__ void __launch_bounds__(kThreads, 1)
    spmm_cc_tile_kernel(const SpmmParams p, const __grid_constant__ CUtensorMap map_b, int groups, int slabs, uint32_t *status) {
    using L = Layout<V>;
    extern __shared__ char raw[];
    char *smem = raw + ((128u - (tc::smem_u32(raw) & 127u)) & 127u);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t full = tc::smem_u32(smem + L::kBars), empty = full + 8 * kStages;
    int *s_off = reinterpret_cast<int *>(smem + kStages * kStageBytes + warp * L::kEntryBytes);
    float *s_val = reinterpret_cast<float *>(s_off + 32);

    // row groups run fastest: the CTAs that are resident together share slabs of B in L2
    const int group = blockIdx.x % groups;
    const int rest = blockIdx.x / groups;
    const int slab = rest % slabs, b = rest / slabs;
    const int x0 = slab * kCols;
    int tiles = (p.K + kTile - 1) / kTile;
    const int zb = p.stride_rhs == 0 ? 0 : b;

    auto issue = [&](int t) {
        const uint32_t bar = full + 8 * (t % kStages);
        tc::mbar_expect_tx(bar, kStageBytes);
        tc::tma_load_3d(tc::smem_u32(smem + (t % kStages) * kStageBytes), &map_b, bar, x0, t * kTile, zb);
    };
    const float *values = static_cast<const float *>(p.values) + (int64_t)b * p.stride_values;

    // Vector-rows are dealt out in the order of row_indices (longest first), one to each CTA in turn, so that all of them
    // get long ones and short ones.
    const int order = warp * groups + group;
    const int row = order < p.m_vec ? __ldg(p.row_indices + order) : -1;
    int cur = row >= 0 ? __ldg(p.row_offsets + row) : 0;
    const int end = row >= 0 ? __ldg(p.row_offsets + row + 1) : 0;

    // A CTA with few entries gathers their rows of B itself instead of streaming the whole slab: nothing is staged and
    // every column counts as gone by.
    int *s_total = reinterpret_cast<int *>(smem + L::kBars + 2 * kStages * 8);
    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            tc::mbar_init(full + 8 * s, 1);
            tc::mbar_init(empty + 8 * s, kWarps);
        }
        tc::fence_mbar_init();
        *s_total = 0;
    }
    __syncthreads();
    if (lane == 0) atomicAdd(s_total, end - cur);
    __syncthreads();
    // 0.8 K entries: both ways measured alike at 95 % sparsity (V = 1 to 8), where 16 rows hold 0.8 K; at 98 % gathering took
    // 0.5 to 0.9 of the time, at 90 % streaming did
    const bool direct = (int64_t)*s_total * 5 < (int64_t)p.K * 4;
    if (direct) tiles = 1;
    else if (threadIdx.x == 0)
        for (int t = 0; t < kStages && t < tiles; ++t) issue(t);

    uint64_t acc[V][2];
#pragma unroll
    for (int v = 0; v < V; ++v) acc[v][0] = acc[v][1] = 0;

    // the next 32 entries of the row, one per lane, are on their way while the entries before them are multiplied
    int col = kNone;
    float val[V];
#pragma unroll
    for (int v = 0; v < V; ++v) val[v] = 0.f;
    auto fetch = [&]() {
        const int j = cur + lane;
        col = kNone;
        if (j < end) {
            col = __ldg(p.col_indices + j);
            VecLoad<float, V>::load(values + (int64_t)j * V, val);
        }
    };
    fetch();

    bool ok = true;
    int t = 0;
    for (; t < tiles; ++t) {
        const int s = t % kStages;
        if (!direct && !__all_sync(0xffffffffu, tc::mbar_wait(full + 8 * s, (t / kStages) & 1))) { ok = false; break; }
        const char *tile = smem + s * kStageBytes + lane * 16;
        const int lo = direct ? kNone : t * kTile;
        bool more;
        do {
            // a run of entries of this tile, or a run of entries whose tiles have gone by: up to the first of another kind
            const unsigned gone = __ballot_sync(0xffffffffu, col < lo);
            const unsigned here = __ballot_sync(0xffffffffu, col >= lo && col - lo < kTile && col != kNone);
            const bool first_gone = gone & 1u;
            const unsigned stop = ~(first_gone ? gone : here);
            const int count = stop ? __ffs(stop) - 1 : 32;
            s_off[lane] = first_gone ? col : (int)((unsigned)(col - lo) * kRowBytes);
            if constexpr (V == 1) {
                s_val[lane] = val[0];
            } else if constexpr (V == 2) {
                reinterpret_cast<float2 *>(s_val)[lane] = make_float2(val[0], val[1]);
            } else {
#pragma unroll
                for (int q = 0; q < V / 4; ++q)
                    reinterpret_cast<float4 *>(s_val)[lane * (V / 4) + q] = make_float4(val[4 * q], val[4 * q + 1], val[4 * q + 2], val[4 * q + 3]);
            }
            cur += count;
            more = !stop || ((gone | here) >> count & 1u);   // the run has ended, this tile's part of the row has not
            fetch();
            __syncwarp();
            auto multiply = [&](const float (&a)[V], const ulonglong2 &f) {
#pragma unroll
                for (int v = 0; v < V; ++v) {
                    const uint64_t av = pack2(a[v], a[v]);
                    fma2(acc[v][0], av, f.x);
                    fma2(acc[v][1], av, f.y);
                }
            };
            auto run = [&](int i, auto n) {   // n entries from the i-th, a multiple of n: all loads, then all sums
                constexpr int U = decltype(n)::value;
                int off[U];
                float a[U][V];
                ulonglong2 f[U];
                if constexpr (U == 4) {
                    const int4 o = *reinterpret_cast<const int4 *>(s_off + i);
                    off[0] = o.x; off[1] = o.y; off[2] = o.z; off[3] = o.w;
                } else if constexpr (U == 2) {
                    const int2 o = *reinterpret_cast<const int2 *>(s_off + i);
                    off[0] = o.x; off[1] = o.y;
                } else {
                    off[0] = s_off[i];
                }
                float w[U * V];
                if constexpr (U * V >= 4) {
#pragma unroll
                    for (int q = 0; q < U * V / 4; ++q) {
                        const float4 x = reinterpret_cast<const float4 *>(s_val + i * V)[q];
                        w[4 * q] = x.x; w[4 * q + 1] = x.y; w[4 * q + 2] = x.z; w[4 * q + 3] = x.w;
                    }
                } else if constexpr (U * V == 2) {
                    const float2 x = *reinterpret_cast<const float2 *>(s_val + i * V);
                    w[0] = x.x; w[1] = x.y;
                } else {
                    w[0] = s_val[i];
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    f[u] = *reinterpret_cast<const ulonglong2 *>(tile + off[u]);
#pragma unroll
                    for (int v = 0; v < V; ++v) a[u][v] = w[u * V + v];
                }
#pragma unroll
                for (int u = 0; u < U; ++u) multiply(a[u], f[u]);
            };
            if (!first_gone) {
                int i = 0;
                for (; i + 4 <= count; i += 4) run(i, std::integral_constant<int, 4>());
                if (count & 2) { run(i, std::integral_constant<int, 2>()); i += 2; }
                if (count & 1) run(i, std::integral_constant<int, 1>());
            } else if (x0 + lane * 4 < p.N) {
                const float *rhs = static_cast<const float *>(p.rhs) + (int64_t)b * p.stride_rhs + x0 + lane * 4;
                constexpr int U = V >= 8 ? 4 : 8;   // rows of B in flight
                for (int i = 0; i < count; i += U) {
                    ulonglong2 f[U];
#pragma unroll
                    for (int u = 0; u < U; ++u)
                        if (i + u < count) f[u] = __ldg(reinterpret_cast<const ulonglong2 *>(rhs + (int64_t)s_off[i + u] * p.N));
#pragma unroll
                    for (int u = 0; u < U; ++u)
                        if (i + u < count) {
                            float a[V];
#pragma unroll
                            for (int v = 0; v < V; ++v) a[v] = s_val[(i + u) * V + v];
                            multiply(a, f[u]);
                        }
                }
            }
            __syncwarp();
        } while (more);
        if (direct) break;
        if (lane == 0) tc::mbar_arrive(empty + 8 * s);
        // the tile before this one has been left by this warp a whole tile ago: the others are seldom waited for here
        if (warp == 0 && t > 0 && t - 1 + kStages < tiles) {
            if (!__all_sync(0xffffffffu, tc::mbar_wait(empty + 8 * ((t - 1) % kStages), ((t - 1) / kStages) & 1))) { ok = false; break; }
            if (lane == 0) issue(t - 1 + kStages);
        }
    }
    if (!ok) {   // no results; thread 0 leaves only when its copies have landed (or the limit is reached again)
        if (lane == 0) atomicOr(status, kStatusTimeout);
        if (threadIdx.x == 0) {
            const int issued = min(tiles, max(kStages, t - 1 + kStages));   // tiles 0 .. t - 2 were replaced
            for (int w = max(0, issued - kStages); w < issued; ++w) tc::mbar_wait(full + 8 * (w % kStages), (w / kStages) & 1);
        }
        return;
    }

    if (row < 0 || x0 + lane * 4 >= p.N) return;
    float *out = static_cast<float *>(p.out) + (int64_t)b * p.stride_out + (int64_t)row * V * p.N + x0 + lane * 4;
#pragma unroll
    for (int v = 0; v < V; ++v) {
        float f[4];
        unpack2(acc[v][0], f[0], f[1]);
        unpack2(acc[v][1], f[2], f[3]);
        store_chunk(out + (int64_t)v * p.N, f);
    }
}

}  // namespace cctile
}  // namespace vs
