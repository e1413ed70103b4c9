// Fixed-mask sparse attention in one kernel per direction: softmax(scale * Q K^T at the mask) V, and its gradients up to dQ.
//
// A vector-row is V <= 8 queries that attend to the SAME list of keys, which is the shape of an m16n8k16 instruction: 16
// gathered keys by 8 queries.  W warps share a vector-row and take its keys in chunks of 32:
//   first pass   S^T[key, query] = K[key, :] . Q^T:  the 16 rows of K are the A operand, read from memory straight into the
//                fragment (a lane reads 32 contiguous bytes of row lane/4; the contraction index is permuted alike in Q).  The
//                scores go to the caller's workspace in fp16, each to the place that the same lane reads again; a lane keeps a
//                running maximum and sum for its two queries.
//   second pass  P = exp(S - maximum) / sum, to the workspace in place of S; O^T[d, query] += V^T[d, key] . P^T[key, query], where P and
//                the rows of V, read as those of K, are transposed in registers (movmatrix).
// No shared memory holds an operand: it is left to L1, which serves the keys that neighbouring vector-rows share (the band of a
// local mask); a CTA therefore holds consecutive vector-rows.
//
// The tensor cores that tcgen05 reaches need 128 rows that share their columns; here 8 do.  Reading 32 bytes per lane matters:
// with 16, eight rows at a time hit the same half of the L1 banks, and reading V^T directly (four rows a lane at one 16-byte
// position) hit a quarter of them: 103 L1 wavefronts per 16 keys, now 80, a quarter of which transpose registers.  Those are what bounds
// it: 70 % of their peak rate, at 54 % of the issue slots (32 heads, sequence 4096, 410 keys: 171 us).
#pragma once
#include <type_traits>

#include "common.cuh"

namespace attention {

using namespace vs;

constexpr int kThreads = 256;
// CTAs per SM, which set the registers a thread may use: the forward kernel at d = 64 gains from warps in flight (128 heads, sequence
// 4096, 410 keys: 741 / 608 / 588 us with 128 / 80 / 64 registers), the backward one until it spills (1247 / 1022 / 1198), d = 128 not at all.
template <int D, bool kBackward> constexpr int kCtasPerSm = D == 64 ? (kBackward ? 3 : 4) : 2;

struct Params {
    int m_vec, V, n, nnz_vec;
    const int32_t *row_offsets;
    const int32_t *col_indices;
    const __half *q, *k, *v;
    __half *out;
    __half *probs;            // [batch][nnz_vec * V]: the probabilities
    const __half *grad_out;   // backward only; `out` is then dQ
    __half *grad_scores;      // backward only: [batch][nnz_vec * V], the gradient of the scores
    float scale;              // positive
};
constexpr float kLargeScore = 64.f;   // of a score times scale and log2(e)

__device__ __forceinline__ void mma16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// Transposes an 8 x 8 matrix of fp16 held as one fragment register per lane.
__device__ __forceinline__ uint32_t transpose8(uint32_t x) {
    uint32_t y;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(y) : "r"(x));
    return y;
}
__device__ __forceinline__ void group_sync(int group, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "r"(threads) : "memory");
}
__device__ __forceinline__ uint32_t pack2(float a, float b) {
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t *>(&h);
}
__device__ __forceinline__ float2 unpack2(uint32_t x) { return __half22float2(*reinterpret_cast<const __half2 *>(&x)); }
__device__ __forceinline__ float exp2_fast(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// 32 bytes, 32-byte aligned: four lanes read 128 consecutive bytes, so that eight rows of a matrix are eight wavefronts.
__device__ __forceinline__ void load32(const __half *src, uint32_t (&r)[8]) {
    asm volatile("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "l"(src));
}
// The lane's pieces of 16 gathered rows: row lane/4 and row lane/4 + 8.
template <int D> struct Rows {
    uint32_t r[2][D / 64][8];
    // base: the matrix, the same for the whole CTA, so that a lane holds a 32-bit offset and no address (fewer than 2^32 elements); col: the columns of a
    // chunk, one per lane; s: which half of the chunk
    __device__ __forceinline__ void fetch(const __half *base, int col, int s, int g) {
        const uint32_t at = (threadIdx.x & 3) * 16;
        const int c0 = __shfl_sync(0xffffffffu, col, 16 * s + g), c1 = __shfl_sync(0xffffffffu, col, 16 * s + 8 + g);
#pragma unroll
        for (int h = 0; h < D / 64; ++h) {
            load32(base + ((uint32_t)c0 * D + 64 * h + at), r[0][h]);
            load32(base + ((uint32_t)c1 * D + 64 * h + at), r[1][h]);
        }
    }
    __device__ __forceinline__ void clear(bool first, bool second) {
#pragma unroll
        for (int h = 0; h < D / 64; ++h)
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                if (first) r[0][h][i] = 0u;
                if (second) r[1][h][i] = 0u;
            }
    }
    // X^T[16 keys, 8 queries]; f: the lane's pieces of the query rows
    __device__ __forceinline__ void times_queries(const uint32_t (&f)[D / 64][8], float (&s)[4]) const {
#pragma unroll
        for (int i = 0; i < 4; ++i) s[i] = 0.f;
#pragma unroll
        for (int h = 0; h < D / 64; ++h)
#pragma unroll
            for (int i = 0; i < 8; i += 2) mma16816(s, r[0][h][i], r[1][h][i], r[0][h][i + 1], r[1][h][i + 1], f[h][i], f[h][i + 1]);
    }
    // acc^T[D, 8 queries] += rows^T . w; b0, b1: the weights, transposed
    __device__ __forceinline__ void weighted(uint32_t b0, uint32_t b1, float (&acc)[D / 64][4][4]) const {
#pragma unroll
        for (int h = 0; h < D / 64; ++h)
#pragma unroll
            for (int j = 0; j < 4; ++j)
                mma16816(acc[h][j], transpose8(r[0][h][2 * j]), transpose8(r[0][h][2 * j + 1]), transpose8(r[1][h][2 * j]), transpose8(r[1][h][2 * j + 1]), b0, b1);
    }
};

// Scores of a chunk of 32 keys against 8 queries; the two halves side by side where the registers allow it.
template <int D> __device__ __forceinline__ void against(const __half *base, int col, int g, const uint32_t (&queries)[D / 64][8], float (&x)[2][4]) {
    if constexpr (D == 64) {
        Rows<D> r0, r1;
        r0.fetch(base, col, 0, g);
        r1.fetch(base, col, 1, g);
        r0.times_queries(queries, x[0]);
        r1.times_queries(queries, x[1]);
    } else {
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            Rows<D> r;
            r.fetch(base, col, s, g);
            r.times_queries(queries, x[s]);
        }
    }
}

// Column of the lane's key in a chunk of 32; column 0 past the row's end, where the caller discards what it loads (and for a column
// outside the matrix, which no valid mask has).
__device__ __forceinline__ int chunk_column(const Params &p, int key, int end) {
    const int c = key < end ? __ldg(p.col_indices + key) : 0;
    return (unsigned)c < (unsigned)p.n ? c : 0;
}

template <int D, int W, bool kBackward>
__global__ void __launch_bounds__(kThreads, (kCtasPerSm<D, kBackward>)) attention_kernel(const Params p) {
    constexpr int kGroups = kThreads / (32 * W);
    constexpr int kPitch = 64 + 4;
    constexpr bool kTwoForms = W > 1 && !kBackward;   // of the second pass
    const int V = p.V;
    __shared__ float red[kGroups][W][8][3];
    __shared__ __align__(16) float part[W > 1 ? kGroups : 1][W > 1 ? W : 1][W > 1 ? 8 : 1][W > 1 ? kPitch : 4];
    const int group = threadIdx.x / (32 * W), w = (threadIdx.x >> 5) % W, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int64_t b = blockIdx.y;
    const __half *kmat = p.k + b * p.n * D, *vmat = p.v + b * p.n * D;
    const __half *q = p.q + b * p.m_vec * V * D + 16 * t;
    const __half *go = kBackward ? p.grad_out + b * p.m_vec * V * D + 16 * t : nullptr;
    __half *out = p.out + b * p.m_vec * V * D;
    // the lane's place in the entry of key 0: queries 2t, 2t+1 of key lane/4
    __half *probs = p.probs + (b * p.nnz_vec + g) * V + 2 * t, *gs = kBackward ? p.grad_scores + (b * p.nnz_vec + g) * V + 2 * t : nullptr;
    const bool stores = 2 * t < V;
    const float sl2 = p.scale * 1.4426950408889634f;

    const int row = blockIdx.x * kGroups + group;
    if (row < p.m_vec) {
        const int beg = min(max(__ldg(p.row_offsets + row), 0), p.nnz_vec);
        const int end = min(max(__ldg(p.row_offsets + row + 1), beg), p.nnz_vec);
        // first pass: scores (and dP) to memory in fp16, and per lane the running maximum and sums
        float mx[2] = {-INFINITY, -INFINITY}, sum[2] = {0.f, 0.f}, dot[2] = {0.f, 0.f};
        {
            uint32_t qf[D / 64][8], gf[kBackward ? D / 64 : 1][8];
#pragma unroll
            for (int h = 0; h < D / 64; ++h) {
                const int64_t at = ((int64_t)row * V + min(g, V - 1)) * D + 64 * h;   // lanes past the V queries: values nobody stores
                load32(q + at, qf[h]);
                if constexpr (kBackward) load32(go + at, gf[h]);
            }
            int next = chunk_column(p, beg + 32 * w + lane, end);
#pragma unroll 1
            for (int key = beg + 32 * w; key < end; key += 32 * W) {
                const int col = next;
                next = chunk_column(p, key + 32 * W + lane, end);
                float x[2][4], dp[2][4];
                against<D>(kmat, col, g, qf, x);
                if constexpr (kBackward) against<D>(vmat, col, g, gf, dp);
                __half *to = probs + (int64_t)key * V;
                __half *tg = kBackward ? gs + (int64_t)key * V : nullptr;
#pragma unroll
                for (int i = 0; i < 4; ++i) {   // 8 keys
                    const uint32_t raw = pack2(x[i >> 1][2 * (i & 1)], x[i >> 1][2 * (i & 1) + 1]);
                    const bool here = key + 8 * i + g < end;
                    if (here && stores) *reinterpret_cast<uint32_t *>(to + 8 * i * V) = raw;
                    const float2 r = unpack2(raw);
                    x[i >> 1][2 * (i & 1)] = here ? r.x : -INFINITY;
                    x[i >> 1][2 * (i & 1) + 1] = here ? r.y : -INFINITY;
                    if constexpr (kBackward) {
                        const uint32_t grad = here ? pack2(dp[i >> 1][2 * (i & 1)], dp[i >> 1][2 * (i & 1) + 1]) : 0u;
                        if (here && stores) *reinterpret_cast<uint32_t *>(tg + 8 * i * V) = grad;
                        const float2 d = unpack2(grad);
                        dp[i >> 1][2 * (i & 1)] = d.x;
                        dp[i >> 1][2 * (i & 1) + 1] = d.y;
                    }
                }
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const float top = fmaxf(mx[i], sl2 * fmaxf(fmaxf(x[0][i], x[0][i + 2]), fmaxf(x[1][i], x[1][i + 2])));
                    const float base = top == -INFINITY ? 0.f : top, keep = exp2_fast(mx[i] - base);
                    sum[i] *= keep;
                    if constexpr (kBackward) dot[i] *= keep;
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float e = exp2_fast(fmaf(x[j >> 1][i + 2 * (j & 1)], sl2, -base));   // the product unrounded, as in the second pass
                        sum[i] += e;
                        if constexpr (kBackward) dot[i] = fmaf(e, dp[j >> 1][i + 2 * (j & 1)], dot[i]);
                    }
                    mx[i] = top;
                }
            }
        }
        // over the lanes that share a query, then over the warps that share the row
        float inv[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            float top = mx[i];
#pragma unroll
            for (int off = 4; off < 32; off <<= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, off));
            const float keep = exp2_fast(mx[i] - (top == -INFINITY ? 0.f : top));
            sum[i] *= keep;
            if constexpr (kBackward) dot[i] *= keep;
#pragma unroll
            for (int off = 4; off < 32; off <<= 1) {
                sum[i] += __shfl_xor_sync(0xffffffffu, sum[i], off);
                if constexpr (kBackward) dot[i] += __shfl_xor_sync(0xffffffffu, dot[i], off);
            }
            mx[i] = top;
        }
        if constexpr (W > 1) {
            if (g == 0) {
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    red[group][w][2 * t + i][0] = mx[i];
                    red[group][w][2 * t + i][1] = sum[i];
                    if constexpr (kBackward) red[group][w][2 * t + i][2] = dot[i];
                }
            }
            group_sync(group, 32 * W);
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                float top = -INFINITY;
#pragma unroll
                for (int x = 0; x < W; ++x) top = fmaxf(top, red[group][x][2 * t + i][0]);
                sum[i] = dot[i] = 0.f;
#pragma unroll
                for (int x = 0; x < W; ++x) {
                    const float e = exp2_fast(red[group][x][2 * t + i][0] - top);   // 0 for a warp without keys; NaN in a row without a finite score
                    sum[i] = fmaf(red[group][x][2 * t + i][1], e, sum[i]);
                    if constexpr (kBackward) dot[i] = fmaf(red[group][x][2 * t + i][2], e, dot[i]);
                }
                mx[i] = top;
            }
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            if constexpr (!kTwoForms) inv[i] = 1.0f / sum[i];
            if constexpr (kBackward) dot[i] *= inv[i];
        }

        // second pass: probabilities (and score gradients) in the place of the scores, and their product with the rows of V (of K)
        float acc[D / 64][4][4];
#pragma unroll
        for (int h = 0; h < D / 64; ++h)
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[h][j][i] = 0.f;
        auto second_pass = [&](auto inside) {   // 1 / sum inside the exponent
            int next = chunk_column(p, beg + 32 * w + lane, end);
#pragma unroll 1
            for (int key = beg + 32 * w; key < end; key += 32 * W) {
                const int col = next;
                next = chunk_column(p, key + 32 * W + lane, end);
                __half *to = probs + (int64_t)key * V;
                __half *tg = kBackward ? gs + (int64_t)key * V : nullptr;
                uint32_t wt[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const bool here = key + 8 * i + g < end;
                    wt[i] = 0u;
                    if (here && stores) {
                        const float2 r = unpack2(*reinterpret_cast<const uint32_t *>(to + 8 * i * V));
                        float p0 = exp2_fast(fmaf(r.x, sl2, -mx[0])), p1 = exp2_fast(fmaf(r.y, sl2, -mx[1]));   // NaN where no score is finite
                        if constexpr (!decltype(inside)::value) {
                            p0 *= inv[0];
                            p1 *= inv[1];
                        }
                        wt[i] = pack2(p0, p1);
                        *reinterpret_cast<uint32_t *>(to + 8 * i * V) = wt[i];
                        if constexpr (kBackward) {
                            const float2 d = unpack2(*reinterpret_cast<const uint32_t *>(tg + 8 * i * V));
                            wt[i] = pack2(p.scale * p0 * (d.x - dot[0]), p.scale * p1 * (d.y - dot[1]));
                            *reinterpret_cast<uint32_t *>(tg + 8 * i * V) = wt[i];
                        }
                    }
                }
                const __half *base = kBackward ? kmat : vmat;
#pragma unroll
                for (int s = 0; s < 2; ++s) {
                    Rows<D> r;
                    r.fetch(base, col, s, g);
                    if (key + 32 > end) r.clear(key + 16 * s + g >= end, key + 16 * s + 8 + g >= end);   // weight 0 times what row 0 may hold
                    r.weighted(transpose8(wt[2 * s]), transpose8(wt[2 * s + 1]), acc);
                }
            }
        };
        // Next to scores of thousands an exponent has no room for the logarithm of the sum: up to 2^-9 of it, the same for all keys of a query, would be
        // lost.  Outside, 1 / sum costs registers that are spent: 128 heads, sequence 4096, 583 -> 591 us, 29 heads, 688, V = 2, two warps to a row, 26.9 -> 28.7.  So
        // forward with several warps to a row it is inside where scores are small enough for an error of 2^-19; with one warp a second body of the loop
        // costs more (600), backward too (142 -> 148 at 110 heads, 424, V = 2).
        if constexpr (kTwoForms) {
            const float l0 = mx[0] + __log2f(sum[0]), l1 = mx[1] + __log2f(sum[1]);
            if (__all_sync(0xffffffffu, fabsf(l0) < kLargeScore && fabsf(l1) < kLargeScore)) {
                mx[0] = l0;
                mx[1] = l1;
                second_pass(std::true_type{});
            } else {
                inv[0] = 1.0f / sum[0];
                inv[1] = 1.0f / sum[1];
                second_pass(std::false_type{});
            }
        } else {
            second_pass(std::false_type{});
        }

        // a lane holds queries 2t, 2t+1 of columns 64 h + 16 (g / 2) + (g & 1) + 2 x (0 .. 7); lane g ^ 1 has those between.  Of the
        // sixteen the even one takes the first eight, the odd one the others
#pragma unroll
        for (int h = 0; h < D / 64; ++h) {
            if (W > 1 && h > 0) group_sync(group, 32 * W);
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                float o[8];
#pragma unroll
                for (int j = 0; j < 2; ++j)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const float low = acc[h][j][i + 2 * e], high = acc[h][j + 2][i + 2 * e];
                        const float got = __shfl_xor_sync(0xffffffffu, g & 1 ? low : high, 4);
                        o[4 * j + 2 * e] = g & 1 ? got : low;
                        o[4 * j + 2 * e + 1] = g & 1 ? high : got;
                    }
                if (2 * t + i < V) {
                    if constexpr (W == 1) {
                        *(reinterpret_cast<uint4 *>(out + ((int64_t)row * V + 2 * t + i) * D) + 8 * h + g) =
                            make_uint4(pack2(o[0], o[1]), pack2(o[2], o[3]), pack2(o[4], o[5]), pack2(o[6], o[7]));
                    } else {
                        float4 *to = reinterpret_cast<float4 *>(&part[group][w][2 * t + i][8 * g]);
                        to[0] = make_float4(o[0], o[1], o[2], o[3]);
                        to[1] = make_float4(o[4], o[5], o[6], o[7]);
                    }
                }
            }
            if constexpr (W > 1) {
                group_sync(group, 32 * W);
                for (int e = threadIdx.x % (32 * W); e < V * 16; e += 32 * W) {
                    const int qi = e / 16, c = (e % 16) * 4;
                    float4 o = *reinterpret_cast<const float4 *>(&part[group][0][qi][c]);
#pragma unroll
                    for (int x = 1; x < W; ++x) {
                        const float4 y = *reinterpret_cast<const float4 *>(&part[group][x][qi][c]);
                        o.x += y.x; o.y += y.y; o.z += y.z; o.w += y.w;
                    }
                    *reinterpret_cast<uint2 *>(out + ((int64_t)row * V + qi) * D + 64 * h + c) = make_uint2(pack2(o.x, o.y), pack2(o.z, o.w));
                }
            }
        }
    }
}

}  // namespace attention
