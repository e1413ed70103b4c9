// A sparse matrix laid out as dense 16-bit tiles, zeros included, in the order in which the multiplying kernels read them:
// [batch][M / 128, rounded up][Kp / 64][part][128 rows][64 columns], Kp = K rounded up to 64.  Rows past M are left as they are.
//
// One part: fp16 values for the pair kernel (spmm_pair.cuh), which otherwise scatters the nonzeros of every tile into shared memory
// itself, again for each 256 columns of the dense operand: 2-byte stores, one per nonzero at V = 1, by a dozen warps beside the tensor
// cores.  Here every SM scatters, once.  Three parts: bf16 parts of fp32 values (spmm_split.cuh).
#pragma once
#include <cuda_bf16.h>

#include "common.cuh"

namespace vs {
namespace densify {

constexpr int kPrepThreads = 256, kPrepValues = 8192;          // of vector-rows at a time: 32 KiB of fp32, 16 of fp16
constexpr int kMaxGroup = 32;                                  // vector-rows of them at most
constexpr uint32_t kTinyInput = (127u - 100u) << 23;

// Eight values as three groups of eight bf16.  Returns whether one of them is too small to be split exactly.
__device__ __forceinline__ bool split8(const float (&x)[8], uint4 (&part)[3]) {
    uint32_t w[3][4];
    bool tiny = false;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float a = x[2 * i], b = x[2 * i + 1];
        tiny |= (__float_as_uint(a) & 0x7fffffffu) - 1u < kTinyInput - 1u || (__float_as_uint(b) & 0x7fffffffu) - 1u < kTinyInput - 1u;
#pragma unroll
        for (int p = 0; p < 3; ++p) {
            const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
            w[p][i] = *reinterpret_cast<const uint32_t *>(&h);
            a -= __uint_as_float(w[p][i] << 16);
            b -= __uint_as_float(w[p][i] & 0xffff0000u);
        }
    }
#pragma unroll
    for (int p = 0; p < 3; ++p) part[p] = make_uint4(w[p][0], w[p][1], w[p][2], w[p][3]);
    return tiny;
}

template <typename T> struct Shared {
    T rows[kPrepValues];
    uint32_t named[kPrepValues / 32];
    int offsets[kMaxGroup + 1];
};

// This CTA's share of the vector-rows, several short ones or a piece of a long one at a time; the entries of such a group lie side by
// side, so the threads walk them together, four loads in flight each, and look up their rows.  Returns whether the thread met a column named
// twice in a vector-row or a value that cannot be split; columns outside the matrix are left out.  `found` is set where the thread
// met a vector-row of 1 .. few - 1 entries.
template <typename T, int V, int kParts>
__device__ __forceinline__ bool lay_out_rows(const SpmmParams &p, int batch_a, int Kp, uint16_t *dst, Shared<T> &sh, int few, bool &found) {
    constexpr int kCols = kPrepValues / V, kChunk = 16 / (int)sizeof(T);
    const int t = threadIdx.x, pieces = (Kp + kCols - 1) / kCols;
    const int group = max(min(kCols / Kp, (int)min((int64_t)kMaxGroup, (int64_t)batch_a * p.m_vec / gridDim.x)), 1), groups = (p.m_vec + group - 1) / group;
    const int k_blocks = Kp / 64, row_tiles = (int)(((int64_t)p.m_vec * V + 127) / 128);
    const int64_t units = (int64_t)batch_a * groups * pieces;
    bool bad = false;
    for (int64_t u = blockIdx.x; u < units; u += gridDim.x) {
        const int c0 = (int)(u % pieces) * kCols, cols = min(kCols, Kp - c0);
        const int64_t r = u / pieces;
        const int row0 = (int)(r % groups) * group, b = (int)(r / groups), count = min(group, p.m_vec - row0);
        for (int i = t; i < count * V * cols / kChunk; i += kPrepThreads) reinterpret_cast<uint4 *>(sh.rows)[i] = make_uint4(0u, 0u, 0u, 0u);
        for (int i = t; i < count * cols / 32; i += kPrepThreads) sh.named[i] = 0u;
        if (t <= count) sh.offsets[t] = __ldg(p.row_offsets + row0 + t);
        __syncthreads();
        if (t < count && sh.offsets[t + 1] > sh.offsets[t] && sh.offsets[t + 1] - sh.offsets[t] < few) found = true;
        const T *values = static_cast<const T *>(p.values) + (int64_t)b * p.stride_values;
        const int end = sh.offsets[count];
        constexpr int U = 4;
        for (int j0 = sh.offsets[0] + t; j0 < end; j0 += U * kPrepThreads) {
            int c[U];
            float a[U][V];
#pragma unroll
            for (int x = 0; x < U; ++x) {
                const int j = j0 + x * kPrepThreads;
                c[x] = j < end ? __ldg(p.col_indices + j) : -1;
                if (j < end) VecLoad<T, V>::load(values + (int64_t)j * V, a[x]);
            }
#pragma unroll
            for (int x = 0; x < U; ++x) {
                const int col = c[x] - c0;
                if (c[x] < 0 || c[x] >= p.K || (unsigned)col >= (unsigned)cols) continue;
                int i = 0;   // the row of the entry: the last one that starts at or before it
                for (int step = kMaxGroup / 2; step > 0; step >>= 1)
                    if (i + step < count && sh.offsets[i + step] <= j0 + x * kPrepThreads) i += step;
                const uint32_t bit = 1u << (col & 31);
                bad |= (atomicOr(&sh.named[(i * cols + col) >> 5], bit) & bit) != 0u;
#pragma unroll
                for (int v = 0; v < V; ++v) store_scalar(&sh.rows[(i * V + v) * cols + col], a[x][v]);
            }
        }
        __syncthreads();
        for (int i = t; i < count * V * (cols / 8); i += kPrepThreads) {
            const int m_in = i / (cols / 8), c = (i % (cols / 8)) * 8;
            uint4 part[kParts];
            if constexpr (kParts == 3) {
                const float4 lo = *reinterpret_cast<const float4 *>(sh.rows + m_in * cols + c), hi = *reinterpret_cast<const float4 *>(sh.rows + m_in * cols + c + 4);
                const float x[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
                bad |= split8(x, part);
            } else {
                part[0] = *reinterpret_cast<const uint4 *>(sh.rows + m_in * cols + c);
            }
            const int64_t m = (int64_t)row0 * V + m_in, tile = ((int64_t)b * row_tiles + m / 128) * k_blocks + (c0 + c) / 64;
#pragma unroll
            for (int s = 0; s < kParts; ++s)
                *reinterpret_cast<uint4 *>(dst + (tile * kParts + s) * (128 * 64) + (m % 128) * 64 + c % 64) = part[s];
        }
        __syncthreads();
    }
    return bad;
}

// verdict: the plan header (common.cuh): word 0 = from min_vectors nonzero vectors on the dense product is the quicker one, words
// 4 ..: one per CTA, nonzero if it met a column twice.
template <int V>
__global__ void __launch_bounds__(kPrepThreads) densify_kernel(const SpmmParams p, int batch_a, int Kp, int64_t min_vectors, uint16_t *dst, int32_t *verdict) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ __align__(16) Shared<__half> sh;
    const bool taken = (int64_t)__ldg(p.row_offsets + p.m_vec) - __ldg(p.row_offsets) >= min_vectors;
    if (blockIdx.x == 0 && threadIdx.x == 0) plan_publish(verdict, taken);
    if (!taken) return;
    bool found = false;
    const int any = __syncthreads_or(lay_out_rows<__half, V, 1>(p, batch_a, Kp, dst, sh, 0, found));
    if (threadIdx.x == 0) verdict[4 + blockIdx.x] = any;
}

}  // namespace densify
}  // namespace vs
