// What the recurrences in chunks of rows share (mamba2_chunk.cu, mlstm_chunk.cu, delta_chunk.cu): which rows a chunk has, asynchronous
// copies, and the 32-bit product of two tiles in shared memory.
#pragma once
#include "common.cuh"

namespace imparo {
namespace chunks {

// chunk number -> request, first row, rows (0: no such chunk); chunks of ROWS rows, p with item_row_start and n_items
template <int ROWS, typename P>
__device__ __forceinline__ int chunk_rows(const P& p, int chunk, int& item, int& first) {
    for (item = 0; item < p.n_items; ++item) {
        const int r0 = p.item_row_start[item], n = p.item_row_start[item + 1] - r0;
        const int chunks = (n + ROWS - 1) / ROWS;
        if (chunk < chunks) {
            first = r0 + chunk * ROWS;
            return min(ROWS, n - chunk * ROWS);
        }
        chunk -= chunks;
    }
    first = 0;
    return 0;
}

__device__ __forceinline__ void cp16(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// ---- products of 64 rows by 64 columns, a patch of 8 x 4 per thread ---------------------------------------------------------------
constexpr int VB = 64;              // columns
constexpr int THREADS = 128;

// acc[8][4] += left[k][l0 ..] x right[k][r0 ..] over k in [0, to): three 16-byte reads of shared memory per 32 operations.
// Every 32 terms are summed by themselves: a third less rounding than one chain of 64 (3% more operations).
// CAUSAL (to = l0 + 8): row l0 + i has the terms up to its own.  Those beyond are left out and not multiplied by zero, so that a
// row that is not finite reaches no earlier one.
template <int LD, bool CAUSAL = false>
__device__ __forceinline__ void product(float2 (&acc)[8][2], const float* left, int l0, const float* right, int r0, int to) {
#pragma unroll 1
    for (int k0 = 0; k0 < to; k0 += 32) {
        float2 part[8][2] = {};
        const int end = min(k0 + 32, CAUSAL ? l0 : to);
#pragma unroll 4
        for (int k = k0; k < end; ++k) {
            const float4 a = *reinterpret_cast<const float4*>(left + k * LD + l0), b = *reinterpret_cast<const float4*>(left + k * LD + l0 + 4);
            const float4 r = *reinterpret_cast<const float4*>(right + k * VB + r0);
            const float2 r01 = make_float2(r.x, r.y), r23 = make_float2(r.z, r.w);
            const float av[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float2 a2 = make_float2(av[i], av[i]);
                part[i][0] = __ffma2_rn(a2, r01, part[i][0]);
                part[i][1] = __ffma2_rn(a2, r23, part[i][1]);
            }
        }
        if (CAUSAL && k0 + 32 > l0) {
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const float4 a = *reinterpret_cast<const float4*>(left + (l0 + u) * LD + l0), b = *reinterpret_cast<const float4*>(left + (l0 + u) * LD + l0 + 4);
                const float4 r = *reinterpret_cast<const float4*>(right + (l0 + u) * VB + r0);
                const float2 r01 = make_float2(r.x, r.y), r23 = make_float2(r.z, r.w);
                const float av[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
                for (int i = u; i < 8; ++i) {
                    const float2 a2 = make_float2(av[i], av[i]);
                    part[i][0] = __ffma2_rn(a2, r01, part[i][0]);
                    part[i][1] = __ffma2_rn(a2, r23, part[i][1]);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int v = 0; v < 2; ++v) acc[i][v] = make_float2(acc[i][v].x + part[i][v].x, acc[i][v].y + part[i][v].y);
    }
}

// ROWS rows of `cols` columns (dst rows of VB floats): zeros beyond n rows and beyond the columns there are
template <int ROWS>
__device__ __forceinline__ void fetch_rows(float* dst, const float* src, size_t stride, int n, int cols) {
    for (int e = threadIdx.x; e < ROWS * (VB / 4); e += THREADS) {
        const int r = e / (VB / 4), v = (e % (VB / 4)) * 4;
        if (r < n && v < cols) cp16(dst + r * VB + v, src + (size_t)r * stride + v);
        else *reinterpret_cast<float4*>(dst + r * VB + v) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
}

}  // namespace chunks
}  // namespace imparo
