// Exact fp32 squared-L2 distances of a small tile of rows against another, in the CPU path's arithmetic (sequential over the
// dimensions, sub / mul / add without FMA: src/cpu/utils/cpu_distance.h:74-81).  Shared by the coarse stage's small batches and the
// IVF-Flat scan.
#pragma once

#include "common.cuh"

namespace psb {
namespace tile {

constexpr int SQ = 32, SC = 64;       // rows of the two sides of a tile
constexpr int kSmallThreads = 128;    // 8 x 16 threads of 4 x 4 pairs

// Floats between staged rows: 4 (mod 32) words or 4 (mod 8) at least, so that eight rows' 16-byte words fall into different banks.
__host__ __device__ __forceinline__ int small_pitch(int dim) { return (dim + 3) / 4 * 4 + ((((dim + 3) / 4) & 1) ? 0 : 4); }
inline size_t small_tile_bytes(int dim) { return (size_t)(SQ + SC) * small_pitch(dim) * 4; }

#ifdef __CUDACC__
__device__ __forceinline__ void async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void async4(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
// One row by the lanes of a warp, the dimensions padded with zeros to a multiple of four.
__device__ __forceinline__ void stage_row(float* dst, const float* __restrict__ src, int dim, bool vec, int lane) {
    if (vec) {
        for (int d = lane; d < dim >> 2; d += 32) async16(dst + d * 4, src + d * 4);
    } else {
        for (int d = lane; d < dim; d += 32) async4(dst + d, src + d);
        if (lane < ((4 - (dim & 3)) & 3)) dst[dim + lane] = 0.0f;
    }
}
__device__ __forceinline__ bool rows_vec(const float* p, int dim) { return (dim & 3) == 0 && (reinterpret_cast<uintptr_t>(p) & 15) == 0; }
template <int THREADS>
__device__ __forceinline__ void stage_rows(float* dst, int pitch, const float* __restrict__ src, int rows, int dim) {
    const bool vec = rows_vec(src, dim);
    for (int r = threadIdx.x >> 5; r < rows; r += THREADS / 32) stage_row(dst + r * pitch, src + (size_t)r * dim, dim, vec, threadIdx.x & 31);
}
__device__ __forceinline__ void stage_wait() {
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
}
// Distance of q (shared memory, 16-byte aligned) to the row x, four elements at a time where vec.
__device__ __forceinline__ float row_distance(const float* __restrict__ q, const float* __restrict__ x, int dim, bool vec) {
    float sum = 0.0f;
    if (vec) {
#pragma unroll 8
        for (int d = 0; d < dim; d += 4) {
            const float4 v = __ldg(reinterpret_cast<const float4*>(x + d));
            const float4 y = *reinterpret_cast<const float4*>(q + d);
            float t = __fsub_rn(y.x, v.x); sum = __fadd_rn(sum, __fmul_rn(t, t));
            t = __fsub_rn(y.y, v.y); sum = __fadd_rn(sum, __fmul_rn(t, t));
            t = __fsub_rn(y.z, v.z); sum = __fadd_rn(sum, __fmul_rn(t, t));
            t = __fsub_rn(y.w, v.w); sum = __fadd_rn(sum, __fmul_rn(t, t));
        }
    } else {
#pragma unroll 8
        for (int d = 0; d < dim; ++d) { const float t = __fsub_rn(q[d], __ldg(x + d)); sum = __fadd_rn(sum, __fmul_rn(t, t)); }
    }
    return sum;
}
// acc[i][j] = distance of q row i to c row 16 j; the zeros behind dim add exact zeros.
__device__ __forceinline__ void tile_distances(const float* __restrict__ q, const float* __restrict__ c, int pitch, int dim, float (&acc)[4][4]) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;
    const int n = (dim + 3) & ~3;
#pragma unroll 2
    for (int d = 0; d < n; d += 4) {
        float4 a[4], b[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const float4*>(q + i * pitch + d);
#pragma unroll
        for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const float4*>(c + 16 * j * pitch + d);
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float t = __fsub_rn(a[i].x, b[j].x); acc[i][j] = __fadd_rn(acc[i][j], __fmul_rn(t, t));
                t = __fsub_rn(a[i].y, b[j].y); acc[i][j] = __fadd_rn(acc[i][j], __fmul_rn(t, t));
                t = __fsub_rn(a[i].z, b[j].z); acc[i][j] = __fadd_rn(acc[i][j], __fmul_rn(t, t));
                t = __fsub_rn(a[i].w, b[j].w); acc[i][j] = __fadd_rn(acc[i][j], __fmul_rn(t, t));
            }
    }
}
#endif

}  // namespace tile
}  // namespace psb
