// Warpgroup tiles of the fused MLP kernels (edge_fused.cu, node_fused.cu): a group
// of 128 threads owns 128 rows, an activation tile [128 x 128] of two swizzled
// slices that is the A operand of the next layer's MMAs, and 128 columns of
// tensor memory.
#pragma once

#include <cuda_bf16.h>

#include <cstdint>

#include "umma.cuh"

namespace pe {
namespace umma {

constexpr int kGroupThreads = 128;        // one thread per row of a tile (TMEM lane)
constexpr uint32_t kSlice = 128u * 128u;  // bytes of a 128-row x 64-column bf16 slice

__device__ __forceinline__ uint32_t sw_off(int row, int chunk) {
    return (uint32_t)row * 128u + ((uint32_t)(chunk ^ (row & 7)) << 4);
}

// barrier of warpgroup g alone (ids 1, 2, ...; 0 is __syncthreads')
__device__ __forceinline__ void group_sync(int g) {
    asm volatile("bar.sync %0, %1;" ::"r"(g + 1), "r"(kGroupThreads) : "memory");
}
// the same barrier, returning whether v holds on every thread of the group
__device__ __forceinline__ bool group_all(int g, bool v) {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "bar.red.and.pred q, %2, %3, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(r)
        : "r"((uint32_t)v), "r"(g + 1), "r"(kGroupThreads)
        : "memory");
    return r != 0;
}

// Rows 0 .. rows - 1 of a K-major bf16 matrix (row length ld) into swizzled slices:
// 16-byte chunk c of row r goes to slice c / 8, chunk c % 8.
__device__ inline void stage_rows(uint8_t* dst, const __nv_bfloat16* __restrict__ src, int ld, int chunks,
                                  int rows = 128) {
    for (int i = threadIdx.x; i < rows * chunks; i += blockDim.x) {
        const int r = i / chunks, c = i % chunks;
        const uint4 v = __ldg(reinterpret_cast<const uint4*>(src + (size_t)r * ld + c * 8));
        *reinterpret_cast<uint4*>(dst + (uint32_t)(c >> 3) * kSlice + sw_off(r, c & 7)) = v;
    }
}

// N fp32 values (columns c0 .. c0 + N - 1 of row r) into the bf16 activation tile
template <int N>
__device__ __forceinline__ void put_bf16_row(uint8_t* sA, int r, int c0, const float (&x)[N]) {
#pragma unroll
    for (int q = 0; q < N / 8; ++q) {
        uint32_t w[4];
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            __nv_bfloat162 b = __floats2bfloat162_rn(x[q * 8 + 2 * h], x[q * 8 + 2 * h + 1]);
            w[h] = *reinterpret_cast<uint32_t*>(&b);
        }
        const int cidx = c0 / 8 + q;  // 16-byte chunk of the 128-column row
        *reinterpret_cast<uint4*>(sA + (uint32_t)(cidx >> 3) * kSlice + sw_off(r, cidx & 7)) =
            make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// N biases from c0 on (a multiple of 4) of a layer in shared memory
template <int N>
__device__ __forceinline__ void get_bias(const float* b, float (&v)[N]) {
#pragma unroll
    for (int i = 0; i < N / 4; ++i) {
        const float4 f = *reinterpret_cast<const float4*>(b + 4 * i);
        v[4 * i] = f.x;
        v[4 * i + 1] = f.y;
        v[4 * i + 2] = f.z;
        v[4 * i + 3] = f.w;
    }
}

// 128 columns of A times those of W (N rows of it): eight MMAs
template <int N = kTileN>
__device__ __forceinline__ void issue_k128(uint32_t tmem, const uint8_t* sA, const uint8_t* sW, bool add = false) {
    const uint32_t a0 = smem_addr(sA), b0 = smem_addr(sW);
#pragma unroll
    for (int s = 0; s < 2; ++s)
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
            umma_bf16<N>(tmem, sw128_desc(a0 + (uint32_t)s * kSlice + kk * 32),
                         sw128_desc(b0 + (uint32_t)s * kSlice + kk * 32), (add || (s | kk)) ? 1u : 0u);
}

}  // namespace umma
}  // namespace pe
