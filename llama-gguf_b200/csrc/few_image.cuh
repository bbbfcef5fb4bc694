// few_image.cuh — the activations of the products of few token rows (gemm_few.cuh), laid out as the shared-memory tiles that they become.
#pragma once
#include "gemm_umma.cuh"

namespace b200 {

// Per token tile and block of 256 elements five slabs of N rows x 128 bytes (SWIZZLE_128B): four of 64 fp16
// elements (in each group of four in the order 0, 2, 1, 3, in which nibbles come out of a word), one with X_s as tf32 pairs (8 high parts, 8 low parts)
__host__ __device__ __forceinline__ size_t few_image_bytes(int T, int N, int K) { return (size_t)((T + N - 1) / N) * (K / 256) * 5 * N * 128; }
// X_s of row r, `b` = the block's image
__device__ __forceinline__ void few_put_sum(uint8_t* b, int N, int r, int s, float sum) {
    const float hi = __uint_as_float(__float_as_uint(sum) & 0xFFFFE000u), lo = __uint_as_float(__float_as_uint(sum - hi) & 0xFFFFE000u);
    uint8_t* q = b + 4 * N * 128;
    *reinterpret_cast<float*>(q + umma_sw128(r, s >> 2) + 4 * (s & 3)) = hi;
    *reinterpret_cast<float*>(q + umma_sw128(r, 2 + (s >> 2)) + 4 * (s & 3)) = lo;
}
// chunk e8 (eight elements) of token t; `sum` = the sum of the chunk's group of 32 elements (read where e8 % 4 == 0)
__device__ __forceinline__ void few_put8(uint8_t* img, int N, int nblk, int t, int e8, const __half (&h)[8], float sum) {
    const int blk = e8 >> 5, c8 = e8 & 31, r = t % N;
    uint8_t* b = img + ((size_t)(t / N) * nblk + blk) * 5 * N * 128;
    const __half2 a0 = __halves2half2(h[0], h[2]), a1 = __halves2half2(h[1], h[3]), a2 = __halves2half2(h[4], h[6]), a3 = __halves2half2(h[5], h[7]);
    uint4 v;
    v.x = *reinterpret_cast<const uint32_t*>(&a0); v.y = *reinterpret_cast<const uint32_t*>(&a1);
    v.z = *reinterpret_cast<const uint32_t*>(&a2); v.w = *reinterpret_cast<const uint32_t*>(&a3);
    *reinterpret_cast<uint4*>(b + (c8 >> 3) * N * 128 + umma_sw128(r, c8 & 7)) = v;
    if ((c8 & 3) == 0) few_put_sum(b, N, r, c8 >> 2, sum);
}
// the sum of the group of 32 elements a lane's chunk of 8 belongs to (lanes 4i .. 4i + 3 hold one group)
__device__ __forceinline__ float few_sum32(const __half (&h)[8]) {
    float s = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; i++) s += __half2float(h[i]);
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    return s + __shfl_xor_sync(0xffffffffu, s, 2);
}

// VEC consecutive elements e .. of token t in every lane (2 or 4; 32 / VEC lanes hold one group of 32)
template <int VEC>
__device__ __forceinline__ void few_put_lane(uint8_t* img, int N, int nblk, int t, int e, const __half (&h)[VEC]) {
    static_assert(VEC == 2 || VEC == 4, "heads of 64 or 128");
    const int blk = e >> 8, c8 = (e >> 3) & 31, r = t % N;
    uint8_t* b = img + ((size_t)(t / N) * nblk + blk) * 5 * N * 128;
    uint8_t* q = b + (c8 >> 3) * N * 128 + umma_sw128(r, c8 & 7) + 2 * (e & 4);
    if constexpr (VEC == 4) {
        const __half2 a0 = __halves2half2(h[0], h[2]), a1 = __halves2half2(h[1], h[3]);
        *reinterpret_cast<uint2*>(q) = make_uint2(*reinterpret_cast<const uint32_t*>(&a0), *reinterpret_cast<const uint32_t*>(&a1));
    } else {      // elements 0, 1 of a group of four: places 0, 2; elements 2, 3: places 1, 3
        __half* o = reinterpret_cast<__half*>(q) + ((e & 2) >> 1);
        o[0] = h[0];
        o[2] = h[1];
    }
    float s = 0.0f;
#pragma unroll
    for (int i = 0; i < VEC; i++) s += __half2float(h[i]);
#pragma unroll
    for (int o = 1; o < 32 / VEC; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((e & 31) == 0) few_put_sum(b, N, r, c8 >> 2, s);
}

}  // namespace b200
