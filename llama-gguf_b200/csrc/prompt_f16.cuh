// prompt_f16.cuh — the products of a prompt in two passes: a weight matrix's GGUF blocks -> fp16 rows in a scratch buffer, then the plain fp16
// product of gemm_tc.cuh.  Same operands as the fused dequant-GEMM (gemm_umma2.cuh: f32 block arithmetic, one rounding to fp16; dequant.rs:
// 205-356), f32 accumulation.
//
// The fused kernel dequantises a weight once per 256 tokens, on warps that share issue slots and shared memory with the tensor pipe (1.25x a
// plain product's step at best, 3x for Q6_K and Q8_0), and a matrix with few row tiles leaves SMs without work.  Here every block is
// unpacked once per prompt chunk, and the product splits K or walks tiles persistently by shape.  Measured at 2048 tokens, 8B layer (Q4_K_M):
// seven fused products 1340 us + SwiGLU 79; here 139 us of unpacking (0.57 GB: 4.1 TB/s) and 90 + 350 + 261 us of products (up to 1.37 PFLOP/s)
// with SwiGLU in the gate / up epilogue.  prefill_gemm in engine.cu draws the line between the two.
#pragma once
#include "gemm_umma.cuh"
#include "prefill.cuh"

namespace b200 {

// One warp unpacks `run` consecutive units of 256 elements: a matrix's rows follow one another without gaps, in blocks and in fp16, so units are counted through
// the matrix and a unit may cross rows of block types of 32.  The run's bytes come in by whole 16-byte words (all in flight), lie in shared memory at their own
// offset, and a lane takes eight (Q8_0) or two times eight elements (K-quants: the low and the high halves of the same bytes) of a unit at a time.  The blocks
// are read before the wait for the kernel before (a product that may still read the scratch rows).
// Bound by DRAM: 0.56 to 1.06 bytes in, 2 out per element.  Runs of eight units, or of two where eight would leave SMs without a block (f16_run_of).  Against a thread per
// eight elements of four rows with 16-bit loads from global memory, whole prompts: 300 tokens through two 8B layers in Q4_K_M 1053 -> 997 us, 700 tokens in Q6_K / Q5_K_M
// 1455 / 1525 -> 1366 / 1372 us, 333 through four 2048-wide ones in Q8_0 624 -> 593 us.
constexpr int F16_RUN = 8, F16_WARPS = 8;
constexpr int F16_BYTES = F16_RUN * 272 + 32;      // of a run, widest type, at any offset of 16
// eight values d sc q - dmin m, each one f32 FMA on a nibble held as subnormal fp16 (q 2^-24), as u2_deq64_q4k computes them
__device__ __forceinline__ uint4 f16_nibbles(uint2 q, int hi, float ds, float cm) {
    uint32_t out[4];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const uint32_t w = (h ? q.y : q.x) >> (4 * hi), e = w & 0x000F000Fu, o = (w >> 8) & 0x000F000Fu;
        const float2 f02 = __half22float2(*reinterpret_cast<const __half2*>(&e)), f13 = __half22float2(*reinterpret_cast<const __half2*>(&o));
        out[2 * h] = umma_pack_h2(fmaf(ds, f02.x, cm), fmaf(ds, f13.x, cm));
        out[2 * h + 1] = umma_pack_h2(fmaf(ds, f02.y, cm), fmaf(ds, f13.y, cm));
    }
    return make_uint4(out[0], out[1], out[2], out[3]);
}
template <int TYPE> struct F16Unit {
    static constexpr int BYTES = TYPE == T_Q4_K ? 144 : TYPE == T_Q5_K ? 176 : TYPE == T_Q6_K ? 210 : 272;
    static constexpr int LANES = TYPE == T_Q8_0 ? 32 : 16;      // lanes per unit
};
// lane i (< LANES) of a unit whose blocks start at blk (shared memory): its elements -> out (the unit's 256 fp16 values); live: elements that exist
template <int TYPE>
__device__ __forceinline__ void f16_unit(const uint8_t* blk, int i, __half* out, int live) {
    if constexpr (TYPE == T_Q4_K) {
        const int gp = i >> 2, c = i & 3, b = 16 * (gp & 1);
        const uint2 h0 = *reinterpret_cast<const uint2*>(blk), h1 = *reinterpret_cast<const uint2*>(blk + 8);      // (blocks are 8-byte aligned at least: umma_eligible)
        const uint4 hdr = make_uint4(h0.x, h0.y, h1.x, h1.y);
        const uint2 q = *reinterpret_cast<const uint2*>(blk + 16 + 32 * gp + 8 * c);
        const float d = half_bits_to_float(hdr.x), dmin = half_bits_to_float(hdr.x >> 16);
        int s0, m0, s1, m1;
        if (gp < 2) {
            s0 = (hdr.y >> b) & 63; m0 = (hdr.z >> b) & 63;
            s1 = (hdr.y >> (b + 8)) & 63; m1 = (hdr.z >> (b + 8)) & 63;
        } else {
            s0 = ((hdr.w >> b) & 15) | (((hdr.y >> (b + 6)) & 3) << 4);
            m0 = ((hdr.w >> (b + 4)) & 15) | (((hdr.z >> (b + 6)) & 3) << 4);
            s1 = ((hdr.w >> (b + 8)) & 15) | (((hdr.y >> (b + 14)) & 3) << 4);
            m1 = ((hdr.w >> (b + 12)) & 15) | (((hdr.z >> (b + 14)) & 3) << 4);
        }
        const uint4 lo = f16_nibbles(q, 0, __fmul_rn(d, (float)s0) * 16777216.0f, -__fmul_rn(dmin, (float)m0));
        const uint4 hi = f16_nibbles(q, 1, __fmul_rn(d, (float)s1) * 16777216.0f, -__fmul_rn(dmin, (float)m1));
        *reinterpret_cast<uint4*>(out + 64 * gp + 8 * c) = lo;
        *reinterpret_cast<uint4*>(out + 64 * gp + 32 + 8 * c) = hi;
    } else if constexpr (TYPE == T_Q8_0) {
        if (8 * i < live) *reinterpret_cast<uint4*>(out + 8 * i) = umma_deq8<true>(TYPE, blk, 64 * (i >> 3), i & 7);
    } else {
        const int gp = i >> 2, c = i & 3;
        const uint4 lo = umma_deq8<true>(TYPE, blk, 64 * gp, c), hi = umma_deq8<true>(TYPE, blk, 64 * gp, c + 4);
        *reinterpret_cast<uint4*>(out + 64 * gp + 8 * c) = lo;
        *reinterpret_cast<uint4*>(out + 64 * gp + 32 + 8 * c) = hi;
    }
}
template <int TYPE>
__global__ void __launch_bounds__(F16_WARPS * 32) rows_to_f16_kernel(const uint8_t* __restrict__ w, long long elems, int run, __half* __restrict__ out) {
    pdl_launch_dependents();
    using U = F16Unit<TYPE>;
    __shared__ __align__(16) uint8_t s_raw[F16_WARPS][(F16_BYTES + 15) & ~15];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long unit0 = ((long long)blockIdx.x * F16_WARPS + warp) * run, units = (elems + 255) / 256;
    const int n = (int)(units - unit0 < run ? units - unit0 : run);
    int off = 0;
    if (n > 0) {
        const long long beg = unit0 * U::BYTES;
        const long long all = (elems / type_block_elems(TYPE)) * type_block_bytes(TYPE);      // bytes of the matrix
        const long long end = beg + (long long)n * U::BYTES < all ? beg + (long long)n * U::BYTES : all;
        const uintptr_t a = (uintptr_t)(w + beg);
        off = (int)(a & 15);
        const int words = (int)((off + (end - beg) + 15) / 16);
        const uint8_t* p = (const uint8_t*)(a & ~(uintptr_t)15);
        constexpr int WORDS = ((F16_RUN * U::BYTES + 30) / 16 + 31) / 32;      // of 16 bytes, per lane
        uint4 raw[WORDS];
#pragma unroll
        for (int k = 0; k < WORDS; k++) {
            const int i = lane + 32 * k;
            if (i >= words) continue;
            const uint8_t* q = p + 16 * i;
            if (q >= w && q + 16 <= w + all) raw[k] = __ldg(reinterpret_cast<const uint4*>(q));
            else {                                          // a word that begins before the matrix or ends behind it
                uint32_t v[4] = {0u, 0u, 0u, 0u};
                for (int j = 0; j < 16; j++)
                    if (q + j >= w && q + j < w + all) v[j >> 2] |= (uint32_t)__ldg(q + j) << (8 * (j & 3));
                raw[k] = make_uint4(v[0], v[1], v[2], v[3]);
            }
        }
#pragma unroll
        for (int k = 0; k < WORDS; k++)
            if (lane + 32 * k < words) *reinterpret_cast<uint4*>(&s_raw[warp][16 * (lane + 32 * k)]) = raw[k];
    }
    __syncwarp();
    pdl_wait();
    constexpr int PER = 32 / U::LANES;
    for (int u = lane / U::LANES; u < n; u += PER) {
        const long long left = elems - (unit0 + u) * 256;
        f16_unit<TYPE>(&s_raw[warp][off + u * U::BYTES], lane % U::LANES, out + (unit0 + u) * 256, left < 256 ? (int)left : 256);
    }
}
inline int f16_run_of(long long elems, int n_sm) { return elems >= 2LL * n_sm * F16_WARPS * F16_RUN * 256 ? F16_RUN : 2; }
inline void (*rows_to_f16_for(int type))(const uint8_t*, long long, int, __half*) {
    return type == T_Q4_K ? rows_to_f16_kernel<T_Q4_K> : type == T_Q5_K ? rows_to_f16_kernel<T_Q5_K> : type == T_Q6_K ? rows_to_f16_kernel<T_Q6_K> : rows_to_f16_kernel<T_Q8_0>;
}

namespace tc16 {
using tc_t = __half;
constexpr bool TC_BF16 = false, TC_W_WAITS = true;
__device__ __forceinline__ void next_grid() { pdl_launch_dependents(); }
__device__ __forceinline__ void wait_grid() { pdl_wait(); }
enum { EPI_STORE = 0, EPI_ADD = 1, EPI_SILU_GLU = 2 };
constexpr bool epi_is_glu(int epi) { return epi == EPI_SILU_GLU; }
constexpr bool epi_is_act(int epi) { return epi == EPI_SILU_GLU; }
template <typename T> __device__ __forceinline__ T from_f(float v);
template <> __device__ __forceinline__ __half from_f<__half>(float v) { return f2h_sat(v); }
// silu(gate) * up (simd.rs:598-649), for an fp16 result
template <int EPI> __device__ __forceinline__ float glu_fast(float g, float up) { return g / (1.0f + expf(-g)) * up; }
template <typename T, int EPI> __device__ __forceinline__ void epi_store(void* Y, size_t idx, float v, float2) {
    if (EPI == EPI_ADD) reinterpret_cast<float*>(Y)[idx] += v;
    else reinterpret_cast<float*>(Y)[idx] = v;
}
template <typename T, int EPI> __device__ __forceinline__ void* seg_rows(void* Y, size_t off) {
    return epi_is_act(EPI) ? (void*)(reinterpret_cast<T*>(Y) + off) : (void*)(reinterpret_cast<float*>(Y) + off);
}
#include "gemm_tc.cuh"

template <int TN, bool PERSISTENT, int EPI, bool PAIR = false>
cudaError_t launch_as(const CUtensorMap& xm, const CUtensorMap& wm, const TcArgs& a, dim3 grid, bool pdl, cudaStream_t st) {
    constexpr size_t smem = tc_smem_bytes<TN, PERSISTENT>(epi_is_glu(EPI));
    auto kern = PERSISTENT ? lp_gemm_tc_kernel<TN, EPI, PAIR> : lp_gemm_tc_split_kernel<(TN > 128 ? 128 : TN), EPI>;
    static bool once[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !once[dev]) {
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64) once[dev] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(TC_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[2];
    int n = 0;
    if (pdl) {
        at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (PAIR || (!PERSISTENT && a.splits > 1)) {
        at[n].id = cudaLaunchAttributeClusterDimension;
        at[n].val.clusterDim.x = PAIR ? 2u : (unsigned)a.splits;
        at[n].val.clusterDim.y = at[n].val.clusterDim.z = 1;
        n++;
    }
    cfg.attrs = at;
    cfg.numAttrs = n;
    return cudaLaunchKernelEx(&cfg, kern, xm, wm, a);
}
template <int EPI> cudaError_t launch_epi(const TcPlan& pl, const CUtensorMap& xm, const CUtensorMap& wm, const TcArgs& a, bool pdl, cudaStream_t st) {
    const int per = epi_is_glu(EPI) ? TC_M / 2 : TC_M, n_mt = (a.N + per - 1) / per, n_nt = (a.R + pl.tn - 1) / pl.tn;
    if (pl.pair) {
        const int two = (n_mt + 1) / 2 * n_nt;
        return launch_as<256, true, EPI, true>(xm, wm, a, dim3(2 * (two < 74 ? two : 74)), pdl, st);
    }
    if (pl.persistent) {
        const dim3 grid(n_mt * n_nt < 148 ? n_mt * n_nt : 148);
        return pl.tn == 256 ? launch_as<256, true, EPI>(xm, wm, a, grid, pdl, st) : launch_as<128, true, EPI>(xm, wm, a, grid, pdl, st);
    }
    const dim3 grid(n_mt * pl.splits, n_nt);
    return pl.tn == 128 ? launch_as<128, false, EPI>(xm, wm, a, grid, pdl, st) : launch_as<64, false, EPI>(xm, wm, a, grid, pdl, st);
}
// Y[t][n] = epi(sum_k x[t][k] w[n][k] + bias[n]), T rows, N outputs (EPI_SILU_GLU: N units from the 2 N rows [gate | up] of w, fp16 Y).
// cudaErrorNotSupported: a tensor map was refused, nothing was launched
inline cudaError_t product(int epi, const __half* x, int ldx, const __half* w, int N, int K, void* y, int ldy, int T, const float* bias, int* err, int pairs, bool pdl, cudaStream_t st) {
    const bool glu = epi_is_glu(epi);
    const TcPlan pl = tc_plan(T, N, K, 1, 0, false, glu, true, false, pairs);
    const int kh = pl.tn == 256 ? TcRing<256>::KH : TcRing<128>::KH;
    CUtensorMap xm, wm;
    if (!tc_map(&xm, x, K, T, ldx, 1, 1, 0, pl.pair ? 128 : pl.tn, kh) || !tc_map(&wm, w, K, N, K, glu ? 2 : 1, 1, 0, glu ? TC_M / 2 : TC_M, kh)) return cudaErrorNotSupported;
    const TcArgs a{y, ldy, T, N, K, 1.0f, err, nullptr, 1, 0, 0, bias, float2{0.0f, 0.0f}, pl.splits, K % TC_K == 0 ? 1 : 0};
    return epi == EPI_STORE ? launch_epi<EPI_STORE>(pl, xm, wm, a, pdl, st) : epi == EPI_ADD ? launch_epi<EPI_ADD>(pl, xm, wm, a, pdl, st) : launch_epi<EPI_SILU_GLU>(pl, xm, wm, a, pdl, st);
}
}  // namespace tc16
}  // namespace b200
