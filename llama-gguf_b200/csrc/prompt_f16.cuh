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

// eight consecutive elements k0 + 8c .. of a Q4_K row (k0 % 64 == 0), as u2_deq64_q4k computes them
__device__ __forceinline__ uint4 f16_deq8_q4k(const uint8_t* row, int k0, int c) {
    const uint8_t* blk = row + (long long)(k0 >> 8) * 144;
    const int gp = (k0 & 255) >> 6, hi = c >> 2, b = 16 * (gp & 1) + 8 * hi;
    const uint4 hdr = __ldg(reinterpret_cast<const uint4*>(blk));
    const uint2 q = __ldg(reinterpret_cast<const uint2*>(blk + 16 + 32 * gp + 8 * (c & 3)));
    const float d = half_bits_to_float(hdr.x), dmin = half_bits_to_float(hdr.x >> 16);
    int s, m;
    if (gp < 2) {
        s = (hdr.y >> b) & 63;
        m = (hdr.z >> b) & 63;
    } else {
        s = ((hdr.w >> b) & 15) | (((hdr.y >> (b + 6)) & 3) << 4);
        m = ((hdr.w >> (b + 4)) & 15) | (((hdr.z >> (b + 6)) & 3) << 4);
    }
    const float ds = __fmul_rn(d, (float)s) * 16777216.0f, cm = -__fmul_rn(dmin, (float)m);      // nibbles as subnormal fp16: q 2^-24
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

// rows x K elements -> fp16 [rows][K].  A thread unpacks one chunk of 8 in F16_ROWS rows (independent loads in flight); bound by DRAM: 0.56 to
// 1.06 bytes in, 2 out per element.  The blocks are read and unpacked before the wait for the kernel before (a product that may still read the scratch rows).
constexpr int F16_ROWS = 4;
__global__ void __launch_bounds__(256) rows_to_f16_kernel(int type, const uint8_t* __restrict__ w, long long row_bytes, int rows, int K, __half* __restrict__ out) {
    pdl_launch_dependents();
    const int ch = blockIdx.x * 256 + threadIdx.x;
    if (ch * 8 >= K) return;
    const int k0 = (ch * 8) & ~63, c = ch & 7, r0 = blockIdx.y * F16_ROWS;
    uint4 v[F16_ROWS];
    if (type == T_Q4_K && (((uintptr_t)w | (uintptr_t)row_bytes) & 15) == 0) {
#pragma unroll
        for (int u = 0; u < F16_ROWS; u++) v[u] = f16_deq8_q4k(w + (long long)min(r0 + u, rows - 1) * row_bytes, k0, c);
    } else {
#pragma unroll
        for (int u = 0; u < F16_ROWS; u++) v[u] = umma_deq8<false>(type, w + (long long)min(r0 + u, rows - 1) * row_bytes, k0, c);
    }
    pdl_wait();
#pragma unroll
    for (int u = 0; u < F16_ROWS; u++)
        if (r0 + u < rows) *reinterpret_cast<uint4*>(out + (size_t)(r0 + u) * K + ch * 8) = v[u];
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

template <int TN, bool PERSISTENT, int EPI>
cudaError_t launch_as(const CUtensorMap& xm, const CUtensorMap& wm, const TcArgs& a, dim3 grid, bool pdl, cudaStream_t st) {
    constexpr size_t smem = tc_smem_bytes<TN, PERSISTENT>(epi_is_glu(EPI));
    auto kern = PERSISTENT ? lp_gemm_tc_kernel<TN, EPI> : lp_gemm_tc_split_kernel<(TN > 128 ? 128 : TN), EPI>;
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
    if (!PERSISTENT && a.splits > 1) {
        at[n].id = cudaLaunchAttributeClusterDimension;
        at[n].val.clusterDim.x = (unsigned)a.splits;
        at[n].val.clusterDim.y = at[n].val.clusterDim.z = 1;
        n++;
    }
    cfg.attrs = at;
    cfg.numAttrs = n;
    return cudaLaunchKernelEx(&cfg, kern, xm, wm, a);
}
template <int EPI> cudaError_t launch_epi(const TcPlan& pl, const CUtensorMap& xm, const CUtensorMap& wm, const TcArgs& a, bool pdl, cudaStream_t st) {
    const int per = epi_is_glu(EPI) ? TC_M / 2 : TC_M, n_mt = (a.N + per - 1) / per, n_nt = (a.R + pl.tn - 1) / pl.tn;
    if (pl.persistent) {
        const dim3 grid(n_mt * n_nt < 148 ? n_mt * n_nt : 148);
        return pl.tn == 256 ? launch_as<256, true, EPI>(xm, wm, a, grid, pdl, st) : launch_as<128, true, EPI>(xm, wm, a, grid, pdl, st);
    }
    const dim3 grid(n_mt * pl.splits, n_nt);
    return pl.tn == 128 ? launch_as<128, false, EPI>(xm, wm, a, grid, pdl, st) : launch_as<64, false, EPI>(xm, wm, a, grid, pdl, st);
}
// Y[t][n] = epi(sum_k x[t][k] w[n][k] + bias[n]), T rows, N outputs (EPI_SILU_GLU: N units from the 2 N rows [gate | up] of w, fp16 Y).
// cudaErrorNotSupported: a tensor map was refused, nothing was launched
inline cudaError_t product(int epi, const __half* x, int ldx, const __half* w, int N, int K, void* y, int ldy, int T, const float* bias, int* err, bool pdl, cudaStream_t st) {
    const bool glu = epi_is_glu(epi);
    const TcPlan pl = tc_plan(T, N, K, 1, 0, false, glu, true);
    const int kh = pl.tn == 256 ? TcRing<256>::KH : TcRing<128>::KH;
    CUtensorMap xm, wm;
    if (!tc_map(&xm, x, K, T, ldx, 1, 1, 0, pl.tn, kh) || !tc_map(&wm, w, K, N, K, glu ? 2 : 1, 1, 0, glu ? TC_M / 2 : TC_M, kh)) return cudaErrorNotSupported;
    const TcArgs a{y, ldy, T, N, K, 1.0f, err, nullptr, 1, 0, 0, bias, float2{0.0f, 0.0f}, pl.splits, K % TC_K == 0 ? 1 : 0};
    return epi == EPI_STORE ? launch_epi<EPI_STORE>(pl, xm, wm, a, pdl, st) : epi == EPI_ADD ? launch_epi<EPI_ADD>(pl, xm, wm, a, pdl, st) : launch_epi<EPI_SILU_GLU>(pl, xm, wm, a, pdl, st);
}
}  // namespace tc16
}  // namespace b200
