// attn_umma.cuh — causal GQA attention of a prompt chunk on the 5th-generation tensor cores (tcgen05 / TMEM).
//
// Same function as prefill_attn_kernel (prefill.cuh) and as the reference's attention_cached applied to T rows
// (src/backend/cpu/ops.rs:1479-1537: s[p] = dot(q, K[p]) * scale, softmax over p <= pos, out = sum s[p] * V[p]; GQA map
// kv_head = head / (n_heads / n_kv), ops.rs:1513), but the two contractions run as tcgen05.mma instead of one warp per
// (token, kv head) on CUDA cores — that kernel was 40 % of a 2048-token prefill and had no tensor instruction at all.
//
// A CTA owns 128 query ROWS = (128 / G tokens) x (the G query heads of one kv head): the rows share every K / V tile.
//   prep   prefill_kv16_kernel rounds the f32 cache rows 0 .. kv_end-1 of the layer to fp16 once per chunk:
//          K16[kv][pos][hd] and the transpose Vt16[kv][hd][pos] (both operands of a tcgen05.mma are K-major), pad rows zeroed;
//   tile   of 64 keys: TMA (SWIZZLE_128B boxes) -> S = Q K^T (tcgen05.mma kind::f16, M = 128, N = 64) into one of two TMEM buffers; two threads
//          per row (32 keys each) scale, mask keys > the query position, agree on the running maximum, and write e = exp(s - max) into a
//          swizzled P tile; O += P V (N = hd) accumulates in TMEM.  O is rescaled only when a row's maximum has grown by more than 2^8 since
//          the last time; the division by the sum comes last.
// Q, K, P and V are carried as fp16 PAIRS (hi + lo, 22 significant bits) and a product as hi hi + lo hi + hi lo: an attention output is an
// average with heavy cancellation, so single-fp16 operands put 2^-12 of relative noise on it — measured: the logits of a 300-token prompt
// moved from 6e-4 to 1.1e-3 of the oracle's.
// Roles: 8 softmax warps, a loader thread (two stages of K and of V^T), an MMA thread that issues the next tile's scores before it waits for this
// tile's probabilities.  What bounds it: the serial chain of a tile -- TMEM load, the two halves' maximum, exponentials, store of P (one buffer, which the products of the tile
// before must have left) -- with one CTA per SM to hide it: 5300 clocks per tile, 1536 of them tensor pipe (6 x 256: M = 128, N = 64, K = hd and back, 29 %
// busy).  The kernel before made two passes over the keys (maximum and sum, then values): 12000 clocks per tile, 358 us per layer of 2048 tokens (32 heads
// over 8) against 157 us now.
// f32 scores / softmax / accumulation.  Every wait is bounded and reports through p.err.
#pragma once
#include <cuda.h>
#include "gemm_umma2.cuh"
#include "ring.cuh"

namespace b200 {

struct AttnUmmaParams {
    const float* qkv;      // [T][ld], q rotated (f32)
    int ld;
    __half* out;           // [T][ldo]: [n_heads][hd] per token, fp16
    int ldo;
    int pos0, T, n_heads, n_kv, G;
    int P;                 // padded position capacity of the fp16 copies (multiple of 128)
    float scale;
    int* err;
};

// fp16 hi / lo pairs of one layer's cache rows 0 .. kv_end-1 (zero up to kv_pad): K16[kv][pos][hd] and the transpose
// Vt16[kv][hd][pos]; hi = fp16(x), lo = fp16(x - hi); the lo halves follow the hi halves (rows n_kv * P ... / n_kv * hd ...).
// grid (kv_pad / 64, n_kv), 256 threads; HD = 64 or 128.
template <int HD>
__global__ void __launch_bounds__(256) prefill_kv16_kernel(const float* __restrict__ kc, const float* __restrict__ vc, int max_seq, int kv_end, int P,
                                                           __half* __restrict__ k16, __half* __restrict__ vt16) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ __half tile[64][HD + 2], tile_lo[64][HD + 2];
    const int kh = blockIdx.y, n_kv = gridDim.y, p0 = blockIdx.x * 64;
    const float* ks = kc + (size_t)kh * max_seq * HD;
    const float* vs = vc + (size_t)kh * max_seq * HD;
    auto half4 = [](float4 f, uint2& hi, uint2& lo) {
        const float v[4] = {fminf(fmaxf(f.x, -65504.0f), 65504.0f), fminf(fmaxf(f.y, -65504.0f), 65504.0f), fminf(fmaxf(f.z, -65504.0f), 65504.0f), fminf(fmaxf(f.w, -65504.0f), 65504.0f)};
        const __half2 a = __floats2half2_rn(v[0], v[1]), b = __floats2half2_rn(v[2], v[3]);
        const float2 af = __half22float2(a), bf = __half22float2(b);
        const __half2 c = __floats2half2_rn(v[0] - af.x, v[1] - af.y), d = __floats2half2_rn(v[2] - bf.x, v[3] - bf.y);
        hi = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
        lo = make_uint2(*reinterpret_cast<const uint32_t*>(&c), *reinterpret_cast<const uint32_t*>(&d));
    };
    // four channels per thread in (NB times, all loads first), eight positions of a channel out (2048 positions of 8 heads: 20 -> 9 us against one by one)
    constexpr int NB = HD / 32;
#pragma unroll
    for (int h = 0; h < 2; h++) {
        float4 k[NB], v[NB];
#pragma unroll
        for (int u = 0; u < NB; u++) {
            const int i = 4 * (threadIdx.x + 256 * (h * NB + u)), pr = i / HD, d = i - pr * HD, pos = p0 + pr;
            const bool ok = pos < kv_end;
            k[u] = ok ? *reinterpret_cast<const float4*>(ks + (size_t)pos * HD + d) : make_float4(0.f, 0.f, 0.f, 0.f);
            v[u] = ok ? *reinterpret_cast<const float4*>(vs + (size_t)pos * HD + d) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int u = 0; u < NB; u++) {
            const int i = 4 * (threadIdx.x + 256 * (h * NB + u)), pr = i / HD, d = i - pr * HD, pos = p0 + pr;
            uint2 hi, lo;
            half4(k[u], hi, lo);
            *reinterpret_cast<uint2*>(k16 + ((size_t)kh * P + pos) * HD + d) = hi;
            *reinterpret_cast<uint2*>(k16 + ((size_t)(n_kv + kh) * P + pos) * HD + d) = lo;
            half4(v[u], hi, lo);
            *reinterpret_cast<uint32_t*>(&tile[pr][d]) = hi.x;
            *reinterpret_cast<uint32_t*>(&tile[pr][d + 2]) = hi.y;
            *reinterpret_cast<uint32_t*>(&tile_lo[pr][d]) = lo.x;
            *reinterpret_cast<uint32_t*>(&tile_lo[pr][d + 2]) = lo.y;
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 8 * HD; i += 256) {      // eight lanes: the 64 positions of a channel
        const int d = i >> 3, pr = 8 * (i & 7);
        uint32_t a[4], b[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const __half2 x = __halves2half2(tile[pr + 2 * u][d], tile[pr + 2 * u + 1][d]), y = __halves2half2(tile_lo[pr + 2 * u][d], tile_lo[pr + 2 * u + 1][d]);
            a[u] = *reinterpret_cast<const uint32_t*>(&x);
            b[u] = *reinterpret_cast<const uint32_t*>(&y);
        }
        *reinterpret_cast<uint4*>(vt16 + ((size_t)kh * HD + d) * P + p0 + pr) = make_uint4(a[0], a[1], a[2], a[3]);
        *reinterpret_cast<uint4*>(vt16 + ((size_t)(n_kv + kh) * HD + d) * P + p0 + pr) = make_uint4(b[0], b[1], b[2], b[3]);
    }
}

constexpr int kAttnTK = 64;   // keys per tile

__device__ __forceinline__ void au_ld32(uint32_t (&v)[32], uint32_t taddr) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
          "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]),
          "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]),
          "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void au_st32(uint32_t taddr, const uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31};" ::"r"(v[0]), "r"(v[1]),
        "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]),
        "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]),
        "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31]), "r"(taddr)
        : "memory");
}
__device__ __forceinline__ float au_ex2(float z) {      // 2^z by the special-function unit (relative error about 2^-22)
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(z));
    return r;
}

template <int HD> struct AttnUmmaSmem {          // Q, two stages of K and of V^T, P: each hi + lo
    static constexpr int Q = 128 * HD * 2, K = kAttnTK * HD * 2, V = HD * kAttnTK * 2, P = 128 * kAttnTK * 2;
    static constexpr int K_AT = 2 * Q, V_AT = K_AT + 4 * K, P_AT = V_AT + 4 * V, MX_AT = P_AT + 2 * P, BAR_AT = MX_AT + 2 * 128 * 4, BYTES = BAR_AT + 128;
};
constexpr int kAttnTcThreads = 320, kAttnLoader = 8, kAttnMma = 9;

template <int HD>
__global__ void __launch_bounds__(kAttnTcThreads, 1) prefill_attn_umma_kernel(const __grid_constant__ CUtensorMap kmap, const __grid_constant__ CUtensorMap vmap,
                                                                            const AttnUmmaParams p) {
    extern __shared__ __align__(1024) uint8_t au_smem[];
    using SM = AttnUmmaSmem<HD>;
    constexpr int NS = HD / 64;                     // 64-element slabs along hd
    pdl_launch_dependents();
    const uint32_t base = umma_smem_u32(au_smem);
    if (base & 1023u) {                             // the swizzle is on absolute address bits (there is no static shared memory in front)
        if (threadIdx.x == 0 && p.err) atomicExch(p.err, 20);
        return;
    }
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int G = p.G, TQ = 128 / G;
    const int qt = (int)gridDim.x - 1 - (int)blockIdx.x;   // heavy (late) query tiles first
    const int kh = blockIdx.y, t0 = qt * TQ;
    const uint32_t bars = base + SM::BAR_AT, s_tmem = bars + 120u;
    const uint32_t k_full = bars, k_empty = bars + 16u, v_full = bars + 32u, v_empty = bars + 48u, s_full = bars + 64u, s_empty = bars + 80u, q_full = bars + 96u,
                   p_full = bars + 104u, pv_done = bars + 112u;
    if (tid == 0) {
        for (int i = 0; i < 2; i++) {
            u2_mbar_init(k_full + 8u * i, 1);
            u2_mbar_init(k_empty + 8u * i, 1);
            u2_mbar_init(v_full + 8u * i, 1);
            u2_mbar_init(v_empty + 8u * i, 1);
            u2_mbar_init(s_full + 8u * i, 1);
            u2_mbar_init(s_empty + 8u * i, 8);      // one arrive per softmax warp
        }
        u2_mbar_init(q_full, 8);
        u2_mbar_init(p_full, 8);
        u2_mbar_init(pv_done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == kAttnMma) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s_tmem), "r"(256) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    uint32_t tmem;
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(tmem) : "r"(s_tmem));
    const uint32_t tO = tmem + 128u;                // S: columns 0..63 and 64..127, O: 128..128+HD-1
    const int nt = (p.pos0 + min(t0 + TQ, p.T) + kAttnTK - 1) / kAttnTK;     // key tiles that the block's queries see
    pdl_wait();
    bool alive = true;
    long long waited = 0;

    if (warp == kAttnLoader) {
        int asked_k = 0, asked_v = 0;
        for (int j = 0; j < nt; j++) {
            const uint32_t b = j & 1, ph = ((j >> 1) & 1) ^ 1;
            u2_wait(k_empty + 8u * b, ph, alive, p.err, 21, waited);
            alive = __all_sync(0xffffffffu, alive);
            if (!alive) break;
            if (u2_elect()) {
                u2_expect_tx(k_full + 8u * b, (uint32_t)(2 * SM::K));
#pragma unroll
                for (int h = 0; h < 2; h++)
#pragma unroll
                    for (int s = 0; s < NS; s++)
                        u2_tma_2d(base + SM::K_AT + (2 * b + h) * SM::K + s * (kAttnTK * 128), &kmap, s * 64, (h * p.n_kv + kh) * p.P + j * kAttnTK, k_full + 8u * b);
            }
            __syncwarp();
            asked_k = j + 1;
            u2_wait(v_empty + 8u * b, ph, alive, p.err, 22, waited);
            alive = __all_sync(0xffffffffu, alive);
            if (!alive) break;
            if (u2_elect()) {
                u2_expect_tx(v_full + 8u * b, (uint32_t)(2 * SM::V));
#pragma unroll
                for (int h = 0; h < 2; h++) u2_tma_2d(base + SM::V_AT + (2 * b + h) * SM::V, &vmap, j * kAttnTK, (h * p.n_kv + kh) * HD, v_full + 8u * b);
            }
            __syncwarp();
            asked_v = j + 1;
        }
        if (!alive) {                           // gave up: what has been asked for lands first (bounded)
            auto land = [&](uint32_t full, int asked) {
                ring_in_flight<2>(asked, [&](int stage, unsigned parity) {
                    bool w = true;
                    u2_wait(full + 8u * stage, parity, w, nullptr, 0, waited);
                });
            };
            land(k_full, asked_k);
            land(v_full, asked_v);
        }
    } else if (warp == kAttnMma) {
        const uint32_t idS = umma_idesc(128, kAttnTK), idO = umma_idesc(128, HD);
        const uint64_t dQ = umma_desc(base), dP = umma_desc(base + SM::P_AT);
        auto scores = [&](int j) {              // S = Q_hi K_hi^T + Q_lo K_hi^T + Q_hi K_lo^T
            const uint32_t b = j & 1, ph = (j >> 1) & 1;
            u2_wait(k_full + 8u * b, ph, alive, p.err, 23, waited);
            u2_wait(s_empty + 8u * b, ph ^ 1u, alive, p.err, 24, waited);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint64_t dK = umma_desc(base + SM::K_AT + 2 * b * SM::K);
            alive = __all_sync(0xffffffffu, alive);
            const bool lead = u2_elect();
            if (lead && alive) {
#pragma unroll
                for (int t = 0; t < 3; t++) {
                    const uint64_t da = dQ + (t == 1 ? SM::Q / 16 : 0), db = dK + (t == 2 ? SM::K / 16 : 0);
#pragma unroll
                    for (int s = 0; s < NS; s++)
#pragma unroll
                        for (int kk = 0; kk < 4; kk++)
                            umma_f16(tmem + b * kAttnTK, da + (uint64_t)(s * (128 * 128 / 16) + 2 * kk), db + (uint64_t)(s * (kAttnTK * 128 / 16) + 2 * kk), idS,
                                     (t > 0 || s > 0 || kk > 0) ? 1u : 0u);
                }
            }
            if (lead) {
                umma_commit(k_empty + 8u * b);
                umma_commit(s_full + 8u * b);
            }
            __syncwarp();
        };
        u2_wait(q_full, 0, alive, p.err, 25, waited);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        scores(0);
        for (int j = 0; j < nt; j++) {
            const uint32_t b = j & 1;
            if (j + 1 < nt) scores(j + 1);
            u2_wait(v_full + 8u * b, (j >> 1) & 1, alive, p.err, 26, waited);
            u2_wait(p_full, j & 1, alive, p.err, 27, waited);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint64_t dV = umma_desc(base + SM::V_AT + 2 * b * SM::V);
            alive = __all_sync(0xffffffffu, alive);
            const bool lead = u2_elect();
            if (lead && alive) {                // O += P_hi V_hi + P_lo V_hi + P_hi V_lo
#pragma unroll
                for (int t = 0; t < 3; t++) {
                    const uint64_t da = dP + (t == 1 ? SM::P / 16 : 0), db = dV + (t == 2 ? SM::V / 16 : 0);
#pragma unroll
                    for (int kk = 0; kk < kAttnTK / 16; kk++) umma_f16(tO, da + (uint64_t)(2 * kk), db + (uint64_t)(2 * kk), idO, (j > 0 || t > 0 || kk > 0) ? 1u : 0u);
                }
            }
            if (lead) {
                umma_commit(v_empty + 8u * b);
                umma_commit(pv_done);
            }
            __syncwarp();
        }
    } else {
        // threads t and t + 128 share query row t & 127 (TMEM lane t & 127): row r = (token t0 + r / G, head kh * G + r % G); they split every tile's 64
        // keys and the head dimension
        const int r = tid & 127, half = tid >> 7, tq = t0 + r / G, g = r % G;
        {   // Q row, f32 -> fp16 hi / lo, swizzled K-major; each thread of the pair converts half of the row's 16-byte chunks
            const float* qrow = p.qkv + (size_t)min(tq, p.T - 1) * p.ld + (size_t)(kh * G + g) * HD;
#pragma unroll
            for (int cc = 0; cc < HD / 16; cc++) {
                const int c = half * (HD / 16) + cc;    // chunk of 8 elements
                const float4 a = *reinterpret_cast<const float4*>(qrow + 8 * c), b = *reinterpret_cast<const float4*>(qrow + 8 * c + 4);
                const float f[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
                uint32_t wh[4], wl[4];
#pragma unroll
                for (int h = 0; h < 4; h++) {
                    const float x0 = fminf(fmaxf(f[2 * h], -65504.0f), 65504.0f), x1 = fminf(fmaxf(f[2 * h + 1], -65504.0f), 65504.0f);
                    const __half2 hi = __floats2half2_rn(x0, x1);
                    const float2 hf = __half22float2(hi);
                    wh[h] = *reinterpret_cast<const uint32_t*>(&hi);
                    wl[h] = umma_pack_h2(x0 - hf.x, x1 - hf.y);
                }
                const uint32_t off = (uint32_t)(c >> 3) * (128 * 128) + umma_sw128(r, c & 7);
                *reinterpret_cast<uint4*>(au_smem + off) = make_uint4(wh[0], wh[1], wh[2], wh[3]);
                *reinterpret_cast<uint4*>(au_smem + SM::Q + off) = make_uint4(wl[0], wl[1], wl[2], wl[3]);
            }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) u2_mbar_arrive(q_full);
        const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
        const int pos_q = p.pos0 + min(tq, p.T - 1);         // this row attends keys 0 .. pos_q
        const float scale2 = p.scale * 1.4426950408889634f;      // scores in powers of two
        float* mx_s = reinterpret_cast<float*>(au_smem + SM::MX_AT);     // [2 halves][128 rows]
        float m = -INFINITY, l = 0.0f;
        for (int j = 0; j < nt; j++) {
            const uint32_t b = j & 1;
            uint32_t v[32];
            u2_wait(s_full + 8u * b, (j >> 1) & 1, alive, p.err, 28, waited);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            au_ld32(v, tmem + b * kAttnTK + lanes + (uint32_t)(half * 32));
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) u2_mbar_arrive(s_empty + 8u * b);
            float s[32];
#pragma unroll
            for (int q = 0; q < 32; q++) s[q] = __uint_as_float(v[q]) * scale2;
            const int seen = pos_q - (j * kAttnTK + half * 32);      // keys 0 .. seen of this half
            if (!__all_sync(0xffffffffu, seen >= 31)) {
#pragma unroll
                for (int q = 0; q < 32; q++) s[q] = q <= seen ? s[q] : -INFINITY;
            }
            float x0 = s[0], x1 = s[1];
#pragma unroll
            for (int q = 2; q < 32; q += 2) {
                x0 = fmaxf(x0, s[q]);
                x1 = fmaxf(x1, s[q + 1]);
            }
            mx_s[half * 128 + r] = fmaxf(x0, x1);
            asm volatile("bar.sync 1, 256;" ::: "memory");
            const float mx = fmaxf(mx_s[r], mx_s[128 + r]);
            if (j > 0) {                            // the products of the tile before are done: P is free, O may be rescaled
                u2_wait(pv_done, (j - 1) & 1, alive, p.err, 29, waited);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            }
            if (__any_sync(0xffffffffu, mx > m + 8.0f)) {          // (the same for both warps of these rows)
                const float mn = fmaxf(m, mx), c = m == -INFINITY ? 0.0f : au_ex2(m - mn);
                l *= c;
                m = mn;
                if (j > 0) {
#pragma unroll 1
                    for (int n = 0; n < HD / 2; n += 32) {
                        uint32_t o[32];
                        const uint32_t at = tO + lanes + (uint32_t)(half * (HD / 2) + n);
                        au_ld32(o, at);
#pragma unroll
                        for (int q = 0; q < 32; q++) o[q] = __float_as_uint(__uint_as_float(o[q]) * c);
                        au_st32(at, o);
                    }
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                }
            }
#pragma unroll
            for (int c = 0; c < 4; c++) {          // 8 keys -> one 16-byte chunk of the row, hi and lo
                uint32_t wh[4], wl[4];
#pragma unroll
                for (int h = 0; h < 4; h++) {
                    const float e0 = au_ex2(s[8 * c + 2 * h] - m), e1 = au_ex2(s[8 * c + 2 * h + 1] - m);      // (key 0 is visible to every row: m is finite)
                    l += e0 + e1;
                    const __half2 hi = __floats2half2_rn(e0, e1);
                    const float2 hf = __half22float2(hi);
                    wh[h] = *reinterpret_cast<const uint32_t*>(&hi);
                    wl[h] = umma_pack_h2(e0 - hf.x, e1 - hf.y);
                }
                const uint32_t off = SM::P_AT + umma_sw128(r, half * 4 + c);
                *reinterpret_cast<uint4*>(au_smem + off) = make_uint4(wh[0], wh[1], wh[2], wh[3]);
                *reinterpret_cast<uint4*>(au_smem + SM::P + off) = make_uint4(wl[0], wl[1], wl[2], wl[3]);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) u2_mbar_arrive(p_full);
            asm volatile("bar.sync 1, 256;" ::: "memory");      // (the maxima have been read)
        }
        mx_s[half * 128 + r] = l;
        asm volatile("bar.sync 1, 256;" ::: "memory");
        const float inv = 1.0f / (mx_s[r] + mx_s[128 + r]);
        u2_wait(pv_done, (nt - 1) & 1, alive, p.err, 30, waited);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        // O row / sum -> fp16; each thread of the pair stores half of the head dimension
        __half* orow = p.out + (size_t)min(tq, p.T - 1) * p.ldo + (size_t)(kh * G + g) * HD + half * (HD / 2);
#pragma unroll
        for (int c0 = 0; c0 < HD / 2; c0 += 32) {
            uint32_t v[32];
            au_ld32(v, tO + lanes + (uint32_t)(half * (HD / 2) + c0));
            if (tq < p.T) {
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    uint32_t w[4];
#pragma unroll
                    for (int h = 0; h < 4; h++) {
                        const __half2 hh = __halves2half2(f2h_sat(__uint_as_float(v[8 * c + 2 * h]) * inv), f2h_sat(__uint_as_float(v[8 * c + 2 * h + 1]) * inv));
                        w[h] = *reinterpret_cast<const uint32_t*>(&hh);
                    }
                    *reinterpret_cast<uint4*>(orow + c0 + 8 * c) = make_uint4(w[0], w[1], w[2], w[3]);
                }
            }
            __syncwarp();
        }
    }
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == kAttnMma) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256) : "memory");
    }
}

// fp16 copies' tensor maps: K16 as {hd, 2 * n_kv * P} (box 64 x 64 keys), Vt16 as {P, 2 * n_kv * hd} (box 64 keys x hd rows), SWIZZLE_128B
inline bool attn_umma_encode(Umma2EncodeFn encode, const __half* k16, const __half* vt16, int n_kv, int hd, int P, CUtensorMap* kmap, CUtensorMap* vmap) {
    const cuuint32_t estr[2] = {1, 1};
    {
        const cuuint64_t dims[2] = {(cuuint64_t)hd, (cuuint64_t)2 * n_kv * P};   // hi rows, then lo rows
        const cuuint64_t strides[1] = {(cuuint64_t)hd * 2};
        const cuuint32_t box[2] = {64, (cuuint32_t)kAttnTK};
        if (encode(kmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, (void*)k16, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return false;
    }
    const cuuint64_t dims[2] = {(cuuint64_t)P, (cuuint64_t)2 * n_kv * hd};   // hi rows, then lo rows
    const cuuint64_t strides[1] = {(cuuint64_t)P * 2};
    const cuuint32_t box[2] = {64, (cuuint32_t)hd};
    return encode(vmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, (void*)vt16, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Other numbers of heads per kv head keep an f32 attention (rows_attn_kernel): padded to the next power of two they would run here too, but with probabilities and values as
// pairs of fp16 in one accumulator over all keys, 2.8e-6 of the logits at 1000 keys for its 4e-7.
inline bool attn_umma_ok(int hd, int n_heads, int n_kv) {
    const int G = n_kv > 0 ? n_heads / n_kv : 0;
    return (hd == 64 || hd == 128) && n_kv > 0 && n_heads % n_kv == 0 && (G == 1 || G == 2 || G == 4 || G == 8);
}

template <int HD>
inline cudaError_t attn_umma_launch_hd(const CUtensorMap& kmap, const CUtensorMap& vmap, const AttnUmmaParams& p, bool pdl, cudaStream_t st) {
    static bool once[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !once[dev]) {
        cudaError_t e = cudaFuncSetAttribute(prefill_attn_umma_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, AttnUmmaSmem<HD>::BYTES);
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64) once[dev] = true;
    }
    const int TQ = 128 / p.G;
    dim3 grid((p.T + TQ - 1) / TQ, p.n_kv);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid; cfg.blockDim = dim3(kAttnTcThreads); cfg.dynamicSmemBytes = AttnUmmaSmem<HD>::BYTES; cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = pdl ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, prefill_attn_umma_kernel<HD>, kmap, vmap, p);
}

}  // namespace b200
