// exact_rows.cuh — a layer's products for several rows at once in f32: GGUF blocks unpacked to f32 (one rounding of scale * quant - minimum), f32 activations,
// f32 sums.  What one row gives through gemv_kernel (gemv.cuh), to the rounding of f32 sums, so the calls whose results must not take the fp16 operands of the
// tensor-core products can take several rows: short prompts, prompts of models whose blocks those products do not know (Q5_0), prompts into an int8 cache (a
// changed rounding before the codes would move codes), and steps of two to seven sequences.  The reference runs all of these token by token
// (src/model/llama.rs:327-345).
//
//   rows_few_kernel    up to 8 rows per weight pass: a warp owns R weight rows and walks K as in gemv.cuh, the rows' x lie in shared memory, an unpacked weight
//                      meets all of them.  Norm before, bias / residual / SwiGLU behind, as gemv_kernel.
//   rows_tile_kernel   64 weight rows x 128 (64) rows of x per CTA, K 32 at a time through shared memory, 8 x 8 (8 x 4) sums per thread, K cut over
//                      gridDim.z where the tiles do not fill the chip; pieces are added in order by the kernel behind (rows_norm_kernel,
//                      rows_qkv_kernel, rows_swiglu_kernel).
// The multiply-adds are packed pairs (fma.rn.f32x2): two along K in the first kernel, two weight rows in the second.
// Measured, token by token -> here: prompts through two layers of a 0.5B model (896 wide, Q5_0 / Q8_0) of 5, 16, 31 tokens 428, 1318, 2545 -> 176, 205, 301 us; of 33, 100, 333,
// 1000, 4000 tokens 2696, 8666, 29785, 94147, 453403 -> 380, 598, 1082, 2597, 10840; two 8B layers in Q4_K_M, 2, 8, 31 tokens 321, 1194, 4628 -> 300, 617, 1874, steps of 2, 4, 7
// sequences 350, 682, 1187 -> 265, 355, 513.  Distance to float64 of 0.5B prompts of 100, 333, 1000 tokens: 2.7e-7, 3.5e-7, 4.1e-7 -> 2.5e-7, 3.3e-7, 4.0e-7 (16 inputs).
#pragma once
#include "attention.cuh"
#include "gemv.cuh"
#include "misc.cuh"

namespace b200 {

__device__ __forceinline__ uint64_t f2_pack(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 f2_unpack(uint64_t v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ void f2_fma(uint64_t& d, uint64_t a, uint64_t b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b)); }
__device__ __forceinline__ void f2_add(uint64_t& d, uint64_t a) { asm("add.rn.f32x2 %0, %0, %1;" : "+l"(d) : "l"(a)); }

struct RowsSeg {
    const uint8_t* w;
    float* out;            // [T][ldo]
    const float* bias;     // optional
    long long row_bytes;
    int type, n_rows, ldo;
};
struct RowsParams {
    RowsSeg seg[3];
    int n_seg, K, T, ldx;
    const float* x;        // [T][ldx]
    const float* norm_w;   // rows_few_kernel: optional RMSNorm of the rows
    float eps;
    int epi;               // rows_few_kernel: EPI_STORE, EPI_RESIDUAL (residual: [T][ldo]), EPI_SWIGLU
    const float* residual;
    int chunk;             // rows_few_kernel: elements of K in shared memory at a time (all, or a multiple of 256)
    int k_split;           // rows_tile_kernel: elements of K per piece (a multiple of 32)
    long long piece;       // rows_tile_kernel: floats between pieces of an output
};

// ---------------------------------------------------------------- few rows
constexpr int kRowsWarps = 8;

// acc[r][t] += w[r][0..3] . x[t][0..3]; xp: row 0's four values in shared memory, rows `ld` floats apart
template <int R, int TT>
__device__ __forceinline__ void rows_fma4(const float (&w)[R][4], const float* xp, int ld, uint64_t (&acc)[R][TT]) {
    uint64_t w0[R], w1[R];
#pragma unroll
    for (int r = 0; r < R; r++) {
        w0[r] = f2_pack(w[r][0], w[r][1]);
        w1[r] = f2_pack(w[r][2], w[r][3]);
    }
#pragma unroll
    for (int t = 0; t < TT; t++) {
        const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(xp + (size_t)t * ld);
#pragma unroll
        for (int r = 0; r < R; r++) {
            f2_fma(acc[r][t], w0[r], x.x);
            f2_fma(acc[r][t], w1[r], x.y);
        }
    }
}

// The lanes' places in a row are gemv.cuh's (rows_dot_k45, rows_dot_q6k, rows_dot_b32); nb blocks from rp[r] on, xs: their elements of x.
template <bool Q5, int R, int TT>
__device__ __forceinline__ void rows_few_k45(const uint8_t* const (&rp)[R], int nb, const float* xs, int ld, int lane, uint64_t (&acc)[R][TT]) {
    constexpr int BB = Q5 ? 176 : 144, QS = Q5 ? 48 : 16;
    const int bl = lane >> 3, p = lane & 7, g = p >> 1, h = p & 1, gg = g & 1;
    for (int b = bl; b < nb; b += 4) {
        uint4 hd[R], q[R], qh[R];
#pragma unroll
        for (int r = 0; r < R; r++) {
            const uint8_t* bp = rp[r] + (size_t)b * BB;
            hd[r] = ldg_stream_u4(bp);
            q[r] = ldg_stream_u4(bp + QS + 16 * p);
            if (Q5) qh[r] = ldg_stream_u4(bp + 16 + 16 * h);
        }
        float d1[R], d2[R], m1[R], m2[R];
#pragma unroll
        for (int r = 0; r < R; r++) {
            const float d = half_bits_to_float(hd[r].x), dmin = half_bits_to_float(hd[r].x >> 16);
            const uint32_t A = (hd[r].y >> (16 * gg)) & 0xFFFFu, B = (hd[r].z >> (16 * gg)) & 0xFFFFu, C = (hd[r].w >> (16 * gg)) & 0xFFFFu;
            uint32_t scp, mnp;
            if (g < 2) {
                scp = A & 0x3F3Fu;
                mnp = B & 0x3F3Fu;
            } else {
                scp = (C & 0x0F0Fu) | ((A >> 2) & 0x3030u);
                mnp = ((C >> 4) & 0x0F0Fu) | ((B >> 2) & 0x3030u);
            }
            d1[r] = d * u8f(scp, 0); d2[r] = d * u8f(scp, 1);
            m1[r] = dmin * u8f(mnp, 0); m2[r] = dmin * u8f(mnp, 1);
        }
        const float* xp = xs + xidx(b * 256 + 64 * g + 16 * h);
#pragma unroll
        for (int wi = 0; wi < 4; wi++) {
            float lo[R][4], hi[R][4];
#pragma unroll
            for (int r = 0; r < R; r++) {
                const uint32_t qw = wi == 0 ? q[r].x : wi == 1 ? q[r].y : wi == 2 ? q[r].z : q[r].w;
                const uint32_t hw = wi == 0 ? qh[r].x : wi == 1 ? qh[r].y : wi == 2 ? qh[r].z : qh[r].w;
                uint32_t a = qw & 0x0F0F0F0Fu, b4 = (qw >> 4) & 0x0F0F0F0Fu;
                if (Q5) {
                    a |= ((hw >> (2 * g)) & 0x01010101u) << 4;
                    b4 |= ((hw >> (2 * g + 1)) & 0x01010101u) << 4;
                }
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    lo[r][k] = fmaf(d1[r], u8f(a, k), -m1[r]);
                    hi[r][k] = fmaf(d2[r], u8f(b4, k), -m2[r]);
                }
            }
            rows_fma4<R, TT>(lo, xp + 4 * wi, ld, acc);
            rows_fma4<R, TT>(hi, xp + 32 + 4 * wi, ld, acc);
        }
    }
}
template <int R, int TT>
__device__ __forceinline__ void rows_few_q6k(const uint8_t* const (&rp)[R], int nb, const float* xs, int ld, int lane, uint64_t (&acc)[R][TT]) {
    const int bl = lane >> 3, t = lane & 7, n = t >> 2, j = t & 3, is = j >> 1;
    for (int b = bl; b < nb; b += 4) {
        uint32_t qa[R][2], qb[R][2], qhv[R][2];
        float ds[R][4];
#pragma unroll
        for (int r = 0; r < R; r++) {
            const uint8_t* bp = rp[r] + (size_t)b * 210;
            const uint8_t* pa = bp + 64 * n + 8 * j;
            const uint8_t* ph = bp + 128 + 32 * n + 8 * j;
#pragma unroll
            for (int w = 0; w < 2; w++) {
                qa[r][w] = ldg_u16(pa + 4 * w) | (ldg_u16(pa + 4 * w + 2) << 16);
                qb[r][w] = ldg_u16(pa + 32 + 4 * w) | (ldg_u16(pa + 32 + 4 * w + 2) << 16);
                qhv[r][w] = ldg_u16(ph + 4 * w) | (ldg_u16(ph + 4 * w + 2) << 16);
            }
            const float d = half_bits_to_float(ldg_u16(bp + 208));
#pragma unroll
            for (int c = 0; c < 4; c++) ds[r][c] = d * (float)ldg_s8(bp + 192 + 8 * n + is + 2 * c);
        }
#pragma unroll
        for (int w = 0; w < 2; w++)
#pragma unroll
            for (int c = 0; c < 4; c++) {
                float v[R][4];
#pragma unroll
                for (int r = 0; r < R; r++) {
                    const uint32_t base = (c & 1) ? qb[r][w] : qa[r][w], hq = qhv[r][w];
                    const uint32_t top = c == 0 ? hq << 4 : c == 1 ? hq << 2 : c == 2 ? hq : hq >> 2;
                    const uint32_t u = ((c < 2 ? base : base >> 4) & 0x0F0F0F0Fu) | (top & 0x30303030u);
#pragma unroll
                    for (int k = 0; k < 4; k++) v[r][k] = ds[r][c] * u8f<32>(u, k);
                }
                rows_fma4<R, TT>(v, xs + xidx(b * 256 + 128 * n + 32 * c + 8 * j + 4 * w), ld, acc);
            }
    }
}
template <int R, int TT>
__device__ __forceinline__ void rows_few_b32(int type, const uint8_t* const (&rp)[R], int nb, const float* xs, int ld, int lane, uint64_t (&acc)[R][TT]) {
    const int bb = (type == T_F32) ? 128 : (type == T_F16) ? 64 : type_block_bytes(type);
    for (int b = lane; b < nb; b += 32) {
        const float* xp = xs + xidx(b * 32);
        if (type == T_Q8_0) {
            uint32_t qv[R][8];
            float d[R];
#pragma unroll
            for (int r = 0; r < R; r++) {
                const uint8_t* bp = rp[r] + (size_t)b * bb;
                d[r] = half_bits_to_float(ldg_u16(bp));
#pragma unroll
                for (int i = 0; i < 8; i++) qv[r][i] = (ldg_u16(bp + 2 + 4 * i) | (ldg_u16(bp + 4 + 4 * i) << 16)) ^ 0x80808080u;
            }
#pragma unroll
            for (int i = 0; i < 8; i++) {
                float v[R][4];
#pragma unroll
                for (int r = 0; r < R; r++)
#pragma unroll
                    for (int k = 0; k < 4; k++) v[r][k] = d[r] * u8f<128>(qv[r][i], k);
                rows_fma4<R, TT>(v, xp + 4 * i, ld, acc);
            }
        } else if (type == T_Q5_0 || type == T_Q4_0) {
            const bool five = type == T_Q5_0;
            uint32_t qv[R][4], qh[R];
            float d[R];
#pragma unroll
            for (int r = 0; r < R; r++) {
                const uint8_t* bp = rp[r] + (size_t)b * bb;
                d[r] = half_bits_to_float(ldg_u16(bp));
                qh[r] = five ? ldg_u16(bp + 2) | (ldg_u16(bp + 4) << 16) : 0u;
                const uint8_t* qs = bp + (five ? 6 : 2);
#pragma unroll
                for (int i = 0; i < 4; i++) qv[r][i] = ldg_u16(qs + 4 * i) | (ldg_u16(qs + 4 * i + 2) << 16);
            }
#pragma unroll
            for (int i = 0; i < 4; i++) {
                float lo[R][4], hi[R][4];
#pragma unroll
                for (int r = 0; r < R; r++) {
                    // the fifth bits as in rows_dot_b32; without them the offset is 8 instead of 16
                    const uint32_t a = (qv[r][i] & 0x0F0F0F0Fu) | ((((qh[r] >> (4 * i)) & 15u) * 0x02040810u) & 0x10101010u);
                    const uint32_t e = ((qv[r][i] >> 4) & 0x0F0F0F0Fu) | ((((qh[r] >> (16 + 4 * i)) & 15u) * 0x02040810u) & 0x10101010u);
                    const float off = five ? 0.0f : 8.0f;
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        lo[r][k] = d[r] * (u8f<16>(a, k) + off);
                        hi[r][k] = d[r] * (u8f<16>(e, k) + off);
                    }
                }
                rows_fma4<R, TT>(lo, xp + 4 * i, ld, acc);
                rows_fma4<R, TT>(hi, xp + 16 + 4 * i, ld, acc);
            }
        } else {
#pragma unroll
            for (int i = 0; i < 8; i++) {
                float v[R][4];
#pragma unroll
                for (int r = 0; r < R; r++) {
                    const uint8_t* bp = rp[r] + (size_t)b * bb;
                    if (type == T_F16) {
                        const uint2 u = ldg_stream_u2(bp + 8 * i);
                        v[r][0] = half_bits_to_float(u.x); v[r][1] = half_bits_to_float(u.x >> 16);
                        v[r][2] = half_bits_to_float(u.y); v[r][3] = half_bits_to_float(u.y >> 16);
                    } else {
                        const uint4 u = ldg_stream_u4(bp + 16 * i);
                        v[r][0] = __uint_as_float(u.x); v[r][1] = __uint_as_float(u.y); v[r][2] = __uint_as_float(u.z); v[r][3] = __uint_as_float(u.w);
                    }
                }
                rows_fma4<R, TT>(v, xp + 4 * i, ld, acc);
            }
        }
    }
}

// What bounds it: instructions, 6.6 per weight at two rows (unpacking three, T / 2 packed multiply-adds), issued in 57 % of the slots by 16 warps per SM of 128 registers (o, q / k / v and
// down, with fewer warps: 39 - 47 %): gate and up of an 8B layer take 46 us where DRAM would take 10.  grid (CTAs, ceil(T / TT)).
template <int R, int TT>
__global__ void __launch_bounds__(kRowsWarps * 32, R * TT <= 16 ? 2 : 1) rows_few_kernel(const __grid_constant__ RowsParams p) {
    constexpr int G = R / 2 > 0 ? R / 2 : 1, NV = R * TT;
    static_assert(NV <= 32 && (NV & (NV - 1)) == 0, "sums of a warp's task");
    extern __shared__ __align__(16) float xs[];
    __shared__ float red[kRowsWarps][TT], inv_s[TT];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tt0 = blockIdx.y * TT, tn = min(TT, p.T - tt0);
    int t0[4];
    t0[0] = 0;
    if (p.epi == EPI_SWIGLU) t0[1] = t0[2] = t0[3] = (p.seg[0].n_rows + G - 1) / G;
    else {
#pragma unroll
        for (int s = 0; s < 3; s++) t0[s + 1] = t0[s] + (s < p.n_seg ? (p.seg[s].n_rows + R - 1) / R : 0);
    }
    const int n_tasks = t0[3], stride = gridDim.x * kRowsWarps;
    auto seg_of = [&](int task) { return p.epi == EPI_SWIGLU ? 0 : task >= t0[2] ? 2 : task >= t0[1] ? 1 : 0; };
    auto ask = [&](int task) {      // a task's weight rows towards L2
        if (task >= n_tasks) return;
        const int s = seg_of(task), per = p.epi == EPI_SWIGLU ? G : R, row0 = (task - t0[s]) * per;
        const long long bytes = (long long)min(per, p.seg[s].n_rows - row0) * p.seg[s].row_bytes;
        for (long long o = (long long)lane * 128; o < bytes; o += 32 * 128) {
            prefetch_l2(p.seg[s].w + (long long)row0 * p.seg[s].row_bytes + o);
            if (p.epi == EPI_SWIGLU) prefetch_l2(p.seg[1].w + (long long)row0 * p.seg[1].row_bytes + o);
        }
    };
    pdl_launch_dependents();
    const int first = blockIdx.x * kRowsWarps + warp;
    if (blockIdx.y == 0) ask(first);
    pdl_wait();
    const int ld = xpad_floats(p.chunk);
    const bool whole = p.chunk >= p.K;
    const float* x = p.x + (size_t)tt0 * p.ldx;
    if (p.norm_w) {                 // 1 / rms of every row
        float ss[TT];
#pragma unroll
        for (int t = 0; t < TT; t++) ss[t] = 0.0f;
        for (int e = tid * 4; e < p.K; e += kRowsWarps * 128) {
#pragma unroll
            for (int t = 0; t < TT; t++) {
                const float4 v = t < tn ? *reinterpret_cast<const float4*>(x + (size_t)t * p.ldx + e) : make_float4(0.f, 0.f, 0.f, 0.f);
                ss[t] += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
                if (whole) *reinterpret_cast<float4*>(xs + (size_t)t * ld + xidx(e)) = v;
            }
        }
#pragma unroll
        for (int t = 0; t < TT; t++) {
            const float s = warp_sum(ss[t]);
            if (lane == 0) red[warp][t] = s;
        }
        __syncthreads();
        if (tid < TT) {
            float tot = 0.0f;
#pragma unroll
            for (int w = 0; w < kRowsWarps; w++) tot += red[w][tid];
            inv_s[tid] = 1.0f / sqrtf(tot / (float)p.K + p.eps);
        }
        __syncthreads();
    }
    auto stage = [&](int k0, int len) {
        for (int e = tid * 4; e < len; e += kRowsWarps * 128) {
            float4 w = make_float4(1.f, 1.f, 1.f, 1.f);
            if (p.norm_w) w = *reinterpret_cast<const float4*>(p.norm_w + k0 + e);
#pragma unroll
            for (int t = 0; t < TT; t++) {
                float4* at = reinterpret_cast<float4*>(xs + (size_t)t * ld + xidx(e));
                float4 v;
                if (p.norm_w && whole) v = *at;
                else v = t < tn ? *reinterpret_cast<const float4*>(x + (size_t)t * p.ldx + k0 + e) : make_float4(0.f, 0.f, 0.f, 0.f);
                if (p.norm_w) {
                    const float inv = inv_s[t];
                    v.x = (v.x * inv) * w.x; v.y = (v.y * inv) * w.y; v.z = (v.z * inv) * w.z; v.w = (v.w * inv) * w.w;
                }
                *at = v;
            }
        }
        __syncthreads();
    };
    if (whole) stage(0, p.K);
    for (int base = blockIdx.x * kRowsWarps; base < n_tasks; base += stride) {      // (the same rounds for every warp: it joins the barriers of the stages)
        const int task = base + warp;
        const bool live = task < n_tasks;
        const uint8_t* rp[R];
        int s = 0, row0 = 0, rows = 0, type = 0;
        if (live) {
            s = seg_of(task);
            const int per = p.epi == EPI_SWIGLU ? G : R;
            row0 = (task - t0[s]) * per;
            rows = min(per, p.seg[s].n_rows - row0);
            type = p.seg[s].type;
#pragma unroll
            for (int r = 0; r < R; r++) {
                const RowsSeg& sg = p.epi == EPI_SWIGLU && r >= G ? p.seg[1] : p.seg[s];
                rp[r] = sg.w + (long long)(row0 + min(p.epi == EPI_SWIGLU && r >= G ? r - G : r, rows - 1)) * sg.row_bytes;
            }
            ask(task + stride);
        }
        uint64_t acc[R][TT];
#pragma unroll
        for (int r = 0; r < R; r++)
#pragma unroll
            for (int t = 0; t < TT; t++) acc[r][t] = 0;
        for (int k0 = 0; k0 < p.K; k0 += p.chunk) {
            const int len = min(p.chunk, p.K - k0);
            if (!whole) {
                __syncthreads();
                stage(k0, len);
            }
            if (!live) continue;
            if (k0) {
                const long long step = (long long)(p.chunk / type_block_elems(type)) * type_block_bytes(type);
#pragma unroll
                for (int r = 0; r < R; r++) rp[r] += step;
            }
            switch (type) {
                case T_Q4_K: rows_few_k45<false, R, TT>(rp, len >> 8, xs, ld, lane, acc); break;
                case T_Q5_K: rows_few_k45<true, R, TT>(rp, len >> 8, xs, ld, lane, acc); break;
                case T_Q6_K: rows_few_q6k<R, TT>(rp, len >> 8, xs, ld, lane, acc); break;
                default: rows_few_b32<R, TT>(type, rp, len >> 5, xs, ld, lane, acc); break;
            }
        }
        if (!live) continue;
        // NV sums over the lanes: halves of what is left go to the lanes that differ in the next bit, then lane l holds sum l / (32 / NV)
        float v[NV];
#pragma unroll
        for (int r = 0; r < R; r++)
#pragma unroll
            for (int t = 0; t < TT; t++) {
                const float2 a = f2_unpack(acc[r][t]);
                v[r * TT + t] = a.x + a.y;
            }
#pragma unroll
        for (int o = 16, n = NV; o > 0; o >>= 1) {
            if (n > 1) {
                n >>= 1;
                const bool up = lane & o;
#pragma unroll
                for (int i = 0; i < NV / 2; i++)
                    if (i < n) {
                        const float give = up ? v[i] : v[i + n], keep = up ? v[i + n] : v[i];
                        v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
                    }
            } else v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
        }
        constexpr int LPV = 32 / NV;
        const int idx = lane / LPV, r = idx / TT, t = idx - r * TT;
        float out = v[0];
        if (p.epi == EPI_SWIGLU) {
            const float upv = __shfl_sync(0xffffffffu, out, (lane + G * TT * LPV) & 31);
            if (lane % LPV == 0 && r < G && r < rows && t < tn) p.seg[0].out[(size_t)(tt0 + t) * p.seg[0].ldo + row0 + r] = silu_f(out) * upv;
        } else if (lane % LPV == 0 && r < rows && t < tn) {
            const RowsSeg& sg = p.seg[s];
            const size_t at = (size_t)(tt0 + t) * sg.ldo + row0 + r;
            if (sg.bias) out += sg.bias[row0 + r];
            if (p.epi == EPI_RESIDUAL) out += p.residual[at];
            sg.out[at] = out;
        }
    }
}

// ---------------------------------------------------------------- tiles
// 16 consecutive elements k0 .. (k0 % 16 == 0) of a weight row: first the words, later the values
struct RowsRaw {
    uint4 a, b, c;
};
__device__ __forceinline__ uint4 ld_u16x8(const uint8_t* q) {
    uint4 v;
    v.x = ldg_u16(q) | (ldg_u16(q + 2) << 16);
    v.y = ldg_u16(q + 4) | (ldg_u16(q + 6) << 16);
    v.z = ldg_u16(q + 8) | (ldg_u16(q + 10) << 16);
    v.w = ldg_u16(q + 12) | (ldg_u16(q + 14) << 16);
    return v;
}
__device__ __forceinline__ void rows_raw(int type, const uint8_t* row, int k0, RowsRaw& w) {
    if (type == T_Q4_K || type == T_Q5_K) {
        const bool five = type == T_Q5_K;
        const uint8_t* b = row + (size_t)(k0 >> 8) * (five ? 176 : 144);
        const int e = k0 & 255;
        w.a = *reinterpret_cast<const uint4*>(b);
        w.b = *reinterpret_cast<const uint4*>(b + (five ? 48 : 16) + (e >> 6) * 32 + (e & 16));
        if (five) w.c = *reinterpret_cast<const uint4*>(b + 16 + (e & 16));
    } else if (type == T_Q6_K) {
        const uint8_t* b = row + (size_t)(k0 >> 8) * 210;
        const int e = k0 & 255, n = e >> 7, l = e & 31, c = (e >> 5) & 3;
        w.a = ld_u16x8(b + n * 64 + l + (c & 1) * 32);
        w.b = ld_u16x8(b + 128 + n * 32 + l);
        w.c.x = ldg_u16(b + 208);
        w.c.y = (uint32_t)ldg_s8(b + 192 + n * 8 + (l >> 4) + 2 * c);
    } else if (type == T_Q8_0) {
        const uint8_t* b = row + (size_t)(k0 >> 5) * 34;
        w.c.x = ldg_u16(b);
        w.a = ld_u16x8(b + 2 + (k0 & 16));
    } else if (type == T_Q5_0 || type == T_Q4_0) {
        const bool five = type == T_Q5_0;
        const uint8_t* b = row + (size_t)(k0 >> 5) * (five ? 22 : 18);
        w.c.x = ldg_u16(b);
        w.c.y = five ? ldg_u16(b + 2) | (ldg_u16(b + 4) << 16) : 0u;
        w.a = ld_u16x8(b + (five ? 6 : 2));
    } else if (type == T_F16) {
        const uint4* q = reinterpret_cast<const uint4*>(row + (size_t)k0 * 2);
        w.a = q[0];
        w.b = q[1];
    }
}
__device__ __forceinline__ void rows_values(int type, const uint8_t* row, int k0, const RowsRaw& w, float (&v)[16]) {
    const uint32_t a[4] = {w.a.x, w.a.y, w.a.z, w.a.w}, b[4] = {w.b.x, w.b.y, w.b.z, w.b.w}, c[4] = {w.c.x, w.c.y, w.c.z, w.c.w};
    if (type == T_Q4_K || type == T_Q5_K) {
        const int j = (k0 & 255) >> 5, sh = 8 * (j & 3);
        const float d = half_bits_to_float(a[0]), dmin = half_bits_to_float(a[0] >> 16);
        uint32_t sc, mn;
        if (j < 4) {
            sc = (a[1] >> sh) & 63u;
            mn = (a[2] >> sh) & 63u;
        } else {
            sc = ((a[3] >> sh) & 15u) | (((a[1] >> sh) & 0xC0u) >> 2);
            mn = ((a[3] >> sh) >> 4 & 15u) | (((a[2] >> sh) & 0xC0u) >> 2);
        }
        const float d1 = d * (float)sc, m1 = dmin * (float)mn;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            uint32_t q = ((j & 1) ? b[i] >> 4 : b[i]) & 0x0F0F0F0Fu;
            if (type == T_Q5_K) q |= ((c[i] >> j) & 0x01010101u) << 4;
#pragma unroll
            for (int k = 0; k < 4; k++) v[4 * i + k] = fmaf(d1, u8f(q, k), -m1);
        }
    } else if (type == T_Q6_K) {
        const int cc = (k0 >> 5) & 3;
        const float ds = half_bits_to_float(c[0]) * (float)(int)c[1];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const uint32_t q = ((cc & 2 ? a[i] >> 4 : a[i]) & 0x0F0F0F0Fu) | (((b[i] >> (2 * cc)) & 0x03030303u) << 4);
#pragma unroll
            for (int k = 0; k < 4; k++) v[4 * i + k] = ds * u8f<32>(q, k);
        }
    } else if (type == T_Q8_0) {
        const float d = half_bits_to_float(c[0]);
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int k = 0; k < 4; k++) v[4 * i + k] = d * u8f<128>(a[i] ^ 0x80808080u, k);
    } else if (type == T_Q5_0 || type == T_Q4_0) {
        const float d = half_bits_to_float(c[0]), off = type == T_Q5_0 ? 0.0f : 8.0f;
        const int hi = k0 & 16;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const uint32_t q = ((hi ? a[i] >> 4 : a[i]) & 0x0F0F0F0Fu) | ((((c[1] >> (hi + 4 * i)) & 15u) * 0x02040810u) & 0x10101010u);
#pragma unroll
            for (int k = 0; k < 4; k++) v[4 * i + k] = d * (u8f<16>(q, k) + off);
        }
    } else if (type == T_F16) {
#pragma unroll
        for (int i = 0; i < 4; i++) {
            v[2 * i] = half_bits_to_float(a[i]); v[2 * i + 1] = half_bits_to_float(a[i] >> 16);
            v[8 + 2 * i] = half_bits_to_float(b[i]); v[9 + 2 * i] = half_bits_to_float(b[i] >> 16);
        }
    } else {
        const float4* q = reinterpret_cast<const float4*>(row + (size_t)k0 * 4);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const float4 f = q[i];
            v[4 * i] = f.x; v[4 * i + 1] = f.y; v[4 * i + 2] = f.z; v[4 * i + 3] = f.w;
        }
    }
}

// Y[z][t][n] = sum over piece z of K.  128 threads: 8 weight rows x TPT rows of x each (weight rows 4 tx .. and 32 + 4 tx .., so that a warp's loads of four
// are 128 bytes in a row); 16 TPT rows of x per CTA, four by four.  Sums run over 16 elements of K, eight of those make a sum of 128, and these are added to the piece's (in shared
// memory): the error of a chain of f32 additions grows with the root of its length (one chain of 4864: 1.7e-6 of the result).  Distance to float64 of prompts of 40, 100, 333, 1000 tokens through two
// layers of a 0.5B model, times that of token by token (16 inputs, +- 0.02): 0.95, 0.94, 0.95, 0.98; with sums of 64 that went straight to the piece's 1.16, 1.14, 1.06, 1.02, in the same time.
// Bound by the FMA pipe: 50 - 54 % of it busy (8 x 8 sums per thread; 29 % with 8 x 4, which waits for shared memory: 129 -> 72 us for 1152 x 1000 x 896).
// grid (tiles of all segments, ceil(T / (16 TPT)), pieces).
template <int TPT> constexpr int kRowsTileSmem = 2 * 32 * (64 + 16 * TPT) * 4 + 128 * 4 * TPT * 8;
constexpr int kRowsBN = 64, kRowsBK = 32, kRowsSum = 4;      // kRowsSum: steps of a sum that goes to the piece's
template <int TPT>
__global__ void __launch_bounds__(128, TPT == 8 ? 2 : 3) rows_tile_kernel(const __grid_constant__ RowsParams p) {
    constexpr int BT = 16 * TPT, XV = BT / 16;      // XV: float4 of x per thread and step
    extern __shared__ __align__(16) float rows_tile_smem[];
    auto ws = reinterpret_cast<float (*)[kRowsBK][kRowsBN]>(rows_tile_smem);
    auto xt = reinterpret_cast<float (*)[kRowsBK][BT]>(rows_tile_smem + 2 * kRowsBK * kRowsBN);
    uint64_t* top = reinterpret_cast<uint64_t*>(rows_tile_smem + 2 * kRowsBK * (kRowsBN + BT)) + threadIdx.x;      // this thread's sums of the piece, 128 apart
    const int tid = threadIdx.x, tx = tid & 7, ty = tid >> 3;
    int s = 0, tile = blockIdx.x;
    while (s < p.n_seg - 1 && tile >= (p.seg[s].n_rows + kRowsBN - 1) / kRowsBN) {
        tile -= (p.seg[s].n_rows + kRowsBN - 1) / kRowsBN;
        s++;
    }
    const RowsSeg& sg = p.seg[s];
    const int n0 = tile * kRowsBN, tt0 = blockIdx.y * BT, type = sg.type;
    const int k_lo = blockIdx.z * p.k_split, k_hi = min(p.K, k_lo + p.k_split);
    const int wr = tid & 63, wk = (tid >> 6) * 16;      // this thread's weight row and 16 of a step's 32 elements
    const uint8_t* row = sg.w + (long long)min(n0 + wr, sg.n_rows - 1) * sg.row_bytes;
    const int xr = tid % BT, xk = (tid / BT) * (4 * XV);     // ... row of x and 4 XV elements
    const float* xrow = p.x + (size_t)min(tt0 + xr, p.T - 1) * p.ldx + xk;
    pdl_launch_dependents();
    RowsRaw raw;
    rows_raw(type, row, k_lo + wk, raw);
    pdl_wait();
    float4 xv[XV];
    auto load_x = [&](int k) {
#pragma unroll
        for (int i = 0; i < XV; i++) xv[i] = *reinterpret_cast<const float4*>(xrow + k + 4 * i);
    };
    auto put = [&](int buf, int k) {
        float v[16];
        rows_values(type, row, k + wk, raw, v);
#pragma unroll
        for (int i = 0; i < 16; i++) ws[buf][wk + i][wr] = v[i];
#pragma unroll
        for (int i = 0; i < XV; i++) {
            xt[buf][xk + 4 * i][xr] = xv[i].x; xt[buf][xk + 4 * i + 1][xr] = xv[i].y;
            xt[buf][xk + 4 * i + 2][xr] = xv[i].z; xt[buf][xk + 4 * i + 3][xr] = xv[i].w;
        }
    };
    load_x(k_lo);
    put(0, k_lo);
    __syncthreads();
    uint64_t tot[4][TPT], acc[4][TPT];
#pragma unroll
    for (int n = 0; n < 4; n++)
#pragma unroll
        for (int t = 0; t < TPT; t++) tot[n][t] = acc[n][t] = 0;
    int step = 0;
    for (int k = k_lo; k < k_hi; k += kRowsBK, step++) {
        const int buf = step & 1;
        const bool more = k + kRowsBK < k_hi;
        if (more) {
            rows_raw(type, row, k + kRowsBK + wk, raw);
            load_x(k + kRowsBK);
        }
#pragma unroll 1
        for (int half = 0; half < kRowsBK; half += 16) {
#pragma unroll 4
            for (int kk = half; kk < half + 16; kk++) {
                const ulonglong2 w0 = *reinterpret_cast<const ulonglong2*>(&ws[buf][kk][4 * tx]), w1 = *reinterpret_cast<const ulonglong2*>(&ws[buf][kk][32 + 4 * tx]);
                float xs[TPT];
#pragma unroll
                for (int i = 0; i < TPT / 4; i++) {
                    const float4 f = *reinterpret_cast<const float4*>(&xt[buf][kk][64 * i + 4 * ty]);
                    xs[4 * i] = f.x; xs[4 * i + 1] = f.y; xs[4 * i + 2] = f.z; xs[4 * i + 3] = f.w;
                }
#pragma unroll
                for (int t = 0; t < TPT; t++) {
                    const uint64_t x2 = f2_pack(xs[t], xs[t]);
                    f2_fma(acc[0][t], w0.x, x2);
                    f2_fma(acc[1][t], w0.y, x2);
                    f2_fma(acc[2][t], w1.x, x2);
                    f2_fma(acc[3][t], w1.y, x2);
                }
            }
#pragma unroll
            for (int n = 0; n < 4; n++)
#pragma unroll
                for (int t = 0; t < TPT; t++) {
                    f2_add(tot[n][t], acc[n][t]);
                    acc[n][t] = 0;
                }
        }
        if (more ? step % kRowsSum == kRowsSum - 1 : step >= kRowsSum) {
#pragma unroll
            for (int n = 0; n < 4; n++)
#pragma unroll
                for (int t = 0; t < TPT; t++) {
                    uint64_t* at = top + (n * TPT + t) * 128;
                    if (step >= kRowsSum) f2_add(tot[n][t], *at);
                    if (more) {
                        *at = tot[n][t];
                        tot[n][t] = 0;
                    }
                }
        }
        if (more) put(buf ^ 1, k + kRowsBK);
        __syncthreads();
    }
    float* out = sg.out + (size_t)blockIdx.z * p.piece;
#pragma unroll
    for (int t = 0; t < TPT; t++) {
        const int tr = tt0 + 64 * (t >> 2) + 4 * ty + (t & 3);
        if (tr >= p.T) continue;
#pragma unroll
        for (int n = 0; n < 4; n++) {
            const float2 f = f2_unpack(tot[n][t]);
            const int at = n0 + (n >> 1) * 32 + 4 * tx + 2 * (n & 1);
            if (at < sg.n_rows) out[(size_t)tr * sg.ldo + at] = f.x;
            if (at + 1 < sg.n_rows) out[(size_t)tr * sg.ldo + at + 1] = f.y;
        }
    }
}

// ---------------------------------------------------------------- attention of a prompt's rows
struct RowsAttn {
    const float* qkv;      // [T][ld], q rotated
    const float* k_cache;  // [n_kv][max_seq][HD], positions 0 .. pos0 + T - 1 valid
    const float* v_cache;
    void* out;             // [T][ldo] of OutT
    int ld, ldo, pos0, T, n_heads, n_kv, max_seq;
    float scale;
};
template <int HD> constexpr int kRowsAttnSmem = (3 * 64 * HD + 64 * 64) * 4;

// Causal GQA attention in f32 (attention_cached, cpu/ops.rs:1479-1537, over the rows of a prompt): a block owns 64 query rows (token, head of one kv head), walks
// the keys 64 at a time with an online softmax; scores and sums as rows_tile_kernel's tiles, 8 keys (HD / 8 channels) x 4 rows per thread.  The tensor-core
// attention of fp16 pairs adds all keys into one accumulator that cuts its sums off: 2.8e-6 of the logits at 1000 keys, against 4e-7 here (sums of 64 keys, then of tiles).
// OutT = __half: prompts with fp16 products whose heads per kv head are no power of two (attn_umma_ok); prompts of 33, 333, 900, 4000 tokens through
// two layers of 14 heads of 64 over 2: 200, 358, 606, 3136 us, with a warp per token and kv head (prefill_attn_kernel) 222, 616, 1387, 16564, with the padded pairs of fp16 188, 241, 303, 924.
// grid (ceil(T G / 64), n_kv), the blocks with the most keys first.
template <int HD, typename OutT = float>
__global__ void __launch_bounds__(128) rows_attn_kernel(const RowsAttn p) {
    extern __shared__ __align__(16) float rows_attn_smem[];
    float *qs = rows_attn_smem, *ks = qs + 64 * HD, *vs = ks + 64 * HD, *ps = vs + 64 * HD;      // [HD][64 rows], [HD][64 keys], [64 keys][HD], [64 keys][64 rows]
    constexpr int NC = HD / 16;              // pairs of channels per thread: 4 tx + 32 i + (0, 1), (2, 3)
    const int tid = threadIdx.x, tx = tid & 7, ty = tid >> 3, G = p.n_heads / p.n_kv, kh = blockIdx.y;
    const int r0 = ((int)gridDim.x - 1 - (int)blockIdx.x) * 64, n_rows = p.T * G;
    pdl_launch_dependents();
    pdl_wait();
    const float* kb = p.k_cache + (size_t)kh * p.max_seq * HD;
    const float* vb = p.v_cache + (size_t)kh * p.max_seq * HD;
    const int lr = tid & 63, lh = (tid >> 6) * (HD / 2);      // this thread's row (key) and half of its channels
    {
        const int r = min(r0 + lr, n_rows - 1);
        const float* q = p.qkv + (size_t)(r / G) * p.ld + (size_t)(kh * G + r % G) * HD + lh;
#pragma unroll
        for (int d = 0; d < HD / 2; d += 4) {
            const float4 f = *reinterpret_cast<const float4*>(q + d);
            qs[(lh + d) * 64 + lr] = f.x; qs[(lh + d + 1) * 64 + lr] = f.y; qs[(lh + d + 2) * 64 + lr] = f.z; qs[(lh + d + 3) * 64 + lr] = f.w;
        }
    }
    int last[4];                             // the last key each of this thread's rows sees
#pragma unroll
    for (int t = 0; t < 4; t++) last[t] = p.pos0 + min(r0 + 4 * ty + t, n_rows - 1) / G;
    const int kv_end = p.pos0 + min(r0 + 63, n_rows - 1) / G + 1;
    uint64_t o[NC][4];
    float m[4], l[4];
#pragma unroll
    for (int t = 0; t < 4; t++) {
        m[t] = -INFINITY;
        l[t] = 0.0f;
#pragma unroll
        for (int c = 0; c < NC; c++) o[c][t] = 0;
    }
    for (int k0 = 0; k0 < kv_end; k0 += 64) {
        __syncthreads();                     // (the tile before has been read)
        {
            const int key = min(k0 + lr, kv_end - 1);
            const float* k = kb + (size_t)key * HD + lh;
#pragma unroll
            for (int d = 0; d < HD / 2; d += 4) {
                const float4 f = *reinterpret_cast<const float4*>(k + d);
                ks[(lh + d) * 64 + lr] = f.x; ks[(lh + d + 1) * 64 + lr] = f.y; ks[(lh + d + 2) * 64 + lr] = f.z; ks[(lh + d + 3) * 64 + lr] = f.w;
            }
#pragma unroll
            for (int i = tid; i < 64 * HD / 4; i += 128) {
                const int row = i / (HD / 4);
                *reinterpret_cast<float4*>(vs + 4 * i) = *reinterpret_cast<const float4*>(vb + (size_t)min(k0 + row, kv_end - 1) * HD + 4 * (i - row * (HD / 4)));
            }
        }
        __syncthreads();
        uint64_t sc[4][4];                   // scores of keys (4 tx + 0, 1), (2, 3), (32 + 4 tx + 0, 1), (2, 3)
#pragma unroll
        for (int n = 0; n < 4; n++)
#pragma unroll
            for (int t = 0; t < 4; t++) sc[n][t] = 0;
#pragma unroll 8
        for (int d = 0; d < HD; d++) {
            const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(ks + d * 64 + 4 * tx), b = *reinterpret_cast<const ulonglong2*>(ks + d * 64 + 32 + 4 * tx);
            const float4 f = *reinterpret_cast<const float4*>(qs + d * 64 + 4 * ty);
            const float x[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
            for (int t = 0; t < 4; t++) {
                const uint64_t x2 = f2_pack(x[t], x[t]);
                f2_fma(sc[0][t], a.x, x2);
                f2_fma(sc[1][t], a.y, x2);
                f2_fma(sc[2][t], b.x, x2);
                f2_fma(sc[3][t], b.y, x2);
            }
        }
        float e[8][4], corr[4];
#pragma unroll
        for (int t = 0; t < 4; t++) {
            float mx = -INFINITY;
#pragma unroll
            for (int n = 0; n < 4; n++) {
                const float2 f = f2_unpack(sc[n][t]);
                const int key = k0 + (n >> 1) * 32 + 4 * tx + 2 * (n & 1);
                e[2 * n][t] = key <= last[t] ? f.x * p.scale : -INFINITY;
                e[2 * n + 1][t] = key + 1 <= last[t] ? f.y * p.scale : -INFINITY;
                mx = fmaxf(mx, fmaxf(e[2 * n][t], e[2 * n + 1][t]));
            }
#pragma unroll
            for (int w = 1; w < 8; w <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, w));
            const float mn = fmaxf(m[t], mx);
            corr[t] = m[t] == -INFINITY ? 0.0f : expf(m[t] - mn);
            float s = 0.0f;
#pragma unroll
            for (int n = 0; n < 8; n++) {
                e[n][t] = e[n][t] == -INFINITY ? 0.0f : expf(e[n][t] - mn);
                s += e[n][t];
            }
            l[t] = l[t] * corr[t] + s;
            m[t] = mn;
        }
#pragma unroll
        for (int n = 0; n < 8; n++)          // key (n >> 2) * 32 + 4 tx + (n & 3)
            *reinterpret_cast<float4*>(ps + ((n >> 2) * 32 + 4 * tx + (n & 3)) * 64 + 4 * ty) = make_float4(e[n][0], e[n][1], e[n][2], e[n][3]);
        __syncwarp();                        // (a warp reads the rows that it has written)
        uint64_t acc[NC][4];
#pragma unroll
        for (int c = 0; c < NC; c++)
#pragma unroll
            for (int t = 0; t < 4; t++) acc[c][t] = 0;
#pragma unroll 4
        for (int k = 0; k < 64; k++) {
            const float4 f = *reinterpret_cast<const float4*>(ps + k * 64 + 4 * ty);
            const float x[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
            for (int i = 0; i < HD / 32; i++) {
                const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(vs + k * HD + 32 * i + 4 * tx);
#pragma unroll
                for (int t = 0; t < 4; t++) {
                    const uint64_t x2 = f2_pack(x[t], x[t]);
                    f2_fma(acc[2 * i][t], v.x, x2);
                    f2_fma(acc[2 * i + 1][t], v.y, x2);
                }
            }
        }
#pragma unroll
        for (int t = 0; t < 4; t++) {
            const uint64_t c2 = f2_pack(corr[t], corr[t]);
#pragma unroll
            for (int c = 0; c < NC; c++) {
                f2_fma(acc[c][t], o[c][t], c2);
                o[c][t] = acc[c][t];
            }
        }
    }
#pragma unroll
    for (int t = 0; t < 4; t++) {
#pragma unroll
        for (int w = 1; w < 8; w <<= 1) l[t] += __shfl_xor_sync(0xffffffffu, l[t], w);
        const int r = r0 + 4 * ty + t;
        if (r >= n_rows) continue;
        OutT* out = reinterpret_cast<OutT*>(p.out) + (size_t)(r / G) * p.ldo + (size_t)(kh * G + r % G) * HD;
        const float inv = 1.0f / l[t];
#pragma unroll
        for (int i = 0; i < HD / 32; i++) {
            const float2 a = f2_unpack(o[2 * i][t]), b = f2_unpack(o[2 * i + 1][t]);
            if constexpr (sizeof(OutT) == 4) *reinterpret_cast<float4*>(out + 32 * i + 4 * tx) = make_float4(a.x * inv, a.y * inv, b.x * inv, b.y * inv);
            else {
                const __half2 lo = __halves2half2(f2h_sat(a.x * inv), f2h_sat(a.y * inv)), hi = __halves2half2(f2h_sat(b.x * inv), f2h_sat(b.y * inv));
                *reinterpret_cast<uint2*>(out + 32 * i + 4 * tx) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
            }
        }
    }
}

// ---------------------------------------------------------------- between the tiles
struct RowsSum {           // pieces of a product: [n][T][ld]
    const float* p;
    int n, ld;
    long long piece;
};
__device__ __forceinline__ float rows_sum(const RowsSum& s, int t, int i) {
    const float* q = s.p + (size_t)t * s.ld + i;
    float v = q[0];
    for (int z = 1; z < s.n; z++) v += q[(size_t)z * s.piece];
    return v;
}
// x[t] += the sum; out[t] = RMSNorm(x[t]) (w != nullptr).  One block of 256 per row.
__global__ void __launch_bounds__(256) rows_norm_kernel(float* __restrict__ x, const RowsSum sum, const float* __restrict__ w, float eps, float* __restrict__ out, int n) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ float red[8];
    const int t = blockIdx.x;
    float* xr = x + (size_t)t * n;
    float ss = 0.0f;
    for (int i = threadIdx.x; i < n; i += 256) {
        float v = xr[i];
        if (sum.n) {
            v += rows_sum(sum, t, i);
            xr[i] = v;
        }
        ss = fmaf(v, v, ss);
    }
    if (!w) return;
    ss = warp_sum(ss);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
    __syncthreads();
    float tot = 0.0f;
    for (int k = 0; k < 8; k++) tot += red[k];
    const float inv = 1.0f / sqrtf(tot / (float)n + eps);
    for (int i = threadIdx.x; i < n; i += 256) out[(size_t)t * n + i] = __fmul_rn(__fmul_rn(xr[i], inv), w[i]);
}
// q | k | v rows = the sum + bias.  grid (ceil(n / 256), T)
__global__ void __launch_bounds__(256) rows_qkv_kernel(const RowsSum sum, const float* __restrict__ bq, const float* __restrict__ bk, const float* __restrict__ bv, int nq, int nk, float* __restrict__ out, int n) {
    pdl_launch_dependents();
    pdl_wait();
    const int i = blockIdx.x * 256 + threadIdx.x, t = blockIdx.y;
    if (i >= n) return;
    const float* b = i < nq ? bq : i < nq + nk ? bk : bv;
    float v = rows_sum(sum, t, i);
    if (b) v += b[i < nq ? i : i < nq + nk ? i - nq : i - nq - nk];
    out[(size_t)t * n + i] = v;
}
// out = silu(gate) up; the sum's rows are gate | up.  grid (ceil(n / 256), T)
__global__ void __launch_bounds__(256) rows_swiglu_kernel(const RowsSum sum, float* __restrict__ out, int n) {
    pdl_launch_dependents();
    pdl_wait();
    const int i = blockIdx.x * 256 + threadIdx.x, t = blockIdx.y;
    if (i < n) out[(size_t)t * n + i] = silu_f(rows_sum(sum, t, i)) * rows_sum(sum, t, n + i);
}

// ---------------------------------------------------------------- host
inline int rows_few_tasks(const RowsParams& p, int R) {
    if (p.epi == EPI_SWIGLU) return (p.seg[0].n_rows + R / 2 - 1) / (R / 2);
    int n = 0;
    for (int s = 0; s < p.n_seg; s++) n += (p.seg[s].n_rows + R - 1) / R;
    return n;
}
template <int R, int TT> constexpr size_t kRowsFewSmem = (R * TT <= 16 ? 110 : 220) << 10;
template <int R, int TT>
inline cudaError_t rows_few_ready() {
    static bool once[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && once[dev]) return cudaSuccess;
    const cudaError_t e = cudaFuncSetAttribute(rows_few_kernel<R, TT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRowsFewSmem<R, TT>);
    if (e == cudaSuccess && dev >= 0 && dev < 64) once[dev] = true;
    return e;
}
template <int R, int TT>
inline cudaError_t rows_few_go(RowsParams& p, int n_sm, bool pdl, cudaStream_t st) {
    // shared memory: all of K where two blocks' rows fit an SM (one block's from 32 sums per warp on), else 256s of it
    const int fit = (int)(kRowsFewSmem<R, TT> / (TT * sizeof(float)));
    p.chunk = xpad_floats(p.K) <= fit ? p.K : (fit - 8) * 16 / 17 / 256 * 256;
    const size_t smem = (size_t)TT * xpad_floats(p.chunk) * sizeof(float);
    if (const cudaError_t e = rows_few_ready<R, TT>()) return e;
    const int want = (rows_few_tasks(p, R) + kRowsWarps - 1) / kRowsWarps, groups = (p.T + TT - 1) / TT;
    const int per_sm = R * TT <= 16 && smem <= (size_t)(110 << 10) ? 2 : 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)std::min(want, std::max(1, per_sm * n_sm / groups)), (unsigned)groups);
    cfg.blockDim = dim3(kRowsWarps * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = pdl ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, rows_few_kernel<R, TT>, p);
}
// The kernels' code on the device (it is loaded at a kernel's first use, and a device that has filled up since has no room for it)
inline cudaError_t rows_load() {
    for (cudaError_t e : {rows_few_ready<4, 2>(), rows_few_ready<2, 2>(), rows_few_ready<1, 2>(), rows_few_ready<4, 4>(), rows_few_ready<2, 4>(), rows_few_ready<1, 4>(), rows_few_ready<4, 8>(),
                          rows_few_ready<2, 8>(), rows_few_ready<1, 8>()})
        if (e != cudaSuccess) return e;
    cudaFuncAttributes a;
    for (const void* f : {(const void*)rows_norm_kernel, (const void*)rows_qkv_kernel, (const void*)rows_swiglu_kernel})
        if (const cudaError_t e = cudaFuncGetAttributes(&a, f)) return e;
    return cudaSuccess;
}
inline cudaError_t rows_few_launch(RowsParams& p, int n_sm, bool pdl, cudaStream_t st) {
    // rounds of the chip's warps times a round's instructions: R weight columns to unpack and multiply, and the rows' x to load whatever R is.  4096 x 14336 with 3 rows: one
    // weight row per warp takes two rounds, 40 us, two take one
    const int full = 2 * n_sm * kRowsWarps, tt = p.T <= 2 ? 2 : p.T <= 4 ? 4 : 8;
    const bool glu = p.epi == EPI_SWIGLU;
    auto cost = [&](int R) { return (rows_few_tasks(p, R) + full - 1) / full * (R * (4 + tt / 2) + (tt == 8 ? 16 : 6)); };
    const int c4 = cost(4), c2 = cost(2), c1 = glu ? c2 + 1 : cost(1);
    const bool four = c4 <= c2 && c4 <= c1, two = c2 <= c1;
    if (p.T <= 2) return four ? rows_few_go<4, 2>(p, n_sm, pdl, st) : two ? rows_few_go<2, 2>(p, n_sm, pdl, st) : rows_few_go<1, 2>(p, n_sm, pdl, st);
    if (p.T <= 4) return four ? rows_few_go<4, 4>(p, n_sm, pdl, st) : two ? rows_few_go<2, 4>(p, n_sm, pdl, st) : rows_few_go<1, 4>(p, n_sm, pdl, st);
    return four ? rows_few_go<4, 8>(p, n_sm, pdl, st) : two ? rows_few_go<2, 8>(p, n_sm, pdl, st) : rows_few_go<1, 8>(p, n_sm, pdl, st);
}

}  // namespace b200
