// gemv.cuh — fused dequant-GEMV for batch-1 decode: y[j] = sum_k deq(W)[j,k] * x[k].
//
// Replaces the reference's one-thread-per-output kernels vec_mat_q4k/q8_0/q6k/q5k
// (src/backend/cuda/kernels.rs:443-509, 519-553, 600-658, 661-735) and the CPU hot
// loop fused_vecmat_dispatch -> simd::dot_q* (src/backend/cpu/ops.rs:1123-1191,
// src/backend/cpu/simd.rs:931-1146).  Weights stay in the GGUF super-block layout,
// untransposed: row j of W is K/bs contiguous blocks.
//
// One launch covers up to three weight matrices that share x (q|k|v, gate|up) and
// fuses what surrounds the GEMV on the decode path:
//   prologue : RMSNorm of x (simd.rs:847-899) when norm_w != nullptr
//   epilogue : +bias (layers.rs:68-74) | +residual (layers.rs:1202-1241) |
//              silu(gate)*up (simd.rs:598-649) | out += w_e * y (moe.rs:363-368)
//
// Work split: a warp owns R=4 consecutive output rows and walks K; x lives in
// shared memory (padded layout, common.cuh:xidx) and each x chunk is reused by the
// 4 rows.  All weight loads of a step are issued before any is consumed
// (8 x 16 B in flight per lane for Q4_K).  Arithmetic is the reference's separated
// form d*sc*sum(q*x) - dmin*m*sum(x) in f32 (simd.rs:1006-1013).
#pragma once
#include "common.cuh"
#include "quant.cuh"

namespace b200 {

constexpr int kGemvWarps = 8;
constexpr int kGemvThreads = kGemvWarps * kWarp;
// rows per warp task: 4, or fewer where 4 would leave warps idle (gemv_rows).  Every row's sum is its own, whatever R is.  896 x 896 in Q5_0: 28 blocks of
// eight warps with 4 rows each, 112 with one.
constexpr int kGemvR = 4;

enum : int { EPI_STORE = 0, EPI_RESIDUAL = 1, EPI_SWIGLU = 2, EPI_SCALED_ACC = 3 };

struct GemvSeg {
    const uint8_t* w;       // n_rows rows of row_bytes
    float* out;             // n_rows outputs
    const float* bias;      // optional
    long long row_bytes;
    long long expert_stride;  // MoE: bytes between experts (0 = dense)
    int type;
    int n_rows;
};

struct GemvParams {
    GemvSeg seg[3];
    int n_seg;
    int K;
    const float* x;         // [K]
    const float* norm_w;    // optional fused RMSNorm weight [K]
    float eps;
    int epi;
    const float* residual;  // EPI_RESIDUAL: out[j] = acc + residual[j]
    // MoE (expert-resident, no host round trip): the slot-th selected expert
    const int* expert_sel;     // device [top_k] or nullptr
    const float* expert_wt;    // device [top_k] (EPI_SCALED_ACC: out[j] += wt * acc)
    int expert_slot;
    // expert parallel (one context per GPU, experts [expert_base, expert_base + expert_count) resident here): a launch whose selected
    // expert lives on another GPU returns at once; EPI_SCALED_ACC writes out[j] = wt * acc (no accumulate, no residual): the
    // weighted output of ONE expert, combined across GPUs by ep_combine_kernel (misc.cuh).  expert_count == 0: off.
    int expert_base, expert_count;
    // n_slots > 1: all selected experts in one launch (the tensor-pipe kernel only, gemv_mma.cuh): slot s reads x + s x_slot and writes out + s out_slot
    int n_slots, x_slot, out_slot;
};

// byte k of w, less `off`, as a float: PRMT drops it into the mantissa of 2^23, one subtraction removes 2^23 + off (exact; an integer conversion runs at a quarter of
// the rate and needs the byte cut out first)
template <int OFF = 0>
__device__ __forceinline__ float u8f(uint32_t w, int k) {
    return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7650 | k)) - (8388608.0f + (float)OFF);
}

// ---- Q4_K / Q5_K: 8 lanes per 256-element block, 16 qs bytes (32 elements) per lane ----
template <bool Q5, int R>
__device__ __forceinline__ void rows_dot_k45(const uint8_t* const (&rp)[R], int nb, const float* xs, int lane,
                                             float (&acc)[R]) {
    constexpr int BB = Q5 ? 176 : 144;
    constexpr int QS = Q5 ? 48 : 16;
    const int bl = lane >> 3, p = lane & 7, g = p >> 1, h = p & 1, gg = g & 1;
    for (int b0 = 0; b0 < nb; b0 += 4) {
        const int b = b0 + bl;
        const bool ok = b < nb;
        const int bc = ok ? b : nb - 1;
        uint4 hd[R], q[R], qh[R];
#pragma unroll
        for (int r = 0; r < R; r++) {
            const uint8_t* bp = rp[r] + (size_t)bc * BB;
            hd[r] = ldg_stream_u4(bp);
            q[r] = ldg_stream_u4(bp + QS + 16 * p);
            if (Q5) qh[r] = ldg_stream_u4(bp + 16 + 16 * h);
        }
        const float* xp = xs + xidx(bc * 256 + 64 * g + 16 * h);
        float xl[16], xh[16];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            float4 a = *reinterpret_cast<const float4*>(xp + 4 * i);
            float4 c = *reinterpret_cast<const float4*>(xp + 32 + 4 * i);
            xl[4 * i] = a.x; xl[4 * i + 1] = a.y; xl[4 * i + 2] = a.z; xl[4 * i + 3] = a.w;
            xh[4 * i] = c.x; xh[4 * i + 1] = c.y; xh[4 * i + 2] = c.z; xh[4 * i + 3] = c.w;
        }
        float sl = 0.0f, sh = 0.0f;
#pragma unroll
        for (int i = 0; i < 16; i++) { sl += xl[i]; sh += xh[i]; }
#pragma unroll
        for (int r = 0; r < R; r++) {
            const float d = half_bits_to_float(hd[r].x);
            const float dmin = half_bits_to_float(hd[r].x >> 16);
            const uint32_t A = (hd[r].y >> (16 * gg)) & 0xFFFFu;
            const uint32_t B = (hd[r].z >> (16 * gg)) & 0xFFFFu;
            const uint32_t C = (hd[r].w >> (16 * gg)) & 0xFFFFu;
            uint32_t scp, mnp;  // (sc[2g], sc[2g+1]) and (m[2g], m[2g+1]) as byte pairs
            if (g < 2) {
                scp = A & 0x3F3Fu;
                mnp = B & 0x3F3Fu;
            } else {
                scp = (C & 0x0F0Fu) | ((A >> 2) & 0x3030u);
                mnp = ((C >> 4) & 0x0F0Fu) | ((B >> 2) & 0x3030u);
            }
            const float d1 = d * (float)(scp & 0xFFu), d2 = d * (float)(scp >> 8);
            const float m1 = dmin * (float)(mnp & 0xFFu), m2 = dmin * (float)(mnp >> 8);
            const uint32_t qw[4] = {q[r].x, q[r].y, q[r].z, q[r].w};
            const uint32_t hw[4] = {qh[r].x, qh[r].y, qh[r].z, qh[r].w};
            float ql = 0.0f, qhh = 0.0f;
#pragma unroll
            for (int wi = 0; wi < 4; wi++) {
                uint32_t lo = qw[wi] & 0x0F0F0F0Fu;
                uint32_t hi = (qw[wi] >> 4) & 0x0F0F0F0Fu;
                if (Q5) {
                    lo |= ((hw[wi] >> (2 * g)) & 0x01010101u) << 4;
                    hi |= ((hw[wi] >> (2 * g + 1)) & 0x01010101u) << 4;
                }
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    ql = fmaf(u8f(lo, k), xl[4 * wi + k], ql);
                    qhh = fmaf(u8f(hi, k), xh[4 * wi + k], qhh);
                }
            }
            const float v = (d1 * ql - m1 * sl) + (d2 * qhh - m2 * sh);
            acc[r] += ok ? v : 0.0f;
        }
    }
}

// ---- Q6_K: 8 lanes per 210-byte block (2-byte aligned: 16-bit loads), 32 elements per lane ----
template <int R>
__device__ __forceinline__ void rows_dot_q6k(const uint8_t* const (&rp)[R], int nb, const float* xs, int lane,
                                             float (&acc)[R]) {
    const int bl = lane >> 3, t = lane & 7, n = t >> 2, j = t & 3, is = j >> 1;
    for (int b0 = 0; b0 < nb; b0 += 4) {
        const int b = b0 + bl;
        const bool ok = b < nb;
        const int bc = ok ? b : nb - 1;
        uint32_t qa[R][2], qb[R][2], qhv[R][2], dd[R];
        int sc[R][4];
#pragma unroll
        for (int r = 0; r < R; r++) {
            const uint8_t* bp = rp[r] + (size_t)bc * 210;
            const uint8_t* pa = bp + 64 * n + 8 * j;
            const uint8_t* ph = bp + 128 + 32 * n + 8 * j;
#pragma unroll
            for (int w = 0; w < 2; w++) {
                qa[r][w] = ldg_u16(pa + 4 * w) | (ldg_u16(pa + 4 * w + 2) << 16);
                qb[r][w] = ldg_u16(pa + 32 + 4 * w) | (ldg_u16(pa + 32 + 4 * w + 2) << 16);
                qhv[r][w] = ldg_u16(ph + 4 * w) | (ldg_u16(ph + 4 * w + 2) << 16);
            }
#pragma unroll
            for (int c = 0; c < 4; c++) sc[r][c] = ldg_s8(bp + 192 + 8 * n + is + 2 * c);
            dd[r] = ldg_u16(bp + 208);
        }
        // x runs: element 128n + 32c + 8j + i, c = 0..3, i = 0..7
        float xv[4][8], xsum[4];
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const float* xp = xs + xidx(bc * 256 + 128 * n + 32 * c + 8 * j);
            float4 a = *reinterpret_cast<const float4*>(xp);
            float4 e = *reinterpret_cast<const float4*>(xp + 4);
            xv[c][0] = a.x; xv[c][1] = a.y; xv[c][2] = a.z; xv[c][3] = a.w;
            xv[c][4] = e.x; xv[c][5] = e.y; xv[c][6] = e.z; xv[c][7] = e.w;
            xsum[c] = ((a.x + a.y) + (a.z + a.w)) + ((e.x + e.y) + (e.z + e.w));
        }
#pragma unroll
        for (int r = 0; r < R; r++) {
            const float d = half_bits_to_float(dd[r]);
            float s[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int w = 0; w < 2; w++) {
                const uint32_t a = qa[r][w], bq = qb[r][w], hq = qhv[r][w];
                const uint32_t q0 = (a & 0x0F0F0F0Fu) | ((hq << 4) & 0x30303030u);
                const uint32_t q1 = (bq & 0x0F0F0F0Fu) | ((hq << 2) & 0x30303030u);
                const uint32_t q2 = ((a >> 4) & 0x0F0F0F0Fu) | (hq & 0x30303030u);
                const uint32_t q3 = ((bq >> 4) & 0x0F0F0F0Fu) | ((hq >> 2) & 0x30303030u);
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    s[0] = fmaf(u8f(q0, k), xv[0][4 * w + k], s[0]);
                    s[1] = fmaf(u8f(q1, k), xv[1][4 * w + k], s[1]);
                    s[2] = fmaf(u8f(q2, k), xv[2][4 * w + k], s[2]);
                    s[3] = fmaf(u8f(q3, k), xv[3][4 * w + k], s[3]);
                }
            }
            float v = 0.0f;
#pragma unroll
            for (int c = 0; c < 4; c++) v += (d * (float)sc[r][c]) * (s[c] - 32.0f * xsum[c]);
            acc[r] += ok ? v : 0.0f;
        }
    }
}

// ---- 32-element block types (Q8_0, Q4_0, Q5_0) and F16/F32: one lane per 32 elements ----
template <int R>
__device__ __forceinline__ void rows_dot_b32(int type, const uint8_t* const (&rp)[R], int K, const float* xs,
                                             int lane, float (&acc)[R]) {
    const int nb = K >> 5;
    const int bb = (type == T_F32) ? 128 : (type == T_F16) ? 64 : type_block_bytes(type);
    for (int b = lane; b < nb; b += 32) {
        float xv[32];
        const float* xp = xs + xidx(b * 32);
#pragma unroll
        for (int i = 0; i < 8; i++) {
            float4 a = *reinterpret_cast<const float4*>(xp + 4 * i);
            xv[4 * i] = a.x; xv[4 * i + 1] = a.y; xv[4 * i + 2] = a.z; xv[4 * i + 3] = a.w;
        }
#pragma unroll
        for (int r = 0; r < R; r++) {
            const uint8_t* bp = rp[r] + (size_t)b * bb;
            float s = 0.0f;
            if (type == T_Q8_0) {
                const float d = half_bits_to_float(ldg_u16(bp));
                uint32_t qv[8];
#pragma unroll
                for (int i = 0; i < 8; i++) qv[i] = (ldg_u16(bp + 2 + 4 * i) | (ldg_u16(bp + 4 + 4 * i) << 16)) ^ 0x80808080u;
#pragma unroll
                for (int i = 0; i < 8; i++)
#pragma unroll
                    for (int k = 0; k < 4; k++) s = fmaf(u8f<128>(qv[i], k), xv[4 * i + k], s);
                s *= d;
            } else if (type == T_Q4_0) {
                const float d = half_bits_to_float(ldg_u16(bp));
                float lo = 0.0f, hi = 0.0f;
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    uint32_t v = ldg_u16(bp + 2 + 2 * i);
                    lo = fmaf((float)((int)(v & 0xF) - 8), xv[2 * i], lo);
                    hi = fmaf((float)((int)((v >> 4) & 0xF) - 8), xv[2 * i + 16], hi);
                    lo = fmaf((float)((int)((v >> 8) & 0xF) - 8), xv[2 * i + 1], lo);
                    hi = fmaf((float)((int)((v >> 12) & 0xF) - 8), xv[2 * i + 17], hi);
                }
                s = d * (lo + hi);
            } else if (type == T_Q5_0) {
                const float d = half_bits_to_float(ldg_u16(bp));
                const uint32_t qh = ldg_u16(bp + 2) | (ldg_u16(bp + 4) << 16);
#pragma unroll
                for (int i = 0; i < 4; i++) {      // bytes 4i .. 4i + 3: elements 4i .. (low nibbles) and 16 + 4i .. (high); bit e of qh is the fifth bit of element e
                    const uint32_t v = ldg_u16(bp + 6 + 4 * i) | (ldg_u16(bp + 8 + 4 * i) << 16);
                    // four bits to bit 4 of four bytes: the products of one bit with 2^4, 2^11, 2^18, 2^25 that land elsewhere are masked off
                    const uint32_t lo = (v & 0x0F0F0F0Fu) | ((((qh >> (4 * i)) & 15u) * 0x02040810u) & 0x10101010u);
                    const uint32_t hi = ((v >> 4) & 0x0F0F0F0Fu) | ((((qh >> (16 + 4 * i)) & 15u) * 0x02040810u) & 0x10101010u);
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        s = fmaf(u8f<16>(lo, k), xv[4 * i + k], s);
                        s = fmaf(u8f<16>(hi, k), xv[16 + 4 * i + k], s);
                    }
                }
                s *= d;
            } else if (type == T_F16) {
#pragma unroll
                for (int i = 0; i < 16; i++) {
                    uint32_t v = ldg_stream_u32(bp + 4 * i);
                    s = fmaf(half_bits_to_float(v), xv[2 * i], s);
                    s = fmaf(half_bits_to_float(v >> 16), xv[2 * i + 1], s);
                }
            } else {  // F32
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    uint4 v = ldg_stream_u4(bp + 16 * i);
                    s = fmaf(__uint_as_float(v.x), xv[4 * i], s);
                    s = fmaf(__uint_as_float(v.y), xv[4 * i + 1], s);
                    s = fmaf(__uint_as_float(v.z), xv[4 * i + 2], s);
                    s = fmaf(__uint_as_float(v.w), xv[4 * i + 3], s);
                }
            }
            acc[r] += s;
        }
    }
}

__device__ __forceinline__ float silu_f(float x) { return x / (1.0f + expf(-x)); }

// Stage x (optionally RMS-normalised) into shared memory in the padded layout.  Rows of up to 4 * kStageV * kGemvThreads elements are loaded once, and their
// norm weights before the wait for the kernel before.
constexpr int kStageV = 4;
struct StageW {
    float4 w[kStageV];
};
__device__ __forceinline__ void stage_w(const GemvParams& p, StageW& sw) {
    if (!p.norm_w || p.K > 4 * kStageV * kGemvThreads) return;
#pragma unroll
    for (int i = 0; i < kStageV; i++) {
        const int e = (threadIdx.x + i * kGemvThreads) * 4;
        if (e < p.K) sw.w[i] = *reinterpret_cast<const float4*>(p.norm_w + e);
    }
}
__device__ __forceinline__ void stage_x(const GemvParams& p, const StageW& sw, float* xs, float* red) {
    const int tid = threadIdx.x;
    if (p.K <= 4 * kStageV * kGemvThreads) {
        float4 v[kStageV];
#pragma unroll
        for (int i = 0; i < kStageV; i++) {
            const int e = (tid + i * kGemvThreads) * 4;
            if (e < p.K) v[i] = *reinterpret_cast<const float4*>(p.x + e);
        }
        float inv = 1.0f;
        if (p.norm_w) {
            float ss = 0.0f;
#pragma unroll
            for (int i = 0; i < kStageV; i++)
                if ((tid + i * kGemvThreads) * 4 < p.K) ss += v[i].x * v[i].x + v[i].y * v[i].y + v[i].z * v[i].z + v[i].w * v[i].w;
            ss = warp_sum(ss);
            if ((tid & 31) == 0) red[tid >> 5] = ss;
            __syncthreads();
            float tot = 0.0f;
#pragma unroll
            for (int w = 0; w < kGemvWarps; w++) tot += red[w];
            inv = 1.0f / sqrtf(tot / (float)p.K + p.eps);
        }
#pragma unroll
        for (int i = 0; i < kStageV; i++) {
            const int e = (tid + i * kGemvThreads) * 4;
            if (e < p.K) {
                if (p.norm_w) {
                    v[i].x = (v[i].x * inv) * sw.w[i].x; v[i].y = (v[i].y * inv) * sw.w[i].y; v[i].z = (v[i].z * inv) * sw.w[i].z; v[i].w = (v[i].w * inv) * sw.w[i].w;
                }
                *reinterpret_cast<float4*>(xs + xidx(e)) = v[i];
            }
        }
        __syncthreads();
        return;
    }
    float inv = 1.0f;
    if (p.norm_w) {
        float ss = 0.0f;
        for (int e = tid * 4; e < p.K; e += kGemvThreads * 4) {
            float4 v = *reinterpret_cast<const float4*>(p.x + e);
            ss += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
        }
        ss = warp_sum(ss);
        if ((tid & 31) == 0) red[tid >> 5] = ss;
        __syncthreads();
        float tot = 0.0f;
#pragma unroll
        for (int w = 0; w < kGemvWarps; w++) tot += red[w];
        inv = 1.0f / sqrtf(tot / (float)p.K + p.eps);
    }
    for (int e = tid * 4; e < p.K; e += kGemvThreads * 4) {
        float4 v = *reinterpret_cast<const float4*>(p.x + e);
        if (p.norm_w) {
            float4 w = *reinterpret_cast<const float4*>(p.norm_w + e);
            v.x = (v.x * inv) * w.x; v.y = (v.y * inv) * w.y; v.z = (v.z * inv) * w.z; v.w = (v.w * inv) * w.w;
        }
        *reinterpret_cast<float4*>(xs + xidx(e)) = v;
    }
    __syncthreads();
}

template <int R>
__global__ void __launch_bounds__(kGemvThreads) gemv_kernel(const __grid_constant__ GemvParams p) {
    static_assert(R == 1 || R == 2 || R == 4, "rows per warp");
    constexpr int G = R / 2 > 0 ? R / 2 : 1;      // (EPI_SWIGLU: R / 2 gate rows and their up rows; never with R = 1)
    extern __shared__ __align__(16) float xs[];
    __shared__ float red[kGemvWarps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;

    // task table: segment s owns tasks [t0[s], t0[s+1]); a task = R rows
    int t0[4];
    t0[0] = 0;
    if (p.epi == EPI_SWIGLU) {
        t0[1] = (p.seg[0].n_rows + G - 1) / G;
        t0[2] = t0[3] = t0[1];
    } else {
#pragma unroll
        for (int s = 0; s < 3; s++) t0[s + 1] = t0[s] + (s < p.n_seg ? (p.seg[s].n_rows + R - 1) / R : 0);
    }
    const int n_tasks = t0[3];

    pdl_launch_dependents();
    if (!p.expert_sel) {  // dense weights do not depend on the predecessor: pull this warp's first rows towards L2
        int task = blockIdx.x * kGemvWarps + warp;
        if (task < n_tasks) {
            if (p.epi == EPI_SWIGLU) {
                const long long off = (long long)task * G;
                const long long bytes = G * p.seg[0].row_bytes;
                for (long long o = (long long)lane * 128; o < bytes; o += 32 * 128) {
                    prefetch_l2(p.seg[0].w + off * p.seg[0].row_bytes + o);
                    prefetch_l2(p.seg[1].w + off * p.seg[1].row_bytes + o);
                }
            } else {
                int s = (task >= t0[2]) ? 2 : (task >= t0[1]) ? 1 : 0;
                const GemvSeg& sg = p.seg[s];
                int row0 = (task - t0[s]) * R;
                int rows = min(R, sg.n_rows - row0);
                const uint8_t* base = sg.w + (long long)row0 * sg.row_bytes;
                long long bytes = (long long)rows * sg.row_bytes;
                for (long long o = (long long)lane * 128; o < bytes; o += 32 * 128) prefetch_l2(base + o);
            }
        }
    }
    StageW sw;
    stage_w(p, sw);
    pdl_wait();
    // MoE: the selected expert is written by the routing kernel (a predecessor): read it only after the wait
    long long eoff = p.expert_sel ? (long long)p.expert_sel[p.expert_slot] : 0;
    if (p.expert_count > 0) {   // expert parallel: not this GPU's expert -> nothing to do (uniform over the grid)
        eoff -= p.expert_base;
        if (eoff < 0 || eoff >= p.expert_count) return;
    }
    stage_x(p, sw, xs, red);

    for (int task = blockIdx.x * kGemvWarps + warp; task < n_tasks; task += gridDim.x * kGemvWarps) {
        const uint8_t* rp[R];
        int type, s = 0, row0, rows;
        if (p.epi == EPI_SWIGLU) {
            const GemvSeg& ga = p.seg[0];
            const GemvSeg& up = p.seg[1];
            row0 = task * G;
            rows = min(G, ga.n_rows - row0);
            type = ga.type;
#pragma unroll
            for (int r = 0; r < R; r++) {
                const GemvSeg& sg = r < G ? ga : up;
                rp[r] = sg.w + eoff * sg.expert_stride + (long long)(row0 + min(r < G ? r : r - G, rows - 1)) * sg.row_bytes;
            }
        } else {
            s = (task >= t0[2]) ? 2 : (task >= t0[1]) ? 1 : 0;
            const GemvSeg& sg = p.seg[s];
            row0 = (task - t0[s]) * R;
            rows = min(R, sg.n_rows - row0);
            type = sg.type;
#pragma unroll
            for (int r = 0; r < R; r++)
                rp[r] = sg.w + eoff * sg.expert_stride + (long long)(row0 + min(r, rows - 1)) * sg.row_bytes;
        }
        float acc[R];
#pragma unroll
        for (int r = 0; r < R; r++) acc[r] = 0.0f;
        switch (type) {
            case T_Q4_K: rows_dot_k45<false, R>(rp, p.K >> 8, xs, lane, acc); break;
            case T_Q5_K: rows_dot_k45<true, R>(rp, p.K >> 8, xs, lane, acc); break;
            case T_Q6_K: rows_dot_q6k(rp, p.K >> 8, xs, lane, acc); break;
            default: rows_dot_b32(type, rp, p.K, xs, lane, acc); break;
        }
#pragma unroll
        for (int r = 0; r < R; r++) acc[r] = warp_sum(acc[r]);
        if (lane == 0) {
            if (p.epi == EPI_SWIGLU) {
                float* out = p.seg[0].out;
#pragma unroll
                for (int r = 0; r < G; r++)
                    if (r < rows) out[row0 + r] = silu_f(acc[r]) * acc[R > 1 ? r + G : r];
            } else {
                const GemvSeg& sg = p.seg[s];
#pragma unroll
                for (int r = 0; r < R; r++) {
                    if (r < rows) {
                        const int jrow = row0 + r;
                        float v = acc[r];
                        if (sg.bias) v += sg.bias[jrow];
                        if (p.epi == EPI_RESIDUAL) v += p.residual[jrow];
                        if (p.epi == EPI_SCALED_ACC) {  // moe.rs:363-368: out (zeros) += w_e * y_e, in selection order
                            const float prev = (p.expert_slot == 0 || p.expert_count > 0) ? 0.0f : sg.out[jrow];
                            v = prev + p.expert_wt[p.expert_slot] * v;
                            if (p.residual && p.expert_count == 0) v += p.residual[jrow];  // last selected expert: + h (layers.rs:1235-1241)
                        }
                        sg.out[jrow] = v;
                    }
                }
            }
        }
    }
}

// Rows per task: as many as still give every one of the chip's warps (two blocks per SM) a task
inline int gemv_tasks(const GemvParams& p, int R) {
    if (p.epi == EPI_SWIGLU) return (p.seg[0].n_rows + R / 2 - 1) / (R / 2);
    int n = 0;
    for (int s = 0; s < p.n_seg; s++) n += (p.seg[s].n_rows + R - 1) / R;
    return n;
}
inline int gemv_rows(const GemvParams& p, int n_sm) {
    for (int R = kGemvR; R > (p.epi == EPI_SWIGLU ? 2 : 1); R /= 2)
        if (gemv_tasks(p, R) >= 2 * n_sm * kGemvWarps) return R;
    return p.epi == EPI_SWIGLU ? 2 : 1;
}

}  // namespace b200
