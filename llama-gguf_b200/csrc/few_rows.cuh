// few_rows.cuh — the kernels between the products of gemm_few.cuh: each adds the pieces of the product before it (FewOut) and writes the image of the next
// one's activations (few_put8).  Same f32 arithmetic as their counterparts in prefill.cuh (RMSNorm simd.rs:847-899, rope cpu/ops.rs:1216-1337, SwiGLU simd.rs:598-649).
// All are bound by latency (a few hundred KB from L2, T blocks): every load of a thread is independent.
#pragma once
#include "gemm_few.cuh"
#include "prefill.cuh"

namespace b200 {

constexpr int kFewNormMax = 8192;      // one chunk of eight per thread, n / 8 threads
// X[t] += the product `add` (where there is one); image (where asked for) = fp16 of rms_norm(X[t]) w
__global__ void __launch_bounds__(1024) few_norm_kernel(float* __restrict__ X, const __grid_constant__ FewOut add, int has_add, const float* __restrict__ w, float eps, uint8_t* __restrict__ img,
                                                        int N, int n) {
    pdl_launch_dependents();
    const int t = blockIdx.x, c = threadIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __shared__ float red[32];
    float v[8], wv[8], s[8];
    if (img) {
        const float4 a = *reinterpret_cast<const float4*>(w + 8 * c), b = *reinterpret_cast<const float4*>(w + 8 * c + 4);
        wv[0] = a.x; wv[1] = a.y; wv[2] = a.z; wv[3] = a.w; wv[4] = b.x; wv[5] = b.y; wv[6] = b.z; wv[7] = b.w;
    }
    FewTile tl{};
    if (has_add) tl = few_tile(add.plan, 0, (8 * c) >> 7, t / add.N);
    pdl_wait();
    float4* xr = reinterpret_cast<float4*>(X + (size_t)t * n + 8 * c);
    const float4 a = xr[0], b = xr[1];
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    if (has_add) {
        few_get<8>(add, 0, tl, t, 8 * c, s);
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] += s[i];
        xr[0] = make_float4(v[0], v[1], v[2], v[3]);
        xr[1] = make_float4(v[4], v[5], v[6], v[7]);
    }
    if (!img) return;
    float ss = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; i++) ss = fmaf(v[i], v[i], ss);
    ss = warp_sum(ss);
    if (lane == 0) red[warp] = ss;
    __syncthreads();
    const float tot = warp_sum(lane < (int)(blockDim.x >> 5) ? red[lane] : 0.0f);
    const float inv = 1.0f / sqrtf(tot / (float)n + eps);
    __half h[8];
#pragma unroll
    for (int i = 0; i < 8; i++) h[i] = f2h_sat(__fmul_rn(__fmul_rn(v[i], inv), wv[i]));
    few_put8(img, N, n / 256, t, c, h, few_sum32(h));
}

// image = silu(gate) up of the products gate (segment 0) and up (segment 1), I wide
__global__ void __launch_bounds__(256) few_swiglu_kernel(const __grid_constant__ FewOut gu, uint8_t* __restrict__ img, int I) {
    pdl_launch_dependents();
    const int nch = I / 8, t = blockIdx.y, c = blockIdx.x * 256 + threadIdx.x;
    if (c >= nch) return;      // (whole warps: I is whole blocks of 256)
    const FewTile tg = few_tile(gu.plan, 0, (8 * c) >> 7, t / gu.N), tu = few_tile(gu.plan, 1, (8 * c) >> 7, t / gu.N);
    pdl_wait();
    float g[8], u[8];
    few_get<8>(gu, 0, tg, t, 8 * c, g);
    few_get<8>(gu, 1, tu, t, 8 * c, u);
    __half h[8];
#pragma unroll
    for (int i = 0; i < 8; i++) h[i] = f2h_sat((g[i] / (1.0f + expf(-g[i]))) * u[i]);
    few_put8(img, gu.N, I / 256, t, c, h, few_sum32(h));
}

// fp16 rows -> image (rows of the tensor-core prompt attention)
__global__ void __launch_bounds__(256) few_image_kernel(const __half* __restrict__ x, int ldx, uint8_t* __restrict__ img, int N, int n) {
    pdl_launch_dependents();
    pdl_wait();
    const int t = blockIdx.y, c = blockIdx.x * 256 + threadIdx.x;
    if (c >= n / 8) return;
    const uint4 a = *reinterpret_cast<const uint4*>(x + (size_t)t * ldx + 8 * c);
    __half h[8];
    *reinterpret_cast<uint4*>(h) = a;
    few_put8(img, N, n / 256, t, c, h, few_sum32(h));
}

// q / k / v of the product qkv (segments 0 - 2) plus their biases: rope, q -> rows of `p.qkv`, k and v -> caches (prefill_rope_kv_kernel's arithmetic).
struct FewRopeArgs {
    FewOut qkv;
    PrefillRopeParams p;
    const float* bias[3];
};
__global__ void __launch_bounds__(256) few_rope_kv_kernel(const __grid_constant__ FewRopeArgs a) {
    pdl_launch_dependents();
    const PrefillRopeParams& p = a.p;
    const int t = blockIdx.x, half = p.hd >> 1;
    __shared__ float cs_s[64], sn_s[64];
    pdl_wait();
    const int pos = p.row_pos ? p.row_pos[t] : p.pos0 + t;
    float* const k_cache = p.row_pos ? p.row_kv[t] + p.k_off : p.k_cache;
    float* const v_cache = p.row_pos ? p.row_kv[t] + p.v_off : p.v_cache;
    const float position = (float)pos / p.rope_scale;
    if ((int)threadIdx.x < half) {
        const float theta = position * p.freq[threadIdx.x];
        cs_s[threadIdx.x] = cosf(theta);
        sn_s[threadIdx.x] = sinf(theta);
    }
    __syncthreads();
    const int n_pairs = (p.n_heads + p.n_kv) * half, n_v = p.n_kv * p.hd, n = t / a.qkv.N;
    float* row = p.qkv + (size_t)t * p.ld;
    for (int i = blockIdx.y * blockDim.x + threadIdx.x; i < n_pairs + n_v; i += blockDim.x * gridDim.y) {
        if (i < n_pairs) {
            const int head = i / half, pi = i - head * half;
            const float c = cs_s[pi], s = sn_s[pi];
            const int i0 = p.neox ? pi : 2 * pi, i1 = p.neox ? pi + half : 2 * pi + 1;
            const bool q = head < p.n_heads;
            const int h = q ? head : head - p.n_heads, sg = q ? 0 : 1;
            const FewTile tl = few_tile(a.qkv.plan, sg, (h * p.hd) >> 7, n);      // (a head lies in one tile: hd is 64 or 128)
            float x0[1], x1[1];
            few_get<1>(a.qkv, sg, tl, t, h * p.hd + i0, x0);
            few_get<1>(a.qkv, sg, tl, t, h * p.hd + i1, x1);
            if (a.bias[sg]) {
                x0[0] += a.bias[sg][h * p.hd + i0];
                x1[0] += a.bias[sg][h * p.hd + i1];
            }
            float* o = q ? row + (size_t)h * p.hd : k_cache + ((size_t)h * p.max_seq + pos) * p.hd;
            o[i0] = __fsub_rn(__fmul_rn(x0[0], c), __fmul_rn(x1[0], s));
            o[i1] = __fadd_rn(__fmul_rn(x0[0], s), __fmul_rn(x1[0], c));
        } else {
            const int j = i - n_pairs, kh = j / p.hd, d = j - kh * p.hd;
            float x[1];
            few_get<1>(a.qkv, 2, few_tile(a.qkv.plan, 2, j >> 7, n), t, j, x);
            if (a.bias[2]) x[0] += a.bias[2][j];
            v_cache[((size_t)kh * p.max_seq + pos) * p.hd + d] = x[0];
        }
    }
}

// Batched decoding: rope, the caches' new rows and attention of one (row, kv head) per block.  The new key and value come from shared memory; the eight
// warps take the positions in turns (four at a time, online softmax as in prefill_attn_kernel) and their sums are merged in the order of the warps.
// One launch where there were two, and eight warps per (row, kv head) where there was one.
struct FewAttnArgs {
    FewOut qkv;
    const float* bias[3];
    const float* freq;
    int n_heads, n_kv, max_seq, neox, A;      // A = n_heads * head size
    float rope_scale, scale;
    const int* row_pos;
    float* const* row_kv;
    long long k_off, v_off;
    uint8_t* img;
};
template <int HD, int GMAX>
__global__ void __launch_bounds__(256) few_attn_kernel(const __grid_constant__ FewAttnArgs a) {
    pdl_launch_dependents();
    constexpr int VEC = HD / 32, UB = 4, NW = 8, HALF = HD / 2;
    __shared__ __align__(16) float s_q[GMAX][HD], s_k[HD], s_v[HD];
    __shared__ __align__(16) float s_acc[NW][GMAX][HD];
    __shared__ float s_m[NW][GMAX], s_l[NW][GMAX], s_cs[HALF], s_sn[HALF];
    const int kh = blockIdx.x, t = blockIdx.y, G = a.n_heads / a.n_kv, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, n = t / a.qkv.N;
    const FewTile tk = few_tile(a.qkv.plan, 1, (kh * HD) >> 7, n), tv = few_tile(a.qkv.plan, 2, (kh * HD) >> 7, n);
    pdl_wait();
    const int pos = a.row_pos[t];
    float* const kb = a.row_kv[t] + a.k_off + (size_t)kh * a.max_seq * HD;
    float* const vb = a.row_kv[t] + a.v_off + (size_t)kh * a.max_seq * HD;
    if (tid < HALF) {
        const float theta = (float)pos / a.rope_scale * a.freq[tid];
        s_cs[tid] = cosf(theta);
        s_sn[tid] = sinf(theta);
    }
    __syncthreads();
    for (int i = tid; i < (G + 1) * HALF + HD; i += 256) {
        if (i < (G + 1) * HALF) {      // pairs of the G query heads, then of the key
            const int hh = i / HALF, pi = i - hh * HALF, i0 = a.neox ? pi : 2 * pi, i1 = a.neox ? pi + HALF : 2 * pi + 1, sg = hh < G ? 0 : 1;
            const int at = (hh < G ? kh * G + hh : kh) * HD;
            const FewTile tl = hh < G ? few_tile(a.qkv.plan, 0, at >> 7, n) : tk;
            float x0[1], x1[1];
            few_get<1>(a.qkv, sg, tl, t, at + i0, x0);
            few_get<1>(a.qkv, sg, tl, t, at + i1, x1);
            if (a.bias[sg]) {
                x0[0] += a.bias[sg][at + i0];
                x1[0] += a.bias[sg][at + i1];
            }
            const float c = s_cs[pi], s = s_sn[pi];
            const float y0 = __fsub_rn(__fmul_rn(x0[0], c), __fmul_rn(x1[0], s)), y1 = __fadd_rn(__fmul_rn(x0[0], s), __fmul_rn(x1[0], c));
            if (hh < G) {
                s_q[hh][i0] = y0;
                s_q[hh][i1] = y1;
            } else {
                s_k[i0] = y0;
                s_k[i1] = y1;
                kb[(size_t)pos * HD + i0] = y0;
                kb[(size_t)pos * HD + i1] = y1;
            }
        } else {
            const int d = i - (G + 1) * HALF;
            float x[1];
            few_get<1>(a.qkv, 2, tv, t, kh * HD + d, x);
            if (a.bias[2]) x[0] += a.bias[2][kh * HD + d];
            s_v[d] = x[0];
            vb[(size_t)pos * HD + d] = x[0];
        }
    }
    __syncthreads();
    float q[GMAX][VEC], acc[GMAX][VEC], m[GMAX], l[GMAX];
#pragma unroll
    for (int g = 0; g < GMAX; g++) {
        m[g] = -INFINITY;
        l[g] = 0.0f;
#pragma unroll
        for (int v = 0; v < VEC; v++) {
            acc[g][v] = 0.0f;
            q[g][v] = g < G ? s_q[g][lane * VEC + v] : 0.0f;
        }
    }
    for (int p0 = warp * UB; p0 <= pos; p0 += NW * UB) {
        float kr[UB][VEC], vr[UB][VEC];
#pragma unroll
        for (int u = 0; u < UB; u++) {
            const int pc = min(p0 + u, pos);      // (clamped, masked below)
            const float* kp = pc == pos ? s_k : kb + (size_t)pc * HD;
            const float* vp = pc == pos ? s_v : vb + (size_t)pc * HD;
#pragma unroll
            for (int v = 0; v < VEC; v += 2) {
                const float2 x = *reinterpret_cast<const float2*>(kp + lane * VEC + v), y = *reinterpret_cast<const float2*>(vp + lane * VEC + v);
                kr[u][v] = x.x; kr[u][v + 1] = x.y;
                vr[u][v] = y.x; vr[u][v + 1] = y.y;
            }
        }
        float s[UB][GMAX];
#pragma unroll
        for (int u = 0; u < UB; u++)
#pragma unroll
            for (int g = 0; g < GMAX; g++) {
                float d = 0.0f;
#pragma unroll
                for (int v = 0; v < VEC; v++) d = fmaf(q[g][v], kr[u][v], d);
                s[u][g] = d;
            }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int u = 0; u < UB; u++)
#pragma unroll
                for (int g = 0; g < GMAX; g++) s[u][g] += __shfl_xor_sync(0xffffffffu, s[u][g], o);
#pragma unroll
        for (int g = 0; g < GMAX; g++) {
            float mb = -INFINITY;
#pragma unroll
            for (int u = 0; u < UB; u++) {
                s[u][g] = p0 + u <= pos ? s[u][g] * a.scale : -INFINITY;
                mb = fmaxf(mb, s[u][g]);
            }
            const float mn = fmaxf(m[g], mb), corr = m[g] == -INFINITY ? 0.0f : expf(m[g] - mn);
            float w[UB], ws = 0.0f;
#pragma unroll
            for (int u = 0; u < UB; u++) {
                w[u] = s[u][g] == -INFINITY ? 0.0f : expf(s[u][g] - mn);
                ws += w[u];
            }
            l[g] = l[g] * corr + ws;
#pragma unroll
            for (int v = 0; v < VEC; v++) {
                float x = acc[g][v] * corr;
#pragma unroll
                for (int u = 0; u < UB; u++) x = fmaf(w[u], vr[u][v], x);
                acc[g][v] = x;
            }
            m[g] = mn;
        }
    }
#pragma unroll
    for (int g = 0; g < GMAX; g++) {
        if (g < G) {
#pragma unroll
            for (int v = 0; v < VEC; v++) s_acc[warp][g][lane * VEC + v] = acc[g][v];
            if (lane == 0) {
                s_m[warp][g] = m[g];
                s_l[warp][g] = l[g];
            }
        }
    }
    __syncthreads();
    if (warp < G) {
        const int g = warp;
        float mx = -INFINITY, sum = 0.0f, out[VEC];
#pragma unroll
        for (int w = 0; w < NW; w++) mx = fmaxf(mx, s_m[w][g]);
#pragma unroll
        for (int v = 0; v < VEC; v++) out[v] = 0.0f;
#pragma unroll
        for (int w = 0; w < NW; w++) {
            const float f = s_m[w][g] == -INFINITY ? 0.0f : expf(s_m[w][g] - mx);      // (a warp without positions)
            sum = fmaf(s_l[w][g], f, sum);
#pragma unroll
            for (int v = 0; v < VEC; v++) out[v] = fmaf(s_acc[w][g][lane * VEC + v], f, out[v]);
        }
        const float inv = 1.0f / sum;
        __half h[VEC];
#pragma unroll
        for (int v = 0; v < VEC; v++) h[v] = f2h_sat(out[v] * inv);
        few_put_lane<VEC>(a.img, a.qkv.N, a.A / 256, t, (kh * G + g) * HD + lane * VEC, h);
    }
}

// the cut tiles of segment 0 -> y (whole ones are there): grid (row tiles, groups of eight tokens)
__global__ void __launch_bounds__(128) few_finish_kernel(const __grid_constant__ FewOut o, float* __restrict__ y, int n_rows) {
    pdl_launch_dependents();
    pdl_wait();
    const int t0 = blockIdx.y * 8, j = blockIdx.x * 128 + threadIdx.x;
    const FewTile tl = few_tile(o.plan, 0, blockIdx.x, t0 / o.N);
    if (tl.b0 == tl.b1 || j >= n_rows) return;
    float v[8][1];
#pragma unroll
    for (int i = 0; i < 8; i++)
        if (t0 + i < o.plan.T) few_get<1>(o, 0, tl, t0 + i, j, v[i]);
#pragma unroll
    for (int i = 0; i < 8; i++)
        if (t0 + i < o.plan.T) y[(size_t)(t0 + i) * o.ldy[0] + j] = v[i][0];
}

}  // namespace b200
