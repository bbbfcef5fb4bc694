// prefill.cuh — the memory-bound kernels around the tcgen05 dequant-GEMM (gemm_umma.cuh) when a prompt is processed T
// tokens at a time: embedding rows, RoPE + KV-cache write, causal GQA attention over the cache, SwiGLU.
// Same arithmetic as the per-token kernels (embed_kernel, attn_decode_item) and as the reference
// (LlamaModel::forward src/model/llama.rs:275-362; ops::rope cpu/ops.rs:1216-1337; attention_cached :1479-1537;
// silu_mul_inplace cpu/simd.rs:598-649), applied to T rows.
#pragma once
#include "attention.cuh"
#include "misc.cuh"
#include "quant.cuh"

namespace b200 {

// X[t][:] = dequantised row tokens[t] of the embedding table (bit-exact), eight elements per thread: one at a time, each read its block's header and scales
// again (2048 rows of 4096 in Q4_K: 34.4 -> 13.6 us, 2.8 TB/s).  Up to 256 rows are split between gridDim.y blocks: what is left there is the latency of the
// token, the block's header and its bytes.
__global__ void prefill_embed_kernel(int type, const uint8_t* __restrict__ table, long long row_bytes, int hidden, const int* __restrict__ tokens,
                                     int vocab, float* __restrict__ X) {
    pdl_launch_dependents();
    pdl_wait();
    const int t = blockIdx.x;
    const int token = min(max(tokens[t], 0), vocab - 1);
    const int be = type_block_elems(type), bb = type_block_bytes(type);
    const uint8_t* row = table + (long long)token * row_bytes;
    if (be >= 32 && hidden % 8 == 0) {      // eight elements of a block per thread
        for (int i = (blockIdx.y * blockDim.x + threadIdx.x) * 8; i < hidden; i += gridDim.y * blockDim.x * 8) {
            const int blk = i / be;
            float v[8];
            dequant_elem8(type, row + (long long)blk * bb, i - blk * be, v);
            float4* o = reinterpret_cast<float4*>(X + (size_t)t * hidden + i);
            o[0] = make_float4(v[0], v[1], v[2], v[3]);
            o[1] = make_float4(v[4], v[5], v[6], v[7]);
        }
        return;
    }
    for (int i = blockIdx.y * blockDim.x + threadIdx.x; i < hidden; i += gridDim.y * blockDim.x) {
        const int blk = i / be;
        X[(size_t)t * hidden + i] = dequant_elem(type, row + (long long)blk * bb, i - blk * be);
    }
}

struct PrefillRopeParams {
    float* qkv;            // [T][ld]: q | k | v raw projections (+bias); q is rotated in place
    int ld;
    float* k_cache;        // [n_kv][max_seq][hd]
    float* v_cache;
    const float* freq;     // [hd/2]
    int pos0, n_heads, n_kv, hd, max_seq, neox;
    float rope_scale;
    // batched decode: row t is the next token of ITS OWN sequence slot -- position row_pos[t], caches at
    // row_kv[t] + k_off / v_off (floats); nullptr = rows are consecutive positions of one sequence (prefill)
    const int* row_pos;
    float* const* row_kv;
    long long k_off, v_off;
};
// one CTA per token: Backend::rope for the token's position pos0 + t, k rows -> cache, v rows -> cache
__global__ void prefill_rope_kv_kernel(const PrefillRopeParams p) {
    pdl_launch_dependents();
    pdl_wait();
    const int t = blockIdx.x, pos = p.row_pos ? p.row_pos[t] : p.pos0 + t;
    float* const k_cache = p.row_pos ? p.row_kv[t] + p.k_off : p.k_cache;
    float* const v_cache = p.row_pos ? p.row_kv[t] + p.v_off : p.v_cache;
    const int half = p.hd >> 1;
    const int n_pairs = (p.n_heads + p.n_kv) * half, n_v = p.n_kv * p.hd;
    const float position = (float)pos / p.rope_scale;
    float* row = p.qkv + (size_t)t * p.ld;
    const float* vraw = row + (size_t)(p.n_heads + p.n_kv) * p.hd;
    // a token's hd / 2 angles once per CTA (every head turns by the same ones; four 2048-wide layers, 333 tokens: 806 -> 798 us)
    __shared__ __align__(16) float cs_s[64], sn_s[64];      // (hd is 64 or 128)
    if ((int)threadIdx.x < half) {
        const float theta = position * p.freq[threadIdx.x];
        cs_s[threadIdx.x] = cosf(theta);
        sn_s[threadIdx.x] = sinf(theta);
    }
    __syncthreads();
    // gridDim.y CTAs share a token's items (each item is independent: same arithmetic whoever computes it): four pairs by two 16-byte loads, three items' loads before the
    // first store.  A pair per thread and iteration was bound by its index arithmetic and by loads that waited
    // for stores (2048 tokens of an 8B layer: 28 -> 18 us, 83 MB).
    const int stride = blockDim.x * gridDim.y, at0 = blockIdx.y * blockDim.x + threadIdx.x, sh = half == 64 ? 4 : 3, n_items = n_pairs >> 2;
    constexpr int NB = 3;
    for (int b0 = at0; b0 < n_items; b0 += NB * stride) {
        float4 a[NB], b[NB];
#pragma unroll
        for (int u = 0; u < NB; u++) {
            const int i = b0 + u * stride;
            if (i >= n_items) continue;
            const int head = i >> sh, pi = (i & ((1 << sh) - 1)) * 4;
            const float* d = row + (size_t)head * p.hd;      // (k heads follow q heads)
            a[u] = *reinterpret_cast<const float4*>(d + (p.neox ? pi : 2 * pi));
            b[u] = *reinterpret_cast<const float4*>(d + (p.neox ? pi + half : 2 * pi + 4));
        }
#pragma unroll
        for (int u = 0; u < NB; u++) {
            const int i = b0 + u * stride;
            if (i >= n_items) continue;
            const int head = i >> sh, pi = (i & ((1 << sh) - 1)) * 4;
            const float4 c = *reinterpret_cast<const float4*>(cs_s + pi), s = *reinterpret_cast<const float4*>(sn_s + pi);
            float* o = head < p.n_heads ? row + (size_t)head * p.hd : k_cache + ((size_t)(head - p.n_heads) * p.max_seq + pos) * p.hd;
            auto lo = [](float x0, float x1, float cc, float ss) { return __fsub_rn(__fmul_rn(x0, cc), __fmul_rn(x1, ss)); };
            auto hi = [](float x0, float x1, float cc, float ss) { return __fadd_rn(__fmul_rn(x0, ss), __fmul_rn(x1, cc)); };
            const float4 x = a[u], y = b[u];
            if (p.neox) {
                *reinterpret_cast<float4*>(o + pi) = make_float4(lo(x.x, y.x, c.x, s.x), lo(x.y, y.y, c.y, s.y), lo(x.z, y.z, c.z, s.z), lo(x.w, y.w, c.w, s.w));
                *reinterpret_cast<float4*>(o + pi + half) = make_float4(hi(x.x, y.x, c.x, s.x), hi(x.y, y.y, c.y, s.y), hi(x.z, y.z, c.z, s.z), hi(x.w, y.w, c.w, s.w));
            } else {
                *reinterpret_cast<float4*>(o + 2 * pi) = make_float4(lo(x.x, x.y, c.x, s.x), hi(x.x, x.y, c.x, s.x), lo(x.z, x.w, c.y, s.y), hi(x.z, x.w, c.y, s.y));
                *reinterpret_cast<float4*>(o + 2 * pi + 4) = make_float4(lo(y.x, y.y, c.z, s.z), hi(y.x, y.y, c.z, s.z), lo(y.z, y.w, c.w, s.w), hi(y.z, y.w, c.w, s.w));
            }
        }
    }
    for (int i = at0; i < n_v / 4; i += stride) {      // (hd is a multiple of 4)
        const int j = 4 * i, kh = j / p.hd, d = j - kh * p.hd;
        *reinterpret_cast<float4*>(v_cache + ((size_t)kh * p.max_seq + pos) * p.hd + d) = *reinterpret_cast<const float4*>(vraw + j);
    }
}

struct PrefillAttnParams {
    const float* qkv;      // [T][ld], q rotated
    int ld;
    const float* k_cache;  // [n_kv][max_seq][hd], positions 0 .. pos0 + T - 1 valid
    const float* v_cache;
    __half* out;           // [T][ldo]: [n_heads][hd] per token, fp16 (input of the O-projection GEMM)
    int ldo;
    int pos0, T, n_heads, n_kv, max_seq;
    float scale;
    const int* row_pos;        // batched decode: see PrefillRopeParams
    float* const* row_kv;
    long long k_off, v_off;
};
// One warp per (token, kv head): the G query heads of the group share every K / V row read (GQA), four cache positions per
// step (16 independent dot products and reductions in flight), block-wise online softmax as in attn_decode_item.
// Causal: token t attends cache positions 0 .. pos0 + t.
template <int HD, int GMAX>
__global__ void __launch_bounds__(128) prefill_attn_kernel(const PrefillAttnParams p) {
    pdl_launch_dependents();
    pdl_wait();
    constexpr int VEC = HD / 32, UB = 4;
    const int lane = threadIdx.x & 31;
    const long long wid = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (wid >= (long long)p.T * p.n_kv) return;
    const int t = (int)(wid / p.n_kv), kh = (int)(wid - (long long)t * p.n_kv);
    const int G = p.n_heads / p.n_kv;
    const int kv_len = (p.row_pos ? p.row_pos[t] : p.pos0 + t) + 1;
    float q[GMAX][VEC], acc[GMAX][VEC], m[GMAX], l[GMAX];
#pragma unroll
    for (int g = 0; g < GMAX; g++) {
        m[g] = -INFINITY;
        l[g] = 0.0f;
#pragma unroll
        for (int v = 0; v < VEC; v++) {
            acc[g][v] = 0.0f;
            q[g][v] = g < G ? p.qkv[(size_t)t * p.ld + (size_t)(kh * G + g) * HD + lane * VEC + v] : 0.0f;
        }
    }
    const float* kb = (p.row_pos ? p.row_kv[t] + p.k_off : p.k_cache) + (size_t)kh * p.max_seq * HD + lane * VEC;
    const float* vb = (p.row_pos ? p.row_kv[t] + p.v_off : p.v_cache) + (size_t)kh * p.max_seq * HD + lane * VEC;
    // the K / V rows of the next four positions are in flight while these four are processed (two register buffers)
    auto load = [&](int pos, float (&kk)[UB][VEC], float (&vv)[UB][VEC]) {
#pragma unroll
        for (int u = 0; u < UB; u++) {
            const int pc = min(pos + u, kv_len - 1);   // clamped: stays in range, masked below
            if constexpr (VEC == 4) {
                const float4 a = *reinterpret_cast<const float4*>(kb + (size_t)pc * HD), b = *reinterpret_cast<const float4*>(vb + (size_t)pc * HD);
                kk[u][0] = a.x; kk[u][1] = a.y; kk[u][2] = a.z; kk[u][3] = a.w;
                vv[u][0] = b.x; vv[u][1] = b.y; vv[u][2] = b.z; vv[u][3] = b.w;
            } else {
                const float2 a = *reinterpret_cast<const float2*>(kb + (size_t)pc * HD), b = *reinterpret_cast<const float2*>(vb + (size_t)pc * HD);
                kk[u][0] = a.x; kk[u][1] = a.y;
                vv[u][0] = b.x; vv[u][1] = b.y;
            }
        }
    };
    float kn[UB][VEC], vn[UB][VEC];
    load(0, kn, vn);
    for (int pos = 0; pos < kv_len; pos += UB) {
        float kr[UB][VEC], vr[UB][VEC];
#pragma unroll
        for (int u = 0; u < UB; u++)
#pragma unroll
            for (int v = 0; v < VEC; v++) { kr[u][v] = kn[u][v]; vr[u][v] = vn[u][v]; }
        if (pos + UB < kv_len) load(pos + UB, kn, vn);
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
            if (g < G) {
                float mb = -INFINITY;
#pragma unroll
                for (int u = 0; u < UB; u++) {
                    s[u][g] = (pos + u < kv_len) ? s[u][g] * p.scale : -INFINITY;
                    mb = fmaxf(mb, s[u][g]);
                }
                const float mn = fmaxf(m[g], mb);
                const float corr = (m[g] == -INFINITY) ? 0.0f : expf(m[g] - mn);
                float w[UB], ws = 0.0f;
#pragma unroll
                for (int u = 0; u < UB; u++) {
                    w[u] = (s[u][g] == -INFINITY) ? 0.0f : expf(s[u][g] - mn);
                    ws += w[u];
                }
                l[g] = l[g] * corr + ws;
#pragma unroll
                for (int v = 0; v < VEC; v++) {
                    float a = acc[g][v] * corr;
#pragma unroll
                    for (int u = 0; u < UB; u++) a = fmaf(w[u], vr[u][v], a);
                    acc[g][v] = a;
                }
                m[g] = mn;
            }
        }
    }
#pragma unroll
    for (int g = 0; g < GMAX; g++) {
        if (g < G) {
            const float inv = 1.0f / l[g];
#pragma unroll
            for (int v = 0; v < VEC; v++) p.out[(size_t)t * p.ldo + (size_t)(kh * G + g) * HD + lane * VEC + v] = f2h_sat(acc[g][v] * inv);
        }
    }
}

// RMSNorm of T rows, output rounded to fp16 for the tensor-core GEMM that consumes it (same f32 arithmetic as
// rms_norm_rows_kernel: ss = sum x^2, inv = 1/sqrt(ss/n + eps), (x*inv)*w; simd.rs:847-899)
// Sums in the order of a block that walks the row: thread t adds the squares of elements t, t + 256, .., then lanes, then warps.
// NV4 > 0: rows of up to 1024 NV4 elements (a multiple of 4, as the buffers' rows are aligned) by float4, all loads of a thread before the first use; the row goes
// through shared memory, where thread t finds the elements of its sum (2048 rows of 4096: 17 -> 10 us; few registers, many blocks).  NV4 = 0: any row.
template <int NV4>
__global__ void __launch_bounds__(256) prefill_rms_norm_kernel(const float* x, const float* w, float eps, __half* out, int n) {
    pdl_launch_dependents();
    pdl_wait();
    constexpr int NV = NV4 > 0 ? NV4 : 1;
    __shared__ float red[8];
    const float* xr = x + (size_t)blockIdx.x * n;
    __half* orow = out + (size_t)blockIdx.x * n;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float ss = 0.0f;
    float4 v[NV], wv[NV];
    if (NV4 > 0) {
        __shared__ __align__(16) float row[1024 * NV];
#pragma unroll
        for (int k = 0; k < NV; k++) {
            const int i = 4 * (threadIdx.x + 256 * k);
            v[k] = i < n ? *reinterpret_cast<const float4*>(xr + i) : make_float4(0.f, 0.f, 0.f, 0.f);
            wv[k] = i < n ? *reinterpret_cast<const float4*>(w + i) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int k = 0; k < NV; k++) *reinterpret_cast<float4*>(row + 4 * (threadIdx.x + 256 * k)) = v[k];
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 4 * NV; k++) {      // (zeros behind the row)
            const float f = row[threadIdx.x + 256 * k];
            ss = fmaf(f, f, ss);
        }
    } else {
        for (int i = threadIdx.x; i < n; i += 256) ss = fmaf(xr[i], xr[i], ss);
    }
    ss = warp_sum(ss);
    if (lane == 0) red[warp] = ss;
    __syncthreads();
    float tot = 0.0f;
    for (int k = 0; k < 8; k++) tot += red[k];
    const float inv = 1.0f / sqrtf(tot / (float)n + eps);
    if (NV4 > 0) {
#pragma unroll
        for (int k = 0; k < NV; k++) {
            const int i = 4 * (threadIdx.x + 256 * k);
            if (i >= n) continue;
            const __half2 a = __halves2half2(f2h_sat(__fmul_rn(__fmul_rn(v[k].x, inv), wv[k].x)), f2h_sat(__fmul_rn(__fmul_rn(v[k].y, inv), wv[k].y)));
            const __half2 b = __halves2half2(f2h_sat(__fmul_rn(__fmul_rn(v[k].z, inv), wv[k].z)), f2h_sat(__fmul_rn(__fmul_rn(v[k].w, inv), wv[k].w)));
            *reinterpret_cast<uint2*>(orow + i) = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
        }
    } else {
        for (int i = threadIdx.x; i < n; i += 256) orow[i] = f2h_sat(__fmul_rn(__fmul_rn(xr[i], inv), w[i]));
    }
}

inline void (*prefill_rms_norm_for(int n))(const float*, const float*, float, __half*, int) {
    return n % 4 || n > 8192 ? prefill_rms_norm_kernel<0> : n <= 1024 ? prefill_rms_norm_kernel<1> : n <= 2048 ? prefill_rms_norm_kernel<2> : n <= 4096 ? prefill_rms_norm_kernel<4> : prefill_rms_norm_kernel<8>;
}

// g[i] = silu(g[i]) * u[i]  (silu rounded to f32 first, then the product: simd.rs:598-649)
__global__ void prefill_swiglu_kernel(const float* __restrict__ g, const float* __restrict__ u, __half* __restrict__ out, long long n) {
    pdl_launch_dependents();
    pdl_wait();
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const float x = g[i];
        out[i] = f2h_sat((x / (1.0f + expf(-x))) * u[i]);
    }
}

// the slot's position after a prompt whose last token was at `next` - 1
__global__ void prefill_advance_kernel(SeqState* st, int next) {
    pdl_launch_dependents();
    pdl_wait();
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        st->pos_cur = next - 1;
        st->pos_next = next;
    }
}

// batched decode: every row's slot stands behind the token at row_pos
__global__ void prefill_advance_rows_kernel(SeqState* const* st, const int* __restrict__ row_pos, int n) {
    pdl_launch_dependents();
    pdl_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        SeqState* s = st[i];
        s->pos_cur = row_pos[i];
        s->pos_next = row_pos[i] + 1;
    }
}

}  // namespace b200
