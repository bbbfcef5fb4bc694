// lp_chunk_scan.cuh — the recurrent scans of prompts in chunks of 32 tokens (f32 throughout).  Included by layerprog.cu inside its anonymous
// namespace, after the scans that go token by token (decoding, and what this file does not take).
//
// A state S [dim][vdim] per (run, head) that every token scales and adds an outer product to is, over a chunk that starts from S0,
//   O_t = z_t (q_t . S0) + p_t sum_{s <= t} M_ts U_s          S' = D S0 + sum_s u_s k_s U_s^T
// with scalars z, p, u, D from the gates and M_ts = (decay from s to t) x (q_t . k_s):
//   matrix memory (MEM)   U = v; a column of ones beside the values gives n . q; the stabiliser m_t = max(m + F_t, mu_t), F and mu local to the chunk
//   state space   (SSD)   U = x, k = B, q = C, step sizes in M and u; + D_skip x
//   delta rule    (DELTA) U = U0 - W S0, U0 = T diag(beta) v, W = T diag(beta e^L) k, T = (1 + A)^-1, A_ts = beta_t (decay) (k_t . k_s), s < t
//                         (each token's write sees the writes before it; T is the substitution over the chunk)
// lp_chunk_prep_kernel does what does not need S0, a block per (chunk, head, run); lp_chunk_scan_kernel walks a run's chunks, a block per (8 state
// columns, head, run) with the columns in shared memory and the next chunk's rows on their way.
// What bounded the token-by-token form: a chain of two reductions per token (1370 clocks for the delta rule at 128 x 128), SMs mostly waiting.
// Here a chunk's reductions are products of 64 x 128 by 8; the chain is per chunk.  1500 tokens, 8 heads of 128 x 128: delta rule 1044 -> 33 + 112 us;
// 4 heads of 64 x 128: memory 656 -> 11 + 75 us (preparation + scan, each launched cold).  The decay from s to t is multiplied up (MEM: its logarithm
// added up) from s on for every s, never a quotient or difference of running products, so it is as exact as one token after the other and a
// decay of 0 stays 0.
#pragma once

constexpr int CS = 32, CS_COLS = 8, CS_THREADS = 256, CS_SCAN_THREADS = 512, CS_STAGES = 3;
enum { CS_MEM = 0, CS_SSD = 1, CS_DELTA = 2 };
struct ChunkScan {
    int H, G, dim, vdim, R;             // heads, heads of q and k, sizes, rows of the step
    const float *Q, *K, *V;             // first column of head 0; rows ld apart, heads dim / vdim apart
    int ldq, ldv;
    const float *ga, *gb;               // gate columns of P (MEM: input, forget; SSD: step; DELTA: write strength, decay), rows ldp apart
    int ldp;
    const float *ca, *cb;               // per head (MEM: biases; SSD, DELTA: A_log, dt_bias)
    const float* skip;                  // SSD: D
    float cap;
    size_t rec_off;
    float *sc, *M, *W, *U0;             // scratch: [3][H][R] scalars, [H][R][32], DELTA: [H][R][dim], [H][R][vdim]
    float* O;
    int ldo;
};

template <int MODE, int DM>
__global__ void __launch_bounds__(CS_THREADS) lp_chunk_prep_kernel(StepMeta sm, ChunkScan g) {
    prev_grid();
    constexpr int PI = DM + 4;
    extern __shared__ __align__(16) float cp_sm[];
    float* qs = cp_sm;                          // [32][PI]
    float* ks = qs + CS * PI;                   // [32][PI]
    float* T = ks + CS * PI;                    // DELTA: A, then T scaled for U0 [32][33]
    float* Tw = T + CS * 33;                    // DELTA: T scaled for W
    float* dec = Tw + CS * 33;                  // [t][s], s <= t: decay from s to t (MEM: its logarithm) [32][33]
    __shared__ float g_s[CS], a_s[CS], b_s[CS], iq[CS], ik[CS];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, h = blockIdx.y, run = blockIdx.z;
    const int r0 = sm.run_start[run] + blockIdx.x * CS, r1 = sm.run_start[run + 1];
    if (r0 >= r1) return;
    const int nt = min(CS, r1 - r0), hk = h * g.G / g.H;
    for (int i = tid; i < CS * (DM / 4); i += CS_THREADS) {
        const int t = i / (DM / 4), d = (i - t * (DM / 4)) * 4;
        const bool in = t < nt && d < g.dim;
        const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
        *reinterpret_cast<float4*>(qs + t * PI + d) = in ? *reinterpret_cast<const float4*>(g.Q + (size_t)(r0 + t) * g.ldq + hk * g.dim + d) : z;
        *reinterpret_cast<float4*>(ks + t * PI + d) = in ? *reinterpret_cast<const float4*>(g.K + (size_t)(r0 + t) * g.ldq + hk * g.dim + d) : z;
    }
    // gates: decay (MEM: its logarithm; none past the end), a / b: what else M and u need
    if (tid < CS) {
        float l = MODE == CS_MEM ? 0.0f : 1.0f, a = 0.0f;
        if (tid < nt) {
            const float* ga = g.ga + (size_t)(r0 + tid) * g.ldp + h;
            const float* gb = g.gb + (size_t)(r0 + tid) * g.ldp + h;
            if (MODE == CS_MEM) {
                a = g.cap * tanhf((*ga + g.ca[h]) / g.cap);
                l = logsigmoid_f(g.cap * tanhf((*gb + g.cb[h]) / g.cap));
            } else if (MODE == CS_SSD) {
                a = softplus_f(*ga + g.cb[h]);
                l = expf(-expf(g.ca[h]) * a);
            } else {
                a = sigmoid_f(*ga);
                l = expf(-expf(g.ca[h]) * softplus_f(*gb + g.cb[h]));
            }
        }
        if (MODE == CS_MEM) {                   // mu_t = the largest i_s + f_(s+1) + ... + f_t of the chunk, composed as (sum of f, mu) pairs
            float L = l, mu = a;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const float pl = __shfl_up_sync(0xffffffffu, L, o), pm = __shfl_up_sync(0xffffffffu, mu, o);
                if (lane >= o) {
                    mu = fmaxf(pm + L, mu);
                    L += pl;
                }
            }
            b_s[tid] = mu;
        }
        g_s[tid] = l;
        a_s[tid] = a;
        __syncwarp();
        float acc = MODE == CS_MEM ? 0.0f : 1.0f;
        dec[tid * 33 + tid] = acc;
#pragma unroll
        for (int t = 1; t < CS; t++)
            if (t > tid) {
                acc = MODE == CS_MEM ? acc + g_s[t] : acc * g_s[t];
                dec[t * 33 + tid] = acc;
            }
    }
    __syncthreads();
    if (MODE == CS_DELTA) {                     // unit norms: four rows of q and of k per warp
        const float qscale = 1.0f / sqrtf((float)g.dim);
        for (int u = warp; u < 2 * CS; u += CS_THREADS / 32) {
            const float* v = (u & 1 ? ks : qs) + (u >> 1) * PI;
            float ss = 0.0f;
            for (int d = lane; d < DM; d += 32) ss += v[d] * v[d];
            ss = wsum(ss);
            if (lane == 0) (u & 1 ? ik : iq)[u >> 1] = ((u & 1) ? 1.0f : qscale) / sqrtf(ss + 1e-6f);
        }
        __syncthreads();
    }
    // q . k (and k . k): a thread's row t against keys s = (tid & 7) + 8 j
    const int t = tid >> 3;
    float qk[4] = {0.f, 0.f, 0.f, 0.f}, kk[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
    for (int d = 0; d < DM; d += 4) {
        const float4 q = *reinterpret_cast<const float4*>(qs + t * PI + d), kt = *reinterpret_cast<const float4*>(ks + t * PI + d);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float4 k = *reinterpret_cast<const float4*>(ks + ((tid & 7) + 8 * j) * PI + d);
            qk[j] = fmaf(q.x, k.x, qk[j]); qk[j] = fmaf(q.y, k.y, qk[j]); qk[j] = fmaf(q.z, k.z, qk[j]); qk[j] = fmaf(q.w, k.w, qk[j]);
            if (MODE == CS_DELTA) { kk[j] = fmaf(kt.x, k.x, kk[j]); kk[j] = fmaf(kt.y, k.y, kk[j]); kk[j] = fmaf(kt.z, k.z, kk[j]); kk[j] = fmaf(kt.w, k.w, kk[j]); }
        }
    }
    const size_t hr = (size_t)h * g.R + r0;
    const float qsc = MODE == CS_MEM ? 1.0f / sqrtf((float)g.dim) : 1.0f;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const int s = (tid & 7) + 8 * j;
        const float dc = s <= t ? dec[t * 33 + s] : 0.0f;
        float m;
        if (MODE == CS_MEM) m = s <= t ? expf(dc + a_s[s] - b_s[t]) * qsc * qk[j] : 0.0f;
        else if (MODE == CS_SSD) m = dc * a_s[s] * qk[j];
        else m = dc * iq[t] * ik[s] * qk[j];
        if (t < nt) g.M[(hr + t) * CS + s] = s < nt ? m : 0.0f;
        if (MODE == CS_DELTA) T[t * 33 + s] = s < t ? a_s[t] * dc * ik[t] * ik[s] * kk[j] : 0.0f;
    }
    if (tid < nt) {
        float *s0 = g.sc + hr + tid, *s1 = s0 + (size_t)g.H * g.R, *s2 = s1 + (size_t)g.H * g.R;
        const float from0 = MODE == CS_MEM ? dec[tid * 33] + g_s[0] : dec[tid * 33] * g_s[0], to_end = dec[(CS - 1) * 33 + tid];     // (rows past the end change nothing)
        if (MODE == CS_MEM) {
            *s0 = from0;
            *s1 = to_end + a_s[tid];
            *s2 = b_s[tid];
        } else {
            *s0 = from0 * (MODE == CS_DELTA ? iq[tid] : 1.0f);
            *s1 = to_end * (MODE == CS_DELTA ? ik[tid] : a_s[tid]);
            *s2 = dec[(CS - 1) * 33] * g_s[0];
        }
    }
    if (MODE != CS_DELTA) return;
    __syncthreads();
    if (warp == 0) {                            // column `lane` of (1 + A)^-1 by substitution
        float x[CS];
#pragma unroll
        for (int i = 0; i < CS; i++) {
            float v0 = 0.0f, v1 = 0.0f;
#pragma unroll
            for (int s = 0; s + 1 < i; s += 2) {
                v0 = fmaf(T[i * 33 + s], x[s], v0);
                v1 = fmaf(T[i * 33 + s + 1], x[s + 1], v1);
            }
            if (i & 1) v0 = fmaf(T[i * 33 + i - 1], x[i > 0 ? i - 1 : 0], v0);
            x[i] = i < lane ? 0.0f : i == lane ? 1.0f : -(v0 + v1);
        }
        __syncwarp();
        const float bu = a_s[lane], bw = bu * dec[lane * 33] * g_s[0] * ik[lane];
#pragma unroll
        for (int i = 0; i < CS; i++) {
            Tw[i * 33 + lane] = x[i] * bw;
            T[i * 33 + lane] = x[i] * bu;
        }
    }
    __syncthreads();
    const int rg = (tid >> 5) * 4;              // rows rg .. rg + 3, four columns per lane
    auto rows4 = [&](const float* A, const float* X, int ldx, bool shared_x, int n, float* out, int ldo) {
        for (int d = lane * 4; d < n; d += 128) {
            float4 acc[4];
#pragma unroll
            for (int u = 0; u < 4; u++) acc[u] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
            for (int s = 0; s < rg + 4; s++) {  // (T is lower triangular)
                const float4 x = (shared_x || s < nt) ? *reinterpret_cast<const float4*>(X + (size_t)s * ldx + d) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const float a = A[(rg + u) * 33 + s];
                    acc[u].x = fmaf(a, x.x, acc[u].x); acc[u].y = fmaf(a, x.y, acc[u].y); acc[u].z = fmaf(a, x.z, acc[u].z); acc[u].w = fmaf(a, x.w, acc[u].w);
                }
            }
#pragma unroll
            for (int u = 0; u < 4; u++)
                if (rg + u < nt) *reinterpret_cast<float4*>(out + (size_t)(rg + u) * ldo + d) = acc[u];
        }
    };
    rows4(Tw, ks, PI, true, g.dim, g.W + hr * g.dim, g.dim);
    rows4(T, g.V + (size_t)r0 * g.ldv + h * g.vdim, g.ldv, false, g.vdim, g.U0 + hr * g.vdim, g.vdim);
}

template <int MODE, int DM> struct CsSmem {
    static constexpr int PI = DM + 4, ROWS = MODE == CS_DELTA ? 3 : 2;                       // staged row blocks: q, k (, W)
    static constexpr int STAGE = ROWS * CS * PI + CS * CS_COLS + CS * 36 + 3 * CS;          // + U0, M (pitch 36), scalars
    static constexpr size_t BYTES = (size_t)(CS_STAGES * STAGE + 2 * DM * CS_COLS + 4 * CS * CS_COLS + 8 * CS) * 4;
};
template <int DM> constexpr size_t cp_smem_bytes() { return (size_t)(2 * CS * (DM + 4) + 3 * CS * 33) * 4; }
__device__ __forceinline__ void cs_sync(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }
__device__ __forceinline__ void cs_arrive(int id, int threads) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory"); }
// RT rows of A (from `a`, pitch PI) times the state S0 [DM][8] (two halves [DM][4]), the key channels d = sl + SL i dealt to SL neighbouring lanes; their partial sums
// are added in a tree that keeps half of the values per step.  out: [RT][8] of this tile.
template <int DM, int PI, int SL, int RT> __device__ __forceinline__ void cs_rows_state(const float* a, const float* S0, int sl, float* out) {
    float acc[8 * RT];
#pragma unroll
    for (int e = 0; e < 8 * RT; e++) acc[e] = 0.0f;
#pragma unroll
    for (int i = 0; i < DM / SL; i++) {
        const int d = i * SL + sl;
        const float4 x = *reinterpret_cast<const float4*>(S0 + d * 4), y = *reinterpret_cast<const float4*>(S0 + DM * 4 + d * 4);
#pragma unroll
        for (int r = 0; r < RT; r++) {
            const float v = a[r * PI + d];
            acc[8 * r] = fmaf(v, x.x, acc[8 * r]); acc[8 * r + 1] = fmaf(v, x.y, acc[8 * r + 1]);
            acc[8 * r + 2] = fmaf(v, x.z, acc[8 * r + 2]); acc[8 * r + 3] = fmaf(v, x.w, acc[8 * r + 3]);
            acc[8 * r + 4] = fmaf(v, y.x, acc[8 * r + 4]); acc[8 * r + 5] = fmaf(v, y.y, acc[8 * r + 5]);
            acc[8 * r + 6] = fmaf(v, y.z, acc[8 * r + 6]); acc[8 * r + 7] = fmaf(v, y.w, acc[8 * r + 7]);
        }
    }
#pragma unroll
    for (int o = SL / 2, n = 4 * RT; o > 0; o >>= 1, n >>= 1) {
        const bool up = (sl & o) != 0;
#pragma unroll
        for (int e = 0; e < n; e++) {
            const float give = up ? acc[e] : acc[e + n], keep = up ? acc[e + n] : acc[e];
            acc[e] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
    }
    const int e0 = sl * (8 * RT / SL);
#pragma unroll
    for (int e = 0; e < 8 * RT / SL; e++) out[e0 + e] = acc[e];
}
// blockIdx.x: 8 columns of the state (MEM: 7 and the column of ones, whose state is n).
// Two groups of eight warps.  The chain (threads 0 .. 255): W S0, U, the state after the chunk; the others: q S0 and the chunk's outputs, from the state before it, beside
// the chain (the state has two buffers), and the copies of the rows two chunks ahead.  1500 tokens, back to back: delta rule 115 -> 109 us, memory 88 -> 73 us against one group of eight
// warps for all of it with the rows one chunk ahead; bound by the chain's shared-memory loads (delta: W S0, U, the update, 2.3 us per chunk).
template <int MODE, int DM>
__global__ void __launch_bounds__(CS_SCAN_THREADS) lp_chunk_scan_kernel(StepMeta sm, ChunkScan g) {
    prev_grid();
    using L = CsSmem<MODE, DM>;
    constexpr int PI = L::PI, VC = MODE == CS_MEM ? CS_COLS - 1 : CS_COLS, SL = MODE == CS_DELTA ? 16 : 32, RT = MODE == CS_DELTA ? 2 : 4;
    extern __shared__ __align__(16) float cs_sm[];
    float* S0 = cs_sm + CS_STAGES * L::STAGE;   // [2 buffers][2 halves][DM][4]
    float* Y = S0 + 2 * DM * CS_COLS;           // [32][8]: W S0
    float* Z = Y + CS * CS_COLS;                // [32][8]: q S0
    float* U = Z + CS * CS_COLS;                // [32][8]
    float* Us = U + CS * CS_COLS;               // [32][8]: u_s U_s
    float* scl = Us + CS * CS_COLS;             // [2 buffers][4][32]: z, p, u, e^-m
    const int tid = threadIdx.x, lane = tid & 31, h = blockIdx.y, run = blockIdx.z, j0 = blockIdx.x * VC;
    const bool chain = tid < 256;
    const int ct = tid & 255;                   // thread of its group
    const int r0 = sm.run_start[run], r1 = sm.run_start[run + 1], hk = h * g.G / g.H;
    float* rec = reinterpret_cast<float*>(sm.run_rec[run] + g.rec_off);
    float* Sg = rec + (size_t)h * g.dim * g.vdim;
    const int flip = MODE == CS_MEM ? sm.run_flip[run] : 0;                                   // MEM: n and m are read from one copy and written to the other (lp_matrix_memory_kernel)
    float* n0 = rec + (size_t)g.H * g.dim * g.vdim;
    const float* nm = n0 + ((size_t)flip * g.H + h) * g.dim;
    float* ng = n0 + ((size_t)(flip ^ 1) * g.H + h) * g.dim;
    float* mg = n0 + (size_t)2 * g.H * g.dim;                                                 // [2][H]
    auto stage = [&](int c0, int buf) {
        float* q = cs_sm + buf * L::STAGE;
        float* k = q + CS * PI;
        float* w = k + CS * PI;                 // (DELTA)
        float* u0 = q + L::ROWS * CS * PI;
        float* m = u0 + CS * CS_COLS;
        float* s = m + CS * 36;
        const int nt = min(CS, r1 - c0);
        const size_t hr = (size_t)h * g.R + c0;
        if (chain) return;                      // (the chain is the longer way)
        for (int i = ct; i < CS * (DM / 4); i += 256) {
            const int t = i / (DM / 4), d = (i - t * (DM / 4)) * 4;
            const bool in = t < nt && d < g.dim;
            const size_t at = in ? (size_t)(c0 + t) * g.ldq + hk * g.dim + d : 0;
            cp_async16(smem_u32(q + t * PI + d), g.Q + at, in ? 16u : 0u);
            cp_async16(smem_u32(k + t * PI + d), g.K + at, in ? 16u : 0u);
            if (MODE == CS_DELTA) cp_async16(smem_u32(w + t * PI + d), in ? g.W + (hr + t) * g.dim + d : g.W, in ? 16u : 0u);
        }
        {
            const int t = ct >> 3, c = ct & 7, j = j0 + c;
            float* dst = u0 + t * CS_COLS + c;
            if (t >= nt || (c < VC && j >= g.vdim)) *dst = 0.0f;
            else if (c >= VC) *dst = 1.0f;
            else cp_async4(dst, MODE == CS_DELTA ? g.U0 + (hr + t) * g.vdim + j : g.V + (size_t)(c0 + t) * g.ldv + h * g.vdim + j);
            cp_async16(smem_u32(m + t * 36 + c * 4), t < nt ? g.M + (hr + t) * CS + c * 4 : g.M, t < nt ? 16u : 0u);
        }
        if (ct < 3 * CS) {
            const int t = ct & 31, row = min(t, nt - 1);                 // (the last row's scalars stand for what is past the end: F and mu of the chunk, D)
            cp_async4(s + ct, g.sc + (size_t)(ct >> 5) * g.H * g.R + hr + row);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // the chain's threads: state row kr, columns c4 .. c4 + 3 of the block's 8
    const int kr = ct >> 1, half = ct & 1, c4 = half * 4;
    const bool mine = chain && kr < DM;
    float st[4] = {0.f, 0.f, 0.f, 0.f};
    if (mine) {
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const int c = c4 + e, j = j0 + c;
            if (kr < g.dim) st[e] = c >= VC ? nm[kr] : j < g.vdim ? Sg[(size_t)kr * g.vdim + j] : 0.0f;
        }
        *reinterpret_cast<float4*>(S0 + half * DM * 4 + kr * 4) = make_float4(st[0], st[1], st[2], st[3]);
    }
    float m_run = MODE == CS_MEM ? mg[flip * g.H + h] : 0.0f;
    const float dskip = MODE == CS_SSD ? g.skip[h] : 0.0f;
    const float qsc = MODE == CS_MEM ? 1.0f / sqrtf((float)g.dim) : 1.0f;
    // (a chunk's rows are asked for two chunks ahead: one is less than their way from L2 takes)
    stage(r0, 0);
    if (r0 + CS < r1) stage(r0 + CS, 1);
    for (int c0 = r0, buf = 0, st3 = 0; c0 < r1; c0 += CS, buf ^= 1, st3 = st3 == CS_STAGES - 1 ? 0 : st3 + 1) {
        const int nt = min(CS, r1 - c0);
        if (c0 + CS < r1) asm volatile("cp.async.wait_group 1;" ::: "memory");
        else asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();                        // this chunk's rows are here, and both groups are done with the chunk before
        if (c0 + 2 * CS < r1) stage(c0 + 2 * CS, st3 == 0 ? 2 : st3 - 1);
        const float* q = cs_sm + st3 * L::STAGE;
        const float* k = q + CS * PI;
        const float* w = k + CS * PI;
        const float* u0 = q + L::ROWS * CS * PI;
        const float* M = u0 + CS * CS_COLS;
        const float* s = M + CS * 36;
        const float* Sb = S0 + buf * DM * CS_COLS;
        float* sc = scl + buf * 4 * CS;
        const int t = ct >> 3, c = ct & 7;
        float D;
        if (MODE == CS_MEM) {
            const float fe = s[CS - 1], m_end = fmaxf(m_run + fe, s[3 * CS - 1]);
            D = expf(m_run + fe - m_end);
            if (!chain && ct < CS) {
                const float f = s[ct], mt = fmaxf(m_run + f, s[2 * CS + ct]);
                sc[ct] = expf(m_run + f - mt) * qsc;
                sc[CS + ct] = expf(s[2 * CS + ct] - mt);
                sc[3 * CS + ct] = expf(-mt);
            }
            if (chain) Us[t * CS_COLS + c] = (t < nt ? expf(s[CS + t] - m_end) : 0.0f) * u0[t * CS_COLS + c];
            m_run = m_end;
        } else {
            D = s[3 * CS - 1];
            if (MODE == CS_SSD && chain) Us[t * CS_COLS + c] = (t < nt ? s[CS + t] : 0.0f) * u0[t * CS_COLS + c];
        }
        if (chain) {
            if (MODE == CS_DELTA) {
                cs_rows_state<DM, PI, SL, RT>(w + (ct / SL) * RT * PI, Sb, ct % SL, Y + (ct / SL) * RT * CS_COLS);
                cs_sync(1, 256);
                const float ut = u0[t * CS_COLS + c] - Y[t * CS_COLS + c];
                U[t * CS_COLS + c] = ut;
                Us[t * CS_COLS + c] = (t < nt ? s[CS + t] : 0.0f) * ut;
                cs_arrive(2, 512);              // (U is there for the outputs)
            }
            cs_sync(1, 256);
            if (mine) {
#pragma unroll
                for (int e = 0; e < 4; e++) st[e] *= D;
#pragma unroll 8
                for (int i = 0; i < CS; i++) {
                    const float kv = k[i * PI + kr];
                    const float4 u = *reinterpret_cast<const float4*>(Us + i * CS_COLS + c4);
                    st[0] = fmaf(kv, u.x, st[0]); st[1] = fmaf(kv, u.y, st[1]); st[2] = fmaf(kv, u.z, st[2]); st[3] = fmaf(kv, u.w, st[3]);
                }
                *reinterpret_cast<float4*>(S0 + (buf ^ 1) * DM * CS_COLS + half * DM * 4 + kr * 4) = make_float4(st[0], st[1], st[2], st[3]);
            }
        } else {
            cs_rows_state<DM, PI, SL, RT>(q + (ct / SL) * RT * PI, Sb, ct % SL, Z + (ct / SL) * RT * CS_COLS);
            if (MODE == CS_DELTA) cs_sync(2, 512);
            else cs_sync(2, 256);
            const float* Uc = MODE == CS_DELTA ? U : u0;
            float a0 = 0.0f, a1 = 0.0f;         // output of (t, c)
#pragma unroll
            for (int i = 0; i < CS; i += 4) {
                const float4 m = *reinterpret_cast<const float4*>(M + t * 36 + i);
                a0 = fmaf(m.x, Uc[i * CS_COLS + c], a0);
                a1 = fmaf(m.y, Uc[(i + 1) * CS_COLS + c], a1);
                a0 = fmaf(m.z, Uc[(i + 2) * CS_COLS + c], a0);
                a1 = fmaf(m.w, Uc[(i + 3) * CS_COLS + c], a1);
            }
            const float z = Z[t * CS_COLS + c], zt = MODE == CS_MEM ? sc[t] : s[t];
            float o = MODE == CS_MEM ? fmaf(zt, z, sc[CS + t] * (a0 + a1)) : fmaf(zt, z, a0 + a1);
            if (MODE == CS_SSD) o = fmaf(dskip, Uc[t * CS_COLS + c], o);
            if (MODE == CS_MEM) {
                const float nq = __shfl_sync(0xffffffffu, o, lane | 7);
                o /= fmaxf(fabsf(nq), sc[3 * CS + t]) + 1e-6f;
            }
            if (t < nt && c < VC && j0 + c < g.vdim) g.O[(size_t)(c0 + t) * g.ldo + h * g.vdim + j0 + c] = o;
        }
    }
    if (mine && kr < g.dim) {
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const int c = c4 + e, j = j0 + c;
            if (c >= VC) {
                if (blockIdx.x == 0) ng[kr] = st[e];
            } else if (j < g.vdim) Sg[(size_t)kr * g.vdim + j] = st[e];
        }
    }
    if (MODE == CS_MEM && blockIdx.x == 0 && tid == 0) mg[(flip ^ 1) * g.H + h] = m_run;
}
