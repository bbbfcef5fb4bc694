// lp_tile_attn.cuh — attention of prompt rows on the 5th-generation tensor cores (bf16 mode).  Included by layerprog.cu inside its anonymous
// namespace.
//
// The hpg = H / G heads of K/V head g meet the same cached rows, so their (token, head) pairs are ONE list of query rows, pair f = (token f / hpg,
// head g hpg + f % hpg); a CTA takes 128 neighbours of the list against tiles of 64 keys:
//   S = Q K^T (M = 128, N = 64) into one of two TMEM buffers; a thread per row reads its 64 scores, masks, caps, keeps the running maximum, writes
//   the probabilities as bf16 into a swizzled tile, and O += P V (M = 128, N = DVP) accumulates in TMEM.  O is rescaled only when a row's
//   maximum has grown by more than 2^8 since the last time (probabilities up to 2^8 lose nothing in bf16; rescaling at every growth: 45 -> 53 us for 2048 queries of
//   16 latent heads); the division comes last.
// Both B operands have the contracted index contiguous, so the cached f32 rows are rounded to bf16 once per layer (lp_keys16_kernel): K16[g]
// [key][DKP] as they are stored (their factors, if they have any, go into F[g][key] and meet the f32 score, as in the mma.sync kernel: 5 us of 70 for 2048 queries of
// 16 heads), and the transpose Vt16[g][channel][key], the keys of every run from the first one that a query of the step sees, in tiles of 64 whose
// missing keys are zeros; TMA brings the tiles.  Roles: 4 softmax warps, a loader thread, an MMA thread; two CTAs share an SM (112 KB
// of shared memory and 256 TMEM columns each), so one CTA's products run under the other's exponentials.
// What bounded the mma.sync kernels (each block converting its own tiles, one tile after the other): 12.5 us per 64-key tile of
// lp_window_attn_tile_kernel, 5 us of lp_row_tile_kernel, where a tile's products need 0.3 us of this pipe and its exponentials 0.5.  Measured:
// 2048 queries, 16 heads over 4, 128 channels, causal 158 -> 53 us (330 TFLOP/s) + 9 us for the copies; prompts of 777, 130 and 41 tokens, 8
// heads over 2: 163 -> 29 + 12 us.  Now bounded by the row's chain of TMEM load, maximum, exponentials and store, two tiles per SM in flight.
// Every wait is bounded and reports through *err.
#pragma once

constexpr int KA_Q = 128, KA_K = 64;
// The keys of a run that its queries of this step see, in tiles of 64: nA tiles from position 0 (kept first tokens), then tiles from `start` on
// (past the kept ones)
__host__ __device__ inline void keys16(const AttnGeom& a, int p0, int len, int& start, int& nA, int& tiles) {
    const int lo = a.chunk ? (p0 / a.window) * a.window : (p0 + 1 > a.window ? p0 + 1 - a.window : 0);
    const int kept = a.keep_first < p0 + len ? a.keep_first : p0 + len;
    nA = (kept + KA_K - 1) / KA_K;
    start = (lo & ~(KA_K - 1)) > nA * KA_K ? lo & ~(KA_K - 1) : nA * KA_K;
    tiles = nA + (p0 + len > start ? (p0 + len - start + KA_K - 1) / KA_K : 0);
}
__device__ __forceinline__ int keys16_tiles(const StepMeta& sm, const AttnGeom& a, int run) {
    int start, nA, tiles;
    keys16(a, sm.run_pos0[run], sm.run_start[run + 1] - sm.run_start[run], start, nA, tiles);
    return tiles;
}

// blockIdx.x: tile of all runs' tiles, blockIdx.y: K/V head.  cols: 64 x all tiles.
template <int DKP, int DVP>
__global__ void __launch_bounds__(256) lp_keys16_kernel(StepMeta sm, AttnGeom a, int n_runs, int cols, bf16* __restrict__ K16, bf16* __restrict__ Vt16,
                                                        float* __restrict__ F) {
    prev_grid();
    __shared__ bf16 sv[DVP][KA_K + 2];
    const int lane = threadIdx.x & 31, g = blockIdx.y, tile = blockIdx.x;
    int run = 0, base = 0;
    for (int r0 = 0; r0 < n_runs; r0 += 32) {        // the run of this tile (every warp for itself)
        int n = r0 + lane < n_runs ? keys16_tiles(sm, a, r0 + lane) : 0, incl = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int up = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += up;
        }
        const unsigned past = __ballot_sync(0xffffffffu, base + incl > tile);
        if (past) {
            const int l = __ffs(past) - 1;
            run = r0 + l;
            base += __shfl_sync(0xffffffffu, incl - n, l);
            break;
        }
        base += __shfl_sync(0xffffffffu, incl, 31);
    }
    const int p0 = sm.run_pos0[run], len = sm.run_start[run + 1] - sm.run_start[run];
    int start, nA, tiles;
    keys16(a, p0, len, start, nA, tiles);
    const int u = tile - base, j0 = u < nA ? u * KA_K : start + (u - nA) * KA_K, end = p0 + len;
    const float* kc = reinterpret_cast<const float*>(sm.run_kv[run] + a.kv_off);
    const float* vc = a.v_in_k ? kc : kc + (size_t)a.cap * a.G * a.dim;
    const float* kinv = a.k_inv ? kc + (size_t)a.cap * a.G * a.dim + g : nullptr;
    const int ldk = a.G * a.dim, ldv = a.v_in_k ? ldk : a.G * a.vdim, vhead = g * (a.v_in_k ? a.dim : a.vdim);
#pragma unroll 4
    for (int i = threadIdx.x; i < KA_K * (DKP / 4); i += 256) {
        const int key = i / (DKP / 4), d = (i - key * (DKP / 4)) * 4, j = j0 + key;
        float4 v = (j < end && d < a.dim) ? *reinterpret_cast<const float4*>(kc + (size_t)j * ldk + g * a.dim + d) : make_float4(0.f, 0.f, 0.f, 0.f);
        *reinterpret_cast<uint2*>(K16 + ((size_t)g * cols + (size_t)tile * KA_K + key) * DKP + d) = make_uint2(pack_bf2(v.x, v.y), pack_bf2(v.z, v.w));
    }
    if (kinv && threadIdx.x < KA_K) F[(size_t)g * cols + (size_t)tile * KA_K + threadIdx.x] = j0 + (int)threadIdx.x < end ? kinv[(size_t)(j0 + threadIdx.x) * a.G] : 0.0f;
#pragma unroll 4
    for (int i = threadIdx.x; i < KA_K * (DVP / 4); i += 256) {
        const int key = i / (DVP / 4), c = (i - key * (DVP / 4)) * 4, j = j0 + key;
        const float4 v = (j < end && c < a.vdim) ? *reinterpret_cast<const float4*>(vc + (size_t)j * ldv + vhead + c) : make_float4(0.f, 0.f, 0.f, 0.f);
        sv[c][key] = __float2bfloat16_rn(v.x);
        sv[c + 1][key] = __float2bfloat16_rn(v.y);
        sv[c + 2][key] = __float2bfloat16_rn(v.z);
        sv[c + 3][key] = __float2bfloat16_rn(v.w);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < DVP * (KA_K / 2); i += 256) {
        const int c = i / (KA_K / 2), k = (i - c * (KA_K / 2)) * 2;
        *reinterpret_cast<uint32_t*>(Vt16 + ((size_t)g * DVP + c) * cols + (size_t)tile * KA_K + k) = *reinterpret_cast<const uint32_t*>(&sv[c][k]);
    }
}

template <int DKP, int DVP> struct KaSmem {
    static constexpr int Q = KA_Q * DKP * 2, K = KA_K * DKP * 2, V = DVP * KA_K * 2, P = KA_Q * KA_K * 2;
    static constexpr int K_AT = Q, V_AT = K_AT + 2 * K, P_AT = V_AT + 2 * V, BAR_AT = P_AT + P, BYTES = BAR_AT + 192;
};
__device__ __forceinline__ uint32_t sw128(int r, int c) {      // 16-byte chunk c of 128-byte row r of a swizzled tile
    return (uint32_t)(r >> 3) * 1024u + (uint32_t)(r & 7) * 128u + (uint32_t)((c ^ (r & 7)) << 4);
}
__device__ __forceinline__ void tc_st32(uint32_t taddr, const uint32_t* v) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31};" ::"r"(v[0]), "r"(v[1]), "r"(v[2]),
        "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]),
        "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]),
        "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31]), "r"(taddr)
        : "memory");
}
// `steps` x 16 of the contracted index, 64 per slab; slabs `sa` / `sb` (>> 4) apart
__device__ __forceinline__ void ka_mma(uint32_t acc, uint64_t da, uint64_t db, uint32_t idesc, int slabs, uint32_t sa, uint32_t sb, bool first) {
    for (int h = 0; h < slabs; h++)
#pragma unroll
        for (int kk = 0; kk < 4; kk++)
            asm volatile(
                "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(acc),
                "l"(da + (uint64_t)(h * sa + 2 * kk)), "l"(db + (uint64_t)(h * sb + 2 * kk)), "r"(idesc), "r"((!first || h > 0 || kk > 0) ? 1u : 0u)
                : "memory");
}

// blockIdx.x = K/V head + G * (blocks from the last queries on), blockIdx.y = run.  out: rows out_ld apart.
template <int DKP, int DVP>
__global__ void __launch_bounds__(192, 2) lp_tile_attn_kernel(const __grid_constant__ CUtensorMap kmap, const __grid_constant__ CUtensorMap vmap, StepMeta sm, AttnGeom a,
                                                              const float* __restrict__ qbuf, const float* __restrict__ P, int ldp, const float* __restrict__ F, int cols,
                                                              bf16* __restrict__ out, int out_ld, float out_scale, int* err) {
    prev_grid();
    extern __shared__ __align__(1024) uint8_t ka_smem[];
    using SM = KaSmem<DKP, DVP>;
    const int run = blockIdx.y, g = blockIdx.x % a.G, bx = blockIdx.x / a.G, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int r0 = sm.run_start[run], len = sm.run_start[run + 1] - r0, p0 = sm.run_pos0[run];
    const int hpg = a.H / a.G, rows = len * hpg, nb = (rows + KA_Q - 1) / KA_Q;
    if (bx >= nb) return;
    const uint32_t base = smem_u32(ka_smem);
    if (base & 1023u) {             // the swizzle is on absolute address bits (there is no static shared memory in front)
        if (tid == 0 && err) atomicExch(err, 9);
        return;
    }
    const uint32_t bars = base + SM::BAR_AT, s_tmem = bars + 128;
    const uint32_t k_full = bars, k_empty = bars + 16, v_full = bars + 32, v_empty = bars + 48, s_full = bars + 64, s_empty = bars + 80, q_full = bars + 96, p_full = bars + 104,
                   pv_done = bars + 112;
    if (tid == 0) {
        for (int i = 0; i < 2; i++) {
            for (uint32_t b : {k_full, k_empty, v_full, v_empty, s_full}) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(b + 8u * i) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 4;" ::"r"(s_empty + 8u * i) : "memory");
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 4;" ::"r"(q_full) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 4;" ::"r"(p_full) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(pv_done) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 5) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s_tmem), "r"(256) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    // this run's place among the tiles, and the tiles that the block's queries see
    int before = 0;
    for (int r = lane; r < run; r += 32) before += keys16_tiles(sm, a, r);
    before = __reduce_add_sync(0xffffffffu, before);
    int start, nA, all;
    keys16(a, p0, len, start, nA, all);
    const int f0 = (nb - 1 - bx) * KA_Q, first = p0 + f0 / hpg, last = p0 + min(f0 + KA_Q - 1, rows - 1) / hpg;
    const int t_lo = max(0, (attn_lo(a, first) - start) / KA_K), n_tiles = nA + (last >= start ? (last - start) / KA_K + 1 - t_lo : 0);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    uint32_t tmem;
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(tmem) : "r"(s_tmem));
    const uint32_t tO = tmem + 128;
    bool alive = true;
    // tile t of the block: its place among the run's tiles, its first position
    auto place = [&](int t) { return t < nA ? t : t + t_lo; };
    auto position = [&](int t) { return t < nA ? t * KA_K : start + (t - nA + t_lo) * KA_K; };
    if (warp == 4) {
        int asked_k = 0, asked_v = 0;
        for (int t = 0; t < n_tiles; t++) {
            const uint32_t b = t & 1, ph = ((t >> 1) & 1) ^ 1;
            const int col = (before + place(t)) * KA_K;
            tc_wait(k_empty + 8u * b, ph, alive, err, 21);
            alive = __all_sync(0xffffffffu, alive);
            if (!alive) break;
            if (tc_elect()) {
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(k_full + 8u * b), "r"((uint32_t)SM::K) : "memory");
                asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(base + SM::K_AT + b * SM::K),
                             "l"(&kmap), "r"(0), "r"(g * cols + col), "r"(0), "r"(k_full + 8u * b)
                             : "memory");
            }
            __syncwarp();
            asked_k = t + 1;
            tc_wait(v_empty + 8u * b, ph, alive, err, 22);
            alive = __all_sync(0xffffffffu, alive);
            if (!alive) break;
            if (tc_elect()) {
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(v_full + 8u * b), "r"((uint32_t)SM::V) : "memory");
                asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(base + SM::V_AT + b * SM::V),
                             "l"(&vmap), "r"(col), "r"(g * DVP), "r"(v_full + 8u * b)
                             : "memory");
            }
            __syncwarp();
            asked_v = t + 1;
        }
        if (!alive) {               // gave up: what has been asked for lands first (bounded)
            auto land = [&](uint32_t full, int asked) {
                ring_in_flight<2>(asked, [&](int stage, unsigned parity) {
                    bool w = true;
                    tc_wait(full + 8u * stage, parity, w, nullptr, 0);
                });
            };
            land(k_full, asked_k);
            land(v_full, asked_v);
        }
    } else if (warp == 5) {
        const uint32_t id_s = tc_idesc(KA_Q, KA_K), id_o = tc_idesc(KA_Q, DVP);
        const uint64_t dq = tc_desc(base), dp = tc_desc(base + SM::P_AT);
        auto scores = [&](int t) {
            const uint32_t b = t & 1, ph = (t >> 1) & 1;
            tc_wait(k_full + 8u * b, ph, alive, err, 23);
            tc_wait(s_empty + 8u * b, ph ^ 1, alive, err, 24);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            alive = __all_sync(0xffffffffu, alive);
            const bool lead = tc_elect();
            if (lead && alive) ka_mma(tmem + b * KA_K, dq, tc_desc(base + SM::K_AT + b * SM::K), id_s, DKP / 64, KA_Q * 8, KA_K * 8, true);
            if (lead) {
                tc_commit(k_empty + 8u * b);
                tc_commit(s_full + 8u * b);
            }
            __syncwarp();
        };
        tc_wait(q_full, 0, alive, err, 25);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        scores(0);
        for (int t = 0; t < n_tiles; t++) {
            const uint32_t b = t & 1, ph = (t >> 1) & 1;
            if (t + 1 < n_tiles) scores(t + 1);
            tc_wait(v_full + 8u * b, ph, alive, err, 26);
            tc_wait(p_full, t & 1, alive, err, 27);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            alive = __all_sync(0xffffffffu, alive);
            const bool lead = tc_elect();
            if (lead && alive) ka_mma(tO, dp, tc_desc(base + SM::V_AT + b * SM::V), id_o, 1, 0, 0, t == 0);
            if (lead) {
                tc_commit(v_empty + 8u * b);
                tc_commit(pv_done);
            }
            __syncwarp();
        }
    } else {
        const int f = min(f0 + tid, rows - 1), tok = f / hpg, h = g * hpg + f - tok * hpg, i = p0 + tok;
        // the query row -> bf16, swizzled
        const float* q = qbuf + ((size_t)(r0 + tok) * a.H + h) * a.dim;
#pragma unroll 4
        for (int c = 0; c < DKP / 8; c++) {
            float4 u = make_float4(0.f, 0.f, 0.f, 0.f), v = u;
            if (c * 8 < a.dim) {          // (dim is a multiple of 16)
                u = *reinterpret_cast<const float4*>(q + c * 8);
                v = *reinterpret_cast<const float4*>(q + c * 8 + 4);
            }
            *reinterpret_cast<uint4*>(ka_smem + (c >> 3) * (KA_Q * 128) + sw128(tid, c & 7)) = make_uint4(pack_bf2(u.x, u.y), pack_bf2(u.z, u.w), pack_bf2(v.x, v.y), pack_bf2(v.z, v.w));
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) tc_arrive(q_full);
        const float L2E = 1.4426950408889634f;
        const bool capped = a.softcap > 0.0f;
        const float sl = a.scale * L2E, cap_in = capped ? a.scale / a.softcap : 0.0f, cap_out = a.softcap * L2E, slope = attn_slope(a, h) * L2E;
        const int lo_i = attn_lo(a, i);
        float m = -INFINITY, l = 0.0f;
        {   // the extra term of the denominator
            float c;
            if (attn_sink(a, h, &c)) { m = c * L2E; l = 1.0f; }
        }
        const uint32_t lanes = (uint32_t)(warp * 32) << 16;
        const float* Fg = F + (size_t)g * cols + (size_t)before * KA_K;      // the keys' factors
        for (int t = 0; t < n_tiles; t++) {
            const uint32_t b = t & 1;
            const int j0 = position(t);
            if (a.k_inv && lane < 2) asm volatile("prefetch.global.L1 [%0];" ::"l"(Fg + place(t) * KA_K + 32 * lane));
            uint32_t raw[KA_K];
            float s[KA_K];
            tc_wait(s_full + 8u * b, (t >> 1) & 1, alive, err, 28);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            tc_ld32(raw, tmem + lanes + b * KA_K);
            tc_ld32(raw + 32, tmem + lanes + b * KA_K + 32);
#pragma unroll
            for (int e = 0; e < KA_K; e++) s[e] = __uint_as_float(raw[e]);
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) tc_arrive(s_empty + 8u * b);
            if (a.k_inv) {
                const float4* f4 = reinterpret_cast<const float4*>(Fg + place(t) * KA_K);
#pragma unroll
                for (int e = 0; e < KA_K; e += 4) {
                    const float4 f = f4[e / 4];
                    s[e] *= f.x; s[e + 1] *= f.y; s[e + 2] *= f.z; s[e + 3] *= f.w;
                }
            }
            if (capped) {
                float big = 0.0f;
#pragma unroll
                for (int e = 0; e < KA_K; e++) {
                    s[e] *= cap_in;
                    big = fmaxf(big, fabsf(s[e]));
                }
                if (!__any_sync(0xffffffffu, big >= SOFT_CAP_SMALL)) {
#pragma unroll
                    for (int e = 0; e < KA_K; e++) s[e] = cap_out * tanh_small(s[e]);
                } else {
#pragma unroll
                    for (int e = 0; e < KA_K; e++) s[e] = fabsf(s[e]) < SOFT_CAP_SMALL ? cap_out * tanh_small(s[e]) : soft_cap_exp(s[e], 2.0f * L2E, cap_out);
                }
            } else {
#pragma unroll
                for (int e = 0; e < KA_K; e++) s[e] *= sl;
            }
            if (slope != 0.0f) {
                const float d = slope * (float)(i - j0);
#pragma unroll
                for (int e = 0; e < KA_K; e++) s[e] = s[e] - (d - slope * (float)e);
            }
            const bool whole = j0 + KA_K - 1 <= i && j0 >= lo_i;
            if (!__all_sync(0xffffffffu, whole)) {
                const int hi = i - j0, lo = lo_i - j0, kf = a.keep_first - j0;
#pragma unroll
                for (int e = 0; e < KA_K; e++) s[e] = (e <= hi && (e >= lo || e < kf)) ? s[e] : -INFINITY;
            }
            float x0 = s[0], x1 = s[1], x2 = s[2], x3 = s[3];
#pragma unroll
            for (int e = 4; e < KA_K; e += 4) {
                x0 = fmaxf(x0, s[e]);
                x1 = fmaxf(x1, s[e + 1]);
                x2 = fmaxf(x2, s[e + 2]);
                x3 = fmaxf(x3, s[e + 3]);
            }
            const float mx = fmaxf(fmaxf(x0, x1), fmaxf(x2, x3));
            if (t > 0) {      // the products of the tile before are done: P is free, O may be rescaled
                tc_wait(pv_done, (t - 1) & 1, alive, err, 29);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            }
            if (__any_sync(0xffffffffu, mx > m + 8.0f)) {
                const float mn = fmaxf(m, mx), c = m == -INFINITY ? 0.0f : ex2_fast(m - mn);
                l *= c;
                m = mn;
                if (t > 0) {
#pragma unroll 1
                    for (int n = 0; n < DVP; n += 32) {
                        uint32_t o[32];
                        tc_ld32(o, tO + lanes + n);
#pragma unroll
                        for (int e = 0; e < 32; e++) o[e] = __float_as_uint(__uint_as_float(o[e]) * c);
                        tc_st32(tO + lanes + n, o);
                    }
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                }
            }
            const float ref = m == -INFINITY ? 0.0f : m;       // (a row without a visible key yet: all weights 0)
            float l0 = 0.0f, l1 = 0.0f;
#pragma unroll
            for (int c = 0; c < KA_K / 8; c++) {
                uint32_t w[4];
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const float u = ex2_fast(s[8 * c + 2 * e] - ref), v = ex2_fast(s[8 * c + 2 * e + 1] - ref);
                    l0 += u;
                    l1 += v;
                    w[e] = pack_bf2(u, v);
                }
                *reinterpret_cast<uint4*>(ka_smem + SM::P_AT + sw128(tid, c)) = make_uint4(w[0], w[1], w[2], w[3]);
            }
            l += l0 + l1;
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) tc_arrive(p_full);
        }
        tc_wait(pv_done, (n_tiles - 1) & 1, alive, err, 29);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const float inv = out_scale / l;
        const size_t r = (size_t)(r0 + tok);
        const float* gate = P + r * ldp + a.g_off;
        bf16* o_row = out + r * out_ld + h * a.vdim;
        const bool mine = f0 + tid < rows, v16 = ((uintptr_t)o_row & 15) == 0;
#pragma unroll 1
        for (int n = 0; n < DVP; n += 32) {
            if (n >= a.vdim) break;
            uint32_t o[32];
            tc_ld32(o, tO + lanes + n);
            if (mine) {
#pragma unroll
                for (int c = 0; c < 32; c += 8) {
                    if (n + c >= a.vdim) break;         // (vdim is a multiple of 8)
                    uint32_t w[4];
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        const int ch = n + c + 2 * e;
                        float u = __uint_as_float(o[c + 2 * e]) * inv, v = __uint_as_float(o[c + 2 * e + 1]) * inv;
                        if (a.vrot) attn_turn_back(a.vrot + r * a.vdim, a.vdim / 2, ch >> 1, u, v);
                        w[e] = pack_bf2(u * attn_gate(a, gate, h, ch), v * attn_gate(a, gate, h, ch + 1));
                    }
                    if (v16) *reinterpret_cast<uint4*>(o_row + n + c) = make_uint4(w[0], w[1], w[2], w[3]);
                    else {
#pragma unroll
                        for (int e = 0; e < 4; e++) *reinterpret_cast<uint32_t*>(o_row + n + c + 2 * e) = w[e];
                    }
                }
            }
            __syncwarp();
        }
    }
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 5) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256) : "memory");
}
