// gemm_tc.cuh — 16-bit products of many rows on the 5th-generation tensor cores.  Included by layerprog.cu (bf16) and engine.cu (fp16), each
// inside a namespace that has defined: next_grid / wait_grid (programmatic launches; empty where there are none), tc_t (the operand type), TC_BF16 (whether it is bfloat16), TC_W_WAITS (whether the kernel before writes the weight rows), the epilogues EPI_STORE, EPI_ADD, ... with
// epi_is_glu, epi_is_act, seg_rows<T, EPI>, epi_store<T, EPI> and glu_fast<EPI>, and from_f<T>.
//
// Y[t][n] = epi(alpha * sum_k X[t][k] W[n][k] + bias[n]).  A tile is TC_M = 128 weight rows (the M of tcgen05.mma) by TN tokens (its N); its
// f32 sums live in TMEM.  A stage holds KH slabs of 64 elements of K (128 bytes = one row of a SWIZZLE_128B atom): one thread asks the TMA
// unit for the stage's weight rows, a second one for its token rows, ONE copy each; an mbarrier ring of TcRing<TN>::N stages runs between
// them and the one thread that issues the MMAs, whose tcgen05.commit hands a stage back.  Rows and columns past the end arrive as zeros
// (a zero-filled box counts its whole size), so ragged shapes need no code in the loop.
//
// What bounds the product: a 128 x 256 tile needs 512 clocks of tensor pipe per 64 elements of K and 48 KB of operands, which arrive at
// about 64 bytes per clock and SM (750 clocks measured per such step); narrower tiles move more bytes per product and exist for products
// that would leave SMs without a tile.  A single thread that issues three copies per 64 elements needs 640 to 720 clocks for them whatever
// TN is, hence two issuing threads, one copy each, and KH = 2 for the narrow tiles.  Measured (f32 results, L2 warm), against the kernel before
// (128 threads that copy with cp.async, one tile per CTA, no split): 2048 x 2048 x 2048 (tokens x rows x K) 37 -> 21 us, the gated 2048 x 16384
// x 2048 195 -> 112 us (1220 TFLOP/s), 32 x 2048 x 2048 20 -> 8.3 us.
//   lp_gemm_tc_kernel        persistent: a CTA per SM walks tiles; two accumulators in TMEM, so the epilogue of a tile runs under the
//                            next tile's products, and the ring never drains between tiles.
//                            With PAIR two CTAs share a tile of 256 x 256: gate and up of an 8B layer, 2048 rows, 357 -> 327 us (1.47 PFLOP/s, 0.91 of
//                            cuBLAS's burst rate), its output and down products 132 -> 118 on average.
//   lp_gemm_tc_rows_kernel   few token rows as M, below.
//   lp_gemm_tc_split_kernel  few tiles: S = 1, 2, 4 or 8 CTAs of a cluster share a tile's K steps; each leaves its partial sums in its own
//                            shared memory and every CTA adds one S-th of the tokens out of all of them (distributed shared memory, always
//                            in CTA order).
// Groups: without `seg`, group z of a batched product reads and writes its own columns (heads); with `seg`, group z has rows [seg[2z],
// seg[2z] + seg[2z + 1]) of X and Y, known on the device only, and its own weight matrix (experts).
// Gated epilogues: the tile's 128 weight rows are 64 units' gate rows and the same units' up rows.
// Every mbarrier wait is bounded: a wait that gives up sets *err, and the CTA goes to its end without further waits.
#pragma once

constexpr int TC_M = 128, TC_K = 64;
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
// K-major SWIZZLE_128B shared-memory matrix descriptor: start >> 4, LBO (unused) = 1, SBO = 1024 bytes between 8-row groups,
// version 1 at bit 46, layout SWIZZLE_128B = 2 at bit 61
__device__ __forceinline__ uint64_t tc_desc(uint32_t saddr) {
    return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
// instruction descriptor: D = f32 (bits 4-5 = 1), A = B = bf16 (1 at bits 7 and 10) or fp16 (0), both K-major, N >> 3 at bit 17, M >> 4 at bit 24
__device__ __forceinline__ uint32_t tc_idesc(int M, int N) {
    return (1u << 4) | (TC_BF16 ? (1u << 7) | (1u << 10) : 0u) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}
__device__ __forceinline__ bool tc_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok)
                 : "r"(bar), "r"(parity)
                 : "memory");
    return ok != 0;
}
// bounded wait; `alive` goes false on the first timeout and every later wait of the thread returns at once
__device__ __forceinline__ void tc_wait(uint32_t bar, uint32_t parity, bool& alive, int* err, int code) {
    if (!alive || tc_try(bar, parity)) return;
    const long long t0 = clock64();
    while (!tc_try(bar, parity)) {
        if (clock64() - t0 > 2000000000LL) {
            alive = false;
            if (err) atomicExch(err, code);
            return;
        }
    }
}
// One lane of a converged warp.  The warps that issue copies and MMAs run their loops whole and elect a lane at the issue: the operands are uniform registers, and
// with a branch on the lane around the loop each of them was moved there by itself (an MMA every 45 clocks at best, whatever its size; 14 like this).
__device__ __forceinline__ bool tc_elect() {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok));
    return ok != 0;
}
// Pairs (cta_group::2): the barrier at `bar` of the cluster's CTA 0
__device__ __forceinline__ uint32_t tc_leader(uint32_t bar) {
    uint32_t p;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(p) : "r"(bar));
    return p;
}
__device__ __forceinline__ uint32_t tc_cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void tc_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void tc_arrive_leader(uint32_t bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(tc_leader(bar)) : "memory");
}
__device__ __forceinline__ void tc_commit_pair(uint32_t bar) {      // the barrier at this place in both CTAs
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"((uint16_t)3) : "memory");
}
// into this CTA's shared memory, counted by the leader's barrier
__device__ __forceinline__ void tc_tma_pair(uint32_t dst, const CUtensorMap* map, int k, int row, int slab, int z, uint32_t leader_bar) {
    asm volatile("cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, %3, %4, %5, %6}], [%7];" ::"r"(dst), "l"(map),
                 "r"(k), "r"(row), "r"(0), "r"(slab), "r"(z), "r"(leader_bar)
                 : "memory");
}
__device__ __forceinline__ void tc_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ void tc_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tc_tma(uint32_t dst, const CUtensorMap* map, int k, int row, int slab, int z, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, %6}], [%7];" ::"r"(dst), "l"(map),
                 "r"(k), "r"(row), "r"(0), "r"(slab), "r"(z), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, uint32_t bytes) {   // bytes = 16, or 0 for a zero chunk
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
// 32 columns of this warp's 32 TMEM lanes
__device__ __forceinline__ void tc_ld32(uint32_t* v, uint32_t taddr) {
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

// the ring: 192 KB of the 227; a stage = KH slabs of 128 weight rows, then KH slabs of TN token rows
template <int TN> struct TcRing {
    static constexpr int KH = TN == 256 ? 1 : 2, W_BYTES = KH * TC_M * 128, X_BYTES = KH * TN * 128, STAGE = W_BYTES + X_BYTES, N = 196608 / STAGE, K = KH * TC_K;
};
// ... of a pair of CTAs: each has its 128 weight rows and half of the 256 token rows
struct TcPairRing {
    static constexpr int W_BYTES = TC_M * 128, X_BYTES = 128 * 128, STAGE = W_BYTES + X_BYTES, N = 196608 / STAGE, K = TC_K;
};
constexpr int TC_EX_BYTES = 32768;      // gated epilogue of the persistent kernel, for each half of its warps: exchanged sums [2][16][64] f32, units [2][32][64] of tc_t
template <int TN, bool PERSISTENT> constexpr size_t tc_smem_bytes(bool glu) {
    return (size_t)TcRing<TN>::N * TcRing<TN>::STAGE + (PERSISTENT && glu ? TC_EX_BYTES : 0) + 1024;
}

struct TcArgs {
    void* Y;
    int ldy, R, N, K;       // seg: R unused, the rows are the group's
    float alpha;
    int* err;
    const int* seg;
    int groups, x_z;        // x_z: 1 when the groups have columns of their own in X
    size_t yz;              // elements between the groups' outputs (without seg)
    const float* bias;
    float2 act;
    int splits, slabs;      // slabs: 1 when the maps have K / 64 as a dimension (K % 64 == 0), 0: one copy per slab
};
enum { TC_EPI_WARPS = 8, TC_LOAD_W = 8, TC_LOAD_X = 9, TC_MMA = 10, TC_THREADS = 352 };

struct TcTile {
    int z, m, row0, t0, rows;     // group, weight-row tile, first row of the group, first token of the tile in the group, rows of the group
};
// the CTA's way through the tiles, token tile fastest; every role walks it by itself
template <int TN> struct TcWalk {
    int z = 0, base = 0;
    __device__ __forceinline__ bool find(const TcArgs& a, int n_mt, int item, TcTile& t) {
        for (; z < a.groups; z++) {
            t.rows = a.seg ? a.seg[2 * z + 1] : a.R;
            const int nt = (t.rows + TN - 1) / TN, per = nt * n_mt;
            if (item - base < per) {
                t.z = z;
                t.row0 = a.seg ? a.seg[2 * z] : 0;
                const int i = item - base;
                t.m = i / nt;
                t.t0 = (i - t.m * nt) * TN;
                return true;
            }
            base += per;
        }
        return false;
    }
};

template <bool PAIR = false>
__device__ __forceinline__ void tc_setup(uint32_t tid, uint32_t warp, uint32_t bar, int stages, uint32_t* s_tmem, int n_acc, uint32_t cols) {
    if (tid == 0) {
        for (int i = 0; i < stages; i++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 2;" ::"r"(bar + 8u * i) : "memory");                                            // full: both loaders
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar + 8u * (stages + i)) : "memory");                                 // empty
        }
        for (int i = 0; i < n_acc; i++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar + 8u * (2 * stages + i)) : "memory");                             // accumulator done
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar + 8u * (2 * stages + n_acc + i)), "r"((uint32_t)(PAIR ? 2 * TC_EPI_WARPS : TC_EPI_WARPS)) : "memory");   // accumulator read (by both CTAs of a pair)
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == TC_MMA) {
        if (PAIR) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(s_tmem)), "r"(cols) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(s_tmem)), "r"(cols) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (PAIR) tc_cluster_sync();      // (the other CTA's barriers are there)
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// a producer that gave up at stage s (its empty parity: ph): the copies that it has asked for land before it goes on (bounded)
template <int NS> __device__ __forceinline__ void tc_drain(uint32_t full, uint32_t s, uint32_t ph) {
    for (uint32_t i = 0; i < NS; i++) {
        bool wait = true;
        tc_wait(full + 8u * i, i < s ? ph ^ 1u : ph, wait, nullptr, 0);
    }
}
// a loader's part of a stage: the weight rows or the token rows of K elements from k on
template <int TN, bool GLU, bool IS_W>
__device__ __forceinline__ void tc_load(uint32_t stage, const CUtensorMap* map, const TcArgs& a, const TcTile& t, int k, uint32_t bar) {
    using Ring = TcRing<TN>;
    constexpr int BYTES = IS_W ? Ring::W_BYTES : Ring::X_BYTES;
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"((uint32_t)BYTES) : "memory");
    const uint32_t dst = stage + (IS_W ? 0u : (uint32_t)Ring::W_BYTES);
    const int row = IS_W ? t.m * (GLU ? TC_M / 2 : TC_M) : t.row0 + t.t0, z = IS_W || a.x_z ? t.z : 0;
    if (a.slabs) {
        tc_tma(dst, map, 0, row, k / TC_K, z, bar);
    } else {
#pragma unroll
        for (int h = 0; h < Ring::KH; h++) tc_tma(dst + h * (BYTES / Ring::KH), map, k + h * TC_K, row, 0, z, bar);
    }
}
template <int TN>
__device__ __forceinline__ void tc_mma_stage(uint32_t acc, uint32_t stage, uint32_t idesc, bool first) {
    using Ring = TcRing<TN>;
    const uint64_t da = tc_desc(stage), db = tc_desc(stage + Ring::W_BYTES);
#pragma unroll
    for (int h = 0; h < Ring::KH; h++) {
#pragma unroll
        for (int kk = 0; kk < TC_K / 16; kk++) {   // 16 elements = 32 bytes along the swizzled row: start address + 2
            const uint32_t accum = (!first || h > 0 || kk > 0) ? 1u : 0u;
            asm volatile(
                "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(acc),
                "l"(da + (uint64_t)(h * TC_M * 8 + 2 * kk)), "l"(db + (uint64_t)(h * TN * 8 + 2 * kk)), "r"(idesc), "r"(accum)
                : "memory");
        }
    }
}

// PAIR: two CTAs of a cluster share a tile of 256 weight rows x 256 tokens (tcgen05.mma.cta_group::2, issued by CTA 0): each brings its own 128 weight rows and half of the
// tokens' rows, 32 KB per 64 elements of K instead of 48, and ends with its own 128 rows.  The sums and their order are the single CTA's.
template <int TN, int EPI, bool PAIR = false>
__global__ void __launch_bounds__(TC_THREADS, 1)
    lp_gemm_tc_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap wmap, const TcArgs a) {
    next_grid();
    extern __shared__ __align__(1024) uint8_t tc_smem[];
    static_assert(!PAIR || TN == 256, "pairs share 256 tokens");
    constexpr int NS = PAIR ? TcPairRing::N : TcRing<TN>::N, STAGE = PAIR ? TcPairRing::STAGE : TcRing<TN>::STAGE, KS = PAIR ? TcPairRing::K : TcRing<TN>::K;
    constexpr bool GLU = epi_is_glu(EPI);
    __shared__ __align__(8) unsigned long long s_bar[2 * NS + 4];
    __shared__ uint32_t s_tmem;
    uint8_t* base = tc_smem + ((1024u - (smem_u32(tc_smem) & 1023u)) & 1023u);   // the swizzle is on absolute address bits
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t bar = smem_u32(&s_bar[0]), full = bar, empty = bar + 8u * NS, acc_full = bar + 16u * NS, acc_empty = acc_full + 16u;
    tc_setup<PAIR>(tid, warp, bar, NS, &s_tmem, 2, 2 * TN);
    const uint32_t rank = PAIR ? tc_cluster_rank() : 0u;
    if (TC_W_WAITS || a.seg || warp != TC_LOAD_W) wait_grid();      // (other weights do not depend on the kernel before)
    const uint32_t tmem = s_tmem, ring = smem_u32(base);
    const int steps = (a.K + KS - 1) / KS, n_own = (a.N + (GLU ? TC_M / 2 : TC_M) - 1) / (GLU ? TC_M / 2 : TC_M), n_mt = PAIR ? (n_own + 1) / 2 : n_own;
    bool alive = true;
    TcWalk<TN> walk;
    TcTile t;
    const int first = PAIR ? blockIdx.x >> 1 : blockIdx.x, stride = PAIR ? gridDim.x >> 1 : gridDim.x;
    auto find = [&](int item) {
        if (!walk.find(a, n_mt, item, t)) return false;
        if (PAIR) t.m = 2 * t.m + rank;      // (one past the last row tile: zeros in, nothing out)
        return true;
    };
    if (warp == TC_LOAD_W || warp == TC_LOAD_X) {
        uint32_t s = 0, ph = 1;
        for (int item = first; alive && find(item); item += stride)
            for (int k = 0; k < steps; k++) {
                tc_wait(empty + 8u * s, ph, alive, a.err, 1);
                alive = __all_sync(0xffffffffu, alive);
                if (!alive) break;
                if (tc_elect()) {
                    if constexpr (PAIR) {
                        const bool is_w = warp == TC_LOAD_W;
                        const int row = is_w ? t.m * (GLU ? TC_M / 2 : TC_M) : t.row0 + t.t0 + (int)rank * 128, z = is_w || a.x_z ? t.z : 0;
                        if (rank == 0)      // both CTAs' bytes
                            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(full + 8u * s), "r"((uint32_t)(2 * (is_w ? TcPairRing::W_BYTES : TcPairRing::X_BYTES))) : "memory");
                        tc_tma_pair(ring + s * STAGE + (is_w ? 0u : (uint32_t)TcPairRing::W_BYTES), is_w ? &wmap : &xmap, a.slabs ? 0 : k * KS, row, a.slabs ? k : 0, z, tc_leader(full + 8u * s));
                    } else if (warp == TC_LOAD_W) tc_load<TN, GLU, true>(ring + s * STAGE, &wmap, a, t, k * KS, full + 8u * s);
                    else tc_load<TN, GLU, false>(ring + s * STAGE, &xmap, a, t, k * KS, full + 8u * s);
                }
                __syncwarp();
                if (++s == NS) { s = 0; ph ^= 1u; }
            }
        if (!alive && rank == 0) tc_drain<NS>(full, s, ph);
    } else if (warp == TC_MMA) {
        const uint32_t idesc = tc_idesc(PAIR ? 2 * TC_M : TC_M, TN);
        uint32_t s = 0, ph = 0, it = 0;
        if (!PAIR || rank == 0)
        for (int item = first; find(item); item += stride, it++) {
            const uint32_t buf = it & 1u;
            tc_wait(acc_empty + 8u * buf, ((it >> 1) & 1u) ^ 1u, alive, a.err, 2);
            if (PAIR) asm volatile("fence.acq_rel.cluster;" ::: "memory");
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            for (int k = 0; k < steps; k++) {
                tc_wait(full + 8u * s, ph, alive, a.err, 3);
                alive = __all_sync(0xffffffffu, alive);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (tc_elect()) {
                    if constexpr (PAIR) {
                        if (alive) {
                            const uint64_t da = tc_desc(ring + s * STAGE), db = tc_desc(ring + s * STAGE + TcPairRing::W_BYTES);
#pragma unroll
                            for (int kk = 0; kk < TC_K / 16; kk++) {
                                const uint32_t accum = (k > 0 || kk > 0) ? 1u : 0u;
                                asm volatile(
                                    "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                                    "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem + buf * TN),
                                    "l"(da + (uint64_t)(2 * kk)), "l"(db + (uint64_t)(2 * kk)), "r"(idesc), "r"(accum)
                                    : "memory");
                            }
                        }
                        tc_commit_pair(empty + 8u * s);
                        if (k == steps - 1) tc_commit_pair(acc_full + 8u * buf);
                    } else {
                        if (alive) tc_mma_stage<TN>(tmem + buf * TN, ring + s * STAGE, idesc, k == 0);
                        tc_commit(empty + 8u * s);
                        if (k == steps - 1) tc_commit(acc_full + 8u * buf);
                    }
                }
                __syncwarp();
                if (++s == NS) { s = 0; ph ^= 1u; }
            }
        }
    } else {
        // warps w and w + 4 read TMEM lanes 32 (w & 3) .. + 31 (= weight rows), every second batch of 32 tokens each
        const int half = warp >> 2, row = tid & (TC_M - 1);
        uint32_t it = 0;
        for (int item = first; find(item); item += stride, it++) {
            const uint32_t buf = it & 1u, acc = tmem + buf * TN + ((uint32_t)((warp & 3) * 32) << 16);
            const int n0 = t.m * (GLU ? TC_M / 2 : TC_M), n = n0 + row, rows = t.rows - t.t0;        // rows: tokens of the tile that exist
            void* Yt = seg_rows<tc_t, EPI>(a.Y, (size_t)(t.row0 + t.t0) * a.ldy + (a.seg ? 0 : t.z * a.yz));
            if constexpr (GLU) {
                tc_wait(acc_full + 8u * buf, (it >> 1) & 1u, alive, a.err, 4);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                float* ex = reinterpret_cast<float*>(base + NS * STAGE + half * (TC_EX_BYTES / 2));      // [2 halves][16 tokens][64 units]
                tc_t* ob = reinterpret_cast<tc_t*>(ex + 2 * 16 * 64);            // [2][32 tokens][64 units]: the units on their way out, 16 bytes per store
                const bool v8 = a.N % 8 == 0 && a.ldy % 8 == 0 && ((uintptr_t)Yt & 15) == 0, up = row >= TC_M / 2;
#pragma unroll 1
                for (int c0 = 32 * half, ph = 0; c0 < TN; c0 += 64, ph ^= 1) {
                    if (c0 >= rows) break;   // uniform over the four warps of a half
                    uint32_t v[32];
                    tc_ld32(v, acc + (uint32_t)c0);
#pragma unroll
                    for (int c = 0; c < 16; c++) ex[(up ? 0 : 16 * 64) + c * 64 + (row & 63)] = __uint_as_float(v[up ? c : 16 + c]);
                    asm volatile("bar.sync %0, 128;" ::"r"(1 + half) : "memory");
#pragma unroll
                    for (int c = 0; c < 16; c++) {
                        const float mine = a.alpha * __uint_as_float(v[up ? 16 + c : c]), other = a.alpha * ex[(up ? 16 * 64 : 0) + c * 64 + (row & 63)];
                        ob[ph * 2048 + (up ? 16 + c : c) * 64 + (row & 63)] = from_f<tc_t>(glu_fast<EPI>(up ? other : mine, up ? mine : other));
                    }
                    asm volatile("bar.sync %0, 128;" ::"r"(1 + half) : "memory");
                    const tc_t* o = ob + ph * 2048;
                    tc_t* y = reinterpret_cast<tc_t*>(Yt) + (size_t)c0 * a.ldy + n0;
                    if (v8) {
#pragma unroll
                        for (int u = 0; u < 2; u++) {
                            const int i = row + u * 128, tt = i >> 3, c = (i & 7) * 8;
                            if (c0 + tt < rows && n0 + c < a.N) *reinterpret_cast<uint4*>(y + (size_t)tt * a.ldy + c) = *reinterpret_cast<const uint4*>(o + tt * 64 + c);
                        }
                    } else {
                        for (int i = row; i < 32 * 64; i += 128)
                            if (c0 + (i >> 6) < rows && n0 + (i & 63) < a.N) y[(size_t)(i >> 6) * a.ldy + (i & 63)] = o[i];
                    }
                }
            } else {
                const bool live = n < a.N;
                const float bn = (a.bias && live) ? a.bias[n] : 0.0f;
                // EPI_ADD: the old sums of 32 tokens are asked for one batch ahead (the first before the products are done), so that no load waits
                // behind a store to the same array
                float old[32];
                auto ask = [&](int c0, float* o) {
#pragma unroll
                    for (int c = 0; c < 32; c++) o[c] = (live && c0 + c < rows) ? reinterpret_cast<const float*>(Yt)[(size_t)(c0 + c) * a.ldy + n] : 0.0f;
                };
                if (EPI == EPI_ADD) ask(32 * half, old);
                tc_wait(acc_full + 8u * buf, (it >> 1) & 1u, alive, a.err, 4);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
                for (int c0 = 32 * half; c0 < TN; c0 += 64) {
                    if (c0 >= rows) break;   // warp-uniform
                    uint32_t v[32];
                    tc_ld32(v, acc + (uint32_t)c0);
                    if (EPI == EPI_ADD) {
                        float nx[32];
                        if (c0 + 64 < TN) ask(c0 + 64, nx);
#pragma unroll
                        for (int c = 0; c < 32; c++)
                            if (live && c0 + c < rows) reinterpret_cast<float*>(Yt)[(size_t)(c0 + c) * a.ldy + n] = old[c] + (a.alpha * __uint_as_float(v[c]) + bn);
#pragma unroll
                        for (int c = 0; c < 32; c++) old[c] = nx[c];
                    } else {
#pragma unroll
                        for (int c = 0; c < 32; c++)
                            if (live && c0 + c < rows) epi_store<tc_t, EPI>(Yt, (size_t)(c0 + c) * a.ldy + n, a.alpha * __uint_as_float(v[c]) + bn, a.act);
                    }
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) {
                if (PAIR) tc_arrive_leader(acc_empty + 8u * buf);
                else tc_arrive(acc_empty + 8u * buf);
            }
        }
    }
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (PAIR) {                                             // nobody leaves while the other's copies, commits or arrivals may still come here
        tc_cluster_sync();
        if (warp == TC_MMA) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * TN) : "memory");
    } else if (warp == TC_MMA) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * TN) : "memory");
}

__device__ __forceinline__ float tc_peer_f32(uint32_t addr, uint32_t rank) {
    uint32_t p;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(p) : "r"(addr), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(p) : "memory");
    return v;
}
template <int TN, int EPI>
__global__ void __launch_bounds__(TC_THREADS, 1)
    lp_gemm_tc_split_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap wmap, const TcArgs a) {
    next_grid();
    if (a.seg) wait_grid();
    extern __shared__ __align__(1024) uint8_t tc_smem[];
    constexpr int NS = TcRing<TN>::N, STAGE = TcRing<TN>::STAGE, KS = TcRing<TN>::K;
    constexpr bool GLU = epi_is_glu(EPI);
    __shared__ __align__(8) unsigned long long s_bar[2 * NS + 2];
    __shared__ uint32_t s_tmem;
    const int S = a.splits, rank = blockIdx.x % S;
    TcTile t;
    t.z = blockIdx.z;
    t.m = blockIdx.x / S;
    t.t0 = blockIdx.y * TN;
    t.row0 = a.seg ? a.seg[2 * t.z] : 0;
    t.rows = a.seg ? a.seg[2 * t.z + 1] : a.R;
    if (t.t0 >= t.rows) return;             // (the whole cluster)
    uint8_t* base = tc_smem + ((1024u - (smem_u32(tc_smem) & 1023u)) & 1023u);
    const int tid = threadIdx.x, warp = tid >> 5;
    const uint32_t bar = smem_u32(&s_bar[0]), full = bar, empty = bar + 8u * NS, acc_full = bar + 16u * NS;
    tc_setup(tid, warp, bar, NS, &s_tmem, 1, TN);
    if (!a.seg && (TC_W_WAITS || warp != TC_LOAD_W)) wait_grid();   // (other weights do not depend on the kernel before)
    const uint32_t tmem = s_tmem, ring = smem_u32(base);
    const int all = (a.K + KS - 1) / KS, k_beg = rank * all / S, k_end = (rank + 1) * all / S;      // (S <= all)
    bool alive = true;
    if (warp == TC_LOAD_W || warp == TC_LOAD_X) {
        uint32_t s = 0, ph = 1;
        for (int k = k_beg; k < k_end; k++) {
            tc_wait(empty + 8u * s, ph, alive, a.err, 1);
            alive = __all_sync(0xffffffffu, alive);
            if (!alive) break;
            if (tc_elect()) {
                if (warp == TC_LOAD_W) tc_load<TN, GLU, true>(ring + s * STAGE, &wmap, a, t, k * KS, full + 8u * s);
                else tc_load<TN, GLU, false>(ring + s * STAGE, &xmap, a, t, k * KS, full + 8u * s);
            }
            __syncwarp();
            if (++s == NS) { s = 0; ph ^= 1u; }
        }
        if (!alive) tc_drain<NS>(full, s, ph);
    } else if (warp == TC_MMA) {
        const uint32_t idesc = tc_idesc(TC_M, TN);
        uint32_t s = 0, ph = 0;
        for (int k = k_beg; k < k_end; k++) {
            tc_wait(full + 8u * s, ph, alive, a.err, 3);
            alive = __all_sync(0xffffffffu, alive);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (tc_elect()) {
                if (alive) tc_mma_stage<TN>(tmem, ring + s * STAGE, idesc, k == k_beg);
                tc_commit(empty + 8u * s);
                if (k == k_end - 1) tc_commit(acc_full);
            }
            __syncwarp();
            if (++s == NS) { s = 0; ph ^= 1u; }
        }
    }
    __syncwarp();
    float* part = reinterpret_cast<float*>(base);           // [TN tokens][128 rows] over the drained ring
    const int rows = min(TN, t.rows - t.t0);
    // K in one piece: nothing to exchange, so the sums go from tensor memory straight to Y, neighbouring lanes to neighbouring columns.  Through shared memory
    // with two cluster barriers this end cost 1 to 4 us of a launch: 32 sequences through two layers of 2048 2943 -> 2867 us, prompts of 777, 130 and 41 rows
    // through three of 1024 626 -> 586 (<64, 0>: 14.1 -> 10.2 us a launch).  Gated units keep the exchange, which pairs two rows of a tile.
    const bool alone = !GLU && S == 1;
    if (warp < TC_EPI_WARPS) {
        const int n = t.m * (GLU ? TC_M / 2 : TC_M) + (tid & (TC_M - 1));
        const bool live = n < a.N;
        const float bn = (alone && a.bias && live) ? a.bias[n] : 0.0f;
        void* Yt = seg_rows<tc_t, EPI>(a.Y, (size_t)(t.row0 + t.t0) * a.ldy + (a.seg ? 0 : t.z * a.yz));
        tc_wait(acc_full, 0, alive, a.err, 4);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
        for (int c0 = 32 * (warp >> 2); c0 < rows; c0 += 64) {
            uint32_t v[32];
            tc_ld32(v, tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c0);
            if (alone) {
                if constexpr (!GLU) {
                    if (EPI == EPI_ADD) {                   // (the old sums first: no load behind a store to the same array)
                        float old[32];
#pragma unroll
                        for (int c = 0; c < 32; c++) old[c] = (live && c0 + c < rows) ? reinterpret_cast<const float*>(Yt)[(size_t)(c0 + c) * a.ldy + n] : 0.0f;
#pragma unroll
                        for (int c = 0; c < 32; c++)
                            if (live && c0 + c < rows) reinterpret_cast<float*>(Yt)[(size_t)(c0 + c) * a.ldy + n] = old[c] + (a.alpha * __uint_as_float(v[c]) + bn);
                    } else {
#pragma unroll
                        for (int c = 0; c < 32; c++)
                            if (live && c0 + c < rows) epi_store<tc_t, EPI>(Yt, (size_t)(c0 + c) * a.ldy + n, a.alpha * __uint_as_float(v[c]) + bn, a.act);
                    }
                }
                continue;
            }
#pragma unroll
            for (int c = 0; c < 32; c++) part[(c0 + c) * TC_M + (tid & (TC_M - 1))] = __uint_as_float(v[c]);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
    if (warp < TC_EPI_WARPS && !alone) {
        const int c_beg = rank * rows / S, c_end = (rank + 1) * rows / S, n0 = t.m * (GLU ? TC_M / 2 : TC_M);
        const uint32_t part_s = smem_u32(part);
        void* Yt = seg_rows<tc_t, EPI>(a.Y, (size_t)(t.row0 + t.t0) * a.ldy + (a.seg ? 0 : t.z * a.yz));
        auto sum = [&](int c, int row) {
            float p[8];
#pragma unroll
            for (int r = 0; r < 8; r++) p[r] = r < S ? tc_peer_f32(part_s + (uint32_t)(c * TC_M + row) * 4u, (uint32_t)r) : 0.0f;
            float v = p[0];
#pragma unroll
            for (int r = 1; r < 8; r++) v += p[r];          // (adds of 0 beyond S)
            return v;
        };
        if constexpr (GLU) {
            const int n = n0 + (tid & 63);
#pragma unroll 2
            for (int c = c_beg + (tid >> 6); c < c_end; c += TC_EPI_WARPS / 2) {
                const float g = a.alpha * sum(c, tid & 63), u = a.alpha * sum(c, (tid & 63) + 64);
                if (n < a.N) reinterpret_cast<tc_t*>(Yt)[(size_t)c * a.ldy + n] = from_f<tc_t>(glu_fast<EPI>(g, u));
            }
        } else {
            const int n = n0 + (tid & (TC_M - 1));
            const bool live = n < a.N;
            const float bn = (a.bias && live) ? a.bias[n] : 0.0f;
#pragma unroll 1
            for (int c = c_beg + 4 * (tid >> 7); c < c_end; c += 8) {
                float old[4], v[4];
#pragma unroll
                for (int u = 0; u < 4; u++)
                    old[u] = (EPI == EPI_ADD && live && c + u < c_end) ? reinterpret_cast<const float*>(Yt)[(size_t)(c + u) * a.ldy + n] : 0.0f;
#pragma unroll
                for (int u = 0; u < 4; u++) v[u] = a.alpha * sum(min(c + u, c_end - 1), tid & (TC_M - 1)) + bn;
#pragma unroll
                for (int u = 0; u < 4; u++)
                    if (live && c + u < c_end) {
                        if (EPI == EPI_ADD) reinterpret_cast<float*>(Yt)[(size_t)(c + u) * a.ldy + n] = old[u] + v[u];
                        else epi_store<tc_t, EPI>(Yt, (size_t)(c + u) * a.ldy + n, v[u], a.act);
                    }
            }
        }
    }
    if (!alone) {                                           // nobody leaves while its partial sums are read
        asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
    }
    if (warp == TC_MMA) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TN) : "memory");
}

// Few token rows whose sums may not be cut along K: the token rows are the M of tcgen05.mma (MR = 64 or 128, those above R are whatever the shared memory holds;
// their sums stay in tensor memory unread) and NT = 16 or 32 weight rows its N, so that 2048 outputs are 128 or 64 CTAs instead of the 16 that tiles of 128 weight rows
// give, each with a quarter of the operand bytes.  Every sum adds its products in the order of K, by the same MMAs of 16: the bits of the other kernels.
// Bound by the operands on their way into shared memory, 128 (R + NT) bytes per 64 elements of K at 64 per clock; the whole ring is asked for at once.
// Warps 0 - 3: epilogue (tensor-memory lane = token row), 4 weight rows, 5 token rows, 6 MMAs.  One CTA per tile of NT outputs.
enum { TR_LOAD_W = 4, TR_LOAD_X = 5, TR_MMA = 6, TR_THREADS = 224, TR_KH = 4, TR_STAGES = 8 };
// stages of 4 slabs: R token rows (a multiple of 8), then NT weight rows; behind the ring what an MMA over MR rows reads beyond the last token rows
__host__ __device__ inline uint32_t tr_stage_bytes(int rows8, int nt) { return (uint32_t)TR_KH * (rows8 + nt) * 128; }
__host__ __device__ inline int tr_stages(int rows8, int nt, int K) {
    const int fit = (int)(196608 / tr_stage_bytes(rows8, nt)), need = (K + TR_KH * TC_K - 1) / (TR_KH * TC_K), most = fit < TR_STAGES ? fit : (int)TR_STAGES;
    return need < most ? need : most;
}
inline size_t tr_smem_bytes(int rows8, int nt, int K, int mr) { return (size_t)tr_stages(rows8, nt, K) * tr_stage_bytes(rows8, nt) + (size_t)mr * 128 + 1024; }

template <int MR, int NT, int EPI>
__global__ void __launch_bounds__(TR_THREADS, 1) lp_gemm_tc_rows_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap wmap, const TcArgs a) {
    static_assert(!epi_is_glu(EPI), "gated units pair two weight rows");
    next_grid();
    extern __shared__ __align__(1024) uint8_t tc_smem[];
    __shared__ __align__(8) unsigned long long s_bar[2 * TR_STAGES + 1];
    __shared__ uint32_t s_tmem;
    uint8_t* base = tc_smem + ((1024u - (smem_u32(tc_smem) & 1023u)) & 1023u);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rows8 = (a.R + 7) & ~7, NS = tr_stages(rows8, NT, a.K), all = (a.K + TC_K - 1) / TC_K, steps = (all + TR_KH - 1) / TR_KH;
    const uint32_t stage_bytes = tr_stage_bytes(rows8, NT), x_bytes = (uint32_t)TR_KH * rows8 * 128, ring = smem_u32(base);
    const uint32_t bar = smem_u32(&s_bar[0]), full = bar, empty = bar + 8u * TR_STAGES, done = bar + 16u * TR_STAGES;
    constexpr uint32_t COLS = 32;
    if (tid == 0) {
        for (int i = 0; i < TR_STAGES; i++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 2;" ::"r"(full + 8u * i) : "memory");      // both loaders
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(empty + 8u * i) : "memory");
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(done) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == TR_MMA) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"(COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (TC_W_WAITS || warp != TR_LOAD_W) wait_grid();       // (other weights do not depend on the kernel before)
    const uint32_t tmem = s_tmem;
    const int n0 = blockIdx.x * NT;
    bool alive = true;
    if (warp == TR_LOAD_W || warp == TR_LOAD_X) {
        const bool is_w = warp == TR_LOAD_W;
        const int rows = is_w ? NT : rows8;
        uint32_t s = 0, ph = 1;
        for (int k = 0; k < steps; k++) {
            tc_wait(empty + 8u * s, ph, alive, a.err, 1);
            alive = __all_sync(0xffffffffu, alive);
            if (!alive) break;
            if (tc_elect()) {
                const uint32_t dst = ring + s * stage_bytes + (is_w ? x_bytes : 0u);
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(full + 8u * s), "r"((uint32_t)TR_KH * rows * 128u) : "memory");
                if (a.slabs) {
                    tc_tma(dst, is_w ? &wmap : &xmap, 0, is_w ? n0 : 0, k * TR_KH, 0, full + 8u * s);
                } else {
#pragma unroll
                    for (int h = 0; h < TR_KH; h++) tc_tma(dst + (uint32_t)h * rows * 128u, is_w ? &wmap : &xmap, (k * TR_KH + h) * TC_K, is_w ? n0 : 0, 0, 0, full + 8u * s);
                }
            }
            __syncwarp();
            if (++s == (uint32_t)NS) { s = 0; ph ^= 1u; }
        }
        if (!alive)      // what has been asked for lands first (bounded)
            for (uint32_t i = 0; i < (uint32_t)NS; i++) {
                bool wait = true;
                tc_wait(full + 8u * i, i < s ? ph ^ 1u : ph, wait, nullptr, 0);
            }
    } else if (warp == TR_MMA) {
        const uint32_t idesc = tc_idesc(MR, NT);
        uint32_t s = 0, ph = 0;
        for (int k = 0; k < steps; k++) {
            tc_wait(full + 8u * s, ph, alive, a.err, 3);
            alive = __all_sync(0xffffffffu, alive);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (tc_elect()) {
                if (alive) {
                    const uint64_t da = tc_desc(ring + s * stage_bytes), db = tc_desc(ring + s * stage_bytes + x_bytes);
#pragma unroll
                    for (int h = 0; h < TR_KH; h++)
                        if (k * TR_KH + h < all) {
#pragma unroll
                            for (int kk = 0; kk < TC_K / 16; kk++) {
                                const uint32_t accum = (k > 0 || h > 0 || kk > 0) ? 1u : 0u;
                                asm volatile(
                                    "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
                                    "l"(da + (uint64_t)(h * rows8 * 8 + 2 * kk)), "l"(db + (uint64_t)(h * NT * 8 + 2 * kk)), "r"(idesc), "r"(accum)
                                    : "memory");
                            }
                        }
                }
                tc_commit(empty + 8u * s);
                if (k == steps - 1) tc_commit(done);
            }
            __syncwarp();
            if (++s == (uint32_t)NS) { s = 0; ph ^= 1u; }
        }
    } else {
        // M = 128: row = lane of tensor memory; M = 64: rows 16 w .. 16 w + 15 in the first half of warp w's lanes
        const int t = MR == 128 ? tid : 16 * warp + lane;
        const bool live = t < a.R && (MR == 128 || lane < 16);
        tc_wait(done, 0, alive, a.err, 4);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        uint32_t v[32];
        tc_ld32(v, tmem + ((uint32_t)(warp * 32) << 16));
        if (live) {
            const size_t at = (size_t)t * a.ldy + n0;
            if (!epi_is_act(EPI) && n0 + NT <= a.N && a.ldy % 4 == 0 && ((uintptr_t)a.Y & 15) == 0 && !a.bias) {
                float4* y = reinterpret_cast<float4*>(reinterpret_cast<float*>(a.Y) + at);
#pragma unroll
                for (int c = 0; c < NT / 4; c++) {
                    const float4 old = EPI == EPI_ADD ? y[c] : make_float4(0.f, 0.f, 0.f, 0.f);
                    float f[4];
#pragma unroll
                    for (int u = 0; u < 4; u++) f[u] = a.alpha * __uint_as_float(v[4 * c + u]) + 0.0f;
                    y[c] = EPI == EPI_ADD ? make_float4(old.x + f[0], old.y + f[1], old.z + f[2], old.w + f[3]) : make_float4(f[0], f[1], f[2], f[3]);
                }
            } else {
#pragma unroll
                for (int c = 0; c < NT; c++)
                    if (n0 + c < a.N) epi_store<tc_t, EPI>(a.Y, at + c, a.alpha * __uint_as_float(v[c]) + (a.bias ? a.bias[n0 + c] : 0.0f), a.act);
            }
        }
    }
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == TR_MMA) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(COLS) : "memory");
}

// ------------------------------------------------------------------------------------------------ host
using TcEncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                                CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
TcEncodeFn tc_encode_fn() {
    static TcEncodeFn fn = []() -> TcEncodeFn {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            return nullptr;
        }
        return (TcEncodeFn)f;
    }();
    return fn;
}
// [groups][parts][rows][K], rows `ld` elements apart, parts (gate and up of a gated matrix) rows * ld, groups z, in boxes of box rows x 64
// elements x all parts; K % 64 == 0: as [groups][K / 64][parts][rows][64], `kh` slabs of 64 per box
bool tc_map(CUtensorMap* map, const void* p, int K, int rows, int ld, int parts, int groups, size_t z, int box, int kh) {
    const TcEncodeFn fn = tc_encode_fn();
    if (!fn) return false;
    const bool slabs = K % TC_K == 0;
    const cuuint64_t dims[5] = {(cuuint64_t)(slabs ? TC_K : K), (cuuint64_t)rows, (cuuint64_t)parts, (cuuint64_t)(slabs ? K / TC_K : 1), (cuuint64_t)groups};
    const cuuint64_t strides[4] = {(cuuint64_t)ld * 2, (cuuint64_t)rows * ld * 2, TC_K * 2, (groups > 1 ? (cuuint64_t)z : (cuuint64_t)ld) * 2};
    const cuuint32_t boxes[5] = {(cuuint32_t)TC_K, (cuuint32_t)box, (cuuint32_t)parts, (cuuint32_t)(slabs ? kh : 1), 1}, one[5] = {1, 1, 1, 1, 1};
    return fn(map, TC_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 5, (void*)p, dims, strides, boxes, one, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Which kernel a product of R rows (of every group; xrows in all groups together when the rows come from `seg`) takes: the least clocks by
// what each one measured, of a step of 64 elements per CTA (operand bytes at 64 per clock) and of what a CTA adds when it is not overlapped
// (filling the ring, epilogue, the exchange of a split), on 148 SMs (74 pairs: a step of 801 clocks where the single CTA's took 875, gate and up of an 8B layer; starting and
// ending together 3000: 1500 rows x 2568 x 1024 lost 2 % of a prompt to pairs that the steps alone spoke for).  Clusters of 8 do not tile the chip's SM groups: 128 of
// their CTAs already took two waves (12.4 us where 64 CTAs in clusters of 4 took 8.3: 32 x 2048 x 2048).
// split: K may be cut over a cluster.  Without, every sum adds its products in the order of K, so that a row's result is the same bits whatever the number of
// rows of the step.
// rows: token rows as M (lp_gemm_tc_rows_kernel), tn weight rows per CTA: for sums that may not be cut (a cut over a cluster is as fast), up to 128 rows
// pair: two CTAs per tile (lp_gemm_tc_kernel), where the single CTAs would not cut K either: a pair adds all of K in one accumulator of tensor memory, which cuts its sums off,
// so in place of a cut it gives other bits and a larger error: 4096 x 700 x 14336 in two cuts, one 8B layer over 24 inputs, 1.0002 +- 0.0001 (Q4_K_M) and 1.0009 +- 0.0001 (Q8_0, 645
// rows) times the distance to float64.  (Time: two 8B layers of 700 rows 1065 us before pairs, 910 with pairs there, 1000 without.)
struct TcPlan {
    bool persistent;
    int tn, splits;
    bool rows, pair;
};
TcPlan tc_plan(int R, int N, int K, int groups, int xrows, bool seg, bool glu, bool split, bool tc_rows_able = false, int pairs = 1) {
    const int n_sm = 148, steps = (K + TC_K - 1) / TC_K, per = glu ? TC_M / 2 : TC_M, n_mt = (N + per - 1) / per;
    auto tiles = [&](int tn) { return (long long)n_mt * (seg ? xrows / tn + (groups + 1) / 2 : groups * ((R + tn - 1) / tn)); };
    TcPlan best{true, 256, 1, false, false};
    long long least = -1;
    auto offer = [&](bool persistent, int tn, int s, long long cost) {
        if (least < 0 || cost < least) { least = cost; best = TcPlan{persistent, tn, s, false, false}; }
    };
    if (tc_rows_able && !split && !seg && !glu && groups == 1 && R <= 128)
        for (int nt : {16, 32}) {
            const long long waves = ((N + nt - 1) / nt + n_sm - 1) / n_sm, step = std::max(2 * (((R + 7) & ~7) + nt), R <= 64 ? 64 + nt : 128 + nt);
            const long long cost = waves * (steps * step + 4500) - 4500 + 18 * 64;
            if (least < 0 || cost < least) { least = cost; best = TcPlan{false, nt, 1, true, false}; }
        }
    for (int tn : {256, 128}) {
        if (tn == 256 && R <= 128) continue;
        const long long waves = (tiles(tn) + n_sm - 1) / n_sm;
        offer(true, tn, 1, waves * steps * (tn == 256 ? 750 : 470) + 17 * tn);
    }
    long long pair_cost = -1;
    if (pairs && R > 128) {
        const long long two = (long long)((n_mt + 1) / 2) * (seg ? xrows / 256 + (groups + 1) / 2 : groups * ((R + 255) / 256)), waves = (two + n_sm / 2 - 1) / (n_sm / 2);
        pair_cost = waves * steps * 680 + 17 * 256 + 3000;
        if (pairs == 2) return TcPlan{true, 256, 1, false, true};
    }
    for (int tn : {128, 64}) {
        if (tn == 128 && R <= 64) continue;
        for (int s : {1, 2, 4, 8}) {
            if (s > 1 && (!split || steps < 4 * s)) break;
            const long long fit = s == 8 ? 112 : s == 4 ? 140 : n_sm, waves = (tiles(tn) * s + fit - 1) / fit;
            offer(false, tn, s, waves * ((steps + s - 1) / s * (tn == 128 ? 470 : 375) + 4500) - 4500 + 18 * tn + (s > 1 ? 1000 : 0));
        }
    }
    if (pair_cost >= 0 && best.splits == 1 && pair_cost < least) return TcPlan{true, 256, 1, false, true};
    return best;
}
