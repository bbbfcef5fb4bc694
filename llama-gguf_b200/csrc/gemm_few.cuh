// gemm_few.cuh — products of few token rows (batched decoding, short prompts) with GGUF weights, straight from the blocks:
//
//   Y[t][j] = sum_k deq(W)[j][k] * X[t][k],   W = rows of Q4_K / Q5_K / Q6_K / Q8_0 blocks, X fp16, f32 sums
//
// (the contraction the reference runs as T GEMVs per matrix: src/model/llama.rs:327-345; block arithmetic src/tensor/quant/dequant.rs:103-109,
// 205-356).  Up to 64 tokens a weight byte meets too few products to matter to the tensor pipe; what counts is unpacking at the rate DRAM delivers.
//
//  * Weights enter the tensor core as INTEGERS: q * sc (6-bit scale times a 4- or 5-bit quant, at most 1953: an fp16 number; int8 scale times 6 bits for Q6_K, which
//    fp16 rounds to even numbers above 2048), one LOP3 and one HFMA2 for two weights.  The block's f32 factor d multiplies the sum of its 256 products instead of every
//    weight, when the block's accumulator is drained (T / 2 FMAs per 256 weights and thread).  The minimum term -dmin sum_s m_s X_s (X_s = sum of the 32
//    activations of sub-block s) is two more K steps of a tf32 product: dmin m_s has 17 bits, X_s is carried as two tf32 numbers.  So Q4_K and
//    Q5_K weights are exact; Q6_K ones are rounded where |q sc| > 2048 (2^-12 of themselves), and Q8_0 ones once, since no factor is common to 256 of them.  Activations
//    are rounded to fp16 (as in gemm_umma2.cuh, which rounds each dequantised weight to fp16 too).
//  * The unpacked operand goes to TENSOR MEMORY (tcgen05.st, thread = weight row) and never through shared memory: 128 x 256 weights written and
//    read back there would cost 1024 clocks of its bandwidth, where DRAM delivers the block in 790.
//  * Activations come as an image of the shared-memory tiles (few_put8): one bulk copy per block of 256, no tensor map.
//  * Work is dealt in (128 rows x 256 elements of K) units, one contiguous range per CTA, weighted by the bytes of a type.  A tile that one CTA
//    covers goes straight to Y; the pieces of a cut tile go to a workspace, and the kernel that reads Y next adds them (FewOut::get), in the order of K.
//
// Roles: 2 groups of 128 threads that unpack every other unit each and add up what its products gave (the sums of the two meet at a piece's end, through
// tensor memory); a warp that loads; a warp that issues the MMAs.  They meet through mbarriers only; every wait is bounded and reports through `err`.
//
// What bounds it: unpacking, about 700 instructions per unit and warp (LOP3 and shifts at half rate), 1450 clocks per unit of Q4_K where DRAM needs 790.  No unit of the
// SM is full meanwhile (counters of gate and up, 32 tokens: issue slots 37 %, tensor pipe 13 %, DRAM 27 % of a cold launch): a scheduler has two unpacking warps, and what
// they wait for is their own chains.  And 5 us of launch, fill and drain.  Measured back to back (weights from DRAM), 32 tokens, the seven products of an 8B layer: gate and up 23.4 us (2.8 TB/s; the
// fused kernel 86), down Q4_K 14.8 (35), Q6_K 18.1, q / k / v 9.3, o 7.5; gate and up in Q8_0 26.4 us (4.7 TB/s), at 64 tokens 27.9 us.
#pragma once
#include <cuda.h>
#include "few_image.cuh"
#include "few_plan.cuh"
#include "gemm_umma2.cuh"

namespace b200 {

// Up to 256 tokens, in token tiles of 64 (the weights of a second tile come from L2).  Prompts through two 8B layers, against the two passes of prompt_f16.cuh or
// the fused kernel, Q4_K_M / Q6_K / Q8_0 / Q5_K_M: 33 tokens 794 / 1005 / 876 / 1025 -> 585 / 645 / 621 / 627 us, 128 tokens 929 / 1060 / 1018 / 1139 -> 695 / 766 /
// 730 / 741, 256 tokens 1024 / 1154 / 1108 / 1238 -> 887 / 1013 / 923 / 957; four 2048-wide layers (ffn 8192), 64 / 128 / 192 / 256 tokens: Q4_K_M 622 / 506 / 561 / 603 -> 390 / 459 / 529 /
// 589; 1024-wide ones (ffn 4096) Q4_K 549 / 362 / 369 / 382 -> 278 / 312 / 349 / 378, Q8_0 324 / 360 / 388 / 380 -> 283 / 317 / 359 / 387.  Every token tile unpacks again,
// so the gain is gone at 256 in the last of these, and a tile or two above in the others.  Batched decoding gains more, since what it replaces is the fused kernel (8 /
// 33 / 128 / 256 sequences, two 8B layers: 439 / 538 / 1284 / 2040 -> 231 / 293 / 581 / 1363).
constexpr int kFewTokens = 256;
constexpr int kFewThreads = 384, kFewLoader = 8, kFewMma = 9;      // (warps 10 and 11 are there for the register split: it goes by warpgroups)
constexpr int kFewRegsWork = 224, kFewRegsServe = 56;              // 256 x 224 + 128 x 56 = 384 x 168, what the block is launched with

struct FewSeg {
    const CUtensorMap* map;              // raw blocks, box = 128 rows x pitch bytes
    int type, n_rows, pitch, block_bytes;
    float* y;                            // [T][ldy]
    int ldy;
};
struct FewArgs {
    FewPlan plan;
    FewSeg seg[kFewMaxSeg];
    const uint8_t* image;
    float* part;                         // [2 grid][N][128]
    int stages_raw, stages_b, raw_stage;
    int* err;
};
// A finished product as its reader sees it.
struct FewOut {
    FewPlan plan;
    const float* y[kFewMaxSeg];
    int ldy[kFewMaxSeg];
    const float* part;
    int N;
};
// V consecutive rows j .. (of one tile) of token t; up to four pieces in flight, added in the order of K
template <int V>
__device__ __forceinline__ void few_get(const FewOut& o, int s, const FewTile& tl, int t, int j, float (&v)[V]) {
    static_assert(V == 1 || V % 4 == 0, "scalars or float4");
    constexpr int VV = V == 1 ? 1 : V / 4;
    auto load = [](const float* p, float (&x)[V]) {
        if constexpr (V == 1) x[0] = __ldcg(p);
        else {
#pragma unroll
            for (int q = 0; q < VV; q++) {
                const float4 a = __ldcg(reinterpret_cast<const float4*>(p) + q);
                x[4 * q] = a.x; x[4 * q + 1] = a.y; x[4 * q + 2] = a.z; x[4 * q + 3] = a.w;
            }
        }
    };
    if (tl.b0 == tl.b1) {
        load(o.y[s] + (size_t)t * o.ldy[s] + j, v);
        return;
    }
    const size_t at = (size_t)(t % o.N) * 128 + (j & 127), pitch = (size_t)o.N * 128;
#pragma unroll
    for (int q = 0; q < V; q++) v[q] = 0.0f;
    for (int b = tl.b0; b <= tl.b1; b += 4) {
        float x[4][V];
#pragma unroll
        for (int i = 0; i < 4; i++)
            if (b + i <= tl.b1) load(o.part + (size_t)(b + i == tl.b0 ? tl.first : 2 * (b + i)) * pitch + at, x[i]);
#pragma unroll
        for (int i = 0; i < 4; i++)
            if (b + i <= tl.b1)
#pragma unroll
                for (int q = 0; q < V; q++) v[q] += x[i][q];
    }
}

// ---- unpacking: one thread, one row, 256 elements -> 128 words of tensor memory at column `ta` of the thread's lane
__device__ __forceinline__ uint32_t few_h2(uint32_t a, uint32_t b, uint32_t c) {      // a * b + c on fp16 pairs
    uint32_t r;
    asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
    return r;
}
__device__ __forceinline__ uint32_t few_add2(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("add.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ uint32_t few_mul2(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
// (no "memory" clobber: loads from shared memory may move across)
__device__ __forceinline__ void few_st32(uint32_t taddr, const uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31};" ::"r"(v[0]), "r"(v[1]),
        "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]),
        "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]),
        "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31]), "r"(taddr));
}
__device__ __forceinline__ void few_st16(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15};" ::"r"(v[0]), "r"(v[1]), "r"(v[2]),
                 "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]),
                 "r"(taddr));
}
__device__ __forceinline__ void few_st4(uint32_t taddr, const uint32_t (&v)[4]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%4], {%0,%1,%2,%3};" ::"r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(taddr));
}
template <int C>
__device__ __forceinline__ void few_ld(uint32_t (&v)[C], uint32_t taddr) {
    static_assert(C == 8 || C == 16, "columns");
    if constexpr (C == 8) {
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                     : "r"(taddr));
    } else {
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                     : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]),
                       "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                     : "r"(taddr));
    }
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// (a & mask) | magic in one instruction: both constants in registers the compiler cannot see through (as immediates they cost two)
struct FewMask {
    uint32_t lo, hi, magic;
    __device__ __forceinline__ FewMask() {
        asm("mov.b32 %0, 0x000F000F;" : "=r"(lo));
        asm("mov.b32 %0, 0x00F000F0;" : "=r"(hi));
        asm("mov.b32 %0, 0x64006400;" : "=r"(magic));
    }
};
__device__ __forceinline__ uint32_t few_pick(uint32_t a, uint32_t mask, uint32_t magic) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(a), "r"(mask), "r"(magic));
    return r;
}
constexpr uint32_t H2_1024 = 0x64006400u, H2_N1024 = 0xE400E400u, H2_16TH = 0x2C002C00u, H2_N64 = 0xD400D400u, H2_N1056 = 0xE420E420u, H2_N1152 = 0xE480E480u;

// Each of these unpacks half h (elements 128 h .. 128 h + 127) of a row's block; wait_a() returns once the operand may be overwritten.
//
// Q4_K / Q5_K: 1024 + q by a mask, times sc, minus 1024 sc: exact.  High nibbles are left in place: (1024 + 16 q) sc / 16 - 64 sc.
// -dmin m_s as two tf32 numbers -> the 16 columns behind the weights.  Returns d.
template <bool Q5, class WaitA>
__device__ __forceinline__ float few_unpack_k45(const uint8_t* row, int h, uint32_t ta, const FewMask& k, WaitA&& wait_a) {
    const uint4* p = reinterpret_cast<const uint4*>(row);
    const uint4 hdr = p[0];
    uint4 raw[4];
#pragma unroll
    for (int i = 0; i < 4; i++) raw[i] = p[(Q5 ? 3 : 1) + 4 * h + i];
    uint32_t qh[8];
    if constexpr (Q5) {
        const uint4 a = p[1], b = p[2];
        const int sh = 4 * h;
        qh[0] = a.x >> sh; qh[1] = a.y >> sh; qh[2] = a.z >> sh; qh[3] = a.w >> sh; qh[4] = b.x >> sh; qh[5] = b.y >> sh; qh[6] = b.z >> sh; qh[7] = b.w >> sh;
    }
    const uint32_t sc = h ? (hdr.w & 0x0F0F0F0Fu) | ((hdr.y >> 2) & 0x30303030u) : hdr.y & 0x3F3F3F3Fu;
    const uint32_t mn = h ? ((hdr.w >> 4) & 0x0F0F0F0Fu) | ((hdr.z >> 2) & 0x30303030u) : hdr.z & 0x3F3F3F3Fu;
#pragma unroll
    for (int gp = 0; gp < 2; gp++) {
        const uint32_t w[8] = {raw[2 * gp].x, raw[2 * gp].y, raw[2 * gp].z, raw[2 * gp].w, raw[2 * gp + 1].x, raw[2 * gp + 1].y, raw[2 * gp + 1].z, raw[2 * gp + 1].w};
        const uint32_t s0 = few_add2(__byte_perm(sc, 0x64646464u, gp ? 0x4242 : 0x4040), H2_N1024);
        const uint32_t s1 = few_add2(__byte_perm(sc, 0x64646464u, gp ? 0x4343 : 0x4141), H2_N1024);
        const uint32_t o0 = few_mul2(s0, H2_N1024), s1h = few_mul2(s1, H2_16TH), o1 = few_mul2(s1, H2_N64);
        uint32_t v[32];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const uint32_t w8 = w[i] >> 8;
            uint32_t l02 = few_pick(w[i], k.lo, k.magic), l13 = few_pick(w8, k.lo, k.magic), h02 = few_pick(w[i], k.hi, k.magic), h13 = few_pick(w8, k.hi, k.magic);
            if constexpr (Q5) {      // bit 2 gp of the byte -> 16, bit 2 gp + 1 -> 16 * 16
                const uint32_t b = qh[i], b8 = b >> 8;
                l02 = few_pick(b << (4 - 2 * gp), 0x00100010u, l02);
                l13 = few_pick(b8 << (4 - 2 * gp), 0x00100010u, l13);
                h02 = few_pick(b << (7 - 2 * gp), 0x01000100u, h02);
                h13 = few_pick(b8 << (7 - 2 * gp), 0x01000100u, h13);
            }
            v[2 * i] = few_h2(l02, s0, o0);
            v[2 * i + 1] = few_h2(l13, s0, o0);
            v[16 + 2 * i] = few_h2(h02, s1h, o1);
            v[16 + 2 * i + 1] = few_h2(h13, s1h, o1);
        }
        if (gp == 0) wait_a();
        few_st32(ta + (uint32_t)(64 * h + 32 * gp), v);
    }
    const float nd = -half_bits_to_float(hdr.x >> 16);
    uint32_t m[4], l[4];
#pragma unroll
    for (int s = 0; s < 4; s++) {
        const float x = nd * (float)((mn >> (8 * s)) & 63u);
        m[s] = __float_as_uint(x) & 0xFFFFE000u;
        l[s] = __float_as_uint(x - __uint_as_float(m[s]));      // 17 bits in all: exact
    }
    few_st4(ta + 128u + 4u * (uint32_t)h, m);
    few_st4(ta + 136u + 4u * (uint32_t)h, l);
    return half_bits_to_float(hdr.x);
}
// Q6_K: blocks of 210 bytes start at any even byte of the 240 that were fetched (the same one for all rows): aligned loads and a funnel shift.
template <int WO>
__device__ __forceinline__ void few_align6(const uint32_t (&a)[20], const uint32_t (&b)[12], const uint32_t (&c)[12], int h, uint32_t sh, uint32_t (&ql)[16], uint32_t (&qh)[8],
                                           uint32_t (&sc)[2], uint32_t& d) {
#pragma unroll
    for (int i = 0; i < 16; i++) ql[i] = __funnelshift_r(a[i + WO], a[i + WO + 1], sh);
#pragma unroll
    for (int i = 0; i < 8; i++) qh[i] = __funnelshift_r(b[i + WO], b[i + WO + 1], sh);
    sc[0] = h ? __funnelshift_r(c[2 + WO], c[3 + WO], sh) : __funnelshift_r(c[WO], c[1 + WO], sh);
    sc[1] = h ? __funnelshift_r(c[3 + WO], c[4 + WO], sh) : __funnelshift_r(c[1 + WO], c[2 + WO], sh);
    d = __funnelshift_r(c[4 + WO], c[5 + WO], sh);
}
template <class WaitA>
__device__ __forceinline__ float few_unpack_q6(const uint8_t* row, int h, int residue, uint32_t ta, const FewMask& k, WaitA&& wait_a) {
    uint32_t ql[16], qh[8], sc[2], d;
    {
        uint32_t a[20], b[12], c[12];
        const uint4* p = reinterpret_cast<const uint4*>(row);
#pragma unroll
        for (int i = 0; i < 5; i++) {
            const uint4 x = p[4 * h + i];
            a[4 * i] = x.x; a[4 * i + 1] = x.y; a[4 * i + 2] = x.z; a[4 * i + 3] = x.w;
        }
#pragma unroll
        for (int i = 0; i < 3; i++) {
            const uint4 x = p[8 + 2 * h + i], y = p[12 + i];
            b[4 * i] = x.x; b[4 * i + 1] = x.y; b[4 * i + 2] = x.z; b[4 * i + 3] = x.w;
            c[4 * i] = y.x; c[4 * i + 1] = y.y; c[4 * i + 2] = y.z; c[4 * i + 3] = y.w;
        }
        const uint32_t sh = (uint32_t)(residue & 2) * 8u;
        switch (residue >> 2) {
            case 0: few_align6<0>(a, b, c, h, sh, ql, qh, sc, d); break;
            case 1: few_align6<1>(a, b, c, h, sh, ql, qh, sc, d); break;
            case 2: few_align6<2>(a, b, c, h, sh, ql, qh, sc, d); break;
            default: few_align6<3>(a, b, c, h, sh, ql, qh, sc, d); break;
        }
    }
    sc[0] ^= 0x80808080u;
    sc[1] ^= 0x80808080u;
#pragma unroll
    for (int hi = 0; hi < 2; hi++) {
        uint32_t o[32];
#pragma unroll
        for (int sec = 0; sec < 2; sec++) {
            const int qq = 2 * hi + sec;
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const int si = 2 * qq + (i >> 2);      // 16 elements share an int8 scale
                const uint32_t s2 = few_add2(__byte_perm(sc[si >> 2], 0x64646464u, 0x4040 | ((si & 3) * 0x0101)), H2_N1152);
                const uint32_t q = ql[8 * sec + i], b = qh[i];
                const uint32_t l0 = hi ? q >> 4 : q, l1 = hi ? q >> 12 : q >> 8;
                const uint32_t h0 = qq <= 2 ? b << (4 - 2 * qq) : b >> (2 * qq - 4), h1 = b >> (4 + 2 * qq);
                const uint32_t e = few_pick(h0, 0x00300030u, few_pick(l0, k.lo, k.magic)), f = few_pick(h1, 0x00300030u, few_pick(l1, k.lo, k.magic));
                o[16 * sec + 2 * i] = few_mul2(few_add2(e, H2_N1056), s2);
                o[16 * sec + 2 * i + 1] = few_mul2(few_add2(f, H2_N1056), s2);
            }
        }
        if (hi == 0) wait_a();
        few_st32(ta + (uint32_t)(64 * h + 32 * hi), o);
    }
    return half_bits_to_float(d);
}
// Q8_0: four blocks of 34 bytes; there is no factor of the 256, so d goes into the weight, rounded to fp16 once.
template <int H, class WaitA>
__device__ __forceinline__ float few_unpack_q8(const uint8_t* row, uint32_t ta, WaitA&& wait_a) {
    const uint4* p = reinterpret_cast<const uint4*>(row);
    constexpr int W0 = (34 * H) / 4;      // first 16-byte word of the half; its bytes start (34 * H) % 4 words into it
    uint32_t w[36];
#pragma unroll
    for (int i = 0; i < 9; i++) {
        const uint4 a = p[W0 + i];
        w[4 * i] = a.x; w[4 * i + 1] = a.y; w[4 * i + 2] = a.z; w[4 * i + 3] = a.w;
    }
#pragma unroll
    for (int g = 0; g < 2; g++) {      // two blocks = 17 words
        uint32_t o[32];
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const int at = (34 * H) % 4 + 17 * g + (k ? 8 : 0);      // word with the block's d: low half (first block) or high half
            const uint32_t d2 = __byte_perm(w[at], 0u, k ? 0x3232 : 0x1010);
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const uint32_t b = (k ? w[at + 1 + i] : __funnelshift_r(w[at + i], w[at + i + 1], 16)) ^ 0x80808080u;
                o[16 * k + 2 * i] = few_mul2(few_add2(__byte_perm(b, 0x64646464u, 0x4240), H2_N1152), d2);
                o[16 * k + 2 * i + 1] = few_mul2(few_add2(__byte_perm(b, 0x64646464u, 0x4341), H2_N1152), d2);
            }
        }
        if (g == 0) wait_a();
        few_st32(ta + (uint32_t)(64 * H + 32 * g), o);
    }
    return 1.0f;
}

__device__ __forceinline__ void few_mma_f16(uint32_t acc, uint32_t a, uint64_t db, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(acc), "r"(a), "l"(db), "r"(idesc),
                 "r"(accumulate)
                 : "memory");
}
__device__ __forceinline__ void few_mma_tf32(uint32_t acc, uint32_t a, uint64_t db, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n\t}" ::"r"(acc), "r"(a), "l"(db), "r"(idesc),
                 "r"(accumulate)
                 : "memory");
}
__device__ __forceinline__ void few_bulk(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}

constexpr int kFewMaxStages = 8;
// bounded wait: polls seldom read the clock
__device__ __forceinline__ void few_wait(uint32_t bar, uint32_t parity, bool& alive, int* err, int code) {
    if (!alive) return;
    uint32_t ok = 0, n = 0;
    long long t0 = 0;
    while (true) {
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, 10000;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
        if (ok) return;
        if ((n++ & 15u) == 0u) {
            const long long t = clock64();
            if (n == 1u) t0 = t;
            else if (t - t0 > 2000000000LL) break;
        }
    }
    alive = false;
    if (err) atomicExch(err, code);
}
// a walk over units: block, row tile, token tile, segment
struct FewCur {
    uint32_t u, blk;
    int m, nt, s;
    __device__ __forceinline__ FewCur(const FewPlan& p, uint32_t at) {
        u = at;
        const uint32_t tile = at / (uint32_t)p.nblk;
        blk = at - tile * (uint32_t)p.nblk;
        m = (int)(tile / (uint32_t)p.n_nt);
        nt = (int)tile - m * p.n_nt;
        s = 0;
        while (s + 1 < p.n_seg && m >= p.tile0[s + 1]) s++;
    }
    __device__ __forceinline__ void next(const FewPlan& p) {
        u++;
        if (++blk != (uint32_t)p.nblk) return;
        blk = 0;
        if (++nt != p.n_nt) return;
        nt = 0;
        if (++m >= p.tile0[s + 1] && s + 1 < p.n_seg) s++;
    }
};
struct FewBars {
    unsigned long long r_full[kFewMaxStages], r_empty[kFewMaxStages], b_full[4], b_empty[4], a_full[2], s_full[2], x_full, x_empty, m_empty;
};

template <int N>
__global__ void __launch_bounds__(kFewThreads, 1) few_gemm_kernel(const __grid_constant__ FewArgs p) {
    extern __shared__ __align__(1024) uint8_t few_smem[];
    __shared__ FewBars bars;
    __shared__ uint32_t s_tmem;
    constexpr int kA = 144, kS = 2 * kA, kMin = kS + 2 * N;       // TMEM columns: two operands (128 + 16), two accumulators, the minimum's
    constexpr uint32_t kSlab = N * 128, kStageB = 5 * kSlab;
    const FewPlan& pl = p.plan;
    uint8_t* base = few_smem + ((1024u - (umma_smem_u32(few_smem) & 1023u)) & 1023u);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t b_rf = umma_smem_u32(bars.r_full), b_re = umma_smem_u32(bars.r_empty), b_bf = umma_smem_u32(bars.b_full), b_be = umma_smem_u32(bars.b_empty);
    const uint32_t b_af = umma_smem_u32(bars.a_full), b_sf = umma_smem_u32(bars.s_full), b_me = umma_smem_u32(&bars.m_empty);
    const uint32_t b_xf = umma_smem_u32(&bars.x_full), b_xe = umma_smem_u32(&bars.x_empty);
    pdl_launch_dependents();
    if (tid == 0) {
        for (int i = 0; i < kFewMaxStages; i++) {
            u2_mbar_init(b_rf + 8u * i, 1);
            u2_mbar_init(b_re + 8u * i, 4);                // the warps of the group that unpacks the unit
        }
        for (int i = 0; i < 4; i++) {
            u2_mbar_init(b_bf + 8u * i, 1);
            u2_mbar_init(b_be + 8u * i, 1);                // tcgen05.commit
        }
        for (int i = 0; i < 2; i++) {
            u2_mbar_init(b_af + 8u * i, 4);
            u2_mbar_init(b_sf + 8u * i, 1);                // tcgen05.commit
        }
        u2_mbar_init(b_xf, 4);                             // a group's sums of a piece are in its accumulator's columns
        u2_mbar_init(b_xe, 4);                             // ... and have been read
        u2_mbar_init(b_me, 4);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == kFewMma) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(umma_smem_u32(&s_tmem)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = s_tmem;
    const uint32_t u_beg = pl.start(blockIdx.x), u_end = pl.start(blockIdx.x + 1);
    const uint32_t nblk = (uint32_t)pl.nblk, SR = (uint32_t)p.stages_raw, SB = (uint32_t)p.stages_b;
    uint8_t* sB = base;
    uint8_t* sR = base + SB * kStageB;
    bool alive = true;

    // The loader's and the MMAs' warp run their loops whole, and one elected lane issues: the operands of copies and MMAs are uniform registers, and with a
    // branch on the lane around the loop the compiler moves each operand there one at a time (45 clocks per MMA issued, 14 to 18 like this at 16 and 32 tokens).
    if (warp >= kFewLoader) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kFewRegsServe));
        if (warp == kFewLoader) {
            for (int s = 0; s < pl.n_seg; s++) asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(p.seg[s].map) : "memory");
            U2Ring rr{0u, 0u}, rb{0u, 0u};
            FewCur cr(pl, u_beg), cb = cr;                    // raw blocks, activations
            auto raw = [&]() {
                const FewSeg& sg = p.seg[cr.s];
                few_wait(b_re + 8u * rr.i, rr.ph ^ 1u, alive, p.err, 31);
                alive = __all_sync(0xffffffffu, alive);
                if (!alive) return;
                if (u2_elect()) {
                    u2_expect_tx(b_rf + 8u * rr.i, (uint32_t)(sg.pitch * 128));
                    u2_tma_2d(umma_smem_u32(sR) + rr.i * (uint32_t)p.raw_stage, sg.map, (((int)cr.blk * sg.block_bytes) & ~15) >> 2, (cr.m - pl.tile0[cr.s]) * 128, b_rf + 8u * rr.i);
                }
                __syncwarp();
                rr.next(SR);
                cr.next(pl);
            };
            while (cr.u < u_end && cr.u - u_beg < SR) raw();  // weights depend on no kernel before: requested before the wait
            pdl_wait();
            asm volatile("fence.proxy.async.global;" ::: "memory");
            while (cb.u < u_end) {
                few_wait(b_be + 8u * rb.i, rb.ph ^ 1u, alive, p.err, 32);
                alive = __all_sync(0xffffffffu, alive);
                if (!alive) break;
                if (u2_elect()) {
                    u2_expect_tx(b_bf + 8u * rb.i, kStageB);
                    few_bulk(umma_smem_u32(sB) + rb.i * kStageB, p.image + ((size_t)cb.nt * nblk + cb.blk) * kStageB, kStageB, b_bf + 8u * rb.i);
                }
                __syncwarp();
                rb.next(SB);
                cb.next(pl);
                if (cr.u < u_end) raw();
            }
            if (!alive) {      // gave up: the copies that may still be on their way land before the block ends
                bool w = true;
                const uint32_t nr = cr.u - u_beg, nb = cb.u - u_beg;
                for (uint32_t t = nr > SR ? nr - SR : 0u; t < nr; t++) few_wait(b_rf + 8u * (t % SR), (t / SR) & 1u, w, nullptr, 0);
                for (uint32_t t = nb > SB ? nb - SB : 0u; t < nb; t++) few_wait(b_bf + 8u * (t % SB), (t / SB) & 1u, w, nullptr, 0);
            }
        } else if (warp == kFewMma) {
            const uint32_t idesc = umma_idesc(128, N), idesc32 = idesc | (2u << 7) | (2u << 10);
            const uint64_t db0 = umma_desc(umma_smem_u32(sB));
            U2Ring rb{0u, 0u};
            uint32_t pieces = 0;
            for (FewCur c(pl, u_beg); c.u < u_end; c.next(pl)) {
                const uint32_t n = c.u - u_beg, g = n & 1u, ph = (n >> 1) & 1u;
                const int type = p.seg[c.s].type;
                const bool mins = type == T_Q4_K || type == T_Q5_K, first = n == 0 || c.blk == 0;
                if (first) {
                    few_wait(b_me, (pieces & 1u) ^ 1u, alive, p.err, 33);      // the minimum's accumulator has been read
                    pieces++;
                }
                few_wait(b_bf + 8u * rb.i, rb.ph, alive, p.err, 34);
                few_wait(b_af + 8u * g, ph, alive, p.err, 36);
                alive = __all_sync(0xffffffffu, alive);
                if (!alive) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t a = tmem + g * kA, acc = tmem + kS + g * N;
                const uint64_t db = db0 + (uint64_t)(rb.i * (kStageB / 16));
                if (u2_elect()) {
    #pragma unroll
                    for (int kk = 0; kk < 16; kk++)
                        few_mma_f16(acc, a + 8u * kk, db + (uint64_t)((kk >> 2) * (kSlab / 16) + 2 * (kk & 3)), idesc, kk > 0 ? 1u : 0u);
                    if (mins) {      // -dmin m (high, low part) times X_s (high, low part); low times low is below f32
                        const uint64_t dx = db + (uint64_t)(4 * (kSlab / 16));
                        few_mma_tf32(tmem + kMin, a + 128u, dx, idesc32, first ? 0u : 1u);
                        few_mma_tf32(tmem + kMin, a + 128u, dx + 2u, idesc32, 1u);
                        few_mma_tf32(tmem + kMin, a + 136u, dx, idesc32, 1u);
                    }
                    umma_commit(b_sf + 8u * g);
                    umma_commit(b_be + 8u * rb.i);
                }
                __syncwarp();
                rb.next(SB);
            }
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kFewRegsWork));
        const int g = warp >> 2, r = tid & 127;
        const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16, ta = tmem + (uint32_t)g * kA + lanes, ts = tmem + kS + (uint32_t)g * N + lanes;
        constexpr int C = N < 32 ? 8 : 16;                // columns per load from tensor memory
        const FewMask masks;
        float acc[N], d = 0.0f;
#pragma unroll
        for (int c = 0; c < N; c++) acc[c] = 0.0f;
        U2Ring rr{(uint32_t)g, 0u};
        if (rr.i >= SR) { rr.i -= SR; rr.ph ^= 1u; }
        bool waited_grid = false, undrained = false;
        uint32_t drains = 0, swaps = 0;                  // units drained, pieces whose sums one group left to the other
        auto drain = [&]() {                              // this group's unit before: its products are done, so its operand may be overwritten
            if (!undrained) return;
            undrained = false;
            few_wait(b_sf + 8u * (uint32_t)g, drains & 1u, alive, p.err, 38);
            drains++;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
            for (int c0 = 0; c0 < N; c0 += C) {
                uint32_t s[C];
                few_ld<C>(s, ts + (uint32_t)c0);
#pragma unroll
                for (int c = 0; c < C; c++) acc[c0 + c] = fmaf(d, __uint_as_float(s[c]), acc[c0 + c]);
            }
        };
        auto nothing = []() {};
        FewCur c(pl, u_beg);
        if (g == 1) c.next(pl);
        while (c.u < u_end) {
            const FewSeg& sg = p.seg[c.s];
            const int type = sg.type, residue = ((int)c.blk * sg.block_bytes) & 15;
            few_wait(b_rf + 8u * rr.i, rr.ph, alive, p.err, 39);
            const uint8_t* row = sR + rr.i * (uint32_t)p.raw_stage + r * sg.pitch;
            float dn;
            if (type == T_Q4_K) {
                dn = few_unpack_k45<false>(row, 0, ta, masks, drain);
                few_unpack_k45<false>(row, 1, ta, masks, nothing);
            } else if (type == T_Q6_K) {
                dn = few_unpack_q6(row, 0, residue, ta, masks, drain);
                few_unpack_q6(row, 1, residue, ta, masks, nothing);
            } else if (type == T_Q5_K) {
                dn = few_unpack_k45<true>(row, 0, ta, masks, drain);
                few_unpack_k45<true>(row, 1, ta, masks, nothing);
            } else {
                dn = few_unpack_q8<0>(row, ta, drain);
                few_unpack_q8<1>(row, ta, nothing);
            }
            d = dn;
            undrained = true;
            const uint32_t beg = c.u - c.blk > u_beg ? c.u - c.blk : u_beg;                       // the piece
            const uint32_t end = c.u - c.blk + nblk < u_end ? c.u - c.blk + nblk : u_end;
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            if (swaps > 0 && c.u < beg + 2u) few_wait(b_xe, (swaps - 1u) & 1u, alive, p.err, 40);  // (this unit's accumulator holds the sums left there)
            __syncwarp();
            if (lane == 0) {
                u2_mbar_arrive(b_re + 8u * rr.i);
                u2_mbar_arrive(b_af + 8u * (uint32_t)g);
            }
            rr.i += 2;
            if (rr.i >= SR) { rr.i -= SR; rr.ph ^= 1u; }
            if (c.u + 2u >= end) {                        // this group's last unit of the piece
                drain();
                if (c.u + 1u < end) {                     // the other group has the last: leave it these sums
#pragma unroll
                    for (int c0 = 0; c0 < N; c0 += 16) {
                        uint32_t s[16];
#pragma unroll
                        for (int q = 0; q < 16; q++) s[q] = __float_as_uint(acc[c0 + q]);
                        few_st16(ts + (uint32_t)c0, s);
                    }
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) u2_mbar_arrive(b_xf);
                    swaps++;                              // (both groups count the pieces of two and more units)
                } else {
                    if (end - beg > 1u) {
                        few_wait(b_xf, swaps & 1u, alive, p.err, 41);
                        swaps++;
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                        for (int c0 = 0; c0 < N; c0 += C) {
                            uint32_t s[C];
                            few_ld<C>(s, tmem + kS + (uint32_t)(g ^ 1) * N + lanes + (uint32_t)c0);
#pragma unroll
                            for (int q = 0; q < C; q++) acc[c0 + q] += __uint_as_float(s[q]);
                        }
                        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                        __syncwarp();
                        if (lane == 0) u2_mbar_arrive(b_xe);
                    }
                    if (type == T_Q4_K || type == T_Q5_K) {
#pragma unroll
                        for (int c0 = 0; c0 < N; c0 += C) {
                            uint32_t s[C];
                            few_ld<C>(s, tmem + kMin + lanes + (uint32_t)c0);
#pragma unroll
                            for (int q = 0; q < C; q++) acc[c0 + q] += __uint_as_float(s[q]);
                        }
                    }
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) u2_mbar_arrive(b_me);
                    if (!waited_grid) {                   // (what the kernel before reads of y and the workspace it has read)
                        pdl_wait();
                        waited_grid = true;
                    }
                    const int t0 = c.nt * N, left = pl.T - t0, j = (c.m - pl.tile0[c.s]) * 128 + r;
                    if (end - beg == nblk) {
                        if (j < sg.n_rows) {
                            float* y = sg.y + (size_t)t0 * sg.ldy + j;
#pragma unroll
                            for (int q = 0; q < N; q++)
                                if (q < left) y[(size_t)q * sg.ldy] = acc[q];
                        }
                    } else {
                        float* q0 = p.part + (size_t)(2u * blockIdx.x + (beg == u_beg ? 0u : 1u)) * N * 128u + r;
#pragma unroll
                        for (int q = 0; q < N; q++)
                            if (q < left) q0[q * 128] = acc[q];
                    }
                }
#pragma unroll
                for (int q = 0; q < N; q++) acc[q] = 0.0f;
            }
            c.next(pl);
            if (c.u < u_end) c.next(pl);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == kFewMma) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
    }
}

inline int few_pitch(int type) { return type == T_Q4_K ? 144 : type == T_Q5_K ? 176 : type == T_Q6_K ? 240 : 272; }      // odd multiples of 16: rows on different banks
template <int N>
inline cudaError_t few_launch_n(const FewArgs& a, size_t smem, bool pdl, cudaStream_t st) {
    static bool once[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !once[dev]) {
        const cudaError_t e = cudaFuncSetAttribute(few_gemm_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, 224 * 1024);
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64) once[dev] = true;
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)a.plan.grid); cfg.blockDim = dim3(kFewThreads); cfg.dynamicSmemBytes = smem; cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = pdl ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, few_gemm_kernel<N>, a);
}
inline cudaError_t few_launch(FewArgs& a, bool pdl, cudaStream_t st) {
    const int N = few_n(a.plan.T), stage_b = 5 * N * 128;
    int pitch = 0;
    for (int s = 0; s < a.plan.n_seg; s++) pitch = a.seg[s].pitch > pitch ? a.seg[s].pitch : pitch;
    a.raw_stage = 128 * pitch;
    a.stages_b = N == 64 ? 2 : 3;
    const int room = 222 * 1024 - 1024 - a.stages_b * stage_b, fit = room / a.raw_stage;
    a.stages_raw = fit < kFewMaxStages ? fit : kFewMaxStages;
    const size_t smem = 1024 + (size_t)a.stages_b * stage_b + (size_t)a.stages_raw * a.raw_stage;
    return N == 16 ? few_launch_n<16>(a, smem, pdl, st) : N == 32 ? few_launch_n<32>(a, smem, pdl, st) : few_launch_n<64>(a, smem, pdl, st);
}

}  // namespace b200
