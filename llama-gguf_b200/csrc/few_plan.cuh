// few_plan.cuh — how a product of few token rows (gemm_few.cuh) is dealt to the blocks of its launch.  Plain arithmetic (compiled by the host compiler in
// tests/test_few_plan_host.py).
#pragma once
#include <stdint.h>

#if defined(__CUDACC__)
#define FEW_FN __host__ __device__ __forceinline__
#else
#define FEW_FN inline
#endif

namespace b200 {

constexpr int kFewMaxSeg = 3;

// Segment s: tiles of 128 rows of one matrix.  A unit = one tile, one token tile, one block of 256 elements of K; units run along K first, then over token
// tiles, row tiles, segments.  CTA b has the units from start(b) to start(b + 1): equal shares of the bytes (cost, in 16 bytes per row), whole units.
// The same for the kernel and for the readers of its result.
struct FewPlan {
    int n_seg, nblk, n_nt, T, grid;      // K / 256, token tiles, tokens, CTAs
    int tile0[kFewMaxSeg + 1];           // first row tile of a segment
    uint32_t cost[kFewMaxSeg];           // of a unit
    uint32_t cost0[kFewMaxSeg + 1];      // of the segments before
    FEW_FN uint32_t start(uint32_t b) const {
        const uint32_t c = cost0[n_seg] * b / (uint32_t)grid;
        int s = 0;
        while (s + 1 < n_seg && c >= cost0[s + 1]) s++;
        return (uint32_t)(tile0[s] * n_nt * nblk) + (c - cost0[s]) / cost[s];
    }
    FEW_FN int cta(int s, uint32_t u) const {      // of unit u of segment s: the last b with start(b) <= u
        const uint32_t end = cost0[s] + (u - (uint32_t)(tile0[s] * n_nt * nblk) + 1u) * cost[s];
        return (int)((end * (uint32_t)grid - 1u) / cost0[n_seg]);
    }
};
// Where rows 128 m .. of segment s are for token tile n: whole in y (b0 == b1), or in the workspace, in pieces of CTAs b0 .. b1.  A CTA has at most two pieces of cut
// tiles: the one its range begins with (slot 2 b), and the one it ends with (slot 2 b + 1, when that is another).
struct FewTile {
    int b0, b1, first;                   // first: slot of the first piece; the others begin their CTA's range
};
FEW_FN FewTile few_tile(const FewPlan& p, int s, int m, int n) {
    const uint32_t u = (uint32_t)(((p.tile0[s] + m) * p.n_nt + n) * p.nblk);
    FewTile t;
    t.b0 = p.cta(s, u);
    t.b1 = p.cta(s, u + (uint32_t)p.nblk - 1u);
    t.first = 2 * t.b0 + (t.b0 != t.b1 && p.start((uint32_t)t.b0) < u ? 1 : 0);
    return t;
}

FEW_FN int few_n(int T) { return T <= 16 ? 16 : T <= 32 ? 32 : 64; }      // tokens of a token tile

// unit_cost[s]: 16-byte words of a row of a unit.  At most n_sm CTAs, with two units each at least (so start() grows with every b, and no CTA is without work).
inline bool few_plan(FewPlan& pl, int n_seg, const int* rows, const int* unit_cost, int K, int T, int n_sm) {
    const int N = few_n(T);
    pl = FewPlan{};
    pl.n_seg = n_seg; pl.nblk = K / 256; pl.T = T; pl.n_nt = (T + N - 1) / N;
    uint64_t tiles = 0, cost = 0;
    uint32_t most = 0;
    for (int s = 0; s < n_seg; s++) {
        pl.tile0[s] = (int)tiles;
        pl.cost[s] = (uint32_t)unit_cost[s];
        pl.cost0[s] = (uint32_t)cost;
        const uint64_t nt = (uint64_t)(rows[s] + 127) / 128;
        tiles += nt;
        cost += nt * (uint64_t)pl.n_nt * (uint64_t)pl.nblk * pl.cost[s];
        if (pl.cost[s] > most) most = pl.cost[s];
        if (cost * (uint64_t)n_sm >> 32) return false;
    }
    for (int s = n_seg; s <= kFewMaxSeg; s++) {
        pl.tile0[s] = (int)tiles;
        pl.cost0[s] = (uint32_t)cost;
    }
    const uint64_t fit = cost / (2 * most);
    pl.grid = (int)(fit < (uint64_t)n_sm ? (fit ? fit : 1) : (uint64_t)n_sm);
    return true;
}

}  // namespace b200
