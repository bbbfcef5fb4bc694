"""csrc/few_plan.cuh on the host: the deal of units to blocks is a partition, readers find every piece of a cut tile in its slot and in the order of K.  A matrix that
can be dealt at 256 rows can be at any smaller number: what the engine asks once, before it lets a model take these products."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "llama-gguf_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <map>
#include <vector>
#include "few_plan.cuh"
using namespace b200;
static unsigned long long st = 12345;
static int rnd(int n) { st = st * 6364136223846793005ull + 1442695040888963407ull; return (int)((st >> 33) % (unsigned)n); }
static int check(int n_seg, const int* rows, const int* cost, int K, int T) {
    FewPlan p;
    if (!few_plan(p, n_seg, rows, cost, K, T, 148)) return 0;
    const uint32_t units = (uint32_t)p.tile0[n_seg] * p.n_nt * p.nblk;
    if (p.start(0) != 0 || p.start(p.grid) != units || p.grid < 1 || p.grid > 148) return 1;
    std::map<int, std::pair<uint32_t, uint32_t>> slots;      // slot -> units
    for (int b = 0; b < p.grid; b++) {
        if (p.start(b) >= p.start(b + 1)) return 2;
        for (uint32_t u = p.start(b); u < p.start(b + 1);) {
            const uint32_t t0 = u / p.nblk * p.nblk, e = t0 + p.nblk < p.start(b + 1) ? t0 + p.nblk : p.start(b + 1);
            if (u != t0 || e != t0 + p.nblk) {
                const int slot = 2 * b + (u == p.start(b) ? 0 : 1);
                if (slots.count(slot)) return 3;
                slots[slot] = {u, e};
            }
            u = e;
        }
    }
    for (int s = 0; s < n_seg; s++)
        for (int m = 0; m < p.tile0[s + 1] - p.tile0[s]; m++)
            for (int n = 0; n < p.n_nt; n++) {
                const FewTile t = few_tile(p, s, m, n);
                uint32_t u = (uint32_t)((p.tile0[s] + m) * p.n_nt + n) * p.nblk;
                const uint32_t e = u + p.nblk;
                if (t.b0 == t.b1) {      // whole: one CTA has it all, and no slot
                    if (p.start(t.b0) > u || p.start(t.b0 + 1) < e) return 4;
                    continue;
                }
                for (int b = t.b0; b <= t.b1; b++) {
                    const int slot = b == t.b0 ? t.first : 2 * b;
                    if (!slots.count(slot) || slots[slot].first != u) return 5;
                    u = slots[slot].second;
                }
                if (u != e) return 6;
            }
    return 0;
}
int main() {
    const int widths[] = {1, 64, 127, 128, 129, 256, 1000, 1024, 4096, 14336, 32000}, costs[] = {9, 11, 15, 17};
    for (int i = 0; i < 4000; i++) {
        int rows[3], cost[3], n = 1 + rnd(3);
        for (int s = 0; s < n; s++) {
            rows[s] = rnd(2) ? widths[rnd(11)] : 1 + rnd(20000);
            cost[s] = costs[rnd(4)];
        }
        const int K = 256 * (1 + (rnd(4) ? rnd(60) : rnd(4))), T = 1 + rnd(256);
        if (int r = check(n, rows, cost, K, T)) return printf("%d: %d segments, rows %d, K %d, T %d\n", r, n, rows[0], K, T), 1;
    }
    for (int rows : {128256, 1 << 20, 1 << 21, 3 << 20})
        for (int K : {4096, 8192, 28672}) {
            FewPlan p;
            const int cost = 17;
            const bool most = few_plan(p, 1, &rows, &cost, K, 256, 148);
            if (most != ((rows + 127) / 128 * 4ull * (K / 256) * 17 * 148 < 1ull << 32)) return printf("bound: rows %d, K %d\n", rows, K), 1;
            for (int T = 1; T <= 256; T++)
                if (most && !few_plan(p, 1, &rows, &cost, K, T, 148)) return printf("rows %d, K %d: %d tokens\n", rows, K, T), 1;
        }
    return 0;
}
"""


def test_plan(tmp_path):
    (tmp_path / "t.cpp").write_text(PROGRAM)
    exe = str(tmp_path / "t")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, "-o", exe, str(tmp_path / "t.cpp")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
