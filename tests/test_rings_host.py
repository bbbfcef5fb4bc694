"""csrc/ring.cuh on the host: a loader that gives up waits for exactly the copies that may still land.  The barriers are simulated (a stage's phase number, completed
by each copy that lands); the loaders of the two prompt-attention kernels are checked for counting each ring by what they asked for."""
import os
import re
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "llama-gguf_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <vector>
#include "ring.cuh"
// copies 0 .. asked - 1 of a ring of N have been asked for; the first `landed` in flight order have landed.  A wait for (stage, parity) returns at once when the
// stage's current phase has the other parity; else it lets copies land until it may return.  0: nothing is in flight afterwards.
template <int N> int left(int asked, int landed) {
    std::vector<int> phase(N, 0);
    for (int t = 0; t < landed; t++) phase[t % N]++;
    int next = landed;
    ring_in_flight<N>(asked, [&](int stage, unsigned parity) {
        while ((unsigned)(phase[stage] & 1) == parity && next < asked) phase[next++ % N]++;
    });
    return asked - next;
}
int main() {
    for (int asked = 0; asked < 200; asked++)
        for (int late = 0; late <= asked; late++) {
            if (late <= 2 && left<2>(asked, asked - late)) return printf("2 stages: %d asked, %d late\n", asked, late), 1;
            if (late <= 3 && left<3>(asked, asked - late)) return printf("3 stages: %d asked, %d late\n", asked, late), 1;
        }
    return 0;
}
"""


def test_every_copy_in_flight_is_waited_for(tmp_path):
    (tmp_path / "t.cpp").write_text(PROGRAM)
    exe = str(tmp_path / "t")
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, "-o", exe, str(tmp_path / "t.cpp")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


@pytest.mark.parametrize("name", ["lp_tile_attn.cuh", "attn_umma.cuh"])
def test_loaders_count_what_they_asked_for(name):
    """Each ring's count moves right behind its copy (before the next wait, which may give up), and both rings are landed."""
    text = open(os.path.join(CSRC, name)).read()
    loader = text.split("int asked_k = 0, asked_v = 0;")[1]
    loader = loader[:loader.index("id_s" if name.startswith("lp") else "idS")]
    order = re.findall(r"(k_empty|v_empty|k_full|v_full) \+ 8u \* b|(asked_[kv]) = |land\((k_full|v_full), (asked_[kv])\)", loader)
    seen = [next(x for x in o if x) if not o[3] else (o[2], o[3]) for o in order]
    first = {}
    for i, x in enumerate(seen):
        first.setdefault(x, i)
    last_copy = {r: max(i for i, x in enumerate(seen) if x == r) for r in ("k_full", "v_full")}
    assert first["k_empty"] < last_copy["k_full"] < first["asked_k"] < first["v_empty"] < last_copy["v_full"] < first["asked_v"]
    assert first[("k_full", "asked_k")] > first["asked_v"] and first[("v_full", "asked_v")] > first["asked_v"]
