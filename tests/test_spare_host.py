"""csrc/spare.cuh on the host, with a device that has so much room: what has to be had takes the room of scratch that can be done without, once, and only
when it has to."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "llama-gguf_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include "spare.cuh"
int main() {
    for (int room = 0; room <= 6; room++)
        for (int scratch = 0; scratch <= 6; scratch++)
            for (int want = 1; want <= 6; want++) {
                int free_ = room, held = scratch, given = 0, asked = 0;
                const int e = alloc_or_give_back([&] { asked++; if (free_ < want) return 2; free_ -= want; return 0; },
                                                 [&] { if (!held) return false; given++; free_ += held; held = 0; return true; });
                const bool fits = want <= room, with = want <= room + scratch;
                if ((e == 0) != with || given != (!fits && scratch ? 1 : 0) || asked != (!fits && scratch ? 2 : 1) || (e && e != 2)) return printf("%d %d %d\n", room, scratch, want), 1;
            }
    return 0;
}
"""


def test_scratch_goes_before_an_allocation_fails(tmp_path):
    (tmp_path / "t.cpp").write_text(PROGRAM)
    exe = str(tmp_path / "t")
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, "-o", exe, str(tmp_path / "t.cpp")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
