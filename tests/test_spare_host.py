"""csrc/spare.cuh on the host.  With a device that has so much room, what has to be had takes the room of scratch that can be done without, once, and only
when it has to; scratch that grows a little with every portion of a conversation is allocated a few times in all."""
import os
import subprocess

import pytest

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


GROWTH = r"""
#include <cstdio>
#include "spare.cuh"
int main() {
    const size_t most = (size_t)1 << 30;
    for (size_t portion : {(size_t)4096, (size_t)100000, (size_t)7777777}) {       // portions that see a little more each time, up to the limit
        size_t have = 0;
        int times = 0;
        for (size_t want = portion; want <= most; want += portion)
            if (want > have) {
                const size_t n = grown(have, want, most);
                if (n < want || n > most) return printf("%zu -> %zu\n", want, n), 1;
                have = n;
                times++;
            }
        if (times > 20) return printf("%d allocations\n", times), 1;               // log2(1 GB / 4096) = 18, the first and the limit
    }
    return 0;
}
"""


@pytest.mark.parametrize("program", [PROGRAM, GROWTH], ids=["gives_back", "grows"])
def test_on_the_host(tmp_path, program):
    (tmp_path / "t.cpp").write_text(program)
    exe = str(tmp_path / "t")
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, "-o", exe, str(tmp_path / "t.cpp")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
