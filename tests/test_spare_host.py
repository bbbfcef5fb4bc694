"""csrc/spare.cuh on the host.  With a device that has so much room, what has to be had takes the room of scratch that can be done without, once, and only
when it has to; scratch that grows a little with every portion of a conversation is allocated a few times in all; scratch that finds no room is asked for seldom, and again
soon after there was room once."""
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

RETRY = r"""
#include <cstdio>
#include "spare.cuh"
int main() {
    SpareRetry r;
    for (int round = 0; round < 2; round++) {
        int asked = 0, last = -1, most = 0;
        for (int call = 0; call < 1000; call++)
            if (r.due()) {
                if (last < 0 && call != 0) return printf("first asked at %d\n", call), 1;
                if (last >= 0) most = std::max(most, call - last - 1);
                last = call;
                asked++;
                r.failed();
            }
        if (asked < 1000 / 65 || asked > 1000 / 65 + 8 || most != 64) return printf("asked %d times, at most %d calls between\n", asked, most), 1;
        while (!r.due()) {}
        r.got();
    }
    return 0;
}
"""


@pytest.mark.parametrize("program", [PROGRAM, GROWTH, RETRY], ids=["gives_back", "grows", "asks_again"])
def test_on_the_host(tmp_path, program):
    (tmp_path / "t.cpp").write_text(program)
    exe = str(tmp_path / "t")
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, "-o", exe, str(tmp_path / "t.cpp")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
