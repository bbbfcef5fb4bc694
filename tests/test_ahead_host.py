"""csrc/ahead.cuh on the host: tokens of a prompt that are queued one behind the other, on a device and (for tensor-parallel contexts) two of them, whose peer may go.

The device is a clock: a step starts when it has been queued and the step before it has ended.  A step behind the peer's last one runs into its bounded wait and raises
the error words; so does every step after it.  The call has to end a few of those waits later, whatever the length of the prompt; and while nothing fails the
device must never stand idle."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "llama-gguf_b200", "csrc")

PROGRAM = r"""
#include <algorithm>
#include <cstdio>
#include "ahead.cuh"
struct Rank {
    int fails_at;                       // first step whose wait runs out
    double host = 0, end = 0, idle = 0, copied[2] = {};
    bool words = false, seen[2] = {};
    int ran = 0, marks = 0, late = 0;   // late: steps behind the first failed one
    int call(int n) {
        return run_ahead(n, [&](int i) {
                host += 0.01;
                if (i > 0 && host > end) idle += host - end;
                const bool bad = i >= fails_at;
                late += words;
                words |= bad;
                end = std::max(end, host) + (bad ? 1000.0 : 0.1);
                ran++;
                return 0;
            }, [&](int j) { copied[j] = end; seen[j] = words; marks++; return 0; },
            [&](int j) { host = std::max(host, copied[j]); return seen[j] ? 7 : 0; });
    }
};
int main() {
    for (int n = 0; n < 70; n++) {
        Rank r{1 << 30};
        if (r.call(n) != 0 || r.ran != n || r.idle > 0) return printf("%d steps: ran %d, idle %g\n", n, r.ran, r.idle), 1;
        if (n <= 2 * kAheadGroup && r.marks) return printf("%d steps: %d marks\n", n, r.marks), 1;
    }
    for (int n : {2 * kAheadGroup + 1, 30, 2000})
        for (int f = 0; f < std::min(n, 40); f++) {      // two ranks: each one's peer stops answering at the same step
            Rank a{f}, b{f};
            const int ea = a.call(n), eb = b.call(n);
            for (const Rank* r : {&a, &b})
                if (r->late > 2 * kAheadGroup - 1) return printf("%d steps, failure at %d: %d more steps\n", n, f, r->late), 1;
            if (ea != eb || (f + 2 * kAheadGroup < n && ea != 7)) return printf("%d steps, failure at %d: %d %d\n", n, f, ea, eb), 1;
        }
    int steps = 0;      // an error of a step itself ends the call at once
    if (run_ahead(20, [&](int i) { steps++; return i == 5 ? 3 : 0; }, [](int) { return 0; }, [](int) { return 0; }) != 3 || steps != 6) return printf("step error\n"), 1;
    return 0;
}
"""


def test_failures_are_noticed(tmp_path):
    (tmp_path / "t.cpp").write_text(PROGRAM)
    exe = str(tmp_path / "t")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, "-o", exe, str(tmp_path / "t.cpp")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
