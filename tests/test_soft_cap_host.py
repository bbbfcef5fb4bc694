"""csrc/soft_cap.cuh on the host, in f32: tanh of small arguments is off by a few 1e-8 of itself (2 ulp = 2.4e-7), down to the smallest."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "llama-gguf_b200", "csrc")

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include <initializer_list>
#include "soft_cap.cuh"
int main() {
    double worst = 0.0;
    for (int i = 0; i <= 2000000; i++) {
        const float x = SOFT_CAP_SMALL * (float)i / 2000000.0f;
        for (float v : {x, -x, x * 1e-6f, x * 1e-30f}) {
            const double want = std::tanh((double)v), d = std::fabs((double)tanh_small(v) - want);
            if (want != 0.0) worst = std::fmax(worst, d / std::fabs(want));
            else if (d != 0.0) return printf("%g\n", v), 1;
        }
    }
    printf("%g\n", worst);
    return worst < 2.4e-7 ? 0 : 1;
}
"""


def test_small_arguments_keep_their_relative_precision(tmp_path):
    (tmp_path / "t.cpp").write_text(PROGRAM)
    exe = str(tmp_path / "t")
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", CSRC, "-o", exe, str(tmp_path / "t.cpp")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
