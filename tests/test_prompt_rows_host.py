"""csrc/prompt_rows.cuh on the host: every kind of rows that a pass writes has its own place, wide enough for what is written there, inside the buffer -- also where the
hidden size is above the feed-forward size, whose sums of few rows go to the place of the gate rows."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "llama-gguf_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include "prompt_rows.cuh"
using namespace b200;
int main() {
    const size_t wide[] = {64, 256, 512, 1024, 4096, 4608, 8192, 14336};
    for (size_t cap : {32, 41, 64, 255, 256, 300, 2048})
        for (size_t hidden : wide)
            for (size_t attn : wide)
                for (size_t ffn : wide) {
                    const size_t qkv = attn + 128;
                    const PromptRows p = prompt_rows(cap, 256, hidden, qkv, attn, ffn);
                    const size_t few = cap < 256 ? cap : 256;
                    const bool ok = p.x + cap * hidden <= p.qkv && p.qkv + cap * qkv <= p.gate && p.gate + cap * ffn <= p.up && p.gate + few * hidden <= p.up &&
                                    p.up + cap * ffn <= p.xn && 2 * p.xn + cap * hidden <= 2 * p.at && 2 * p.at + cap * attn <= 2 * p.act && 2 * p.act + cap * ffn <= 2 * p.floats;
                    const bool aligned = (p.qkv | p.gate | p.up | p.xn | p.at | p.act) % 4 == 0;      // 16 bytes
                    if (!ok || !aligned) return printf("cap %zu, hidden %zu, attention %zu, ffn %zu\n", cap, hidden, attn, ffn), 1;
                }
    return 0;
}
"""


def test_places(tmp_path):
    (tmp_path / "t.cpp").write_text(PROGRAM)
    exe = str(tmp_path / "t")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, "-o", exe, str(tmp_path / "t.cpp")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
