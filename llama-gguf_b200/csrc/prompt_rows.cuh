// prompt_rows.cuh — where the activation rows of a pass of many rows lie in their buffer.  Plain arithmetic (compiled by the host compiler in
// tests/test_prompt_rows_host.py).
#pragma once
#include <algorithm>
#include <cstddef>

namespace b200 {

// Offsets in floats, for chunks of up to `cap` rows.  Products of up to `few` rows leave the sums that X still lacks where the gate rows go (the product they belong to
// is added before the next gate product starts): that place holds `few` rows of the wider of the two, so a model whose hidden size is above its feed-forward size has
// room for both.
struct PromptRows {
    size_t x, qkv, gate, up, xn, at, act, floats;      // f32: residual stream, q / k / v, gate (or those sums), up; fp16: normed rows, attention, gated units
};
inline PromptRows prompt_rows(size_t cap, size_t few, size_t hidden, size_t qkv, size_t attn, size_t ffn) {
    PromptRows p;
    p.x = 0;
    p.qkv = p.x + cap * hidden;
    p.gate = p.qkv + cap * qkv;
    p.up = p.gate + std::max(cap * ffn, std::min(cap, few) * hidden);
    p.xn = p.up + cap * ffn;
    p.at = p.xn + cap * hidden / 2;
    p.act = p.at + cap * attn / 2;
    p.floats = p.act + (cap * ffn + 1) / 2;
    return p;
}

}  // namespace b200
