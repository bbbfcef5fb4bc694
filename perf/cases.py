"""Workloads to time: what programs that use this package have it do, through its public entry points.

GGUF models (GpuOnlyInference): prompts through forward_batch, decoding through forward (one sequence) and decode_batch (many), over
block types, block sizes, cache formats and experts.  Layer-program models (LayerProgramInference): prompts through step, decoding through
forward and decode_batch.  Every pass starts from empty sequence slots (reset) and is fed given tokens, so that it can be repeated and its
logits compared.  Weights are random: N(0, 1 / fan_in) for bf16 matrices, random blocks of the same spread for GGUF matrices.

`exact` restates each model in float64 with torch, whole sequences at a time."""
import math
import zlib

import numpy as np
import torch

import llama_gguf_b200 as B
from llama_gguf_b200 import gefovik, lazilorn, madudra, mefurax
from llama_gguf_b200.presets import PRESETS, make_desc, tensor_plan

DESIGNS = {"gefovik": gefovik, "lazilorn": lazilorn, "madudra": madudra, "mefurax": mefurax}


# ---------------------------------------------------------------------------------------------------------------- cases
def listed():
    return [
        # a short chat turn with an 8B model: the prompt, then the answer token by token with host logits (the headline model, whole)
        dict(name="chat_8b", family="gguf", preset="llama-3-8b", layers=32, vocab=128256, mix="Q4_K_M", kv="f32", batch=1, prompt=128, decode=16),
        # the smallest call: a few tokens through two layers of a 0.5B model with the int8 cache
        dict(name="small_chat_int8", family="gguf", preset="qwen2.5-0.5b", layers=2, vocab=4096, mix="Q4_K_M", kv="int8", batch=1, prompt=5, decode=4),
        # a full prompt chunk through two 8B-shaped layers
        dict(name="prompt_2048", family="gguf", preset="llama-3-8b", layers=2, vocab=4096, mix="Q4_K_M", kv="f32", batch=1, prompt=2048, decode=0),
        # an ordinary prompt of odd length through a small model's layers in Q8_0
        dict(name="prompt_333_q8", family="gguf", preset="tinyllama-1.1b", layers=4, vocab=4096, mix="Q8_0", kv="f32", batch=1, prompt=333, decode=0),
        # a long document and an answer about it: prompt and decoding with many keys
        dict(name="document_6000", family="gguf", preset="llama-3-8b", layers=2, vocab=4096, mix="Q4_K_M", kv="f32", batch=1, prompt=6000, decode=24),
        # a server's decode steps: 32 sequences at once through four 8B-shaped layers
        dict(name="batch_32", family="gguf", preset="llama-3-8b", layers=4, vocab=4096, mix="Q4_K_M", kv="f32", batch=32, prompt=0, decode=6),
        # decoding with a mixture of experts, one layer of 8 experts
        dict(name="experts_decode", family="gguf", preset="mixtral-8x7b", layers=1, vocab=4096, mix="Q5_K_M", kv="f32", batch=1, prompt=0, decode=8),
        # a scored prompt (every 16th row's logits) through softmax + latent attention, gated layers and experts
        dict(name="gefovik_prompt_2048", family="gefovik", width=2048, pattern="aD,lM", heads=16, kv_heads=4, ff=8192, eff=2048, vocab=2048, lens="2048",
             decode=0, stride=16, compute="bfloat16"),
        # three prompts of odd lengths in one step: rotary and windowed mixers, experts beside an always-on one
        dict(name="mefurax_prompts", family="mefurax", width=1024, pattern="b,b,a", heads=8, kv_heads=2, ff=4096, eff=1024, vocab=2048, lens="777,130,41",
             decode=0, stride=8, compute="bfloat16"),
        # a prompt through both recurrent mixers: windowed attention beside a matrix memory, gated delta rule
        dict(name="lazilorn_prompt_1500", family="lazilorn", width=1024, pattern="p,d", heads=8, kv_heads=2, ff=4096, eff=0, vocab=2048, lens="1500",
             decode=0, stride=16, compute="bfloat16"),
        # one sequence: prompt and answer through latent attention, state-space layers, residual streams and experts
        dict(name="madudra_chat", family="madudra", width=1024, pattern="l,m,m,k", heads=8, kv_heads=0, ff=0, eff=1024, vocab=2048, lens="300", decode=24,
             stride=64, compute="bfloat16"),
        # a server's step: 32 prompts together, then decode steps of all
        dict(name="gefovik_batch_32", family="gefovik", width=2048, pattern="aD,lM", heads=16, kv_heads=4, ff=8192, eff=2048, vocab=2048,
             lens=",".join(["48"] * 32), decode=8, stride=48, compute="bfloat16"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["prompt", "prompt", "chat", "batch", "experts", "lp_prompt", "lp_prompt", "lp_chat", "lp_batch"])
    if kind in ("prompt", "chat", "batch", "experts"):
        c = dict(family="gguf", preset=rng.choice(["llama-3-8b", "tinyllama-1.1b", "qwen2.5-0.5b"]), layers=rng.choice([1, 2, 3, 4]),
                 vocab=rng.choice([2048, 4096, 5000, 8192]), mix=rng.choice(["Q4_K_M", "Q4_K_M", "Q8_0", "Q6_K", "Q5_K_M"]), kv="f32", batch=1)
        if c["preset"] == "qwen2.5-0.5b":
            c["mix"] = rng.choice(["Q4_K_M", "Q8_0"])
        if kind == "prompt":
            c.update(prompt=_log(rng, 33, 4000), decode=0)
        elif kind == "chat":
            c.update(prompt=_log(rng, 2, 2000), decode=rng.randint(2, 24), kv=rng.choice(["f32", "f32", "int8"]))
            if c["kv"] == "int8":
                c["prompt"] = min(c["prompt"], 40 + c["prompt"] % 20)
        elif kind == "batch":
            c.update(preset=rng.choice(["llama-3-8b", "tinyllama-1.1b"]), batch=_log(rng, 2, 64), prompt=0, decode=rng.randint(2, 8))
        else:
            c.update(preset="mixtral-8x7b", layers=1, mix=rng.choice(["Q5_K_M", "Q4_K_M"]), prompt=0, decode=rng.randint(2, 16))
        return c
    f = rng.choice(["gefovik", "mefurax", "lazilorn", "madudra"])
    w = rng.choice([1024, 2048])
    pattern = {"gefovik": ["aD,lM", "aM,lD", "aD,aM", "lM,lD"], "mefurax": ["b,b,a", "b,a", "a,b"], "lazilorn": ["p,d", "d,p", "p"],
               "madudra": ["l,m,k", "l,m,m,k", "l,m"]}[f]
    c = dict(family=f, width=w, pattern=rng.choice(pattern), heads=w // 128, kv_heads=0 if f == "madudra" else w // 512,
             ff=0 if f == "madudra" else 4 * w, eff=0 if f == "lazilorn" else w, vocab=2048, compute="bfloat16")
    if kind == "lp_prompt":
        lens = [_log(rng, 33, 3000)] + [_log(rng, 17, 400) for _ in range(rng.choice([0, 0, 1, 2]))]
        c.update(lens=",".join(map(str, lens)), decode=0, stride=rng.choice([8, 16, 32]))
    elif kind == "lp_chat":
        c.update(lens=str(_log(rng, 2, 1500)), decode=rng.randint(4, 32), stride=64, compute=rng.choice(["bfloat16", "bfloat16", "bfloat16", "float32"]))
        if c["compute"] == "float32":
            c["lens"] = str(min(int(c["lens"]), 200 + int(c["lens"]) % 57))
    else:
        n = _log(rng, 2, 48)
        c.update(lens=",".join(str(rng.randint(8, 64)) for _ in range(n)), decode=rng.randint(2, 10), stride=64)
    return c


# ---------------------------------------------------------------------------------------------------------------- inputs
def _gen(seed, name):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1000003 + zlib.crc32(name.encode())) & 0x7FFFFFFFFFFFFFFF)
    return g


def _randn(seed, name, *shape):
    return torch.randn(shape, generator=_gen(seed, name), device="cuda")


def _tokens(seed, name, n, vocab):
    return np.random.default_rng([int(seed), zlib.crc32(name.encode())]).integers(0, vocab, n).astype(np.uint32)


def _f16(v):
    return int(np.array([v], dtype=np.float16).view(np.int16)[0])


def _preset(case):
    return dict(PRESETS[case["preset"]], n_layers=case["layers"], vocab=case["vocab"])


def _gguf_tensor(seed, name, ttype, ne):
    """On the device: f32 values, or int16 words of the blocks [blocks, words]."""
    n = int(np.prod(ne))
    if name.endswith("norm.weight"):
        return 1.0 + 0.1 * _randn(seed, name, n)
    if name.endswith(".bias"):
        return 0.1 * _randn(seed, name, n)
    sigma = 1.0 if name == "token_embd.weight" else ne[0] ** -0.5
    if ttype == B.F32:
        return sigma * _randn(seed, name, n)
    be, bb = B.BLOCK[ttype]
    raw = torch.randint(-32768, 32768, (n // be, bb // 2), generator=_gen(seed, name), device="cuda", dtype=torch.int16)
    at, scales = {B.Q4_K: (0, (sigma / 200.0, 7.5 * sigma / 200.0)), B.Q5_K: (0, (sigma / 400.0, 15.5 * sigma / 400.0)),
                  B.Q6_K: (104, (sigma / 1400.0,)), B.Q8_0: (0, (sigma / 74.0,)), B.Q5_0: (0, (sigma / 9.2,))}[ttype]
    for k, s in enumerate(scales):
        raw[:, at + k] = _f16(s)
    return raw


def _lp_config(case):
    s, mid = case, []
    W = s["width"]
    for ch in s["pattern"].split(","):
        if s["family"] == "gefovik":
            mlp = {"kind": "dense", "ff": s["ff"]} if ch[1] == "D" else {"kind": "moe", "router": {"experts": 8, "identity": 2, "top": 2}, "expert": {"ff": s["eff"]}}
            if ch[0] == "a":
                mid.append({"type": "attention", "mlp": mlp, "mixer": {"heads": s["heads"], "kv_heads": s["kv_heads"], "dim": 128, "vdim": 128,
                                                                       "scale": 128 ** -0.5, "softcap": 50.0, "q_temp": {"coef": 0.1, "every": 1024}}})
            else:
                mid.append({"type": "latent_attention", "mlp": mlp, "mixer": {"heads": s["heads"], "dim": 96, "vdim": 128, "kv_rank": 128, "scale": 96 ** -0.5}})
        elif s["family"] == "mefurax":
            mlp = {"kind": "dense", "ff": s["ff"]} if not mid else {"kind": "moe", "router": {"experts": 8, "top": 2}, "expert": {"ff": s["eff"]}, "shared": {"ff": s["eff"]}}
            m = {"heads": s["heads"], "kv_heads": s["kv_heads"], "dim": 128, "vdim": 128, "mask": {"size": 1024}, "scale": 128 ** -0.5, "v_mix": True}
            m.update({"conv": 4} if ch == "a" else {"rot": {"dims": 64, "base": 10000.0}, "softcap": 50.0})
            mid.append({"type": "attention" if ch == "a" else "attention_2", "mixer": m, "mlp": mlp})
        elif s["family"] == "lazilorn":
            mlp = {"kind": "dense", "ff": s["ff"]}
            if ch == "p":
                mid.append({"type": "parallel", "mlp": mlp,
                            "mixer": {"left": {"heads": s["heads"], "kv_heads": s["kv_heads"], "dim": 128, "vdim": 128, "mask": {"size": 1024, "keep_first": 4},
                                               "scale": 128 ** -0.5},
                                      "right": {"heads": s["heads"] // 2, "dim": 64, "vdim": 128, "gate_cap": 15.0}, "left_scale": 0.7, "right_scale": 0.7}})
            else:
                mid.append({"type": "delta", "mlp": mlp, "mixer": {"heads": s["heads"], "kv_heads": s["kv_heads"], "dim": 128, "vdim": 128, "conv": 4}})
        else:
            mlp = {"kind": "moe", "router": {"experts": 8, "top": 2, "scale": 1.0}, "expert": {"ff": s["eff"]}}
            if ch == "m":
                mid.append({"type": "mamba2", "mlp": mlp, "mixer": {"heads": W // 64, "vdim": 128, "state": 128, "groups": 1, "conv": 4, "norm_groups": 1}})
            else:
                m = {"heads": s["heads"], "dim": 64, "rot_dim": 32, "vdim": 128, "q_rank": 512 if W == 1024 else 768, "kv_rank": 96, "mask": {"size": 1024},
                     "scale": 96 ** -0.5, "rot": {"dims": 32, "base": 10000.0, "scaling": {"factor": 4.0, "original": 4096, "fast": 32.0, "slow": 1.0}}}
                if ch == "k":
                    m["kv_from"] = 0
                mid.append({"type": "latent_attention", "mixer": m, "mlp": mlp})
    cfg = {"architecture": s["family"].capitalize(), "width": W, "vocab": s["vocab"], "norm": {"eps": 1e-6}, "embedding": {"scale": 1.0}, "layers": mid}
    cfg.update({"lazilorn": {"logit_scale": 1.0, "loop": {"start": 0, "stop": 0, "times": 1}}, "mefurax": {"postln_alpha": 2.0},
                "madudra": {"residual_mult": 0.5, "streams": 4}}.get(s["family"], {}))
    return cfg


def _lp_tensor(cfg, seed, name, shape):
    last = name.split(".")[-1]
    if ".hc" in name:
        if last == "mix":
            return torch.eye(shape[0], device="cuda") + 0.05 * _randn(seed, name, *shape)
        return torch.full(shape, 1.0 / shape[0] if last == "in" else 1.0, device="cuda")
    r = _randn(seed, name, *shape)
    if name == "embed":      # rows lean towards two experts of every mixture, as trained routers are decided on most tokens (near ties would be coin tosses)
        for i, L in enumerate(cfg["layers"]):
            if L["mlp"]["kind"] == "moe":
                n = L["mlp"]["router"]["experts"] + L["mlp"]["router"].get("identity", 0)
                router = _lp_tensor(cfg, seed, "l%d.mlp.router" % i, (n, shape[1])).float()
                two = torch.rand((shape[0], n), generator=_gen(seed, "choice%d" % i), device="cuda").topk(2, -1)[1]
                r = r + 8.0 * router[two[:, 0]] + 7.5 * router[two[:, 1]]
        return r.bfloat16()
    if len(shape) == 2 and last != "conv":
        return (r * shape[-1] ** -0.5).bfloat16()
    if last == "conv":
        return 0.5 * r
    if name.endswith("f.b"):
        return 2.5 + 0.5 * r
    if last in ("A_log", "dt_bias", "b") and len(shape) == 1:
        return 0.5 * r - 0.75
    if last == "correction":
        return 0.1 * r
    if cfg["architecture"] == "Mefurax" and (last in ("norm1", "norm2", "vmix") or name == "final.norm"):
        return 0.1 * r + (0.4 if last == "vmix" else 0.0)
    return 1.0 + 0.1 * r


def _lens(case):
    return [int(v) for v in case["lens"].split(",")]


def _lp_want(case):
    """Rows of the prompt step whose logits are asked for: every `stride`th of a run and its last."""
    want, at = [], 0
    for n in _lens(case):
        want += [at + r for r in range(n) if r % case["stride"] == case["stride"] - 1 or r == n - 1]
        at += n
    return want


def _lp_inputs(case, seed):
    lens = _lens(case)
    return [_tokens(seed, "prompt%d" % i, n, case["vocab"]) for i, n in enumerate(lens)], [_tokens(seed, "step%d" % t, len(lens), case["vocab"]) for t in range(case["decode"])]


def prepare(case, seed):
    if case["family"] == "gguf":
        p = _preset(case)
        desc = make_desc(p, max(64, case["prompt"] + case["decode"] + 8), case["batch"])

        def feed(upload):
            for name, t, ne in tensor_plan(p, case["mix"]):
                upload(name, t, ne, _gguf_tensor(seed, name, t, ne).cpu().numpy())
        gpu = B.GpuOnlyInference(desc, None, feeder=feed, kv_format=case["kv"])
        prompt = _tokens(seed, "prompt", case["prompt"], case["vocab"])
        steps = [_tokens(seed, "step%d" % t, case["batch"], case["vocab"]) for t in range(case["decode"])]
        return dict(case=case, gpu=gpu, prompt=prompt, steps=steps)
    cfg, mod = _lp_config(case), DESIGNS[case["family"]]
    lens = _lens(case)
    program, layers = mod.parse_config(cfg, max(lens) + case["decode"] + 8, len(lens), case["compute"])

    def feed(upload):
        for name, shape in mod.tensor_shapes(cfg).items():
            t = _lp_tensor(cfg, seed, name, shape)
            ne = list(reversed(shape)) if shape else [1]
            if t.dtype == torch.bfloat16:
                upload(name, B.BF16, ne, t.view(torch.int16).cpu().numpy().view(np.uint16))
            else:
                upload(name, B.F32, ne, t.reshape(shape or (1,)).cpu().numpy())
    gpu = B.LayerProgramInference(program, layers, feeder=feed)
    prompts, steps = _lp_inputs(case, seed)
    return dict(case=case, gpu=gpu, runs=[(i, [int(x) for x in t]) for i, t in enumerate(prompts)], want=_lp_want(case), steps=steps)


def run(state):
    case, gpu, out = state["case"], state["gpu"], []
    if case["family"] == "gguf":
        n = case["batch"]
        for s in range(n):
            gpu.reset(s)
        if case["prompt"]:
            out.append(gpu.forward_batch(state["prompt"]))
    else:
        n = len(state["runs"])
        for s in range(n):
            gpu.reset(s)
        out.append(gpu.step(state["runs"], state["want"]))
    for t in state["steps"]:
        out.append(gpu.forward(int(t[0])) if n == 1 else gpu.decode_batch(list(range(n)), t))
    return out


# ---------------------------------------------------------------------------------------------------------------- work and tolerance
def work(case):
    """Bytes: weights once per call that uses them (calls follow one another), cached rows a decoded token reads, logits.  Operations: products of
    the weights a token meets, scores and sums of attention."""
    if case["family"] == "gguf":
        p = _preset(case)
        body = body_bytes = head = head_bytes = 0.0
        for name, t, ne in tensor_plan(p, case["mix"]):
            n = float(np.prod(ne))
            if len(ne) == 3:
                n *= p["n_experts_used"] / p["n_experts"]
            be, bb = B.BLOCK[t]
            if name == "output.weight" or (p.get("tied") and name == "token_embd.weight"):
                head, head_bytes = n, n / be * bb
            elif name != "token_embd.weight":
                body, body_bytes = body + n, body_bytes + n / be * bb
        P, D, nb, L = case["prompt"], case["decode"], case["batch"], case["layers"]
        keys = sum(range(1, P + 1)) + nb * sum(range(P + 1, P + D + 1))
        calls = (1 if P else 0) + D
        row = 2 * p["n_kv_heads"] * p["head_dim"] * (1 if case["kv"] == "int8" else 4)
        rows_out = (1 if P else 0) + nb * D
        flops = 2.0 * body * (P + nb * D) + 2.0 * head * rows_out + 4.0 * L * p["n_heads"] * p["head_dim"] * keys
        nbytes = calls * (body_bytes + head_bytes) + L * row * (P + nb * sum(range(P + 1, P + D + 1))) + 4.0 * rows_out * case["vocab"]
        return {"bytes": nbytes, "flops": flops}
    cfg, mod = _lp_config(case), DESIGNS[case["family"]]
    size = 4 if case["compute"] == "float32" else 2
    dense = expert = head = 0.0
    for name, shape in mod.tensor_shapes(cfg).items():
        n = float(np.prod(shape)) if len(shape) == 2 else 0.0
        if name == "head" or (name == "embed" and case["family"] == "gefovik"):
            head = n
        elif ".mlp.e" in name:
            expert += n
        elif name != "embed":
            dense += n
    lens, D = _lens(case), case["decode"]
    n_prompt, want = sum(lens), len(_lp_want(case))
    rows = n_prompt + len(lens) * D
    flops = 2.0 * (dense + expert * 2 / 8) * rows + 2.0 * head * (want + len(lens) * D)
    for L in cfg["layers"]:
        m = L["mixer"].get("left", L["mixer"])
        if L["type"] in ("mamba2", "delta"):
            flops += 6.0 * m["heads"] * m["vdim"] * (m.get("state") or m["dim"]) * rows
            continue
        if "right" in L["mixer"]:
            r = L["mixer"]["right"]
            flops += 6.0 * r["heads"] * r["dim"] * r["vdim"] * rows
        span = (m.get("mask") or {}).get("size", 1 << 30)
        keys = sum(min(i + 1, span) for n in lens for i in range(n + D))
        flops += 2.0 * m["heads"] * (m["dim"] + m.get("rot_dim", 0) + m["vdim"]) * keys
    met = min(1.0, 2 * len(lens) / 8)
    nbytes = size * (dense + expert + head) + D * size * (dense + expert * met + head) + 4.0 * (want + len(lens) * D) * case["vocab"]
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """About four times the distance to `exact`: 32-bit sums 1e-6 (a few per call in a row), fp16 operands of prompts and of 8 and more sequences
    1.1e-3, a changed rounding of int8 cache rows 5e-3 to 2e-2, bf16 activations through two to four layers 4e-3."""
    if case["family"] == "gguf":
        if case["kv"] == "int8":
            return {"rel": 0.03, "max": 0.4}
        return {"rel": 4.5e-3, "max": 0.05} if case["prompt"] >= 32 or case["batch"] >= 8 else {"rel": 1e-5, "max": 3e-4}
    if case["compute"] == "float32":
        return {"rel": 2e-5, "max": 1e-3}
    return {"rel": 0.016, "max": 0.4}


# ---------------------------------------------------------------------------------------------------------------- in 64 bits
F = torch.float64


def _dequant(raw, ttype, ne):
    """Block words on the device -> float64 [rows, ne0] (one more leading axis for experts)."""
    if raw.dtype != torch.int16:
        return raw.to(F).reshape(list(reversed(ne)))
    u = raw.view(torch.uint8)
    half = lambda at: raw[:, at:at + 1].contiguous().view(torch.float16).to(F)  # noqa: E731
    if ttype in (B.Q4_K, B.Q5_K):
        d, dm, sb = half(0), half(1), u[:, 4:16].to(torch.int32)
        sc, mn = [], []
        for j in range(8):
            if j < 4:
                sc.append(sb[:, j] & 63)
                mn.append(sb[:, j + 4] & 63)
            else:
                sc.append((sb[:, j + 4] & 15) | ((sb[:, j - 4] >> 6) << 4))
                mn.append((sb[:, j + 4] >> 4) | ((sb[:, j] >> 6) << 4))
        qs = u[:, -128:].reshape(-1, 4, 32)
        q = torch.stack([qs & 15, qs >> 4], 2).reshape(-1, 8, 32)
        if ttype == B.Q5_K:
            qh = u[:, 16:48].unsqueeze(1)
            q = q + 16 * ((qh >> torch.arange(8, device="cuda", dtype=torch.uint8).view(1, 8, 1)) & 1)
        w = (d * torch.stack(sc, 1).to(F)).unsqueeze(2) * q.to(F) - (dm * torch.stack(mn, 1).to(F)).unsqueeze(2)
    elif ttype == B.Q6_K:
        ql, qh = u[:, :128].reshape(-1, 2, 64), u[:, 128:192].reshape(-1, 2, 32)
        sc = u[:, 192:208].view(torch.int8).to(F).reshape(-1, 2, 8)
        parts = []
        for k in range(4):
            lo = ql[:, :, (k & 1) * 32:(k & 1) * 32 + 32]
            lo = (lo & 15) if k < 2 else (lo >> 4)
            q = (lo | (((qh >> (2 * k)) & 3) << 4)).to(F) - 32.0
            parts.append(q * sc[:, :, 2 * k:2 * k + 2].repeat_interleave(16, 2))
        w = half(104).unsqueeze(2) * torch.cat(parts, 2)
    elif ttype == B.Q8_0:
        w = half(0) * u[:, 2:].view(torch.int8).to(F)
    else:
        bits = u[:, 2:6].to(torch.int64)
        qh = bits[:, 0] | (bits[:, 1] << 8) | (bits[:, 2] << 16) | (bits[:, 3] << 24)
        hi = ((qh.unsqueeze(1) >> torch.arange(32, device="cuda")) & 1) << 4
        q = torch.cat([u[:, 6:] & 15, u[:, 6:] >> 4], 1).to(torch.int64) | hi
        w = half(0) * (q.to(F) - 16.0)
    return w.reshape(list(reversed(ne)))


def _rms(x, w, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _ln(x, w, eps):
    x = x - x.mean(-1, keepdim=True)
    return _rms(x, w, eps)


def _attend(q, k, v, scale, see=None, bias=None, cap=0.0, sink=None):
    """q [T, H, d], k [T, G, d], v [T, G, dv] -> [T, H, dv]; see(i, j): which keys, beside j <= i; 512 queries at a time."""
    T, H, _ = q.shape
    kk, vv = (x.repeat_interleave(H // x.shape[1], 1).transpose(0, 1) for x in (k, v))
    out = []
    for a in range(0, T, 512):
        b = min(T, a + 512)
        i, j = torch.arange(a, b, device="cuda").view(-1, 1), torch.arange(b, device="cuda").view(1, -1)
        s = q[a:b].transpose(0, 1) @ kk[:, :b].transpose(1, 2) * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        if bias is not None:
            s = s - bias.view(-1, 1, 1) * (i - j)
        ok = (j <= i) if see is None else (j <= i) & see(i, j)
        s = s.masked_fill(~ok, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink.view(-1, 1, 1).expand(H, b - a, 1)], 2)
        pr = torch.softmax(s, 2)[:, :, :b]
        out.append((pr @ vv[:, :b]).transpose(0, 1))
    return torch.cat(out)


def _turn(x, freqs, pairs, mult=1.0):
    """x [T, H, d]: position t turns the first 2 len(freqs) channels; pairs: neighbours (2i, 2i + 1), else (i, i + half)."""
    n = len(freqs)
    a = torch.arange(x.shape[0], device="cuda", dtype=F).view(-1, 1, 1) * torch.tensor(freqs, device="cuda", dtype=F)
    c, s = torch.cos(a) * mult, torch.sin(a) * mult
    u, w = (x[..., 0:2 * n:2], x[..., 1:2 * n:2]) if pairs else (x[..., :n], x[..., n:2 * n])
    out = x.clone()
    if pairs:
        out[..., 0:2 * n:2], out[..., 1:2 * n:2] = u * c - w * s, w * c + u * s
    else:
        out[..., :n], out[..., n:2 * n] = u * c - w * s, w * c + u * s
    return out


def _exact_gguf(case, seed):
    p = _preset(case)
    plan = {name: (t, ne) for name, t, ne in tensor_plan(p, case["mix"])}
    get = lambda name: _dequant(_gguf_tensor(seed, name, *plan[name]), *plan[name])  # noqa: E731
    eps, hd, nh, nkv = p["norm_eps"], p["head_dim"], p["n_heads"], p["n_kv_heads"]
    freqs = [p["rope_base"] ** (-2.0 * i / hd) for i in range(hd // 2)]
    prompt = _tokens(seed, "prompt", case["prompt"], case["vocab"])
    steps = [_tokens(seed, "step%d" % t, case["batch"], case["vocab"]) for t in range(case["decode"])]
    emb = get("token_embd.weight")
    seqs = [np.concatenate([prompt] + [s[b:b + 1] for s in steps]) for b in range(case["batch"])]
    xs = [emb[torch.from_numpy(s.astype(np.int64)).cuda()] for s in seqs]
    for i in range(p["n_layers"]):
        b = "blk.%d." % i
        w = {n: get(b + n) for n in ("attn_norm.weight", "ffn_norm.weight", "attn_q.weight", "attn_k.weight", "attn_v.weight", "attn_output.weight")}
        if p.get("bias"):
            w.update({n: get(b + n) for n in ("attn_q.bias", "attn_k.bias", "attn_v.bias")})
        for n, x in enumerate(xs):
            h = _rms(x, w["attn_norm.weight"], eps)
            q, k, v = (h @ w["attn_%s.weight" % c].T + (w["attn_%s.bias" % c] if p.get("bias") else 0.0) for c in "qkv")
            q, k = (_turn(y.reshape(len(x), -1, hd), freqs, not p["rope_neox"]) for y in (q, k))
            o = _attend(q, k, v.reshape(len(x), nkv, hd), hd ** -0.5)
            xs[n] = x + o.reshape(len(x), nh * hd) @ w["attn_output.weight"].T
        names = ("ffn_gate_exps", "ffn_up_exps", "ffn_down_exps") if p.get("n_experts") else ("ffn_gate", "ffn_up", "ffn_down")
        gate, up, down = (get(b + n + ".weight") for n in names)
        for n, x in enumerate(xs):
            h = _rms(x, w["ffn_norm.weight"], eps)
            if p.get("n_experts"):
                z, at = (h @ get(b + "ffn_gate_inp.weight").T).topk(p["n_experts_used"], -1)
                wt, y = torch.softmax(z, -1), torch.zeros_like(x)
                for e in range(p["n_experts"]):
                    t, c = torch.nonzero(at == e, as_tuple=True)
                    he = h[t]
                    y.index_add_(0, t, wt[t, c].unsqueeze(1) * ((torch.nn.functional.silu(he @ gate[e].T) * (he @ up[e].T)) @ down[e].T))
            else:
                y = (torch.nn.functional.silu(h @ gate.T) * (h @ up.T)) @ down.T
            xs[n] = x + y
    head = emb if p.get("tied") else get("output.weight")
    norm = get("output_norm.weight")
    P, nb = case["prompt"], case["batch"]
    lg = [_rms(x[max(0, P - 1):], norm, eps) @ head.T for x in xs]
    out = [lg[0][0]] if P else []
    for t in range(case["decode"]):
        r = t + (1 if P else 0)
        out.append(lg[0][r] if nb == 1 else torch.stack([v[r] for v in lg]))
    return out


def _mixture(h, W, pre, mlp, choice, weight, unit):
    """Chosen experts' outputs; weight(values at the choice, the choice)."""
    top = mlp["router"]["top"]
    at = torch.sort(choice, dim=-1, descending=True, stable=True)[1][:, :top]
    wt, y = weight(at), torch.zeros_like(h)
    for e in range(choice.shape[1]):
        t, c = torch.nonzero(at == e, as_tuple=True)
        if len(t):
            y.index_add_(0, t, wt[t, c].unsqueeze(1) * (unit(h[t], pre + "e%d." % e) if e < mlp["router"]["experts"] else h[t]))
    return y


def _conv(u, f):
    """u [T, C], f [C, taps]: the last column meets the current token."""
    taps = f.shape[1]
    pad = torch.cat([torch.zeros(taps - 1, u.shape[1], device="cuda", dtype=F), u])
    return sum(pad[j:j + len(u)] * f[:, j] for j in range(taps))


def _gefovik(cfg, W, x):
    eps, T = 1e-6, len(x)
    pos = torch.arange(T, device="cuda", dtype=F).view(-1, 1, 1)
    for i, L in enumerate(cfg["layers"]):
        m, a, f = L["mixer"], "l%d.mix." % i, "l%d.mlp." % i
        H = m["heads"]
        q = (x @ W[a + "q"].T).reshape(T, H, -1)
        if L["type"] == "attention":
            k = (x @ W[a + "k"].T).reshape(T, m["kv_heads"], -1)
            q = _rms(q, 1.0, eps) * (1.0 + m["q_temp"]["coef"] * torch.log(torch.floor((pos + 1) / m["q_temp"]["every"]) + 1.0))
            o = _attend(q, _rms(k, 1.0, eps), k, m["scale"], cap=m["softcap"])
        else:
            c = _rms(x @ W[a + "dkv"].T, W[a + "dkv.norm"], eps)
            o = _attend(q, (c @ W[a + "uk"].T).reshape(T, H, -1), (c @ W[a + "uv"].T).reshape(T, H, -1), m["scale"], sink=W[a + "sink"])
            o = o * torch.sigmoid(x @ W[a + "g"].T).unsqueeze(2)
        x = x + _ln(o.reshape(T, -1) @ W[a + "o"].T, W["l%d.norm1" % i], eps)
        if L["mlp"]["kind"] == "dense":
            y = (torch.relu(x @ W[f + "gate"].T) * (x @ W[f + "up"].T)) @ W[f + "down"].T
        else:
            s = torch.softmax(x @ W[f + "router"].T, -1)
            y = _mixture(x, W, f, L["mlp"], s + W[f + "correction"], lambda at: s.gather(1, at),
                         lambda h, n: (torch.nn.functional.silu(h @ W[n + "gate"].T) * (h @ W[n + "up"].T)) @ W[n + "down"].T)
        x = x + _ln(y, W["l%d.norm2" % i], eps)
    return _ln(x, W["final.norm"], eps) @ W["embed"].T


def _mefurax(cfg, W, x):
    eps, T, al, first = 1e-6, len(x), cfg["postln_alpha"], None
    for i, L in enumerate(cfg["layers"]):
        m, a, f = L["mixer"], "l%d.mix." % i, "l%d.mlp." % i
        H, G, size = m["heads"], m["kv_heads"], m["mask"]["size"]
        q, k, v = (x @ W[a + n].T for n in "qkv")
        if L["type"] == "attention":
            q, k, v = (_conv(u + W[a + n + ".b"], W[a + n + ".conv"]) for n, u in zip("qkv", (q, k, v)))
            q, k = (_rms(u, W[a + n + ".norm"], eps) for n, u in zip("qk", (q, k)))
        else:
            fr = [m["rot"]["base"] ** (-2.0 * j / m["rot"]["dims"]) for j in range(m["rot"]["dims"] // 2)]
            q, k = (_rms(_turn(u.reshape(T, n, -1), fr, True), 1.0, eps) for u, n in ((q, H), (k, G)))
        if first is None:
            first = v
        else:
            v = (1.0 - W[a + "vmix"]) * v + W[a + "vmix"] * first
        q, k, v = q.reshape(T, H, -1), k.reshape(T, G, -1), v.reshape(T, G, -1)
        if L["type"] == "attention":
            o = _attend(q, k, v, m["scale"], lambda i, j: i - j < size, torch.tensor([2.0 ** (-8.0 * (h + 1) / H) for h in range(H)], device="cuda", dtype=F))
        else:
            o = _attend(q, k, v, m["scale"], lambda i, j: i // size == j // size, cap=m["softcap"]) * torch.sigmoid(x @ W[a + "g"].T).unsqueeze(2)
        x = _rms(al * x + o.reshape(T, -1) @ W[a + "o"].T, 1.0 + W["l%d.norm1" % i], eps)
        if L["mlp"]["kind"] == "dense":
            y = (torch.nn.functional.gelu(x @ W[f + "gate"].T, approximate="tanh") * (x @ W[f + "up"].T)) @ W[f + "down"].T
        else:
            unit = lambda h, n: torch.relu(h @ W[n + "up"].T).square() @ W[n + "down"].T  # noqa: E731
            z = x @ W[f + "router"].T
            y = _mixture(x, W, f, L["mlp"], z, lambda at: torch.softmax(z.gather(1, at), -1), unit) + unit(x, f + "shared.")
        x = _rms(al * x + y, 1.0 + W["l%d.norm2" % i], eps)
    return _rms(x, 1.0 + W["final.norm"], eps) @ W["head"].T


def _lazilorn(cfg, W, x):
    eps, T, width = 1e-6, len(x), cfg["width"]
    sg, silu = torch.sigmoid, torch.nn.functional.silu
    ang = torch.arange(T, device="cuda", dtype=F).view(-1, 1) * 10000.0 ** (-2.0 * torch.arange(width // 2, device="cuda", dtype=F) / width)
    x = x + torch.stack([torch.sin(ang), torch.cos(ang)], 2).reshape(T, width)
    for i, L in enumerate(cfg["layers"]):
        m, a = L["mixer"], "l%d.mix." % i
        h = _rms(x, W["l%d.norm1" % i], eps)
        if L["type"] == "parallel":
            le, ri = m["left"], m["right"]
            l, r = a + "left.", a + "right."
            q, k, v = ((h @ W[l + n].T).reshape(T, le["heads"] if n == "q" else le["kv_heads"], -1) for n in "qkv")
            q, k = _rms(q, W[l + "q.norm"], eps), _rms(k, W[l + "k.norm"], eps)
            o = _attend(q, k, v, le["scale"], lambda i, j: (i - j < le["mask"]["size"]) | (j < le["mask"]["keep_first"]))
            left = (o.reshape(T, -1) * sg(h @ W[l + "g"].T)) @ W[l + "o"].T
            H, d, dv, cap = ri["heads"], ri["dim"], ri["vdim"], ri["gate_cap"]
            q, k, v = ((h @ W[r + n].T).reshape(T, H, -1) for n in "qkv")
            q = q * d ** -0.5
            ig = cap * torch.tanh((h @ W[r + "i"].T + W[r + "i.b"]) / cap)
            fg = torch.nn.functional.logsigmoid(cap * torch.tanh((h @ W[r + "f"].T + W[r + "f.b"]) / cap))
            # closed form of the memory in 64 bits: weight of token s at token t is exp(i_s + f_(s+1) + ... + f_t), over exp(m_t)
            cum = torch.cumsum(fg, 0)
            u = torch.maximum(torch.cummax(ig - cum, 0)[0], torch.zeros(1, device="cuda", dtype=F))       # m_t - cum_t (m starts at 0)
            o = []
            for t0 in range(0, T, 256):
                t1 = min(T, t0 + 256)
                wt = (ig - cum)[:t1].T.unsqueeze(1) - u[t0:t1].T.unsqueeze(2)                                # [H, t, s]
                ok = torch.arange(t1, device="cuda").view(1, 1, -1) <= torch.arange(t0, t1, device="cuda").view(1, -1, 1)
                s = torch.exp(wt.masked_fill(~ok, -math.inf)) * (q[t0:t1].transpose(0, 1) @ k[:t1].permute(1, 2, 0))
                den = torch.maximum(s.sum(2).abs(), torch.exp(-(u + cum)[t0:t1].T)) + 1e-6
                o.append((s @ v[:t1].transpose(0, 1) / den.unsqueeze(2)).transpose(0, 1))
            o = _rms(torch.cat(o), 1.0, eps).reshape(T, H * dv) * W[r + "norm"] * sg(h @ W[r + "g"].T)
            x = x + m["left_scale"] * left + m["right_scale"] * (o @ W[r + "o"].T)
        else:
            H, G, d, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
            q, k, v = (silu(_conv(h @ W[a + n].T, W[a + n + ".conv"])).reshape(T, H if n == "v" else G, -1) for n in "qkv")
            q = (q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * d ** -0.5).repeat_interleave(H // G, 1)
            k = (k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, 1)
            beta = sg(h @ W[a + "b"].T)
            g = torch.exp(-torch.exp(W[a + "A_log"]) * torch.nn.functional.softplus(h @ W[a + "a"].T + W[a + "dt_bias"]))
            S, o = torch.zeros(H, d, dv, device="cuda", dtype=F), []
            for t in range(T):
                S = S * g[t].view(-1, 1, 1)
                S = torch.baddbmm(S, k[t].unsqueeze(2), (beta[t].unsqueeze(1) * (v[t] - torch.bmm(k[t].unsqueeze(1), S).squeeze(1))).unsqueeze(1))
                o.append(torch.bmm(q[t].unsqueeze(1), S).squeeze(1))
            o = (_rms(torch.stack(o), W[a + "norm"], eps)).reshape(T, H * dv) * silu(h @ W[a + "g"].T)
            x = x + o @ W[a + "o"].T
        x = x + torch.relu(_rms(x, W["l%d.norm2" % i], eps) @ W["l%d.mlp.up" % i].T).square() @ W["l%d.mlp.down" % i].T
    return _rms(x, W["final.norm"], eps) @ W["head"].T


def _stretched(rot):
    """Rotary frequencies slowed by `factor` where the wavelength is long against the original context, and the factor on cos and sin."""
    dims, base, sc = rot["dims"], rot["base"], rot["scaling"]
    at = [dims * math.log(sc["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base)) for turns in (sc["fast"], sc["slow"])]
    lo, hi = max(math.floor(at[0]), 0), min(math.ceil(at[1]), dims - 1)
    out = []
    for i in range(dims // 2):
        r = min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0)
        f = base ** (-2.0 * i / dims)
        out.append(f / sc["factor"] * r + f * (1.0 - r))
    return out, 0.1 * math.log(sc["factor"]) + 1.0


def _madudra(cfg, W, x):
    eps, T = 1e-6, len(x)
    silu = torch.nn.functional.silu
    X, rows = x.unsqueeze(0).repeat(cfg["streams"], 1, 1), {}

    def sub(X, pre, norm, fn):
        y = fn(_ln(torch.einsum("s,stw->tw", W[pre + "in"], X), W[norm], eps))
        return torch.einsum("st,srw->trw", W[pre + "mix"], X) + cfg["residual_mult"] * W[pre + "out"].view(-1, 1, 1) * y

    for i, L in enumerate(cfg["layers"]):
        m, a, f = L["mixer"], "l%d.mix." % i, "l%d.mlp." % i

        def latent(h):
            H, d, rd, rank = m["heads"], m["dim"], m["rot_dim"], m["kv_rank"]
            fr, mult = _stretched(m["rot"])
            q = (_rms(h @ W[a + "dq"].T, W[a + "dq.norm"], eps) @ W[a + "uq"].T).reshape(T, H, d + rd)
            if m.get("kv_from") is None:
                c = h @ W[a + "dkv"].T
                rows[i] = (_rms(c[:, :rank], W[a + "dkv.norm"], eps), _turn(c[:, rank:].unsqueeze(1), fr, False, mult))
            c, kr = rows[i if m.get("kv_from") is None else m["kv_from"]]
            k = torch.cat([(c @ W[a + "uk"].T).reshape(T, H, d), kr.expand(T, H, rd)], 2)
            q = torch.cat([q[..., :d], _turn(q[..., d:], fr, False, mult)], 2)
            o = _attend(q, k, (c @ W[a + "uv"].T).reshape(T, H, -1), m["scale"], lambda i, j: i - j < m["mask"]["size"])
            return (o.reshape(T, -1) * torch.sigmoid(h @ W[a + "g"].T)) @ W[a + "o"].T

        def scan(h):
            H, vd, N, G = m["heads"], m["vdim"], m["state"], m["groups"]
            inner = H * vd
            y = h @ W[a + "in"].T
            z, c, dt = y[:, :inner], y[:, inner:2 * inner + 2 * G * N], y[:, 2 * inner + 2 * G * N:]
            c = silu(_conv(c, W[a + "conv"]) + W[a + "conv.b"])
            u = c[:, :inner].reshape(T, H, vd)
            Bm, Cm = (v.reshape(T, G, N).repeat_interleave(H // G, 1) for v in (c[:, inner:inner + G * N], c[:, inner + G * N:]))
            dt = torch.nn.functional.softplus(dt + W[a + "dt_bias"])
            cum = torch.cumsum(-torch.exp(W[a + "A_log"]) * dt, 0)
            o = []
            for t0 in range(0, T, 128):          # closed form: token s weighs exp(cum_t - cum_s) dt_s at token t
                t1 = min(T, t0 + 128)
                wt = cum[t0:t1].T.unsqueeze(2) - cum[:t1].T.unsqueeze(1)
                ok = torch.arange(t1, device="cuda").view(1, 1, -1) <= torch.arange(t0, t1, device="cuda").view(1, -1, 1)
                s = torch.exp(wt.masked_fill(~ok, -math.inf)) * dt[:t1].T.unsqueeze(1) * (Cm[t0:t1].transpose(0, 1) @ Bm[:t1].permute(1, 2, 0))
                o.append((s @ u[:t1].transpose(0, 1)).transpose(0, 1))
            o = torch.cat(o) + W[a + "D"].view(1, -1, 1) * u
            o = (o.reshape(T, inner) * silu(z)).reshape(T, m["norm_groups"], -1)
            return (_rms(o, 1.0, eps).reshape(T, inner) * W[a + "norm"]) @ W[a + "o"].T

        def experts(h):
            s = torch.softmax(h @ W[f + "router"].T, -1)
            return _mixture(h, W, f, L["mlp"], s, lambda at: s.gather(1, at) * L["mlp"]["router"]["scale"],
                            lambda u, n: torch.nn.functional.gelu(u @ W[n + "up"].T) @ W[n + "down"].T)

        X = sub(X, "l%d.hc1." % i, "l%d.norm1" % i, latent if L["type"] == "latent_attention" else scan)
        X = sub(X, "l%d.hc2." % i, "l%d.norm2" % i, experts)
    return _ln(X.sum(0), W["final.norm"], eps) @ W["head"].T


def exact(case, seed):
    if case["family"] == "gguf":
        return _exact_gguf(case, seed)
    cfg, mod = _lp_config(case), DESIGNS[case["family"]]
    W = {n: _lp_tensor(cfg, seed, n, s).to(F) for n, s in mod.tensor_shapes(cfg).items()}
    prompts, steps = _lp_inputs(case, seed)
    model = {"gefovik": _gefovik, "mefurax": _mefurax, "lazilorn": _lazilorn, "madudra": _madudra}[case["family"]]
    first, then = [], []
    for b, p in enumerate(prompts):
        toks = np.concatenate([p] + [s[b:b + 1] for s in steps]).astype(np.int64)
        lg = model(cfg, W, W["embed"][torch.from_numpy(toks).cuda()])
        first.append(lg[[r for r in range(len(p)) if r % case["stride"] == case["stride"] - 1 or r == len(p) - 1]])
        then.append(lg[len(p):])
    return [torch.cat(first)] + [then[0][t] if len(prompts) == 1 else torch.stack([v[t] for v in then]) for t in range(len(steps))]
