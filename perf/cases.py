"""The work this framework is used for, as cases that can be timed: training steps of the dense native trainers, the routed
expert feed-forward with its gradients, prompts and decode steps of the resident inference engine.

``listed()`` names the cases, ``draw(rng)`` gives more of the same ranges, ``prepare`` makes what a program holds before the
call, ``run`` makes one call through the public entry points, ``work`` counts what the call cannot do without and ``exact``
restates it in 64-bit PyTorch.
"""
from __future__ import annotations

import math

import numpy as np
import torch
import torch.nn.functional as F

BF, F32, F64 = torch.bfloat16, torch.float32, torch.float64


# ------------------------------------------------------------------------------------------------ cases
def listed() -> list[dict]:
    return [
        # one optimizer step of a toy GPT (the size of the smoke test): the step is a chain of short launches
        _gpt("gpt_toy_step", 2, 4, 2048, 4, 256, "gpt2_qknorm_softcap_zloss"),
        # the benchmark's workload: GPT-2 124M with QK norm, soft-cap and z-loss, micro-batch 16 x 1024
        _gpt("gpt2_124m_step", 12, 12, 50257, 16, 1024, "gpt2_qknorm_softcap_zloss"),
        # a mid-sized plain GPT-2 on sequences whose length fits no tile
        _gpt("gpt_ragged_step", 6, 8, 50257, 5, 777, "gpt2"),
        # layers of the Llama-3-8B shape at its training length: the largest products and attention
        _llama("llama_8b_layers_step", 2, 32, 8, 128, 14336, 32000, 2, 4096, 0, False, False),
        # a small Llama with sliding windows, grouped heads of 64, QK norm and a tied head, ragged length
        _llama("llama_window_step", 8, 16, 4, 64, 2816, 32000, 3, 1531, 512, True, True),
        # expert feed-forward of a layer of the MoE decoder shape (64 experts of 1024, top 8), forward and backward
        dict(name="moe_64_experts", kind="moe", tokens=8192, width=2048, experts=64, top=8, ff=1024),
        # the same of a toy MoE on a short ragged batch
        dict(name="moe_8_experts_short", kind="moe", tokens=611, width=512, experts=8, top=2, ff=1344),
        # a long prompt through Glimmer blocks with sliding windows (one period of three local and one global layer,
        # the width of the serving benchmark)
        _serve("prompt_glimmer_8k", "prompt", "glimmer", 4, 32, 8, 128, 14336, 32768, 1, 8191, 1024, "bf16", 1),
        # a short chat prompt of odd length through a Llama of the same width: time to first token
        _serve("prompt_llama_short", "prompt", "llama", 8, 16, 4, 128, 5632, 32000, 1, 317, 0, "bf16", 1),
        # single-stream decoding, sixteen tokens
        _serve("decode_llama_single", "decode", "llama", 8, 16, 4, 128, 5632, 32000, 1, 1023, 0, "bf16", 16),
        # batched decoding over caches of different lengths at the width of Llama-3-8B
        _serve("decode_llama_batch", "decode", "llama", 4, 32, 8, 128, 14336, 32000, 32, 3071, 0, "bf16", 16),
        # a few streams of Glimmer blocks whose projections stay in Q4_K blocks
        _serve("decode_glimmer_q4k", "decode", "glimmer", 4, 16, 4, 128, 5632, 32768, 4, 2047, 4096, "q4_k", 16),
    ]


def _gpt(name, layers, heads, vocab, batch, seq, variant) -> dict:
    return dict(name=name, kind="gpt", layers=layers, heads=heads, vocab=vocab, batch=batch, seq=seq, variant=variant)


def _llama(name, layers, heads, kv_heads, dim, ff, vocab, batch, seq, window, qk_norm, tied) -> dict:
    return dict(name=name, kind="llama", layers=layers, heads=heads, kv_heads=kv_heads, dim=dim, ff=ff, vocab=vocab, batch=batch, seq=seq,
                window=window, qk_norm=qk_norm, tied=tied)


def _serve(name, kind, blocks, layers, heads, kv_heads, dim, ff, vocab, batch, context, window, weights, steps) -> dict:
    return dict(name=name, kind=kind, blocks=blocks, layers=layers, heads=heads, kv_heads=kv_heads, dim=dim, ff=ff, vocab=vocab, batch=batch,
                context=context, window=window, weights=weights, steps=steps)


def _spread(rng, lo: int, hi: int) -> int:
    """A whole number in [lo, hi], even over the logarithm."""
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng) -> dict:
    kind = rng.choice(["gpt", "gpt", "llama", "llama", "moe", "moe", "prompt", "prompt", "decode", "decode", "decode"])
    if kind == "gpt":
        c = _gpt("", rng.randint(2, 12), rng.randint(4, 12), rng.choice([2048, 32000, 50257]), _spread(rng, 1, 16), _spread(rng, 65, 1024),
                 rng.choice(["gpt2", "gpt2_qknorm", "gpt2_stable", "gpt2_softcap", "gpt2_qknorm_softcap_zloss"]))
    elif kind == "llama":
        dim = rng.choice([64, 128])
        heads = rng.choice([8, 16, 32])
        seq = _spread(rng, 130, 4096)
        while True:
            c = _llama("", rng.randint(1, 8), heads, heads // rng.choice([1, 2, 4]), dim, 64 * _spread(rng, 16, 224), rng.choice([4096, 32000]),
                       rng.randint(1, 4), seq, rng.choice([0, max(64, seq // 3)]), rng.random() < 0.5, rng.random() < 0.3)
            if work(c)["flops"] < 2.5e13 and _n_params(c) < 6e8:
                break
            seq = max(130, seq * 3 // 4)
    elif kind == "moe":
        width, experts = rng.choice([512, 1024, 2048]), rng.choice([4, 8, 16, 32, 64])
        c = dict(kind="moe", tokens=_spread(rng, 64, 8192), width=width, experts=experts, top=rng.randint(1, min(8, experts)), ff=64 * _spread(rng, 4, 16))
    else:
        blocks = rng.choice(["llama", "glimmer"])
        dim = rng.choice([64, 128])
        heads = rng.choice([8, 16, 32]) * (128 // dim)
        wide = heads * dim > 2048
        ff = 256 * rng.randint(8, 20) * (2 if wide else 1)
        layers = rng.randint(2, 4) if wide or blocks == "glimmer" else rng.randint(2, 8)
        if kind == "prompt":
            c = _serve("", kind, blocks, layers, heads, heads // 4, dim, ff, 32000, 1, _spread(rng, 17, 8191), rng.choice([512, 1024]) if blocks == "glimmer" else 0, "bf16", 1)
        else:
            q4 = rng.random() < 0.3
            c = _serve("", kind, blocks, layers, heads, heads // 4, dim, ff, 32000, _spread(rng, 1, 8 if q4 else 32), _spread(rng, 64, 3071),
                       4096 if blocks == "glimmer" else 0, "q4_k" if q4 else "bf16", 16)
    c.pop("name", None)
    return c


# ------------------------------------------------------------------------------------------------ weights
def _gen(seed: int) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(seed)


def _randn(g, shape, std: float, mean: float = 0.0, dtype=F32) -> torch.Tensor:
    return torch.randn(shape, generator=g, device="cuda", dtype=F32).mul_(std).add_(mean).to(dtype)


def _padded(vocab: int) -> int:
    return (vocab + 127) // 128 * 128


def _train_specs(c: dict) -> list[tuple[str, tuple, bool, float, float]]:
    """(name, shape, weight decay, std, mean) of a trained model's tensors in their flat order."""
    L, H, V, std = c["layers"], c["heads"], _padded(c["vocab"]), 0.02
    out = 0.02 / math.sqrt(2 * L)
    if c["kind"] == "gpt":
        C = 64 * H
        s = [("wte", (V, C), True, std, 0.0), ("wpe", (c["seq"], C), True, std, 0.0)]
        for i in range(L):
            p = f"h.{i}."
            s += [(p + "ln_1.weight", (C,), False, 0.02, 1.0), (p + "ln_1.bias", (C,), False, 0.02, 0.0),
                  (p + "attn.c_attn.weight", (3 * C, C), True, std, 0.0), (p + "attn.c_attn.bias", (3 * C,), False, 0.02, 0.0),
                  (p + "attn.c_proj.weight", (C, C), True, out, 0.0), (p + "attn.c_proj.bias", (C,), False, 0.02, 0.0),
                  (p + "ln_2.weight", (C,), False, 0.02, 1.0), (p + "ln_2.bias", (C,), False, 0.02, 0.0),
                  (p + "mlp.c_fc.weight", (4 * C, C), True, std, 0.0), (p + "mlp.c_fc.bias", (4 * C,), False, 0.02, 0.0),
                  (p + "mlp.c_proj.weight", (C, 4 * C), True, out, 0.0), (p + "mlp.c_proj.bias", (C,), False, 0.02, 0.0)]
        s += [("ln_f.weight", (C,), False, 0.02, 1.0), ("ln_f.bias", (C,), False, 0.02, 0.0)]
    else:
        C, K, D, f = H * c["dim"], c["kv_heads"], c["dim"], c["ff"]
        s = [("tok_embeddings", (V, C), True, std, 0.0)]
        for i in range(L):
            p = f"layers.{i}."
            s += [(p + "attn_norm", (C,), False, 0.02, 1.0), (p + "wqkv", ((H + 2 * K) * D, C), True, std, 0.0), (p + "wo", (C, H * D), True, out, 0.0),
                  (p + "ffn_norm", (C,), False, 0.02, 1.0), (p + "w_gate_up", (2 * f, C), True, std, 0.0), (p + "w_down", (C, f), True, out, 0.0)]
        s += [("norm", (C,), False, 0.02, 1.0)] + ([] if c["tied"] else [("lm_head", (V, C), True, std, 0.0)])
    return [x for x in s if x[2]] + [x for x in s if not x[2]]


def _n_params(c: dict) -> int:
    return sum(math.prod(s[1]) for s in _train_specs(c))


def _train_master(c: dict, seed: int) -> dict[str, torch.Tensor]:
    g = _gen(seed)
    out = {}
    for name, shape, _, std, mean in _train_specs(c):
        t = _randn(g, shape, std, mean)
        if name in ("wte", "tok_embeddings", "lm_head"):
            t[c["vocab"]:] = 0
        out[name] = t
    return out


def _train_batch(c: dict, seed: int) -> tuple[torch.Tensor, torch.Tensor]:
    """Token ids with some of the skew of text (low ids are drawn more often) and their successors."""
    g = torch.Generator().manual_seed(seed + 1)
    u = torch.rand(c["batch"], c["seq"] + 1, generator=g)
    ids = (c["vocab"] * u ** 1.5).to(torch.int32).clamp_(0, c["vocab"] - 1)
    return ids[:, :-1].contiguous(), ids[:, 1:].contiguous()


def _serve_tensors(c: dict, seed: int):
    """(name, bf16 tensor or None, Q4_K blocks or None, weights in 64 bits) of a served model, one at a time. The head favours one
    successor of every token by several standard deviations of the other logits, as a trained model's does."""
    g = _gen(seed)
    L, H, K, D, f, V = c["layers"], c["heads"], c["kv_heads"], c["dim"], c["ff"], _padded(c["vocab"])
    C, glimmer = H * D, c["blocks"] == "glimmer"
    qkv = (H + 2 * K) * D + (H * D if glimmer else 0)
    emb = _randn(g, (V, C), 1.0, dtype=BF)
    emb[c["vocab"]:] = 0
    yield "tok_embeddings", emb, None
    small = 0.02 / math.sqrt(2 * L)
    for i in range(L):
        p = f"layers.{i}."
        yield p + "attn_norm", _randn(g, (C,), 0.02, 0.0 if glimmer else 1.0, BF), None
        yield p + "wqkv", *_projection(c, g, qkv, C, 0.02)
        yield p + "wo", *_projection(c, g, C, H * D, small)
        if glimmer:
            yield p + "post_attn_norm", _randn(g, (C,), 0.02, -0.85, BF), None
        yield p + "ffn_norm", _randn(g, (C,), 0.02, 0.0 if glimmer else 1.0, BF), None
        yield p + "w_gate_up", *_projection(c, g, 2 * f, C, 0.02)
        yield p + "w_down", *_projection(c, g, C, f, small)
        if glimmer:
            yield p + "post_ffn_norm", _randn(g, (C,), 0.02, -0.85, BF), None
    yield "norm", _randn(g, (C,), 0.02, 1.0, BF), None
    head = _randn(g, (V, C), 0.92)
    head[_successor(c, torch.arange(c["vocab"], device="cuda"))] += 0.4 * emb[:c["vocab"]].float()
    head *= (5.1 if glimmer else 1.0) / math.sqrt(C)
    head[c["vocab"]:] = 0
    yield "lm_head", head.to(BF), None


def _successor(c: dict, token):
    """The token a served model puts after ``token``: a permutation of the vocabulary."""
    return (token + 7919) % c["vocab"]


def _projection(c: dict, g, n: int, k: int, std: float):
    """(bf16 weights, None), or (the weights in 64 bits, Q4_K blocks of them): random 4-bit values around the middle of their
    range, 6-bit scales and offsets per 32 values."""
    if c["weights"] == "bf16":
        return _randn(g, (n, k), std, dtype=BF), None
    nb = n * k // 256
    scale = torch.randint(32, 64, (nb, 8), generator=g, device="cuda", dtype=torch.uint8)
    q = torch.randint(0, 256, (nb, 128), generator=g, device="cuda", dtype=torch.uint8)
    d = torch.tensor([std / 220.0], dtype=torch.float16, device="cuda")
    dmin = torch.tensor([std / 220.0 * 7.5], dtype=torch.float16, device="cuda")
    raw = torch.empty(nb, 144, dtype=torch.uint8, device="cuda")
    raw[:, 0:2], raw[:, 2:4] = d.view(torch.uint8), dmin.view(torch.uint8)
    raw[:, 4:8] = (scale[:, :4] & 63) | ((scale[:, 4:] >> 4) << 6)
    raw[:, 8:12] = raw[:, 4:8]
    raw[:, 12:16] = (scale[:, 4:] & 15) | ((scale[:, 4:] & 15) << 4)
    raw[:, 16:] = q
    four = torch.stack([q.view(nb, 4, 32) & 15, q.view(nb, 4, 32) >> 4], 2).view(nb, 8, 32)
    w = (scale[..., None].double() * (d.double() * four.double() - dmin.double())).view(n, k)
    return w, raw.view(-1)


def _prompts(c: dict, seed: int) -> list[list[int]]:
    g = torch.Generator().manual_seed(seed + 1)
    n = [c["context"]] + [int(v) for v in torch.randint(max(8, c["context"] // 24), c["context"] + 1, (c["batch"] - 1,), generator=g)]
    return [torch.randint(0, c["vocab"], (k,), generator=g).tolist() for k in n]


def _moe_inputs(c: dict, seed: int) -> dict[str, torch.Tensor]:
    g = _gen(seed)
    T, d, E, k, f = (c[n] for n in ("tokens", "width", "experts", "top", "ff"))
    x = _randn(g, (T, d), 1.0, dtype=BF)
    logits = x.float() @ _randn(g, (d, E), d ** -0.5) + _randn(g, (E,), 0.5)     # some experts are more popular than others
    w, idx = torch.softmax(logits, -1).topk(k, dim=-1)
    return dict(x=x, w1=_randn(g, (E, d, f), 0.02, dtype=BF), w2=_randn(g, (E, f, d), 0.02, dtype=BF), w3=_randn(g, (E, d, f), 0.02, dtype=BF),
                weights=w / w.sum(-1, keepdim=True), indices=idx, dout=_randn(g, (T, d), 1.0, dtype=BF))


# ------------------------------------------------------------------------------------------------ prepare, run
def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    if kind == "moe":
        t = _moe_inputs(case, seed)
        for n in ("x", "w1", "w2", "w3", "weights"):
            t[n].requires_grad_(True)
        return dict(kind=kind, **t)
    return _prepare_training(case, seed) if kind in ("gpt", "llama") else _prepare_serving(case, seed)


def _prepare_training(c: dict, seed: int) -> dict:
    from neuralfn_b200.trainers.dense_gpt import DenseGPTTrainer
    if c["kind"] == "gpt":
        from neuralfn_b200.models.gpt2 import GPT2Config
        cfg = GPT2Config.variant(c["variant"], n_layer=c["layers"], n_head=c["heads"], d_model=64 * c["heads"], vocab_size=c["vocab"], max_seq_len=c["seq"])
    else:
        from neuralfn_b200.models.llama import LlamaConfig
        cfg = LlamaConfig(n_layer=c["layers"], n_head=c["heads"], n_kv_head=c["kv_heads"], d_model=c["heads"] * c["dim"], d_ff=c["ff"],
                          vocab_size=c["vocab"], max_seq_len=c["seq"], window=c["window"], qk_norm=c["qk_norm"], tie_embeddings=c["tied"])
    trainer = DenseGPTTrainer(cfg, c["batch"], c["seq"])
    for name, t in _train_master(c, seed).items():
        trainer.layout.view(trainer.opt.master, name).copy_(t)
    trainer.opt.publish_params()
    tokens, targets = _train_batch(c, seed)
    cuts = _cuts([n for n, *_ in _train_specs(c)], trainer.layout.offsets, trainer.layout.n_used)
    return dict(kind="train", trainer=trainer, tokens=tokens.pin_memory(), targets=targets.pin_memory(),
                grads=[trainer.bufs.grads[a:b] for a, b in cuts])


def _cuts(names: list[str], offsets: dict[str, int], end: int) -> list[tuple[int, int]]:
    """The flat buffer in pieces: embeddings, the matrices of each layer, what follows."""
    marks = sorted({offsets[n] for n in names if n in ("wte", "wpe", "tok_embeddings", "lm_head") or n.endswith((".attn.c_attn.weight", ".wqkv"))}
                   | {offsets["ln_f.weight"] if "ln_f.weight" in offsets else offsets["norm"]}
                   | {offsets[n] for n in names if n in ("h.0.ln_1.weight", "layers.0.attn_norm")}) + [end]
    return list(zip(marks[:-1], marks[1:]))


def _prepare_serving(c: dict, seed: int) -> dict:
    from neuralfn_b200.serving import EngineConfig, ResidentEngine
    max_seq = (c["context"] + c["steps"] + 2 + 63) // 64 * 64
    size = dict(n_layer=c["layers"], d_model=c["heads"] * c["dim"], n_head=c["heads"], n_kv_head=c["kv_heads"], head_dim=c["dim"], d_ff=c["ff"],
                vocab=c["vocab"], max_seq=max_seq, max_batch=c["batch"])
    if c["blocks"] == "glimmer":
        cfg = EngineConfig.glimmer(window=c["window"], **size)
    else:
        cfg = EngineConfig(family=1, padded_vocab=_padded(c["vocab"]), rope_theta=500000.0, tie_embeddings=0, **size)
    engine = ResidentEngine(cfg)
    for name, t, blocks in _serve_tensors(c, seed):
        if blocks is not None:
            engine.set_tensor_kquant(name, "Q4_K", blocks)
        else:
            engine.set_tensor(name, t)
    engine.finalize()
    prompts = _prompts(c, seed)
    first = [engine.prefill(s, p) for s, p in enumerate(prompts)] if c["kind"] == "decode" else []
    return dict(kind=c["kind"], engine=engine, prompts=prompts, first=first, steps=c["steps"])


def run(state: dict):
    kind = state["kind"]
    if kind == "train":
        trainer = state["trainer"]
        loss = trainer.train_step(state["tokens"], state["targets"])
        return dict(loss=loss, grads=state["grads"], master=trainer.opt.master, params=trainer.bufs.params)
    if kind == "moe":
        from neuralfn_b200.ops.moe import moe_experts
        wrt = [state[n] for n in ("x", "w1", "w2", "w3", "weights")]
        out = moe_experts(*wrt, state["indices"])
        return [out.detach(), *torch.autograd.grad(out, wrt, state["dout"])]
    engine, prompts = state["engine"], state["prompts"]
    if kind == "prompt":
        token = engine.prefill(0, prompts[0])
        return dict(token=token, logits=engine.last_logits(0))
    slots = range(len(prompts))
    for s in slots:                                  # back to the end of the prompts: the answer is drawn again
        engine.truncate(s, len(prompts[s]))
    tokens, answer = dict(enumerate(state["first"])), []
    for _ in range(state["steps"]):
        tokens = engine.decode(tokens)
        answer.append([tokens[s] for s in slots])
    return dict(tokens=np.array(answer), logits=[engine.last_logits(s) for s in slots])


# ------------------------------------------------------------------------------------------------ work, tolerance
def work(case: dict) -> dict:
    c = case
    if c["kind"] == "moe":
        T, d, E, k, f = (c[n] for n in ("tokens", "width", "experts", "top", "ff"))
        return dict(bytes=2 * (2 * 3 * E * d * f + 4 * T * d) + 4 * 2 * T * k + 8 * T * k, flops=3 * 2 * 3 * T * k * d * f)
    C, H, L = (c["heads"] * c.get("dim", 64)), c["heads"], c["layers"]
    if c["kind"] in ("gpt", "llama"):
        B, T, n = c["batch"], c["seq"], _n_params(c)
        head = _padded(c["vocab"]) * C
        if c["kind"] == "gpt":
            mat, seen = n - c["seq"] * C, T * (T + 1) / 2
        else:
            w = c["window"] or T
            mat, seen = n if c["tied"] else n - head, sum(min(t + 1, w) for t in range(T))
        # parameters in bf16 read once, gradients written once, fp32 master weights and two moments read and written, parameters written
        return dict(bytes=n * (2 + 2 + 24 + 2) + 2 * 4 * B * T, flops=6.0 * mat * B * T + 12.0 * L * B * seen * C)
    K, D, f, V = c["kv_heads"], c["dim"], c["ff"], _padded(c["vocab"])
    layer = C * ((H + 2 * K) * D + (C if c["blocks"] == "glimmer" else 0)) + C * C + 3 * C * f
    wide = 144 / 256 if c["weights"] == "q4_k" else 2.0
    lens = [c["context"]] if c["kind"] == "prompt" else [len(p) for p in _prompts(c, 0)]
    if c["kind"] == "prompt":
        n = c["context"]
        local, whole = sum(min(t + 1, c["window"] or n) for t in range(n)), n * (n + 1) / 2
        seen = sum(whole if not c["window"] or (i + 1) % 4 == 0 else local for i in range(L))
        return dict(bytes=L * layer * wide + V * C * 2.0 + 2 * n * C + L * n * 2 * K * D * 2, flops=2.0 * n * L * layer + 4.0 * C * seen + 2.0 * V * C)
    cached = sum(n + s + 1 for n in lens for s in range(c["steps"]))
    return dict(bytes=c["steps"] * (L * layer * wide + V * C * 2.0) + cached * L * 2 * K * D * 2,
                flops=2.0 * c["steps"] * len(lens) * (L * layer + V * C) + 4.0 * C * L * cached)


def tolerance(case: dict) -> dict:
    if case["kind"] in ("gpt", "llama"):
        return dict(rel=0.03, max=0.9)
    if case["kind"] == "moe":
        return dict(rel=0.02, max=0.2)
    return dict(rel=0.03, max=0.3)


# ------------------------------------------------------------------------------------------------ 64-bit restatement
def exact(case: dict, seed: int):
    if case["kind"] == "moe":
        return _exact_moe(case, seed)
    if case["kind"] in ("gpt", "llama"):
        return _exact_training(case, seed)
    return _exact_serving(case, seed)


def _exact_moe(c: dict, seed: int):
    t = _moe_inputs(c, seed)
    x, w1, w2, w3, wt, dout = (t[n].double() for n in ("x", "w1", "w2", "w3", "weights", "dout"))
    idx = t["indices"]
    out, dx, dw = torch.zeros_like(x), torch.zeros_like(x), torch.zeros_like(wt)
    g1, g2, g3 = torch.zeros_like(w1), torch.zeros_like(w2), torch.zeros_like(w3)
    for e in range(c["experts"]):
        rows, place = (idx == e).nonzero(as_tuple=True)
        xe, de, s = x[rows], dout[rows], wt[rows, place][:, None]
        a, b = xe @ w1[e], xe @ w3[e]
        sg = torch.sigmoid(a)
        h = a * sg * b
        y = h @ w2[e]
        out.index_add_(0, rows, s * y)
        dw[rows, place] = (y * de).sum(-1)
        dh = (s * de) @ w2[e].T
        g2[e] = h.T @ (s * de)
        db, da = dh * a * sg, dh * b * (sg + a * sg * (1 - sg))
        g1[e], g3[e] = xe.T @ da, xe.T @ db
        dx.index_add_(0, rows, da @ w1[e].T + db @ w3[e].T)
    return [out, dx, g1, g2, g3, dw]


def _rope(x: torch.Tensor, theta: float, pos: torch.Tensor) -> torch.Tensor:
    """Rotates halves; x [..., positions, dim]."""
    half = x.shape[-1] // 2
    ang = pos.double()[:, None] * theta ** (-torch.arange(half, device=x.device, dtype=F64) / half)
    cos, sin, a, b = ang.cos(), ang.sin(), x[..., :half], x[..., half:]
    return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)


def _rms(x: torch.Tensor, eps: float) -> torch.Tensor:
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)


def _attend(q, k, v, window: int, first: int = 0) -> torch.Tensor:
    """q [heads, n, dim] at positions first ..; k, v [kv heads, positions, dim]: causal, with a sliding window if it is not 0."""
    out, group = [], q.shape[0] // k.shape[0]
    i = first + torch.arange(q.shape[1], device=q.device)[:, None]
    j = torch.arange(k.shape[1], device=q.device)[None, :]
    hidden = (j > i) | ((i - j >= window) if window else torch.zeros_like(j > i))
    for h in range(k.shape[0]):
        s = (q[h * group:(h + 1) * group] @ k[h].T) / math.sqrt(q.shape[-1])
        out.append(torch.softmax(s.masked_fill(hidden, -math.inf), -1) @ v[h])
    return torch.cat(out)


def _exact_training(c: dict, seed: int):
    specs, master = _train_specs(c), _train_master(c, seed)
    p = {n: t.to(BF).double().requires_grad_(True) for n, t in master.items()}
    tokens, targets = (t.cuda().long() for t in _train_batch(c, seed))
    variant = c.get("variant", "")
    cap = 30.0 if "softcap" in variant else 0.0
    z = 1e-4 if "zloss" in variant or "stable" in variant else 0.0
    loss = 0.0
    for b in range(c["batch"]):
        x = _gpt_hidden(c, p, tokens[b]) if c["kind"] == "gpt" else _llama_hidden(c, p, tokens[b])
        logits = x @ p["wte" if c["kind"] == "gpt" else "tok_embeddings" if c["tied"] else "lm_head"][:c["vocab"]].T
        if cap:
            logits = cap * torch.tanh(logits / cap)
        lse = torch.logsumexp(logits, -1)
        part = (lse - logits.gather(1, targets[b][:, None])[:, 0] + z * lse * lse).sum() / (c["batch"] * c["seq"])
        part.backward()
        loss += float(part.detach())
    offsets, end = {}, 0
    for n, shape, *_ in specs:
        offsets[n], end = end, end + (math.prod(shape) + 7) // 8 * 8
    flat, new = torch.zeros(end, dtype=F64, device="cuda"), torch.zeros(end, dtype=F64, device="cuda")
    norm = math.sqrt(sum(float(t.grad.square().sum()) for t in p.values()))
    clip = min(1.0, 1.0 / (norm + 1e-6))
    for n, shape, decay, *_ in specs:                # first step of AdamW: lr 6e-4 / 60 in the warm-up, moments corrected for their start
        g, w = p[n].grad.flatten(), master[n].double().flatten()
        flat[offsets[n]:offsets[n] + g.numel()] = g
        new[offsets[n]:offsets[n] + g.numel()] = w - 1e-5 * (g * clip / ((g * clip).abs() + 1e-8) + (0.1 if decay else 0.0) * w)
    cuts = _cuts([s[0] for s in specs], offsets, end)
    return dict(loss=loss, grads=[flat[a:b] for a, b in cuts], master=new, params=new)


def _gpt_hidden(c: dict, p: dict, tok: torch.Tensor) -> torch.Tensor:
    H, C, T = c["heads"], 64 * c["heads"], tok.numel()
    x = p["wte"][tok] + p["wpe"][:T]
    for i in range(c["layers"]):
        n = f"h.{i}."
        y = F.layer_norm(x, (C,), p[n + "ln_1.weight"], p[n + "ln_1.bias"], 1e-5) @ p[n + "attn.c_attn.weight"].T + p[n + "attn.c_attn.bias"]
        q, k, v = (t.view(T, H, 64).transpose(0, 1) for t in y.split(C, -1))
        if "qknorm" in c["variant"] or "stable" in c["variant"]:
            q, k = _rms(q, 1e-6), _rms(k, 1e-6)
        x = x + _attend(q, k, v, 0).transpose(0, 1).reshape(T, C) @ p[n + "attn.c_proj.weight"].T + p[n + "attn.c_proj.bias"]
        y = F.layer_norm(x, (C,), p[n + "ln_2.weight"], p[n + "ln_2.bias"], 1e-5) @ p[n + "mlp.c_fc.weight"].T + p[n + "mlp.c_fc.bias"]
        x = x + F.gelu(y, approximate="tanh") @ p[n + "mlp.c_proj.weight"].T + p[n + "mlp.c_proj.bias"]
    return F.layer_norm(x, (C,), p["ln_f.weight"], p["ln_f.bias"], 1e-5)


def _llama_hidden(c: dict, p: dict, tok: torch.Tensor) -> torch.Tensor:
    H, K, D, T = c["heads"], c["kv_heads"], c["dim"], tok.numel()
    pos = torch.arange(T, device=tok.device)
    x = p["tok_embeddings"][tok]
    for i in range(c["layers"]):
        n = f"layers.{i}."
        y = (_rms(x, 1e-5) * p[n + "attn_norm"]) @ p[n + "wqkv"].T
        q, k, v = (t.reshape(T, -1, D).transpose(0, 1) for t in y.split([H * D, K * D, K * D], -1))
        if c["qk_norm"]:
            q, k = _rms(q, 1e-6), _rms(k, 1e-6)
        a = _attend(_rope(q, 1e4, pos), _rope(k, 1e4, pos), v, c["window"])
        x = x + a.transpose(0, 1).reshape(T, H * D) @ p[n + "wo"].T
        g, u = ((_rms(x, 1e-5) * p[n + "ffn_norm"]) @ p[n + "w_gate_up"].T).split(c["ff"], -1)
        x = x + (F.silu(g) * u) @ p[n + "w_down"].T
    return _rms(x, 1e-5) * p["norm"]


@torch.no_grad()
def _exact_serving(c: dict, seed: int):
    w = {n: t.double() for n, t, _ in _serve_tensors(c, seed)}
    prompts, chain, logits = _prompts(c, seed), [], []
    for prompt in prompts:
        seq = list(prompt)
        for _ in range(c["steps"] if c["kind"] == "decode" else 0):
            seq.append(_successor(c, seq[-1]))
        out = _served_logits(c, w, torch.tensor(seq, device="cuda"), len(seq) - len(prompt) + 1)
        chain.append(out.argmax(-1).tolist())
        logits.append(out[-1].cpu())
        if any(t != _successor(c, s) for s, t in zip(seq[len(prompt) - 1:], chain[-1])):
            return None
    if c["kind"] == "prompt":
        return dict(token=chain[0][0], logits=logits[0])
    return dict(tokens=np.array([[row[s + 1] for row in chain] for s in range(c["steps"])]), logits=logits)


def _served_logits(c: dict, w: dict, tok: torch.Tensor, last: int) -> torch.Tensor:
    """Logits of the last positions of one sequence."""
    H, K, D, T, glimmer = c["heads"], c["kv_heads"], c["dim"], tok.numel(), c["blocks"] == "glimmer"
    pos, off = torch.arange(T, device=tok.device), 1.0 if glimmer else 0.0
    x = w["tok_embeddings"][tok]
    if glimmer:
        x = _rms(x, 1e-5)
    for i in range(c["layers"]):
        n, local = f"layers.{i}.", not glimmer or (i + 1) % 4 != 0
        y = (_rms(x, 1e-5) * (off + w[n + "attn_norm"])) @ w[n + "wqkv"].T
        q, k, v = (t.reshape(T, -1, D).transpose(0, 1) for t in y[:, :(H + 2 * K) * D].split([H * D, K * D, K * D], -1))
        if glimmer:
            q, k = 3.87 * _rms(q, 1e-6), _rms(k, 1e-6)
        if local:
            q, k = _rope(q, 5e5, pos), _rope(k, 5e5, pos)
        a = torch.cat([_attend(q[:, s:s + 1024], k[:, :s + 1024], v[:, :s + 1024], c["window"] if local else 0, s) for s in range(0, T, 1024)], 1)
        a = a.transpose(0, 1).reshape(T, H * D)
        if glimmer:
            a = a * torch.sigmoid(y[:, (H + 2 * K) * D:])
        a = a @ w[n + "wo"].T
        x = x + (_rms(a, 1e-8) * (1.0 + w[n + "post_attn_norm"]) if glimmer else a)
        g, u = ((_rms(x, 1e-5) * (off + w[n + "ffn_norm"])) @ w[n + "w_gate_up"].T).split(c["ff"], -1)
        a = (F.silu(g) * u) @ w[n + "w_down"].T
        x = x + (_rms(a, 1e-8) * (1.0 + w[n + "post_ffn_norm"]) if glimmer else a)
    out = (_rms(x[T - last:], 1e-5) * w["norm"]) @ w["lm_head"][:c["vocab"]].T
    return 20.0 * torch.tanh(0.19611613513818404 * out / 20.0) if glimmer else out
