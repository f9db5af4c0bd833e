"""The work whose time matters to a user of this framework, as measurable cases.

Each case goes through a public entry point on sizes of the models that the framework serves: the
LLaMA-3.2-1B and LLaMA-3-8B shapes with ternary weights (operators and decoder), and layers of 1B
size of the models of mixer layers (Petulix, Femolix): few enough that BF16 rounding and changed
choices of experts stay small in the logits.  Weights and inputs are drawn from a seed.

  kind "gemv"     a projection of one or a few vectors on prepared weights, FP16 or INT8 activations
  kind "gemm"     a projection of a batch of tokens on prepared weights
  kind "prompt"   a prompt through the ternary decoder, logits of its last token
  kind "step"     one token of one sequence behind a context, FP16 activations (the INT8 option rounds
                  activations so coarsely that two correct implementations' logits differ by a
                  tenth behind 16 layers; its kernel is measured by itself)
  kind "batch"    one lock-step token of several sequences
  kind "mixed"    a prompt through a model of mixer layers, then given tokens one at a time

exact() computes the same outputs in 64 bits with torch operations alone.
"""
from __future__ import annotations

import math

import torch

import ternary_llm_b200 as tl
from ternary_llm_b200 import mixed
from ternary_llm_b200.tllm_format import TernaryTensor, TllmConfig, TllmFile

GROUP = 128

# LLaMA-3.2-1B; four layers of LLaMA-3-8B (one stage of eight) with the 1B model's vocabulary
LLAMA = {
    "1b": dict(vocab_size=128256, hidden_dim=2048, intermediate_dim=8192, n_layers=16, n_heads=32, n_kv_heads=8, head_dim=64),
    "8b-4l": dict(vocab_size=128256, hidden_dim=4096, intermediate_dim=14336, n_layers=4, n_heads=32, n_kv_heads=8, head_dim=128),
}
MAX_SEQ = 4096
MAX_SEQ_BATCH = 2048


def listed():
    return [
        # the smallest call of a decode step: one KV projection of the 1B model, quantised activations
        dict(name="gemv_int8_512x2048", kind="gemv", rows=512, cols=2048, batch=1, int8=True),
        # a few sequences in lock step through the 8B down projection, the longest rows of that model
        dict(name="gemv_b4_4096x14336", kind="gemv", rows=4096, cols=14336, batch=4, int8=False),
        # a short ragged prompt, or the step of a larger batch, through the 8B output projection
        dict(name="gemm_37x4096x4096", kind="gemm", m=37, rows=4096, cols=4096),
        # a long prompt through the 8B up projection, the largest matrix of that model
        dict(name="gemm_2048x14336x4096", kind="gemm", m=2048, rows=14336, cols=4096),
        # an ordinary question to the 1B model
        dict(name="prompt_1b_300", kind="prompt", model="1b", tokens=300),
        # a document in front of the 8B model's layers (head size 128)
        dict(name="prompt_8b4l_2000", kind="prompt", model="8b-4l", tokens=2000),
        # the next token of a conversation with the 1B model, as a program that samples itself asks for it
        dict(name="step_1b_1500", kind="step", model="1b", context=1500),
        # a small server: one token for each of 24 sequences of the 1B model
        dict(name="batch_1b_24x300", kind="batch", model="1b", context=300, sequences=24),
        # a document (prompt alone) through latent attention, selective scan and gated recurrence
        dict(name="petulix_2000", kind="mixed", design="petulix", tokens=2000, steps=0),
        # an answer of that model: a question, then token by token
        dict(name="petulix_100_24", kind="mixed", design="petulix", tokens=100, steps=24),
        # a prompt in front of delta rule, chunk-local beside linear attention, and experts
        dict(name="femolix_1000", kind="mixed", design="femolix", tokens=1000, steps=0),
        # an answer of that model
        dict(name="femolix_100_24", kind="mixed", design="femolix", tokens=100, steps=24),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    kind = rng.choice(["gemv", "gemv", "gemm", "gemm", "prompt", "prompt", "step", "batch", "mixed", "mixed"])
    if kind == "gemv":
        batch = rng.choice([1, 1, 1, 2, 3, 4, 6, 8, 12, 16])
        return dict(kind=kind, rows=_log_int(rng, 96, 14336), cols=GROUP * _log_int(rng, 8, 112), batch=batch,
                    int8=batch == 1 and rng.random() < 0.5)
    if kind == "gemm":
        return dict(kind=kind, m=_log_int(rng, 9, 2048), rows=_log_int(rng, 256, 14336), cols=GROUP * _log_int(rng, 8, 112))
    if kind == "prompt":
        return dict(kind=kind, model=rng.choice(["1b", "8b-4l"]), tokens=_log_int(rng, 16, 1500))
    if kind == "step":
        return dict(kind=kind, model=rng.choice(["1b", "8b-4l"]), context=_log_int(rng, 16, 2000))
    if kind == "batch":
        return dict(kind=kind, model=rng.choice(["1b", "8b-4l"]), context=_log_int(rng, 16, 500), sequences=rng.randint(2, 32))
    return dict(kind=kind, design=rng.choice(["petulix", "femolix"]), tokens=_log_int(rng, 16, 2000), steps=rng.choice([0, 0, 8, 16]))


# ---- inputs ------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _ternary(rows, cols, gen):
    """Masks and scales of a ternary matrix: about 41 % zeros, even signs, scales near those of
    weights of standard deviation 0.02."""
    words = torch.randint(-2 ** 31, 2 ** 31, (5, rows, cols // 32), generator=gen, device="cuda", dtype=torch.int64).to(torch.int32)
    nz = words[0] & words[1] | words[2] & words[3] | words[4] & (words[0] | words[2])
    sign = torch.randint(-2 ** 31, 2 ** 31, nz.shape, generator=gen, device="cuda", dtype=torch.int64).to(torch.int32) & nz
    scales = 0.02 * (0.9 + 0.5 * torch.rand(rows, cols // GROUP, generator=gen, device="cuda"))
    return nz.contiguous(), sign.contiguous(), scales.to(torch.float16)


def _llama(case, seed):
    """(model, token generator) of a ternary case."""
    cfg = TllmConfig(**LLAMA[case["model"]], max_seq_len=MAX_SEQ_BATCH if case["kind"] == "batch" else MAX_SEQ)
    gen = _gen(seed)

    def dense(rows, cols):
        return (torch.randn(rows, cols, generator=gen, device="cuda") * 0.02).to(torch.float16)

    def norm():
        return (1.0 + 0.1 * torch.randn(cfg.hidden_dim, generator=gen, device="cuda")).to(torch.float16)

    m = TllmFile(cfg, dense(cfg.vocab_size, cfg.hidden_dim))
    for _ in range(cfg.n_layers):
        layer = {name: TernaryTensor(*_ternary(rows, cols, gen)) for name, rows, cols in cfg.proj_shapes()}
        layer["attn_norm"], layer["ffn_norm"] = norm(), norm()
        m.layers.append(layer)
    m.final_norm, m.lm_head = norm(), dense(cfg.vocab_size, cfg.hidden_dim)
    return m, gen


# Petulix and Femolix at the width of the 1B model: two layers of each mixer, one of each combination
WIDTH, FF, VOCAB = 2048, 8192, 32000


def _petulix():
    kinds = [
        {"type": "latent_attention", "mixer": {"heads": 16, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 512,
                                               "rot": {"base": 10000.0, "dims": 64}, "scale": 192 ** -0.5}},
        {"type": "mamba1", "mixer": {"inner": 4096, "state": 16, "dt_rank": 128, "conv": 4}},
        {"type": "rglru", "mixer": {"width": 2048, "blocks": 16, "conv": 4}},
    ]
    return {"architecture": "Petulix", "vocab": VOCAB, "width": WIDTH, "norm": {"eps": 1e-5}, "loop": None,
            "layers": [dict(kinds[i % 3], mlp={"kind": "dense", "ff": FF}) for i in range(6)]}


def _femolix():
    dense = {"kind": "dense", "ff": FF}
    moe = {"kind": "moe", "router": {"experts": 32, "top": 4}, "expert": {"ff": FF // 4}}
    delta = {"type": "delta", "mixer": {"heads": 16, "kv_heads": 8, "dim": 128, "vdim": 128, "conv": 4}}
    both = {"type": "parallel", "mixer": {
        "left": {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "mask": {"size": 1024}, "rot": {"base": 10000.0, "dims": 128},
                 "scale": 128 ** -0.5}, "left_scale": 0.5, "right_scale": 0.5,
        "right": {"heads": 8, "dim": 128, "vdim": 128, "decay": [1 - 2.0 ** -(3 + 6 * i / 7) for i in range(8)]}}}
    kinds = [dict(delta, mlp=dense), dict(both, mlp=moe), dict(both, mlp=dense), dict(delta, mlp=moe)]
    return {"architecture": "Femolix", "vocab": VOCAB, "width": WIDTH, "norm": {"eps": 1e-5}, "postln_alpha": 2.0, "logit_softcap": 30.0,
            "layers": [kinds[i % 4] for i in range(4)]}


def _mixed(case, seed):
    """(design, configuration, tensors by name, tokens) of a mixed case."""
    cls, cfg = (mixed.Petulix, _petulix()) if case["design"] == "petulix" else (mixed.Femolix, _femolix())
    tensors = mixed.random_tensors(cls.tensor_shapes(cfg), seed, "cuda")
    tokens = torch.randint(0, VOCAB, (case["tokens"] + case["steps"],), generator=_gen(seed + 1), device="cuda", dtype=torch.int64)
    return cls, cfg, tensors, tokens.to(torch.int32)


def _operator(case, seed):
    """(masks and scales, activations) of a gemv or gemm case."""
    gen = _gen(seed)
    w = _ternary(case["rows"], case["cols"], gen)
    return w, torch.randn(case.get("m") or case["batch"], case["cols"], generator=gen, device="cuda").to(torch.float16)


def _quantise(x):
    """Absmax quantisation of a vector to INT8: (whole numbers, scale)."""
    scale = x.abs().max() / 127.0
    return torch.clamp(torch.round(x / scale), -127, 127), scale


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("gemv", "gemm"):
        w, x = _operator(case, seed)
        s = dict(case, w=tl.PreparedWeight(*w, case["rows"], case["cols"], register=False, keep_source=False), x=x,
                 y=torch.empty(x.shape[0], case["rows"], dtype=torch.float16, device="cuda"))
        if case.get("int8"):
            q, scale = _quantise(x[0].float())
            s["q"], s["scale"] = q.to(torch.int8), float(scale)
        return s
    if kind == "mixed":
        cls, cfg, tensors, tokens = _mixed(case, seed)
        n = case["tokens"]
        dec = tl.Decoder(cls.from_config(cfg, tensors), max_seq_len=max(512, n + case["steps"]))
        return dict(case, dec=dec, prompt=tokens[:n].clone(), given=[tokens[i:i + 1].clone() for i in range(n, n + case["steps"])],
                    logits=torch.empty(1 + case["steps"], VOCAB, dtype=torch.float32, device="cuda"))
    model, gen = _llama(case, seed)
    vocab = model.config.vocab_size
    b = case.get("sequences", 1)
    dec = tl.Decoder(model, max_batch=b, int8_decode=False)
    # the decoder's logits are a view of its own buffer, which a program that keeps them copies
    logits = torch.empty((b, vocab) if kind == "batch" else (vocab,), dtype=torch.float16, device="cuda")
    if kind == "prompt":
        prompt = torch.randint(0, vocab, (case["tokens"],), generator=gen, device="cuda", dtype=torch.int32)
        return dict(case, dec=dec, prompt=prompt, logits=logits)
    contexts = torch.randint(0, vocab, (b, case["context"]), generator=gen, device="cuda", dtype=torch.int32)
    last = torch.randint(0, vocab, (b,), generator=gen, device="cuda", dtype=torch.int32)
    for i in range(b):
        dec.forward_seq(i, contexts[i], 0)
    return dict(case, dec=dec, last=last, logits=logits)


def run(state):
    kind = state["kind"]
    if kind == "gemv":
        if state["int8"]:
            tl.ternary_gemv_int8_packed(state["w"], state["q"], state["scale"], state["y"])
        else:
            tl.ternary_gemv_packed(state["w"], state["x"], state["y"], batch=state["batch"])
        return state["y"]
    if kind == "gemm":
        tl.ternary_gemm_packed(state["x"], state["w"], state["y"], state["m"])
        return state["y"]
    dec = state["dec"]
    out = state["logits"]
    if kind == "prompt":
        return out.copy_(dec.forward(state["prompt"], 0))
    if kind == "step":
        return out.copy_(dec.forward(state["last"], state["context"]))
    if kind == "batch":
        return out.copy_(dec.forward_batch(state["last"], state["context"]))
    out[0].copy_(dec.forward(state["prompt"], 0))
    for i, token in enumerate(state["given"]):
        out[1 + i].copy_(dec.forward(token, state["tokens"] + i))
    return out


# ---- what a pass cannot do without --------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind in ("gemv", "gemm"):
        m, n, k = case.get("m") or case["batch"], case["rows"], case["cols"]
        weights = n * k // 4 + 2 * n * (k // GROUP)
        return {"bytes": weights + m * k * (1 if case.get("int8") else 2) + 2 * m * n, "flops": 2 * m * n * k}
    if kind == "mixed":
        return _mixed_work(case)
    c = TllmConfig(**LLAMA[case["model"]])
    params = sum(rows * cols for _, rows, cols in c.proj_shapes()) * c.n_layers
    head = c.vocab_size * c.hidden_dim
    b, ctx = case.get("sequences", 1), case.get("context", 0)
    tokens = case["tokens"] if kind == "prompt" else b
    rows_out = b if kind == "batch" else 1
    seen = tokens * (tokens + 1) // 2 if kind == "prompt" else b * (ctx + 1)     # (query, position) pairs of a head
    kv = 4 * c.n_kv_heads * c.head_dim * c.n_layers                              # bytes of a position's keys and values
    return {"bytes": params // 4 + params // 64 + 2 * head + kv * (tokens + b * ctx) + 2 * tokens * c.hidden_dim + 2 * rows_out * c.vocab_size,
            "flops": 2 * params * tokens + 2 * head * rows_out + 4 * c.n_heads * c.head_dim * seen * c.n_layers}


def _mixed_work(case):
    cfg = _petulix() if case["design"] == "petulix" else _femolix()
    shapes = (mixed.Petulix if case["design"] == "petulix" else mixed.Femolix).tensor_shapes(cfg)
    n, steps = case["tokens"], case["steps"]
    dense = sum(math.prod(s) for name, s in shapes.items() if name not in ("embed", "head") and ".mlp.e" not in name)
    expert = used = 0
    for layer in cfg["layers"]:
        if layer["mlp"]["kind"] == "moe":
            r = layer["mlp"]["router"]
            one = 3 * WIDTH * layer["mlp"]["expert"]["ff"]
            expert += r["top"] * one
            used += min(r["experts"], r["top"] * n) * one          # experts that a prompt's tokens reach
    head = VOCAB * WIDTH
    pairs = n * (n + 1) // 2
    if case["design"] == "petulix":
        attend = 2 * 2 * 16 * (192 + 128)
        cache = 2 * 2 * 576
        state = 2 * 4 * 4096 * 16 + 2 * 4 * 2048
    else:
        full, rest = divmod(n, 1024)
        pairs = full * 1024 * 1025 // 2 + rest * (rest + 1) // 2
        attend = 2 * 2 * 16 * 256
        cache = 2 * 2 * 4 * 256
        state = 2 * 4 * 16 * 128 * 128 + 2 * 4 * 8 * 128 * 128
    read = 2 * (dense + used + head) + cache * n + state
    flops = 2 * (dense + expert) * n + 2 * head + attend * pairs
    read += steps * (2 * (dense + expert + head) + cache * n + 2 * state)
    flops += steps * (2 * (dense + expert + head) + attend * n)
    return {"bytes": read + 4 * VOCAB * (1 + steps), "flops": flops}


def tolerance(case):
    """About four times what the present code is off exact(): FP16 results of an operator, FP16
    rounding between the operators of a decoder, BF16 rounding between those of a mixed model."""
    if case["kind"] in ("gemv", "gemm"):
        return {"rel": 1e-3}
    if case.get("design") == "petulix":
        return {"rel": 0.03}
    return {"rel": 0.011}


# ---- the same outputs in 64 bits ----------------------------------------------------------
F = torch.float64


def _matrix(w):
    """A ternary matrix as 64-bit numbers."""
    nz, sign, scales = w
    shifts = torch.arange(32, device=nz.device, dtype=torch.int32)
    out = torch.empty(nz.shape[0], nz.shape[1] * 32, dtype=F, device=nz.device)
    for r in range(0, nz.shape[0], 4096):
        t = ((nz[r:r + 4096, :, None] >> shifts) & 1) * (2 * ((sign[r:r + 4096, :, None] >> shifts) & 1) - 1)
        out[r:r + 4096] = t.reshape(t.shape[0], -1).to(F)
    return out.view(nz.shape[0], -1, GROUP).mul_(scales.to(F)[:, :, None]).view(nz.shape[0], -1)


def _norm(x, w, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * w.to(F)


def _causal(q, k, v, scale, sink=None, chunk=0):
    """q [n, H, d], k [n, G, d], v [n, G, e]: causal attention, optionally with exp(sink) in the
    denominator or within chunks of positions."""
    n, heads, group = q.shape[0], q.shape[1], q.shape[1] // k.shape[1]
    i = torch.arange(n, device=q.device)
    hidden = i[None, :] > i[:, None]
    if chunk:
        hidden |= i[None, :] // chunk != i[:, None] // chunk
    out = torch.empty(n, heads, v.shape[2], dtype=F, device=q.device)
    for h in range(heads):
        s = (q[:, h] @ k[:, h // group].T * scale).masked_fill_(hidden, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].to(F).expand(n, 1)], dim=1)
        out[:, h] = torch.softmax(s, dim=1)[:, :n] @ v[:, h // group]
    return out


def _exact_llama(model, tokens):
    """Logits behind the last of tokens [sequences, n]."""
    c = model.config
    b, n = tokens.shape
    res = model.embedding[tokens.long()].to(F)
    i = torch.arange(c.head_dim // 2, device="cuda", dtype=F)
    angle = torch.arange(n, device="cuda", dtype=F)[:, None] * c.rope_theta ** (-2 * i / c.head_dim)
    cos, sin = torch.cos(angle)[:, None, :], torch.sin(angle)[:, None, :]

    def linear(x, *names):
        return [x @ _matrix((layer[t].nonzero_masks, layer[t].sign_masks, layer[t].scales)).T for t in names]

    def rotate(x):
        u, v = x[..., 0::2], x[..., 1::2]
        return torch.stack([u * cos - v * sin, u * sin + v * cos], dim=-1).reshape(x.shape)

    for layer in model.layers:
        q, k, v = linear(_norm(res, layer["attn_norm"], c.rms_norm_eps), "q_proj", "k_proj", "v_proj")
        heads = [rotate(q.view(b, n, c.n_heads, -1)), rotate(k.view(b, n, c.n_kv_heads, -1)), v.view(b, n, c.n_kv_heads, -1)]
        a = torch.stack([_causal(*(t[s] for t in heads), c.head_dim ** -0.5).reshape(n, -1) for s in range(b)])
        res = res + linear(a, "o_proj")[0]
        gate, up = linear(_norm(res, layer["ffn_norm"], c.rms_norm_eps), "gate_proj", "up_proj")
        res = res + linear(torch.nn.functional.silu(gate) * up, "down_proj")[0]
    return _norm(res[:, -1], model.final_norm, c.rms_norm_eps) @ model.lm_head.to(F).T


def _half_turn(x, base):
    """Rotation by position of the whole last axis, entry i paired with i + half."""
    n, half = x.shape[0], x.shape[-1] // 2
    i = torch.arange(half, device=x.device, dtype=F)
    angle = torch.arange(n, device=x.device, dtype=F)[:, None] * base ** (-i / half)
    angle = angle.view((n,) + (1,) * (x.dim() - 2) + (half,))
    u, v = x[..., :half], x[..., half:]
    return torch.cat([u * torch.cos(angle) - v * torch.sin(angle), v * torch.cos(angle) + u * torch.sin(angle)], dim=-1)


def _conv(x, w):
    """Causal convolution per channel, w [channels, taps]."""
    n, taps = x.shape[0], w.shape[1]
    padded = torch.cat([x.new_zeros(taps - 1, x.shape[1]), x])
    return sum(padded[j:j + n] * w[:, j] for j in range(taps))


def _exact_mixer(kind, m, W, h, eps):
    n, silu, softplus = h.shape[0], torch.nn.functional.silu, torch.nn.functional.softplus
    if kind == "latent_attention":
        heads, d, r, e, rank = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
        q, kv = (h @ W["q"].T).view(n, heads, d + r), h @ W["dkv"].T
        latent, base = _norm(kv[:, :rank], W["dkv.norm"], eps), m["rot"]["base"]
        q = torch.cat([q[:, :, :d], _half_turn(q[:, :, d:], base)], dim=2)
        k = torch.cat([(latent @ W["uk"].T).view(n, heads, d), _half_turn(kv[:, rank:], base)[:, None].expand(n, heads, r)], dim=2)
        o = _causal(q, k, (latent @ W["uv"].T).view(n, heads, e), m["scale"], sink=W["sink"])
        return (o * torch.sigmoid(h @ W["g"].T)[:, :, None]).reshape(n, -1) @ W["o"].T
    if kind == "mamba1":
        inner, st, dr = m["inner"], m["state"], m["dt_rank"]
        x, z = (h @ W["in"].T).split(inner, dim=1)
        x = silu(_conv(x, W["conv"]) + W["conv.b"])
        p = x @ W["x"].T
        dt = softplus(p[:, :dr] @ W["dt"].T + W["dt.b"])
        a, y, S = -torch.exp(W["A_log"]), torch.empty_like(x), x.new_zeros(inner, st)
        dx = dt * x
        for t in range(n):
            S = torch.exp(dt[t][:, None] * a) * S + dx[t][:, None] * p[t, dr:dr + st]
            y[t] = S @ p[t, dr + st:]
        return ((y + W["D"] * x) * silu(z)) @ W["o"].T
    if kind == "rglru":
        nb, y = m["blocks"], torch.nn.functional.gelu(h @ W["y"].T + W["y.b"], approximate="tanh")
        u = _conv(h @ W["x"].T + W["x.b"], W["conv"]) + W["conv.b"]
        r, i = (torch.sigmoid(torch.einsum("nbi,boi->nbo", u.view(n, nb, -1), W[g]) + W[g + ".b"]).reshape(n, -1) for g in ("ra", "ri"))
        log_a = -8.0 * r * softplus(W["lam"])
        a, x = torch.exp(log_a), torch.sqrt(-torch.expm1(2 * log_a)) * i * u
        S, out = x.new_zeros(x.shape[1]), torch.empty_like(x)
        for t in range(n):
            S = a[t] * S + x[t]
            out[t] = S
        return (out * y) @ W["o"].T
    if kind == "delta":
        heads, g, d, e = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        q, k, v = (silu(_conv(h @ W[t].T, W[t + ".conv"])) for t in "qkv")
        q, k = (t.view(n, g, d) * torch.rsqrt((t.view(n, g, d) ** 2).sum(-1, keepdim=True) + 1e-6) for t in (q, k))
        q, k = (t.repeat_interleave(heads // g, dim=1) for t in (q * d ** -0.5, k))
        v, beta = v.view(n, heads, e), torch.sigmoid(h @ W["b"].T)
        decay = torch.exp(-torch.exp(W["A_log"]) * softplus(h @ W["a"].T + W["dt_bias"]))
        S, o = h.new_zeros(heads, d, e), torch.empty_like(v)
        for t in range(n):
            S = S * decay[t][:, None, None]
            S = S + k[t][:, :, None] * (beta[t][:, None] * (v[t] - (k[t][:, None] @ S)[:, 0]))[:, None]
            o[t] = (q[t][:, None] @ S)[:, 0]
        return (_norm(o, W["norm"], eps).reshape(n, -1) * silu(h @ W["g"].T)) @ W["o"].T
    left, right = m["left"], m["right"]
    L, R = ({k[len(p):]: v for k, v in W.items() if k.startswith(p)} for p in ("left.", "right."))
    q, k = (_half_turn(_norm((h @ L[t].T).view(n, -1, left["dim"]), L[t + ".norm"], eps), left["rot"]["base"]) for t in "qk")
    o = _causal(q, k, (h @ L["v"].T).view(n, -1, left["vdim"]), left["scale"], chunk=left["mask"]["size"])
    y = m["left_scale"] * (o.reshape(n, -1) @ L["o"].T)
    q, k, v = (silu(h @ R[t].T).view(n, right["heads"], -1) for t in "qkv")
    decay = torch.tensor(right["decay"], device=h.device, dtype=torch.float32).to(F)[:, None, None]
    S, o = h.new_zeros(right["heads"], right["dim"], right["vdim"]), torch.empty_like(v)
    for t in range(n):
        S = decay * S + k[t][:, :, None] * v[t][:, None]
        o[t] = (q[t][:, None] @ S)[:, 0]
    return y + m["right_scale"] * ((_norm(o.reshape(n, -1), R["norm"], eps) * torch.sigmoid(h @ R["g"].T)) @ R["o"].T)


def _exact_mixed(case, seed):
    _, cfg, tensors, tokens = _mixed(case, seed)
    eps, petulix = cfg["norm"]["eps"], case["design"] == "petulix"
    act = (lambda t: torch.nn.functional.gelu(t, approximate="tanh")) if petulix else torch.nn.functional.silu

    def take(prefix):
        return {name[len(prefix):]: t.to(F) for name, t in tensors.items() if name.startswith(prefix) and ".mlp." not in name}

    def gated(x, p):
        return (act(x @ tensors[p + "gate"].to(F).T) * (x @ tensors[p + "up"].to(F).T)) @ tensors[p + "down"].to(F).T

    def feed_forward(x, mlp, p):
        if mlp["kind"] == "dense":
            return gated(x, p)
        z, chosen = torch.topk(x @ tensors[p + "router"].to(F).T, mlp["router"]["top"], dim=1)
        weight, out = torch.softmax(z, dim=1), torch.zeros_like(x)
        for e in range(mlp["router"]["experts"]):
            t, s = torch.nonzero(chosen == e, as_tuple=True)
            if len(t):
                out[t] += weight[t, s][:, None] * gated(x[t], f"{p}e{e}.")
        return out

    x = tensors["embed"][tokens.long()].to(F)
    for i, layer in enumerate(cfg["layers"]):
        p = f"l{i}."
        W, mix = take(p), take(p + "mix.")
        if petulix:
            x = x + _norm(_exact_mixer(layer["type"], layer["mixer"], mix, _norm(x, W["norm1"], eps), eps), W["norm1b"], eps)
            x = x + _norm(feed_forward(_norm(x, W["norm2"], eps), layer["mlp"], p + "mlp."), W["norm2b"], eps)
        else:
            alpha = cfg["postln_alpha"]
            x = _norm(alpha * x + _exact_mixer(layer["type"], layer["mixer"], mix, x, eps), W["norm1"], eps)
            x = _norm(alpha * x + feed_forward(x, layer["mlp"], p + "mlp."), W["norm2"], eps)
    x = _norm(x[case["tokens"] - 1:], tensors["final.norm"], eps)
    if petulix:
        return x @ tensors["embed"].to(F).T
    cap = cfg["logit_softcap"]
    return cap * torch.tanh(x @ tensors["head"].to(F).T / cap)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("gemv", "gemm"):
        w, x = _operator(case, seed)
        x = x.to(F)
        if case.get("int8"):
            q, scale = _quantise(x[0].float())
            x = (q.to(F) * float(scale))[None, :]
        return x @ _matrix(w).T
    if kind == "mixed":
        return _exact_mixed(case, seed)
    model, gen = _llama(case, seed)
    vocab = model.config.vocab_size
    if kind == "prompt":
        tokens = torch.randint(0, vocab, (case["tokens"],), generator=gen, device="cuda", dtype=torch.int32)
        return _exact_llama(model, tokens[None])[0]
    b = case.get("sequences", 1)
    contexts = torch.randint(0, vocab, (b, case["context"]), generator=gen, device="cuda", dtype=torch.int32)
    last = torch.randint(0, vocab, (b,), generator=gen, device="cuda", dtype=torch.int32)
    logits = _exact_llama(model, torch.cat([contexts, last[:, None]], dim=1))
    return logits[0] if kind == "step" else logits
