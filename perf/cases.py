"""The work that users of this library have it do, as measurable cases.

Every case goes through the library's public entry points: the fused all-reduce + residual + RMSNorm op (one rank, as
``bench.py`` runs it on one GPU), the bf16 and block-scaled e4m3 linear layers, decode and prompt attention, the e4m3
feed-forward block of the 70B-shaped model, and a whole decode step of the 8B-shaped model replayed from its CUDA
graph. Sizes are those of the Llama-3-8B / 70B shapes (whole, or one rank's share at TP=2 and TP=8) and of the fused
op's own sweep (hidden 4096 to 8192, 1 to 8192 tokens); token counts and sequence lengths are ragged where a serving
program's are.
"""
from __future__ import annotations

import math

import torch

import torch_dist_ext_b200 as tdx
from torch_dist_ext_b200.models.llama import LlamaConfig, TPLlama
from torch_dist_ext_b200.ops import activation, attention, gemm
from torch_dist_ext_b200.parallel import comm

DEV = "cuda"
HEAD = 128
EPS = 1e-6
TYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}

# (out features, in features) of the projections of the 8B shape at TP=1 and TP=8, and of its sharded lm-head
LINEAR = [(6144, 4096), (4096, 4096), (28672, 4096), (4096, 14336), (768, 4096), (4096, 512), (3584, 4096), (4096, 1792),
          (16032, 4096)]
# the same of the 70B shape (e4m3 weights) at TP=2 and TP=8
LINEAR_FP8 = [(5120, 8192), (8192, 4096), (28672, 8192), (8192, 14336), (1280, 8192), (8192, 1024), (7168, 8192), (8192, 3584)]
# (query heads, KV heads): the 8B shape, and one rank's share at TP=8 of the 8B and of the 70B shape
HEADS = [(32, 8), (4, 1), (8, 1)]
MOST_FLOPS = 0.96e12


def listed():
    return [
        # the op a tensor-parallel decoder layer calls twice, at the headline message (128 tokens x 4096, bf16)
        dict(name="norm_128x4096", kind="norm", tokens=128, hidden=4096, dtype="bf16", out="same"),
        # a long prompt's rows, quantised for the e4m3 projection that follows (one scale per 128 columns)
        dict(name="norm_8192x7168_fp8", kind="norm", tokens=8192, hidden=7168, dtype="bf16", out="block"),
        # gate/up projection of a decode batch: streams 235 MB of weights
        dict(name="linear_64x28672", kind="linear", tokens=64, n=28672, k=4096, dtype="bf16"),
        # down projection of an odd-sized prompt
        dict(name="linear_1999x4096", kind="linear", tokens=1999, n=4096, k=14336, dtype="bf16"),
        # one rank's gate/up projection of the 70B shape, decode batch 64
        dict(name="fp8_64x7168", kind="fp8_linear", tokens=64, n=7168, k=8192),
        # the same projection at TP=2 for a 2048-token prompt
        dict(name="fp8_2048x28672", kind="fp8_linear", tokens=2048, n=28672, k=8192),
        # one sequence, one rank's heads: the latency of a lone user's step
        dict(name="decode_attn_1x2000", kind="decode_attn", batch=1, length=2000, hq=8, hkv=1),
        # a full batch of ragged sequences
        dict(name="decode_attn_64x2048", kind="decode_attn", batch=64, length=2048, hq=32, hkv=8),
        # a short odd prompt on one rank's heads, and a long one on all heads
        dict(name="prompt_attn_1337", kind="prompt_attn", s=1337, hq=8, hkv=1),
        dict(name="prompt_attn_8192", kind="prompt_attn", s=8192, hq=32, hkv=8),
        # norm -> gate/up -> silu*mul -> down -> norm of the 70B shape on one rank of eight, 2048-token prompt
        dict(name="mlp_fp8_2048", kind="mlp_fp8", tokens=2048, hidden=8192, ffn=3584),
        # four layers and the sharded lm-head of the 8B shape on one rank of eight, batch 16 over 2048 positions
        dict(name="decode_step_16", kind="decode_step", batch=16, length=2048, layers=4),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["norm", "linear", "linear", "fp8_linear", "fp8_linear", "decode_attn", "prompt_attn", "mlp_fp8", "decode_step"])
    if kind == "norm":
        return dict(kind=kind, tokens=_log_int(rng, 1, 8192), hidden=rng.choice([4096, 5120, 7168, 8192]),
                    dtype=rng.choice(["bf16", "bf16", "fp16", "fp32"]), out=rng.choice(["same", "same", "token", "block"]))
    if kind == "linear":
        n, k = rng.choice(LINEAR)
        return dict(kind=kind, tokens=_log_int(rng, 1, min(8192, int(MOST_FLOPS / (2.0 * n * k)))), n=n, k=k,
                    dtype=rng.choice(["bf16", "bf16", "bf16", "fp16"]))
    if kind == "fp8_linear":
        n, k = rng.choice(LINEAR_FP8)
        return dict(kind=kind, tokens=_log_int(rng, 1, min(8192, int(MOST_FLOPS / (2.0 * n * k)))), n=n, k=k)
    if kind == "decode_attn":
        hq, hkv = rng.choice(HEADS)
        return dict(kind=kind, batch=_log_int(rng, 1, 64), length=_log_int(rng, 17, 2048 if hkv > 1 else 8192), hq=hq, hkv=hkv)
    if kind == "prompt_attn":
        hq, hkv = rng.choice(HEADS)
        return dict(kind=kind, s=_log_int(rng, 16, 8192), hq=hq, hkv=hkv)
    if kind == "mlp_fp8":
        return dict(kind=kind, tokens=_log_int(rng, 1, 4096), hidden=8192, ffn=3584)
    return dict(kind=kind, batch=_log_int(rng, 1, 64), length=_log_int(rng, 64, 2048), layers=rng.choice([2, 3, 4]))


# ---- inputs: plain torch, from the seed alone ---------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _randn(g, *shape, std=1.0, mean=0.0, dtype=torch.bfloat16):
    x = torch.empty(*shape, dtype=torch.float32, device=DEV)
    return x.normal_(mean, std, generator=g).to(dtype)


def _quant_rows(x):
    """e4m3 rows with one fp32 scale per 128 columns."""
    t, k = x.shape
    b = x.float().view(t, k // 128, 128)
    scale = b.abs().amax(-1, keepdim=True).clamp_min(1e-10) / 448.0
    return (b / scale).clamp(-448, 448).to(torch.float8_e4m3fn).view(t, k), scale.squeeze(-1).contiguous()


def _quant_weight(w):
    """e4m3 weights with one fp32 scale per 128 x 128 block."""
    n, k = w.shape
    b = w.float().view(n // 128, 128, k // 128, 128)
    scale = b.abs().amax(dim=(1, 3), keepdim=True).clamp_min(1e-10) / 448.0
    return (b / scale).clamp(-448, 448).to(torch.float8_e4m3fn).view(n, k), scale.view(n // 128, k // 128).contiguous()


def _norm_inputs(case, seed):
    g, dt = _gen(seed), TYPES[case["dtype"]]
    t, h = case["tokens"], case["hidden"]
    return dict(x=_randn(g, t, h, dtype=dt), res=_randn(g, t, h, dtype=dt), gamma=_randn(g, h, std=0.1, mean=1.0, dtype=dt))


def _linear_inputs(case, seed):
    g, dt = _gen(seed), TYPES[case["dtype"]]
    return dict(a=_randn(g, case["tokens"], case["k"], dtype=dt), w=_randn(g, case["n"], case["k"], std=0.02, dtype=dt))


def _fp8_inputs(case, seed):
    g = _gen(seed)
    aq, a_scale = _quant_rows(_randn(g, case["tokens"], case["k"]))
    wq, w_scale = _quant_weight(_randn(g, case["n"], case["k"], std=0.02))
    return dict(aq=aq, a_scale=a_scale, wq=wq, w_scale=w_scale)


def _decode_attn_inputs(case, seed):
    g = _gen(seed)
    b, n, hq, hkv = case["batch"], case["length"], case["hq"], case["hkv"]
    lens = torch.randint(n // 2 + 1, n + 1, (b,), device=DEV, generator=g, dtype=torch.int32)
    lens[0] = n
    return dict(q=_randn(g, b, hq, HEAD), k=_randn(g, b, n, hkv, HEAD), v=_randn(g, b, n, hkv, HEAD), lens=lens)


def _prompt_attn_inputs(case, seed):
    # views into the fused qkv projection of the prompt, as the model passes them
    g = _gen(seed)
    s, hq, hkv = case["s"], case["hq"], case["hkv"]
    qkv = _randn(g, s, (hq + 2 * hkv) * HEAD)
    q, k, v = qkv.split([hq * HEAD, hkv * HEAD, hkv * HEAD], dim=1)
    return dict(q=q.view(s, hq, HEAD), k=k.view(s, hkv, HEAD), v=v.view(s, hkv, HEAD))


def _mlp_inputs(case, seed):
    g = _gen(seed)
    t, h, f = case["tokens"], case["hidden"], case["ffn"]
    wgu, sgu = _quant_weight(_randn(g, 2 * f, h, std=0.02))
    wd, sd = _quant_weight(_randn(g, h, f, std=0.02))
    return dict(x=_randn(g, t, h), res=_randn(g, t, h), g1=_randn(g, h, std=0.02, mean=1.0), g2=_randn(g, h, std=0.02, mean=1.0),
                wgu=wgu, sgu=sgu, wd=wd, sd=sd)


_STEP = dict(hidden=4096, hq=4, hkv=1, ffn=1792, vocab=16032, theta=5e5, eps=1e-5)


def _step_inputs(case, seed):
    g, c = _gen(seed), _STEP
    b, n = case["batch"], case["length"]
    layers = []
    for _ in range(case["layers"]):
        layers.append(dict(
            ln1=_randn(g, c["hidden"], std=0.02, mean=1.0), ln2=_randn(g, c["hidden"], std=0.02, mean=1.0),
            wqkv=_randn(g, (c["hq"] + 2 * c["hkv"]) * HEAD, c["hidden"], std=0.02),
            wo=_randn(g, c["hidden"], c["hq"] * HEAD, std=0.02),
            wgu=_randn(g, 2 * c["ffn"], c["hidden"], std=0.02), wd=_randn(g, c["hidden"], c["ffn"], std=0.02),
            k=_randn(g, b, n, c["hkv"], HEAD), v=_randn(g, b, n, c["hkv"], HEAD)))
    positions = torch.randint(n // 2, n, (b,), device=DEV, generator=g)
    positions[0] = n - 1
    return dict(layers=layers, embed=_randn(g, c["vocab"], c["hidden"], std=0.02), lm_head=_randn(g, c["vocab"], c["hidden"], std=0.02),
                final_norm=_randn(g, c["hidden"], std=0.02, mean=1.0), positions=positions,
                tokens=torch.randint(0, c["vocab"], (b,), device=DEV, generator=g))


_INPUTS = dict(norm=_norm_inputs, linear=_linear_inputs, fp8_linear=_fp8_inputs, decode_attn=_decode_attn_inputs,
               prompt_attn=_prompt_attn_inputs, mlp_fp8=_mlp_inputs, decode_step=_step_inputs)


def _environment():
    try:
        comm.get_comm()
    except RuntimeError:
        tdx.setup_env(0, 1)


def prepare(case, seed):
    _environment()
    state = dict(_INPUTS[case["kind"]](case, seed), case=case)
    if case["kind"] == "norm":
        state["ws"] = tdx.get_workspace(state["x"])
    if case["kind"] == "decode_step":
        state["model"] = _load_model(case, state)
        state["layers"] = None          # the model holds the weights and the caches from here on
    return state


def _load_model(case, st):
    """The 8B-shaped model's share of one rank of eight with these weights and caches, its step captured."""
    b, n = case["batch"], case["length"]
    cfg = LlamaConfig.shard_of(LlamaConfig.llama3_8b(), 8, n_layers=case["layers"])
    model = TPLlama(cfg, max_batch=b, max_seq=n)
    for i, src in enumerate(st["layers"]):
        L = model.layers[i]
        L["ln1"].copy_(src["ln1"])
        L["ln2"].copy_(src["ln2"])
        for name in ("wqkv", "wo", "wgu", "wd"):
            L[name].w.copy_(src[name])
        model.k_cache[i].copy_(src["k"])
        model.v_cache[i].copy_(src["v"])
    model.embed.copy_(st.pop("embed"))
    model.lm_head.copy_(st.pop("lm_head"))
    model.final_norm.copy_(st.pop("final_norm"))
    saved = [(k[:, 0].clone(), v[:, 0].clone()) for k, v in zip(model.k_cache, model.v_cache)]
    model.capture_decode(b, n)
    for (k0, v0), k, v in zip(saved, model.k_cache, model.v_cache):      # the warm-up appended at position 0
        k[:, 0].copy_(k0)
        v[:, 0].copy_(v0)
    return model


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "norm":
        x, res, gamma = state["x"], state["res"], state["gamma"]
        if case["out"] == "same":
            return tdx.allreduce_rms(0, 1, x, res, gamma, EPS, state["ws"])
        return tdx.allreduce_rms_fp8(x, res, gamma, EPS, state["ws"], block_scaled=case["out"] == "block")
    if kind == "linear":
        return gemm.linear(state["a"], state["w"])
    if kind == "fp8_linear":
        return gemm.linear_fp8_blockscaled(state["aq"], state["a_scale"], state["wq"], state["w_scale"])
    if kind == "decode_attn":
        return attention.decode_attention(state["q"], state["k"], state["v"], state["lens"], case["length"])
    if kind == "prompt_attn":
        return attention.prefill_attention(state["q"], state["k"], state["v"])
    if kind == "mlp_fp8":
        x, xs, res = tdx.allreduce_rms_fp8(state["x"], state["res"], state["g1"], EPS, block_scaled=True)
        gu = gemm.linear_fp8_blockscaled(x, xs, state["wgu"], state["sgu"])
        act, act_scale = activation.silu_mul(gu, quant_block128=True)
        y = gemm.linear_fp8_blockscaled(act, act_scale, state["wd"], state["sd"])
        return tdx.allreduce_rms_fp8(y, res, state["g2"], EPS, block_scaled=True)
    # The next tokens are the arg-max of these logits: with random weights their two best are often closer than a
    # rounding step of the hidden state, so what is handed on for comparison is the logits and the appended caches.
    model = state["model"]
    model.decode(state["tokens"], state["positions"])
    return dict(logits=gemm.linear(model.last_hidden, model.lm_head, out_dtype=torch.float32), k=model.k_cache, v=model.v_cache)


# ---- what a pass cannot do without ----------------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind == "norm":
        n, e = case["tokens"] * case["hidden"], TYPES[case["dtype"]].itemsize
        out = n * e if case["out"] == "same" else n + 4 * case["tokens"] * (1 if case["out"] == "token" else case["hidden"] // 128)
        return dict(bytes=3 * n * e + case["hidden"] * e + out, flops=6 * n)
    if kind == "linear":
        m, n, k = case["tokens"], case["n"], case["k"]
        return dict(bytes=2 * (m * k + n * k + m * n), flops=2 * m * n * k)
    if kind == "fp8_linear":
        m, n, k = case["tokens"], case["n"], case["k"]
        return dict(bytes=m * k + n * k + 4 * (m * k // 128 + n * k // 128 ** 2) + 2 * m * n, flops=2 * m * n * k)
    if kind == "decode_attn":
        b, n, hq, hkv = case["batch"], case["length"], case["hq"], case["hkv"]
        seen = n + (b - 1) * 0.75 * n           # lengths are spread over the upper half of the range
        return dict(bytes=4 * seen * hkv * HEAD + 4 * b * hq * HEAD + 4 * b, flops=4 * seen * hq * HEAD)
    if kind == "prompt_attn":
        s, hq, hkv = case["s"], case["hq"], case["hkv"]
        return dict(bytes=2 * s * HEAD * (2 * hq + 2 * hkv), flops=4 * (s * (s + 1) / 2) * hq * HEAD)
    if kind == "mlp_fp8":
        t, h, f = case["tokens"], case["hidden"], case["ffn"]
        return dict(bytes=t * h * (2 + 2 + 2 + 1) + 4 * t * h // 128 + 3 * f * h, flops=6 * t * h * f)
    c, b, n = _STEP, case["batch"], case["length"]
    per_layer = c["hidden"] * HEAD * (c["hq"] + 2 * c["hkv"]) + c["hidden"] * c["hq"] * HEAD + 3 * c["hidden"] * c["ffn"]
    weights = case["layers"] * per_layer + c["vocab"] * c["hidden"]
    seen = n + (b - 1) * 0.75 * n
    kv = case["layers"] * seen * c["hkv"] * HEAD * 2
    return dict(bytes=2 * weights + 2 * kv + 2 * b * c["hidden"] + 4 * b * c["vocab"],
                flops=2 * b * weights + case["layers"] * 4 * seen * c["hq"] * HEAD)


def tolerance(case):
    kind = case["kind"]
    if kind == "norm":
        if case["out"] != "same":
            return dict(rel=4e-3, max=0.15)     # a value on the edge of an e4m3 step lands one step (1/8) off
        return dict(rel=2e-6, max=2e-5) if case["dtype"] == "fp32" else dict(rel=4e-3, max=0.02)
    if kind in ("linear", "fp8_linear"):
        return dict(rel=7e-3, max=0.03)         # one rounding to 16 bits
    if kind in ("decode_attn", "prompt_attn"):
        return dict(rel=9e-3, max=0.1)          # 16-bit probabilities and one rounding to 16 bits
    if kind == "mlp_fp8":
        return dict(rel=1.2e-2, max=0.3)
    return dict(rel=2.5e-2, max=0.2)            # rounding to 16 bits in every layer


# ---- the same in plain torch, 64 bits ---------------------------------------------------------------------------------
def _e4m3(y, columns):
    """(e4m3 values, scales) of rows ``y`` in 64 bits, one scale per ``columns`` columns."""
    t, h = y.shape
    b = y.view(t, h // columns, columns)
    scale = b.abs().amax(-1, keepdim=True).clamp_min(1e-10) / 448.0
    q = (b / scale).clamp(-448, 448).float().to(torch.float8_e4m3fn)
    return q.view(t, h), scale.squeeze(-1)


def _rows(q, scale):
    t, h = q.shape
    return (q.double().view(t, scale.shape[1], -1) * scale.double().unsqueeze(-1)).view(t, h)


def _norm64(x, res, gamma, eps):
    """(normalised rows, residual): the residual is stored in the data type, the norm is of the stored values."""
    r = (x.double() + res.double()).to(gamma.dtype)
    y = r.double()
    return y * torch.rsqrt(y.square().mean(-1, keepdim=True) + eps) * gamma.double(), r


def _weight64(wq, scale):
    n, k = wq.shape
    return (wq.double().view(n // 128, 128, k // 128, 128) * scale.double().view(n // 128, 1, k // 128, 1)).view(n, k)


def _attend64(q, k, v, mask=None):
    """One KV head: ``q [R, 128]``, ``k``/``v [N, 128]`` in 64 bits."""
    p = (q @ k.t()) / math.sqrt(HEAD)
    if mask is not None:
        p.masked_fill_(mask, float("-inf"))
    return torch.softmax(p, -1) @ v


def exact(case, seed):
    st = _INPUTS[case["kind"]](case, seed)
    kind = case["kind"]
    if kind == "norm":
        y, r = _norm64(st["x"], st["res"], st["gamma"], EPS)
        if case["out"] == "same":
            return y, r.double()
        q, scale = _e4m3(y, case["hidden"] if case["out"] == "token" else 128)
        return q.double(), scale, r.double()
    if kind == "linear":
        return st["a"].double() @ st["w"].double().t()
    if kind == "fp8_linear":
        return _rows(st["aq"], st["a_scale"]) @ _weight64(st["wq"], st["w_scale"]).t()
    if kind == "decode_attn":
        b, hq, hkv = case["batch"], case["hq"], case["hkv"]
        out = torch.empty(b, hq, HEAD, dtype=torch.float64, device=DEV)
        g = hq // hkv
        for i in range(b):
            n = int(st["lens"][i])
            for h in range(hkv):
                out[i, h * g:(h + 1) * g] = _attend64(st["q"][i, h * g:(h + 1) * g].double(), st["k"][i, :n, h].double(), st["v"][i, :n, h].double())
        return out
    if kind == "prompt_attn":
        s, hq, hkv = case["s"], case["hq"], case["hkv"]
        out = torch.empty(s, hq, HEAD, dtype=torch.float64, device=DEV)
        mask = torch.ones(s, s, dtype=torch.bool, device=DEV).triu(1)
        for h in range(hq):
            kv = h // (hq // hkv)
            out[:, h] = _attend64(st["q"][:, h].double(), st["k"][:, kv].double(), st["v"][:, kv].double(), mask)
        return out
    if kind == "mlp_fp8":
        # in 64 bits between the points where the block's entry points hand on 16-bit or e4m3 rows
        f = case["ffn"]
        y, res = _norm64(st["x"], st["res"], st["g1"], EPS)
        gu = (_rows(*_e4m3(y, 128)) @ _weight64(st["wgu"], st["sgu"]).t()).to(torch.bfloat16).double()
        act = (torch.nn.functional.silu(gu[:, :f]) * gu[:, f:]).to(torch.bfloat16).double()
        act = _rows(*_e4m3(act, 128))
        down = (act @ _weight64(st["wd"], st["sd"]).t()).to(torch.bfloat16)
        y, res = _norm64(down, res, st["g2"], EPS)
        q, scale = _e4m3(y, 128)
        return q.double(), scale, res.double()
    return _step64(case, st)


def _step64(case, st):
    c, b = _STEP, case["batch"]
    hq, pos, rows = c["hq"], st["positions"], torch.arange(case["batch"], device=DEV)
    inv = 1.0 / (c["theta"] ** (torch.arange(0, HEAD, 2, dtype=torch.float64, device=DEV) / HEAD))
    ang = pos.double()[:, None, None] * inv
    cos, sin = ang.cos(), ang.sin()

    def rotate(x):
        lo, hi = x[..., :HEAD // 2], x[..., HEAD // 2:]
        return torch.cat([lo * cos - hi * sin, hi * cos + lo * sin], -1)

    def norm(x, gamma):
        return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + c["eps"]) * gamma.double()

    res = st["embed"][st["tokens"]].double()
    ks, vs = [], []
    for L in st["layers"]:
        qkv = (norm(res, L["ln1"]) @ L["wqkv"].double().t()).view(b, hq + 2, HEAD)
        q, k, v = rotate(qkv[:, :hq]), rotate(qkv[:, hq:hq + 1]), qkv[:, hq + 1:]
        kc, vc = L["k"].double(), L["v"].double()
        kc[rows, pos], vc[rows, pos] = k, v
        attn = torch.stack([_attend64(q[i], kc[i, :int(pos[i]) + 1, 0], vc[i, :int(pos[i]) + 1, 0]) for i in range(b)])
        res = res + attn.view(b, hq * HEAD) @ L["wo"].double().t()
        gu = norm(res, L["ln2"]) @ L["wgu"].double().t()
        res = res + (torch.nn.functional.silu(gu[:, :c["ffn"]]) * gu[:, c["ffn"]:]) @ L["wd"].double().t()
        ks.append(kc)
        vs.append(vc)
    return dict(logits=norm(res, st["final_norm"]) @ st["lm_head"].double().t(), k=ks, v=vs)
