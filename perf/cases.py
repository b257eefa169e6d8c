"""What this framework is timed on: the calls that a program which serves models with it makes, over the sizes it meets.

Kinds of case (one dict of plain values each; sizes from the repository's tests and benchmark, or generic):

  decode     attn_decode: one token's attention over the KV caches of a batch (fp16 or bf16 caches, one length or ragged)
  host_step  HostDecodeStep: the same from pinned host buffers - copy in, rotary + cache insert, attention, copy out
  prefill    attn_prefill_causal: causal attention of whole prompts
  ffn_q8     the FFN half of a generation step, Q8_0 weights: norm -> gate|up with SwiGLU -> down projection, replayed
             as a CUDA graph, which is how Llama (and any engine step) drives these launches
  ffn_f16    the same with fp16 weights
  ffn_prompt the FFN half of a layer for all tokens of a prompt: norm -> GEMM -> SwiGLU -> GEMM
  step       Llama.forward: one generation step of a Q8_0 model, batch of sequences at different positions
  prompt     Llama.prefill: ragged prompts of a Q8_0 model, all tokens at once

`exact` states every kind in float64 torch from the same inputs.
"""
import importlib.util
import math
import os
import sys

import torch

DEV = "cuda"
GOLDEN = 0.6180339887498949


def _package():
    """The package's directory name carries a hyphen: load it by path under its import name."""
    name = "llm_infer_b200"
    if name not in sys.modules:
        here = os.path.join(os.getcwd(), "llm-infer_b200")
        spec = importlib.util.spec_from_file_location(name, os.path.join(here, "__init__.py"), submodule_search_locations=[here])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    from llm_infer_b200 import attention, model
    return attention, model


# ------------------------------------------------------------------------------------------------------------ cases
def _decode(name, batch, heads, kv_heads, dim, kv, q, kvt, ragged):
    return dict(name=name, kind="decode", batch=batch, heads=heads, kv_heads=kv_heads, dim=dim, kv=kv, q=q, kvt=kvt, ragged=ragged)


def listed():
    return [
        # the smallest decode call: one sequence of a 1.1B-shaped model, short context; latency and launches
        _decode("decode_b1_kv512_d64", 1, 32, 4, 64, 512, "f32", "f16", False),
        # the headline shape: batched decode of an 8B-shaped layer
        _decode("decode_b16_kv4096", 16, 32, 8, 128, 4096, "f16", "f16", False),
        # a serving batch with every sequence at its own length, bf16 caches
        _decode("decode_b7_ragged_bf16", 7, 32, 8, 128, 2999, "f32", "bf16", True),
        # one long context (512 MiB of KV): streaming
        _decode("decode_b1_kv131072", 1, 32, 8, 128, 131072, "f16", "f16", False),
        # an attention block driven from host buffers, token by token
        dict(name="host_step_b8_kv2048", kind="host_step", batch=8, heads=32, kv_heads=8, dim=128, kv=2048),
        # whole prompts, 8B-shaped, bf16
        dict(name="prefill_b4_s2048_bf16", kind="prefill", batch=4, seq=2048, heads=32, kv_heads=8, dim=128, dtype="bf16", out="bf16"),
        # one short ragged-length prompt of a head_dim-64 model, fp32 result
        dict(name="prefill_b1_s333_d64", kind="prefill", batch=1, seq=333, heads=32, kv_heads=4, dim=64, dtype="f16", out="f32"),
        # FFN of a generation step at batch 8, Q8_0 (activations prepared by the norm, down projection split over CTAs)
        dict(name="ffn_q8_b8", kind="ffn_q8", batch=8, n=4096, hidden=14336),
        # FFN of a single user's generation step, the engine's own fp16 weights
        dict(name="ffn_f16_b1", kind="ffn_f16", batch=1, n=4096, hidden=14336),
        # FFN of a layer over the tokens of a prompt (1003: no multiple of any tile)
        dict(name="ffn_prompt_f16_m1003", kind="ffn_prompt", tokens=1003, n=4096, hidden=14336),
        # a whole generation step: four layers of the 8B shape, full classifier, 8 sequences at ragged positions
        dict(name="step_8b_q8_b8", kind="step", batch=8, layers=4, n=4096, hidden=14336, heads=32, kv_heads=8, dim=128,
             vocab=128256, low=128, high=2048),
        # the prompt phase of the same batch: 8 prompts, two layers
        dict(name="prompt_8b_q8_b8", kind="prompt", batch=8, layers=2, n=4096, hidden=14336, heads=32, kv_heads=8, dim=128,
             vocab=128256, low=128, high=2048),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "host_step", "prefill", "prefill", "ffn_q8", "ffn_f16", "ffn_prompt", "step", "prompt"])
    heads, kv_heads, dim = rng.choice([(32, 8, 128), (32, 4, 64), (32, 8, 128), (8, 2, 128), (16, 16, 64), (64, 8, 128), (24, 2, 128)])
    if kind == "decode":
        batch = _log(rng, 1, 48)
        kv = _log(rng, 64, max(65, min(131072, 131072 * 8 // (kv_heads * batch))))
        q, kvt = rng.choice([("f32", "f16"), ("f16", "f16"), ("f32", "bf16"), ("bf16", "bf16")])
        return {k: v for k, v in _decode("", batch, heads, kv_heads, dim, kv, q, kvt, rng.random() < 0.5).items() if k != "name"}
    if kind == "host_step":
        return dict(kind=kind, batch=_log(rng, 1, 16), heads=heads, kv_heads=kv_heads, dim=dim, kv=_log(rng, 64, 4096))
    if kind == "prefill":
        batch = _log(rng, 1, 4)
        dtype = rng.choice(["f16", "bf16"])
        return dict(kind=kind, batch=batch, seq=_log(rng, 40, 4096 // batch), heads=heads, kv_heads=kv_heads, dim=dim,
                    dtype=dtype, out=rng.choice(["f32", dtype]))
    n, hidden = rng.choice([(4096, 14336), (2048, 5632), (4096, 11008), (2048, 8192)])
    if kind in ("ffn_q8", "ffn_f16"):
        return dict(kind=kind, batch=rng.randint(1, 8), n=n, hidden=hidden)
    if kind == "ffn_prompt":
        return dict(kind=kind, tokens=_log(rng, 17, 4096), n=n, hidden=hidden)
    heads, kv_heads, dim = (32, 8, 128) if n == 4096 else (32, 4, 64)
    return dict(kind=kind, batch=rng.randint(1, 8), layers=rng.randint(1, 2), n=n, hidden=hidden, heads=heads, kv_heads=kv_heads,
                dim=dim, vocab=rng.choice([32000, 32768, 50257]), low=_log(rng, 16, 128), high=_log(rng, 129, 1800))


def _lengths(case):
    """Ragged lengths of the batch: spread over the range, a function of the case alone."""
    if case["kind"] == "decode":
        lo, hi = max(1, case["kv"] // 8), case["kv"]
    else:
        lo, hi = case["low"], case["high"]
    return [lo + int((hi - lo + 1) * ((i + 1) * GOLDEN % 1.0)) for i in range(case["batch"])]


# ----------------------------------------------------------------------------------------------------------- inputs
_T = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _randn(g, *shape, dtype=torch.float32):
    """N(0, 1), cast once; large tensors leading index by leading index."""
    if math.prod(shape) <= 1 << 27:
        return torch.randn(shape, generator=g, device=DEV).to(dtype)
    out = torch.empty(shape, dtype=dtype, device=DEV)
    flat = out.view(-1)
    for i in range(0, flat.numel(), 1 << 27):
        part = flat[i:i + (1 << 27)]
        part.copy_(torch.randn(part.numel(), generator=g, device=DEV))
    return out


def _norm_weight(g, *shape):
    return 1.0 + 0.1 * torch.randn(shape, generator=g, device=DEV)


def _f16_matrix(g, rows, n):
    return (torch.randn((rows, n), generator=g, device=DEV) * n ** -0.5).half()


def _q8_matrix(g, rows, n, std=None):
    """GGML Q8_0 blocks uint8 [rows, n/32*34] of roughly normal weights of standard deviation n^-0.5 (or std)."""
    std = n ** -0.5 if std is None else std
    out = torch.empty((rows, n // 32, 34), dtype=torch.uint8, device=DEV)
    step = max(1, (1 << 26) // n)
    for r in range(0, rows, step):
        m = min(step, rows - r)
        q = (torch.randn((m, n // 32, 32), generator=g, device=DEV) * 40.0).round_().clamp_(-127, 127).to(torch.int8)
        d = (torch.rand((m, n // 32, 1), generator=g, device=DEV) * 0.4 + 0.8).mul_(std / 40.0).half()
        out[r:r + m, :, :2] = d.view(torch.uint8)
        out[r:r + m, :, 2:] = q.view(torch.uint8)
    return out.view(rows, n // 32 * 34)


def _q8_value(w):
    """Q8_0 blocks [rows, n/32*34] -> float64 [rows, n]."""
    b = w.view(w.shape[0], -1, 34)
    d = b[..., :2].contiguous().view(torch.float16).double()
    return (d * b[..., 2:].contiguous().view(torch.int8).double()).view(w.shape[0], -1)


def _attention_inputs(case, seed):
    g = _gen(seed)
    B, H, Hkv, D = case["batch"], case["heads"], case["kv_heads"], case["dim"]
    if case["kind"] == "prefill":
        S, t = case["seq"], _T[case["dtype"]]
        return _randn(g, B, S, H, D, dtype=t), _randn(g, B, S, Hkv, D, dtype=t), _randn(g, B, S, Hkv, D, dtype=t)
    T, t = case["kv"], _T[case.get("kvt", "f16")]
    return _randn(g, B, H, D, dtype=_T[case.get("q", "f32")]), _randn(g, B, T, Hkv, D, dtype=t), _randn(g, B, T, Hkv, D, dtype=t)


def _host_token(case, seed):
    """q, k, v of the current token of every sequence, one after the other, as the host holds them."""
    B, H, Hkv, D = case["batch"], case["heads"], case["kv_heads"], case["dim"]
    g = torch.Generator().manual_seed(int(seed) + 1)
    return torch.randn(B * (H + 2 * Hkv) * D, generator=g)


def _ffn_inputs(case, seed):
    g, n, hidden, q8 = _gen(seed), case["n"], case["hidden"], case["kind"] == "ffn_q8"
    matrix = _q8_matrix if q8 else _f16_matrix
    rows = case.get("batch", case.get("tokens"))
    return dict(x=_randn(g, rows, n), norm=_norm_weight(g, n), w13=matrix(g, 2 * hidden, n), w2=matrix(g, n, hidden))


def _model_weights(case, seed):
    g, L, n, hidden = _gen(seed), case["layers"], case["n"], case["hidden"]
    q_dim, kv_dim = case["heads"] * case["dim"], case["kv_heads"] * case["dim"]
    m = lambda rows, cols: torch.stack([_q8_matrix(g, rows, cols) for _ in range(L)])  # noqa: E731
    return dict(embed=_q8_matrix(g, case["vocab"], n, 1.0), wcls=_q8_matrix(g, case["vocab"], n), rms_final=_norm_weight(g, n),
                rms_att=_norm_weight(g, L, n), rms_ffn=_norm_weight(g, L, n), wq=m(q_dim, n), wk=m(kv_dim, n), wv=m(kv_dim, n),
                wo=m(n, q_dim), w1=m(hidden, n), w3=m(hidden, n), w2=m(n, hidden))


def _cache_rows(case):
    return (case["high"] + 128 + 63) // 64 * 64


def _tokens(case, seed):
    g = torch.Generator().manual_seed(int(seed) + 2)
    if case["kind"] == "step":
        return torch.randint(0, case["vocab"], (case["batch"],), generator=g, dtype=torch.int32)
    return [torch.randint(0, case["vocab"], (n,), generator=g).tolist() for n in _lengths(case)]


def _history(case, seed):
    """K and V of the tokens that the step's sequences already hold."""
    g = _gen(int(seed) + 3)
    shape = (case["layers"], case["batch"], _cache_rows(case), case["kv_heads"], case["dim"])
    return _randn(g, *shape, dtype=torch.float16), _randn(g, *shape, dtype=torch.float16)


EPS, THETA = 1e-5, 500000.0


def _graph(launches):
    """The launches as a CUDA graph, warmed once outside the capture."""
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        launches()
    torch.cuda.current_stream().wait_stream(side)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        launches()
    return graph


def prepare(case, seed):
    A, M = _package()
    kind = case["kind"]
    s = {"kind": kind}
    if kind == "decode":
        q, k, v = _attention_inputs(case, seed)
        B, H, Hkv, D = case["batch"], case["heads"], case["kv_heads"], case["dim"]
        lens = torch.tensor(_lengths(case), dtype=torch.int32, device=DEV) if case["ragged"] else None
        s.update(q=q, k=k, v=v, lens=lens, out=torch.empty((B, H, D), device=DEV), ws=A.DecodeWorkspace(B, H, Hkv, D))
    elif kind == "host_step":
        _, k, v = _attention_inputs(case, seed)
        B, T = case["batch"], case["kv"]
        last = torch.full((B,), T - 1, dtype=torch.int32, device=DEV)
        out = torch.empty((B, case["heads"], case["dim"]), pin_memory=True)
        s.update(step=A.HostDecodeStep(_host_token(case, seed).pin_memory(), k, v, last, last, out, n_heads=case["heads"],
                                       theta=THETA, kv_early=True), k=k, v=v)
    elif kind == "prefill":
        q, k, v = _attention_inputs(case, seed)
        s.update(q=q, k=k, v=v, out=torch.empty(q.shape, dtype=_T[case["out"]], device=DEV))
    elif kind == "ffn_prompt":
        s.update(_ffn_inputs(case, seed))
        m, n, hidden = case["tokens"], case["n"], case["hidden"]
        pair = lambda c: tuple(torch.empty((m, c), dtype=torch.float16, device=DEV) for _ in range(2))  # noqa: E731
        s.update(pn=pair(n), ph=pair(hidden), gate_up=torch.empty((m, 2 * hidden), device=DEV), out=torch.empty((m, n), device=DEV))
    elif kind in ("ffn_q8", "ffn_f16"):
        w = _ffn_inputs(case, seed)
        B, n, hidden, q8 = case["batch"], case["n"], case["hidden"], kind == "ffn_q8"
        act = torch.int32 if q8 else torch.float32
        xb, hb = torch.empty((B, n), dtype=act, device=DEV), torch.empty((B, hidden), dtype=act, device=DEV)
        # the split that Llama takes for the down projection of this batch
        chunks, split = hidden // 256, max(1, -(-B * (hidden * 4 + 64) // (140 * 1024)))
        while split <= chunks and chunks % split:
            split += 1
        split = split if split <= chunks else 1
        out = torch.empty((split, B, n) if split > 1 else (B, n), device=DEV)
        w13, w2 = (A.repack_q8_0(w["w13"]), A.repack_q8_0(w["w2"])) if q8 else (w["w13"], w["w2"])
        gemv = A.gemv_q8_0 if q8 else A.gemv_f16

        def launches():
            A.rmsnorm(w["x"], w["norm"], EPS, out=xb)
            gemv(xb, w13, out=hb, swiglu=True)
            gemv(hb, w2, out=out, k_split=split)

        s.update(graph=_graph(launches), out=out, keep=(w["x"], w["norm"], w13, w2, xb, hb))
    else:
        c = case
        cfg = M.ModelConfig(dim=c["n"], hidden_dim=c["hidden"], n_layers=c["layers"], n_heads=c["heads"], n_kv_heads=c["kv_heads"],
                            head_dim=c["dim"], vocab_size=c["vocab"], max_seq_len=_cache_rows(c), norm_eps=EPS, rope_theta=THETA)
        s["model"] = m = M.Llama(cfg, _model_weights(c, seed), c["batch"], weight_type="q8_0")
        if kind == "step":
            k, v = _history(c, seed)
            m.capture()
            m.k_cache.copy_(k)
            m.v_cache.copy_(v)
            s.update(tokens=_tokens(c, seed).to(DEV), pos=_lengths(c))
        else:
            s["prompts"] = _tokens(c, seed)
    return s


def run(state):
    A, _ = _package()
    s, kind = state, state["kind"]
    if kind == "decode":
        return A.attn_decode(s["q"], s["k"], s["v"], s["lens"], out=s["out"], workspace=s["ws"])
    if kind == "host_step":
        return s["step"](), s["k"], s["v"]
    if kind == "prefill":
        return A.attn_prefill_causal(s["q"], s["k"], s["v"], out=s["out"])
    if kind == "ffn_prompt":
        A.rmsnorm_pair(s["x"], s["norm"], EPS, out=s["pn"])
        A.gemm_f16(*s["pn"], s["w13"], out=s["gate_up"])
        A.swiglu_pair(s["gate_up"], out=s["ph"])
        return A.gemm_f16(*s["ph"], s["w2"], out=s["out"])
    if kind in ("ffn_q8", "ffn_f16"):
        s["graph"].replay()
        return s["out"]
    m = s["model"]
    if kind == "step":
        m.forward(s["tokens"], s["pos"])
    else:
        m.prefill(s["prompts"])
    return m.logits, m.k_cache, m.v_cache


# ------------------------------------------------------------------------------------------- what it cannot do without
def work(case):
    kind, B = case["kind"], case.get("batch", 1)
    if kind in ("decode", "host_step"):
        H, Hkv, D = case["heads"], case["kv_heads"], case["dim"]
        rows = sum(_lengths(case)) if case.get("ragged") else B * case["kv"]
        qb = {"f32": 4, "f16": 2, "bf16": 2}[case.get("q", "f32")]
        return {"bytes": rows * Hkv * D * 4 + B * H * D * (qb + 4) + (B * Hkv * D * 12 if kind == "host_step" else 0),
                "flops": 4 * rows * H * D}
    if kind == "prefill":
        S, H, Hkv, D = case["seq"], case["heads"], case["kv_heads"], case["dim"]
        return {"bytes": B * S * D * (2 * H + 4 * Hkv + H * (4 if case["out"] == "f32" else 2)), "flops": 2 * B * H * S * (S + 1) * D}
    n, hidden = case["n"], case["hidden"]
    if kind in ("ffn_q8", "ffn_f16", "ffn_prompt"):
        rows = case.get("tokens", B)
        return {"bytes": 3 * n * hidden * (34 / 32 if kind == "ffn_q8" else 2) + rows * n * 8, "flops": 6 * rows * n * hidden}
    H, Hkv, D, L, V = case["heads"], case["kv_heads"], case["dim"], case["layers"], case["vocab"]
    layer = n * (H + 2 * Hkv) * D + n * H * D + 3 * n * hidden
    lens = _lengths(case)
    if kind == "step":
        kv = sum(p + 1 for p in lens)
        return {"bytes": (L * layer + V * n) * 34 / 32 + L * kv * Hkv * D * 4 + B * V * 4,
                "flops": 2 * B * (L * layer + V * n) + 4 * L * kv * H * D}
    T = sum(lens)
    return {"bytes": (L * layer + V * n) * 34 / 32 + L * T * Hkv * D * 4 + B * V * 4,
            "flops": 2 * T * L * layer + 2 * B * V * n + L * sum(2 * p * (p + 1) for p in lens) * H * D}


def tolerance(case):
    """About four times the distance from float64 that was measured over the ranges (in brackets)."""
    kind = case["kind"]
    if kind == "decode":  # fp32 sums of products whose probabilities carry 22 (fp16) or 16 bits (bf16) (2.4e-6, 3.2e-6)
        return {"rel": 1e-5 if case["kvt"] == "f16" else 1.5e-5}
    if kind == "host_step":  # the rotated query is fp16 (2.1e-4)
        return {"rel": 8e-4}
    if kind == "prefill":  # a 16-bit result carries its own rounding (2.0e-4, 1.6e-3)
        return {"rel": {"f32": 1e-5 if case["dtype"] == "f16" else 5e-5, "f16": 8e-4, "bf16": 6.4e-3}[case["out"]]}
    if kind == "ffn_q8":  # (2.8e-7; the sums' order moves it)
        return {"rel": 4e-6}
    if kind == "ffn_f16":  # (1.8e-6)
        return {"rel": 7e-6}
    if kind == "ffn_prompt":  # the tensor cores' fp32 accumulation over 14336 terms (5.1e-5)
        return {"rel": 2e-4}
    if kind == "step":  # logits 3.5e-7; cache rows are fp16, a few ties of which move (3.5e-7)
        return {"rel": 5e-6}
    return {"rel": 4.5e-4}  # prompt: logits 4.6e-5, cache rows 1.1e-4 (fp16 ties)


# -------------------------------------------------------------------------------------------------------- in float64
def _attend(q, k, v):
    """q [H, D], k / v [T, Hkv, D] -> [H, D]"""
    H, D = q.shape
    Hkv = k.shape[1]
    q = q.double().view(Hkv, H // Hkv, D)
    p = torch.softmax(torch.einsum("hgd,thd->hgt", q, k.double()) / math.sqrt(D), dim=-1)
    return torch.einsum("hgt,thd->hgd", p, v.double()).reshape(H, D)


def _causal(q, k, v):
    """q [S, H, D], k / v [S, Hkv, D] -> [S, H, D]"""
    S, H, D = q.shape
    Hkv = k.shape[1]
    G = H // Hkv
    later = torch.ones((S, S), dtype=torch.bool, device=q.device).triu_(1)
    out = torch.empty((S, H, D), dtype=torch.float64, device=q.device)
    for h in range(H):
        s = (q[:, h].double() @ k[:, h // G].double().T / math.sqrt(D)).masked_fill_(later, -math.inf)
        out[:, h] = torch.softmax(s, dim=-1) @ v[:, h // G].double()
    return out


def _rotate(x, pos):
    """x [T, heads, D] float64 at positions pos [T]: adjacent pairs; the angle is the product of two fp32 numbers."""
    T, _, D = x.shape
    e = (torch.arange(0, D, 2, dtype=torch.float32, device=x.device) / D).double()
    freq = 1.0 / torch.pow(torch.tensor(THETA, dtype=torch.float64, device=x.device), e).float()
    angle = (pos.float()[:, None] * freq[None, :]).double()
    c, s = angle.cos()[:, None, :], angle.sin()[:, None, :]
    a, b = x[..., 0::2], x[..., 1::2]
    return torch.stack([a * c - b * s, a * s + b * c], dim=-1).reshape(x.shape)


def _rms(x, w):
    return x / torch.sqrt((x * x).mean(dim=-1, keepdim=True) + EPS) * w.double()


def _silu_mul(gu):
    g, u = gu.chunk(2, dim=-1)
    return g / (1.0 + torch.exp(-g)) * u


def exact(case, seed):
    kind = case["kind"]
    if kind == "decode":
        q, k, v = _attention_inputs(case, seed)
        lens = _lengths(case) if case["ragged"] else [case["kv"]] * case["batch"]
        return torch.stack([_attend(q[b], k[b, :n], v[b, :n]) for b, n in enumerate(lens)])
    if kind == "host_step":
        _, k, v = _attention_inputs(case, seed)
        B, H, Hkv, D, T = case["batch"], case["heads"], case["kv_heads"], case["dim"], case["kv"]
        tok = _host_token(case, seed).to(DEV).double()
        q, kn, vn = (t.view(B, -1, D) for t in tok.split([B * H * D, B * Hkv * D, B * Hkv * D]))
        pos = torch.full((B,), T - 1, device=DEV)
        k[:, T - 1], v[:, T - 1] = _rotate(kn, pos).half(), vn.half()
        q = _rotate(q, pos)
        return torch.stack([_attend(q[b], k[b], v[b]) for b in range(B)]), k.double(), v.double()
    if kind == "prefill":
        q, k, v = _attention_inputs(case, seed)
        return torch.stack([_causal(q[b], k[b], v[b]) for b in range(case["batch"])])
    if kind in ("ffn_q8", "ffn_f16", "ffn_prompt"):
        w = _ffn_inputs(case, seed)
        value = _q8_value if kind == "ffn_q8" else torch.Tensor.double
        h = _silu_mul(_rms(w["x"].double(), w["norm"]) @ value(w["w13"]).T)
        w2 = value(w["w2"])
        if kind == "ffn_prompt":
            return h @ w2.T
        B, hidden = case["batch"], case["hidden"]
        chunks, split = hidden // 256, max(1, -(-B * (hidden * 4 + 64) // (140 * 1024)))
        while split <= chunks and chunks % split:
            split += 1
        if split > chunks or split == 1:
            return h @ w2.T
        return torch.stack([a @ b.T for a, b in zip(h.chunk(split, dim=1), w2.chunk(split, dim=1))])
    w = _model_weights(case, seed)
    B, L, H, Hkv, D = case["batch"], case["layers"], case["heads"], case["kv_heads"], case["dim"]
    lens, rows = _lengths(case), _cache_rows(case)
    if kind == "step":
        toks, pos = _tokens(case, seed).to(DEV).long(), torch.tensor(lens, device=DEV)
        kc, vc = _history(case, seed)
    else:
        toks = torch.tensor([t for p in _tokens(case, seed) for t in p], device=DEV)
        pos = torch.cat([torch.arange(n, device=DEV) for n in lens])
        kc = torch.zeros((L, B, rows, Hkv, D), dtype=torch.float16, device=DEV)
        vc = torch.zeros_like(kc)
    starts = [sum(lens[:b]) for b in range(B + 1)]
    x = _q8_value(w["embed"][toks])
    T = x.shape[0]
    for l in range(L):
        xb = _rms(x, w["rms_att"][l])
        q = _rotate((xb @ _q8_value(w["wq"][l]).T).view(T, H, D), pos)
        k = _rotate((xb @ _q8_value(w["wk"][l]).T).view(T, Hkv, D), pos).half()  # the caches hold fp16
        v = (xb @ _q8_value(w["wv"][l]).T).view(T, Hkv, D).half()
        att = torch.empty((T, H, D), dtype=torch.float64, device=DEV)
        for b in range(B):
            if kind == "step":
                kc[l, b, lens[b]], vc[l, b, lens[b]] = k[b], v[b]
                att[b] = _attend(q[b], kc[l, b, :lens[b] + 1], vc[l, b, :lens[b] + 1])
            else:
                at = slice(starts[b], starts[b] + lens[b])
                kc[l, b, :lens[b]], vc[l, b, :lens[b]] = k[at], v[at]
                att[at] = _causal(q[at], k[at], v[at])
        x = x + att.view(T, H * D) @ _q8_value(w["wo"][l]).T
        xb = _rms(x, w["rms_ffn"][l])
        gu = torch.cat([xb @ _q8_value(w["w1"][l]).T, xb @ _q8_value(w["w3"][l]).T], dim=1)
        x = x + _silu_mul(gu) @ _q8_value(w["w2"][l]).T
    if kind == "prompt":
        x = x[[starts[b] + lens[b] - 1 for b in range(B)]]
    logits = _rms(x, w["rms_final"]) @ _q8_value(w["wcls"]).T
    return logits, kc.double(), vc.double()
