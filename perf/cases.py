"""The work that is timed: single layers of the models that this engine serves, called through its C ABI the way a host
program calls them, and whole engine steps through the Python front end.

Each kind of case is one piece of a serving step:

  attn     paged attention over a flattened batch of requests (decode rows first, then prompt chunks)
  mlp      pre-norm, first projection with its activation, second projection (gated SiLU, or OPT's ReLU with biases)
  qkv      pre-norm, packed projection, rotary embedding, write of keys and values into the paged cache
  head     final norm, vocabulary projection, sampling
  step     one decode step of a whole OPT model with its logits
  design   a whole layer-list model: a prompt step of several requests, then decode steps, with their logits

Sizes are those of the models and workloads that this repository names (opt-125m, Llama 3.2 1B, 3.1 8B and 70B heads, the
w2048 layer-list design of the benchmark) and ragged ones of the same ranges.
"""
import json
import math
import os
import struct
import tempfile

import numpy as np
import torch

from kge_loader import load

kge = load()
DT = {"bf16": torch.bfloat16, "fp16": torch.float16}


# ------------------------------------------------------------------------------------------------------------- cases

def listed():
    attn = dict(kind="attn", dtype="bf16", heads=32, kv=8, hd=128, block=64)
    mlp = dict(kind="mlp", dtype="bf16", act="silu")
    return [
        # 64 concurrent requests of the 8B model generate at 2k-in / 256-out: one layer's decode attention
        dict(attn, name="attn-decode-8b", reqs=64, ctx_lo=2048, ctx_hi=2304, new=1, prompts=0, chunk=0, prior=0),
        # 32 short chats on the 1B model, with blocks of 16 tokens (the front end's default): little work for the whole chip
        dict(attn, name="attn-decode-1b", hd=64, block=16, reqs=32, ctx_lo=96, ctx_hi=256, new=1, prompts=0, chunk=0, prior=0),
        # a prompt step: four whole 2k prompts fill the token budget of 8192
        dict(attn, name="attn-prefill-8b", reqs=0, ctx_lo=0, ctx_hi=0, new=1, prompts=4, chunk=2048, prior=0),
        # a mixed step in float16: decode rows beside two odd chunks of long prompts whose beginnings are already cached
        dict(attn, name="attn-mixed-fp16", dtype="fp16", block=16, reqs=37, ctx_lo=50, ctx_hi=3000, new=1, prompts=2, chunk=1011, prior=2777),
        # one token of opt-125m: the smallest projections there are
        dict(mlp, name="mlp-opt125m-1", act="relu", rows=1, width=768, ff=3072),
        # the 8B model's feed-forward in a decode step of 64 requests: weights stream from memory
        dict(mlp, name="mlp-8b-64", rows=64, width=4096, ff=14336),
        # the same in a full prompt step
        dict(mlp, name="mlp-8b-8192", rows=8192, width=4096, ff=14336),
        # attention front half of an 8B decode step
        dict(kind="qkv", name="qkv-8b-64", dtype="bf16", rows=64, width=4096, heads=32, kv=8, hd=128, bias=False, block=64),
        # attention front half with biases, in float16, for an odd number of prompt tokens
        dict(kind="qkv", name="qkv-fp16-1339", dtype="fp16", rows=1339, width=2048, heads=32, kv=8, hd=64, bias=True, block=16),
        # next tokens of 32 requests of the 1B model, drawn with temperature, top-k and top-p as each asks
        dict(kind="head", name="head-1b-32", dtype="bf16", rows=32, width=2048, vocab=128256),
        # the minimal deployment: opt-125m, one request, one token at a time
        dict(kind="step", name="step-opt125m-1", layers=12, width=768, heads=12, ff=3072, vocab=50272, reqs=1, ctx_lo=190, ctx_hi=190),
        # two prompts through the four-layer pattern of the benchmark's design, then four decode steps
        dict(kind="design", name="design-w2048", width=2048, reqs=2, ctx_lo=1000, ctx_hi=1300, decode=4),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["attn", "attn", "attn", "mlp", "mlp", "qkv", "qkv", "head", "step", "design"])
    dtype = rng.choice(["bf16", "bf16", "bf16", "fp16"])
    if kind == "attn":
        hd, block = rng.choice([64, 128, 128]), rng.choice([16, 32, 64])
        kv = rng.choice([4, 8])
        heads = kv * rng.choice([1, 4, 8])
        c = dict(kind=kind, dtype=dtype, heads=heads, kv=kv, hd=hd, block=block, new=1)
        mode = rng.choice(["decode", "prefill", "mixed"])
        hi = _log(rng, 64, 4096)
        c.update(reqs=_log(rng, 1, 64) if mode != "prefill" else 0, ctx_lo=max(1, hi // rng.choice([1, 2, 20])), ctx_hi=hi)
        if mode == "decode":
            c.update(prompts=0, chunk=0, prior=0)
        else:
            prompts = _log(rng, 1, 8)
            c.update(prompts=prompts, chunk=_log(rng, 17, 8192 // prompts if heads <= 32 else 4096 // prompts), prior=rng.choice([0, 0, _log(rng, 10, 2000)]))
        return c
    if kind == "mlp":
        width, ff, act = rng.choice([(768, 3072, "relu"), (2048, 8192, "silu"), (4096, 14336, "silu")])
        return dict(kind=kind, dtype=dtype, act=act, rows=_log(rng, 1, 4096), width=width, ff=ff)
    if kind == "qkv":
        width, heads, kv, hd = rng.choice([(2048, 32, 8, 64), (4096, 32, 8, 128), (2048, 16, 4, 128)])
        return dict(kind=kind, dtype=dtype, rows=_log(rng, 1, 4096), width=width, heads=heads, kv=kv, hd=hd, bias=rng.choice([False, True]), block=rng.choice([16, 64]))
    if kind == "head":
        width, vocab = rng.choice([(768, 50272), (2048, 128256), (4096, 32000)])
        return dict(kind=kind, dtype=dtype, rows=_log(rng, 1, 64), width=width, vocab=vocab)
    if kind == "step":
        hi = _log(rng, 32, 600)
        return dict(kind=kind, layers=rng.randint(2, 12), width=768, heads=12, ff=3072, vocab=50272, reqs=_log(rng, 1, 32), ctx_lo=max(2, hi // 2), ctx_hi=hi)
    hi = _log(rng, 150, 1300)
    return dict(kind=kind, width=2048, reqs=rng.randint(1, 2), ctx_lo=max(2, hi // 2), ctx_hi=hi, decode=rng.randint(1, 4))


# ----------------------------------------------------------------------------------------------------- inputs, shared

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(1_000_003 + seed)


def _randn(g, shape, std, dtype, mean=0.0):
    return (torch.randn(shape, generator=g, device="cuda", dtype=torch.float32) * std + mean).to(dtype)


def _call(st, name, *args):
    """One entry point of the C ABI on torch's current stream; tensors are passed by their device pointer."""
    fn = getattr(st["lib"], name)
    rc = fn(*[a.data_ptr() if isinstance(a, torch.Tensor) else a for a in args], st["stream"])
    if rc < 0:
        kge.check(rc, name)


def _names(case):
    f16 = case["dtype"] == "fp16"
    n = dict(gemm="kge_gemm_f16" if f16 else "kge_gemm_bf16", gate="kge_gemm_silu_gate_ws_f16" if f16 else "kge_gemm_silu_gate_ws_bf16")
    for k in ("rmsnorm", "layernorm", "rope_kvwrite", "paged_attn", "sample"):
        n[k] = f"kge_{k}" + ("_f16" if f16 else "")
    return n


def _base(case):
    return {"case": case, "lib": kge.lib(), "stream": torch.cuda.current_stream().cuda_stream, "fn": _names(case)}


def _gemm_ws(T, N, K):
    n = max(1024, kge.lib().kge_gemm_workspace_bytes(T, N, K))
    return torch.zeros(n, dtype=torch.uint8, device="cuda"), n


def _rms64(x, w, eps):
    return x / torch.sqrt(x.pow(2).mean(-1, keepdim=True) + eps) * w


def _ln64(x, w, b, eps):
    return torch.nn.functional.layer_norm(x, (x.shape[-1],), w, b, eps)


# ---------------------------------------------------------------------------------------------------------- attention

def _attn_shape(case, seed):
    """Context and query lengths of the flattened batch: decode requests first, then prompt chunks."""
    r = np.random.default_rng(seed + 17)
    ctx = r.integers(case["ctx_lo"], case["ctx_hi"] + 1, case["reqs"]).tolist() if case["reqs"] else []
    q = [case["new"]] * len(ctx)
    for i in range(case["prompts"]):
        n = case["chunk"] - (i * 7 % 5 if case["prior"] else 0)
        q.append(max(1, n))
        ctx.append(q[-1] + (case["prior"] + 131 * i if case["prior"] else 0))
    return ctx, q


def _attn_inputs(case, seed):
    g, dt = _gen(seed), DT[case["dtype"]]
    ctx, q = _attn_shape(case, seed)
    B, T, H, KV, hd, bs = len(ctx), sum(q), case["heads"], case["kv"], case["hd"], case["block"]
    per = [(c + bs - 1) // bs for c in ctx]
    blocks = sum(per) + 1
    order = torch.randperm(blocks - 1, generator=g, device="cuda").add_(1).to(torch.int32)      # block 0 is the null block
    table = torch.zeros(B, max(per), dtype=torch.int32, device="cuda")
    at = 0
    for b, n in enumerate(per):
        table[b, :n] = order[at:at + n]
        at += n
    qkv = _randn(g, (T, (H + 2 * KV) * hd), 1.0, dt)
    kc = _randn(g, (blocks, KV, bs, hd), 1.0, dt)
    vc = _randn(g, (blocks, KV, bs, hd), 1.0, dt)
    return dict(ctx=ctx, q=q, B=B, T=T, table=table, qkv=qkv, kc=kc, vc=vc)


def _attn_prepare(case, seed):
    st, i = _base(case), _attn_inputs(case, seed)
    st.update(i)
    st["lens"] = torch.tensor(i["ctx"], dtype=torch.int32, device="cuda")
    st["qsl"] = torch.tensor(np.concatenate([[0], np.cumsum(i["q"])]), dtype=torch.int32, device="cuda")
    st["maxq"], st["maxc"] = max(i["q"]), max(i["ctx"])
    st["out"] = torch.empty(i["T"], case["heads"] * case["hd"], dtype=DT[case["dtype"]], device="cuda")
    st["nws"] = st["lib"].kge_attn_workspace_bytes(i["B"], case["heads"], case["hd"], st["maxc"])
    st["ws"] = torch.empty(max(16, st["nws"]), dtype=torch.uint8, device="cuda")
    return st


def _attn_run(st):
    c = st["case"]
    _call(st, st["fn"]["paged_attn"], st["out"], st["qkv"], st["qkv"].shape[1], st["kc"], st["vc"], st["table"], st["table"].shape[1], st["lens"], st["qsl"],
          st["B"], st["T"], st["maxq"], st["maxc"], c["heads"], c["kv"], c["hd"], c["block"], c["hd"] ** -0.5, st["ws"], st["nws"])
    return st["out"]


def _attend64(q, k, v, scale, first):
    """q [n, H, hd] whose first row sits at position `first`; k, v [ctx, KV, hd]; causal, float64."""
    n, H, hd = q.shape
    KV = k.shape[1]
    out = torch.empty(n, H, v.shape[-1], dtype=torch.float64, device=q.device)
    pos = torch.arange(n, device=q.device)[:, None] + first
    hidden = torch.arange(k.shape[0], device=q.device)[None, :] > pos
    for h in range(H):
        s = (q[:, h] @ k[:, h * KV // H].T) * scale
        s.masked_fill_(hidden, -math.inf)
        out[:, h] = torch.softmax(s, -1) @ v[:, h * KV // H]
    return out


def _attn_exact(case, seed):
    i = _attn_inputs(case, seed)
    H, KV, hd, bs = case["heads"], case["kv"], case["hd"], case["block"]
    outs, at = [], 0
    for b in range(i["B"]):
        n, c = i["q"][b], i["ctx"][b]
        rows = i["table"][b, :(c + bs - 1) // bs].long()
        k, v = (x[rows].permute(0, 2, 1, 3).reshape(-1, KV, hd)[:c].double() for x in (i["kc"], i["vc"]))
        q = i["qkv"][at:at + n, :H * hd].double().view(n, H, hd)
        outs.append(_attend64(q, k, v, hd ** -0.5, c - n).reshape(n, H * hd))
        at += n
    return torch.cat(outs)


def _attn_work(case, seed=0):
    ctx, q = _attn_shape(case, seed)
    H, KV, hd = case["heads"], case["kv"], case["hd"]
    return {"bytes": float(sum(ctx) * KV * hd * 4 + sum(q) * H * hd * 4),
            "flops": float(sum(4 * H * hd * n * (c - n + (n + 1) / 2) for c, n in zip(ctx, q)))}


# ---------------------------------------------------------------------------------------------------- feed-forward layer

def _mlp_inputs(case, seed):
    g, dt, T, d, f = _gen(seed), DT[case["dtype"]], case["rows"], case["width"], case["ff"]
    i = dict(x=_randn(g, (T, d), 1.5, dt), nw=_randn(g, (d,), 0.1, dt, 1.0))
    if case["act"] == "silu":
        i.update(w1=_randn(g, (2 * f, d), d ** -0.5, dt), w2=_randn(g, (d, f), 2 * f ** -0.5, dt))
    else:
        i.update(nb=_randn(g, (d,), 0.1, dt), w1=_randn(g, (f, d), d ** -0.5, dt), b1=_randn(g, (f,), 0.1, dt), w2=_randn(g, (d, f), f ** -0.5, dt),
                 b2=_randn(g, (d,), 0.1, dt))
    return i


def _mlp_prepare(case, seed):
    st = _base(case)
    st.update(_mlp_inputs(case, seed))
    T, d, f, dt = case["rows"], case["width"], case["ff"], DT[case["dtype"]]
    st["h"], st["a"], st["y"] = (torch.empty(T, n, dtype=dt, device="cuda") for n in (d, f, d))
    st["ws1"], st["n1"] = _gemm_ws(T, f, d)
    st["ws2"], st["n2"] = _gemm_ws(T, d, f)
    return st


def _mlp_run(st):
    c, fn = st["case"], st["fn"]
    T, d, f = c["rows"], c["width"], c["ff"]
    if c["act"] == "silu":
        _call(st, fn["rmsnorm"], st["h"], st["x"], st["nw"], T, d, 1e-5)
        _call(st, fn["gate"], st["a"], st["h"], st["w1"], T, f, d, st["ws1"], st["n1"])
        _call(st, fn["gemm"], st["y"], st["a"], st["w2"], None, T, d, f, 0, st["ws2"], st["n2"])
    else:
        _call(st, fn["layernorm"], st["h"], st["x"], None, st["nw"], st["nb"], T, d, 1e-5)
        _call(st, fn["gemm"], st["a"], st["h"], st["w1"], st["b1"], T, f, d, 1, st["ws1"], st["n1"])
        _call(st, fn["gemm"], st["y"], st["a"], st["w2"], st["b2"], T, d, f, 0, st["ws2"], st["n2"])
    return st["y"]


def _mlp_exact(case, seed):
    i = _mlp_inputs(case, seed)
    w1, w2 = i["w1"].double(), i["w2"].double()
    outs = []
    for x in i["x"].split(2048):
        if case["act"] == "silu":
            g, u = (_rms64(x.double(), i["nw"].double(), 1e-5) @ w1.T).chunk(2, -1)
            outs.append((torch.nn.functional.silu(g) * u) @ w2.T)
        else:
            h = _ln64(x.double(), i["nw"].double(), i["nb"].double(), 1e-5)
            outs.append(torch.relu(h @ w1.T + i["b1"].double()) @ w2.T + i["b2"].double())
    return torch.cat(outs)


def _mlp_work(case):
    T, n = case["rows"], (3 if case["act"] == "silu" else 2) * case["width"] * case["ff"]
    return {"bytes": 2.0 * (n + 2 * T * case["width"]), "flops": 2.0 * T * n}


# ------------------------------------------------------------------------------------------------- attention front half

def _qkv_inputs(case, seed):
    g, dt, T, d, hd = _gen(seed), DT[case["dtype"]], case["rows"], case["width"], case["hd"]
    n, bs = (case["heads"] + 2 * case["kv"]) * hd, case["block"]
    i = dict(x=_randn(g, (T, d), 1.5, dt), nw=_randn(g, (d,), 0.1, dt, 1.0), w=_randn(g, (n, d), d ** -0.5, dt), b=_randn(g, (n,), 0.3, dt) if case["bias"] else None)
    ang = torch.arange(8192, device="cuda", dtype=torch.float64)[:, None] * 500000.0 ** (-torch.arange(0, hd, 2, device="cuda", dtype=torch.float64) / hd)[None, :]
    i["cs"] = torch.cat([ang.cos(), ang.sin()], -1).to(dt)
    i["pos"] = torch.randint(0, 8192, (T,), generator=g, device="cuda", dtype=torch.int32)
    i["blocks"] = (T + bs - 1) // bs + 3
    i["slots"] = torch.randperm((i["blocks"] - 1) * bs, generator=g, device="cuda")[:T] + bs
    return i


def _qkv_prepare(case, seed):
    st = _base(case)
    st.update(_qkv_inputs(case, seed))
    T, d, hd, dt = case["rows"], case["width"], case["hd"], DT[case["dtype"]]
    st["n"] = (case["heads"] + 2 * case["kv"]) * hd
    st["h"], st["qkv"] = torch.empty(T, d, dtype=dt, device="cuda"), torch.empty(T, st["n"], dtype=dt, device="cuda")
    st["kc"], st["vc"] = (torch.zeros(st["blocks"], case["kv"], case["block"], hd, dtype=dt, device="cuda") for _ in range(2))
    st["ws"], st["nws"] = _gemm_ws(T, st["n"], d)
    return st


def _qkv_run(st):
    c, fn = st["case"], st["fn"]
    T, d = c["rows"], c["width"]
    _call(st, fn["rmsnorm"], st["h"], st["x"], st["nw"], T, d, 1e-5)
    _call(st, fn["gemm"], st["qkv"], st["h"], st["w"], st["b"], T, st["n"], d, 0, st["ws"], st["nws"])
    _call(st, fn["rope_kvwrite"], st["qkv"], st["cs"], st["pos"], st["slots"], st["kc"], st["vc"], T, c["heads"], c["kv"], c["hd"], c["block"])
    return {"qkv": st["qkv"], "k": st["kc"], "v": st["vc"]}


def _qkv_exact(case, seed):
    i = _qkv_inputs(case, seed)
    T, H, KV, hd, bs = case["rows"], case["heads"], case["kv"], case["hd"], case["block"]
    y = _rms64(i["x"].double(), i["nw"].double(), 1e-5) @ i["w"].double().T
    if i["b"] is not None:
        y = y + i["b"].double()
    y = y.view(T, H + 2 * KV, hd)
    cos, sin = (t[:, None, :] for t in i["cs"].double()[i["pos"].long()].chunk(2, -1))
    a, b = y[:, :H + KV].chunk(2, -1)
    y[:, :H + KV] = torch.cat([a * cos - b * sin, b * cos + a * sin], -1)
    kc, vc = (torch.zeros(i["blocks"], KV, bs, hd, dtype=torch.float64, device="cuda") for _ in range(2))
    kc[i["slots"] // bs, :, i["slots"] % bs] = y[:, H:H + KV]
    vc[i["slots"] // bs, :, i["slots"] % bs] = y[:, H + KV:]
    return {"qkv": y.reshape(T, -1), "k": kc, "v": vc}


def _qkv_work(case):
    T, d, n = case["rows"], case["width"], (case["heads"] + 2 * case["kv"]) * case["hd"]
    return {"bytes": 2.0 * (n * d + T * d + T * n + 2 * T * case["kv"] * case["hd"]), "flops": 2.0 * T * n * d}


# --------------------------------------------------------------------------------------------------- vocabulary and tokens

def _head_inputs(case, seed):
    g, dt, R, d, V = _gen(seed), DT[case["dtype"]], case["rows"], case["width"], case["vocab"]
    return dict(x=_randn(g, (R, d), 1.5, dt), nw=_randn(g, (d,), 0.1, dt, 1.0), w=_randn(g, (V, d), 2.5 * d ** -0.5, dt))


def _head_prepare(case, seed):
    st = _base(case)
    st.update(_head_inputs(case, seed))
    R, d, V, dt = case["rows"], case["width"], case["vocab"], DT[case["dtype"]]
    st["h"], st["logits"] = torch.empty(R, d, dtype=dt, device="cuda"), torch.empty(R, V, dtype=dt, device="cuda")
    st["ids"] = torch.empty(R, dtype=torch.int32, device="cuda")
    want = [(0.0, 0, 1.0), (0.7, 20, 0.8), (1.0, 0, 0.95), (0.6, 50, 1.0)]          # (temperature, top_k, top_p): greedy and usual settings
    rows = [want[(r + seed) % 4] for r in range(R)]
    st["temp"] = torch.tensor([t for t, _, _ in rows], dtype=torch.float32, device="cuda")
    st["topk"] = torch.tensor([k for _, k, _ in rows], dtype=torch.int32, device="cuda")
    st["topp"] = torch.tensor([p for _, _, p in rows], dtype=torch.float32, device="cuda")
    st["seeds"] = torch.randint(1, 1 << 62, (R,), generator=_gen(seed + 1), device="cuda")
    st["ws"], st["nws"] = _gemm_ws(R, V, d)
    st["ns"] = st["lib"].kge_sample_workspace_bytes(R, V)
    st["sws"] = torch.empty(max(16, st["ns"]), dtype=torch.uint8, device="cuda")
    return st


def _head_run(st):
    c, fn = st["case"], st["fn"]
    R, d, V = c["rows"], c["width"], c["vocab"]
    _call(st, fn["rmsnorm"], st["h"], st["x"], st["nw"], R, d, 1e-5)
    _call(st, fn["gemm"], st["logits"], st["h"], st["w"], None, R, V, d, 0, st["ws"], st["nws"])
    _call(st, fn["sample"], st["ids"], st["logits"], R, V, V, st["temp"], st["topk"], st["topp"], None, st["seeds"], 11, st["sws"], st["ns"])
    return {"logits": st["logits"], "tokens": st["ids"]}


def _head_exact(case, seed):
    i = _head_inputs(case, seed)
    return {"logits": _rms64(i["x"].double(), i["nw"].double(), 1e-5) @ i["w"].double().T, "tokens": None}


def _head_work(case):
    R, d, V = case["rows"], case["width"], case["vocab"]
    return {"bytes": 2.0 * (V * d + R * d + R * V), "flops": 2.0 * R * V * d}


# ------------------------------------------------------------------------------------------------------------ whole models

def _write_model(path, cfg, W):
    """config.json and one safetensors file: header length, JSON header, raw values."""
    with open(os.path.join(path, "config.json"), "w") as f:
        json.dump(cfg, f)
    head, at = {}, 0
    for k, v in W.items():
        n = v.numel() * 2
        head[k] = {"dtype": "BF16", "shape": list(v.shape), "data_offsets": [at, at + n]}
        at += n
    js = json.dumps(head).encode()
    with open(os.path.join(path, "model.safetensors"), "wb") as f:
        f.write(struct.pack("<Q", len(js)) + js)
        for v in W.values():
            v.contiguous().view(torch.int16).cpu().numpy().tofile(f)


def _engine(cfg, W, **kw):
    room = "/dev/shm" if os.path.isdir("/dev/shm") and os.access("/dev/shm", os.W_OK) else None
    try:
        with tempfile.TemporaryDirectory(dir=room) as d:
            _write_model(d, cfg, W)
            return kge.LLM(d, **kw)
    except OSError:
        with tempfile.TemporaryDirectory() as d:
            _write_model(d, cfg, W)
            return kge.LLM(d, **kw)


class _Batch:
    """Step metadata of requests whose blocks lie one after another in the pool: what a host scheduler keeps."""

    def __init__(self, spans, ids, bs):
        # spans: (first position, end position) of each request in this step; ids: its whole token list
        longest = max(len(t) for t in ids)
        self.per = (longest + bs - 1) // bs
        table = 1 + np.arange(len(spans) * self.per, dtype=np.int32).reshape(len(spans), self.per)
        pos = [np.arange(a, b, dtype=np.int32) for a, b in spans]
        slots = [table[r, p // bs].astype(np.int64) * bs + p % bs for r, p in enumerate(pos)]
        qsl = np.concatenate([[0], np.cumsum([b - a for a, b in spans])]).astype(np.int32)
        self.args = (np.concatenate([np.asarray(t[a:b], dtype=np.int32) for t, (a, b) in zip(ids, spans)]), np.concatenate(pos), qsl,
                     np.asarray([b for _, b in spans], dtype=np.int32), table, self.per, np.concatenate(slots), qsl[1:] - 1)


def _tokens(case, seed, extra):
    r = np.random.default_rng(seed + 29)
    lens = r.integers(case["ctx_lo"], case["ctx_hi"] + 1, case["reqs"])
    return [r.integers(3, case.get("vocab", 32000) - 1, n + extra).tolist() for n in lens]


def _opt_weights(case, seed):
    g, d, f, V = _gen(seed), case["width"], case["ff"], case["vocab"]
    bf = torch.bfloat16
    W = {"model.decoder.embed_tokens.weight": _randn(g, (V, d), 0.05, bf), "model.decoder.embed_positions.weight": _randn(g, (2050, d), 0.05, bf)}

    def norm(name):
        W[name + ".weight"], W[name + ".bias"] = _randn(g, (d,), 0.1, bf, 1.0), _randn(g, (d,), 0.1, bf)

    def lin(name, n, k):
        W[name + ".weight"], W[name + ".bias"] = _randn(g, (n, k), k ** -0.5, bf), _randn(g, (n,), 0.05, bf)
    for i in range(case["layers"]):
        p = f"model.decoder.layers.{i}."
        for n in ("q_proj", "k_proj", "v_proj", "out_proj"):
            lin(p + "self_attn." + n, d, d)
        lin(p + "fc1", f, d)
        lin(p + "fc2", d, f)
        norm(p + "self_attn_layer_norm")
        norm(p + "final_layer_norm")
    norm("model.decoder.final_layer_norm")
    return W


def _step_prepare(case, seed):
    W, ids, bs = _opt_weights(case, seed), _tokens(case, seed, 0), 16
    cfg = dict(model_type="opt", architectures=["OPTForCausalLM"], vocab_size=case["vocab"], hidden_size=case["width"], num_hidden_layers=case["layers"],
               num_attention_heads=case["heads"], ffn_dim=case["ff"], max_position_embeddings=2048, do_layer_norm_before=True, word_embed_proj_dim=case["width"],
               activation_function="relu", tie_word_embeddings=True, bos_token_id=2, eos_token_id=2, pad_token_id=1)
    blocks = max(len(ids) * ((max(map(len, ids)) + bs - 1) // bs), 2048 // bs) + 1
    llm = _engine(cfg, W, max_model_len=2048, max_num_seqs=32, max_num_batched_tokens=2048, block_size=bs, num_gpu_blocks_override=blocks, enable_prefix_caching=False)
    for r in range(len(ids)):           # the contexts are in the cache before the timed step
        spans = [(0, len(t) - 1) for t in ids]
        b = _Batch(spans, ids, bs)
        qsl = b.args[2]
        a, e = qsl[r], qsl[r + 1]
        llm.raw_step(b.args[0][a:e], b.args[1][a:e], [0, e - a], b.args[3][r:r + 1], b.args[4][r:r + 1], b.per, b.args[6][a:e], [e - a - 1])
    return {"case": case, "llm": llm, "batch": _Batch([(len(t) - 1, len(t)) for t in ids], ids, bs).args}


def _step_run(st):
    tokens, logits = st["llm"].raw_step(*st["batch"], want_logits=True)
    return {"logits": logits, "tokens": tokens}


def _step_exact(case, seed):
    W = {k: v.double() for k, v in _opt_weights(case, seed).items()}
    H, d = case["heads"], case["width"]
    hd = d // H

    def lin(x, name):
        return x @ W[name + ".weight"].T + W[name + ".bias"]

    def norm(x, name):
        return _ln64(x, W[name + ".weight"], W[name + ".bias"], 1e-5)
    out = []
    for t in _tokens(case, seed, 0):
        n = len(t)
        x = W["model.decoder.embed_tokens.weight"][torch.tensor(t, device="cuda")] + W["model.decoder.embed_positions.weight"][2:n + 2]
        for i in range(case["layers"]):
            p = f"model.decoder.layers.{i}."
            h = norm(x, p + "self_attn_layer_norm")
            q, k, v = (lin(h, f"{p}self_attn.{m}_proj").view(n, H, hd) for m in "qkv")
            x = x + lin(_attend64(q, k, v, hd ** -0.5, 0).reshape(n, d), p + "self_attn.out_proj")
            x = x + lin(torch.relu(lin(norm(x, p + "final_layer_norm"), p + "fc1")), p + "fc2")
        out.append(norm(x[-1:], "model.decoder.final_layer_norm") @ W["model.decoder.embed_tokens.weight"].T)
    return {"logits": torch.cat(out), "tokens": None}


def _step_work(case):
    d, f, V, B = case["width"], case["ff"], case["vocab"], case["reqs"]
    n = case["layers"] * (4 * d * d + 2 * d * f) + V * d
    ctx = B * (case["ctx_lo"] + case["ctx_hi"]) / 2
    return {"bytes": 2.0 * (n + case["layers"] * 2 * ctx * d) + 4.0 * B * V, "flops": 2.0 * B * n + 4.0 * case["layers"] * ctx * d}


# ------------------------------------------------------------------------------------------------------ a layer-list model
# Four layers of two kinds: attention within chunks of positions beside a matrix memory, and gated linear recurrences after a
# short convolution; dense units and routed experts in turn.

_D = dict(heads=16, kv=4, dim=128, chunk=1024, m_heads=4, m_dim=128, m_vdim=256, r_width=2560, r_blocks=16, conv=4, ff=8192, experts=16, top=2, eff=1024, sff=2048,
          vocab=32000, cap=15.0, eps=1e-5)
_LAYERS = (("parallel", "dense"), ("rglru", "moe"), ("rglru", "dense"), ("parallel", "moe"))


def _design_config(case):
    z = _D
    par = {"left": {"dim": z["dim"], "heads": z["heads"], "kv_heads": z["kv"], "mask": {"size": z["chunk"]}, "scale": z["dim"] ** -0.5, "vdim": z["dim"]},
           "left_scale": 1.0, "right": {"dim": z["m_dim"], "gate_cap": z["cap"], "heads": z["m_heads"], "vdim": z["m_vdim"]}, "right_scale": 1.0}
    mixers = {"parallel": par, "rglru": {"blocks": z["r_blocks"], "conv": z["conv"], "width": z["r_width"]}}
    mlps = {"dense": {"ff": z["ff"], "kind": "dense"},
            "moe": {"expert": {"ff": z["eff"]}, "kind": "moe", "router": {"experts": z["experts"], "top": z["top"]}, "shared": {"ff": z["sff"]}}}
    return {"architecture": "Safupel", "layers": [{"mixer": mixers[m], "mlp": mlps[f], "type": m} for m, f in _LAYERS], "logit_scale": 1.0, "norm": {"eps": z["eps"]},
            "vocab": z["vocab"], "width": case["width"]}


def _design_weights(case, seed):
    g, D, z, bf = _gen(seed), case["width"], _D, torch.bfloat16
    W = {"embed": _randn(g, (z["vocab"], D), 1.0, bf), "final.norm": _randn(g, (D,), 0.2, bf), "head": _randn(g, (z["vocab"], D), D ** -0.5, bf)}

    def mat(name, *shape):
        W[name] = _randn(g, shape, shape[-1] ** -0.5, bf)

    def vec(name, *shape, std=0.3, mean=0.0):
        W[name] = _randn(g, shape, std, bf, mean)
    for i, (mixer, mlp) in enumerate(_LAYERS):
        p = f"l{i}."
        vec(p + "norm1", D, std=0.2)
        if mixer == "rglru":
            w, nb = z["r_width"], z["r_blocks"]
            for n in "yx":
                mat(f"{p}mix.{n}", w, D)
                vec(f"{p}mix.{n}.b", w)
            vec(p + "mix.conv", w, z["conv"], std=0.5)
            vec(p + "mix.conv.b", w)
            for n in ("ra", "ri"):
                mat(f"{p}mix.{n}", nb, w // nb, w // nb)
                vec(f"{p}mix.{n}.b", nb, w // nb)
            vec(p + "mix.lam", w, std=1.0, mean=-1.5)
            mat(p + "mix.o", D, w)
        else:
            H, KV, hd, mh, md, mv = z["heads"], z["kv"], z["dim"], z["m_heads"], z["m_dim"], z["m_vdim"]
            for n, rows in (("left.q", H * hd), ("left.k", KV * hd), ("left.v", KV * hd), ("right.q", mh * md), ("right.k", mh * md), ("right.v", mh * mv), ("right.g", mh * mv)):
                mat(f"{p}mix.{n}", rows, D)
            mat(p + "mix.left.o", D, H * hd)
            mat(p + "mix.right.o", D, mh * mv)
            vec(p + "mix.right.norm", mh * mv, std=0.2, mean=1.0)
            for n in "if":
                mat(f"{p}mix.right.{n}", mh, D)
                vec(f"{p}mix.right.{n}.b", mh)
        if mlp == "dense":
            mat(p + "mlp.up", z["ff"], D)
            mat(p + "mlp.down", D, z["ff"])
        else:
            W[p + "mlp.router"] = _randn(g, (z["experts"], D), 2.0 * D ** -0.5, bf)
            for n, e in [(f"e{x}", z["eff"]) for x in range(z["experts"])] + [("shared", z["sff"])]:
                mat(f"{p}mlp.{n}.gate", e, D)
                mat(f"{p}mlp.{n}.up", e, D)
                mat(f"{p}mlp.{n}.down", D, e)
    return W


def _design_prepare(case, seed):
    ids, bs = _tokens(case, seed, case["decode"]), 64
    blocks = max(len(ids) * ((max(map(len, ids)) + bs - 1) // bs), 4096 // bs) + 1
    llm = _engine(_design_config(case), _design_weights(case, seed), max_model_len=4096, max_num_seqs=8, max_num_batched_tokens=4096, block_size=bs,
                  num_gpu_blocks_override=blocks, enable_prefix_caching=False)
    n = case["decode"]
    batches = [_Batch([(0, len(t) - n) for t in ids], ids, bs).args]
    batches += [_Batch([(len(t) - n + k, len(t) - n + k + 1) for t in ids], ids, bs).args for k in range(n)]
    return {"case": case, "llm": llm, "batches": batches}


def _design_run(st):
    steps = [st["llm"].raw_step(*b, want_logits=True) for b in st["batches"]]
    return {"logits": [s[1] for s in steps], "tokens": [s[0] for s in steps]}


def _design_forward64(W, ids):
    z = _D
    T, dev = len(ids), "cuda"
    x = W["embed"][torch.tensor(ids, device=dev)]

    def rms(v, w):
        return v / torch.sqrt(v.pow(2).mean(-1, keepdim=True) + z["eps"]) * w

    def unit(h, p):
        return (torch.nn.functional.silu(h @ W[p + "gate"].T) * (h @ W[p + "up"].T)) @ W[p + "down"].T
    for i, (mixer, mlp) in enumerate(_LAYERS):
        p = f"l{i}."
        h = rms(x, 1.0 + W[p + "norm1"])
        if mixer == "rglru":
            w, nb = z["r_width"], z["r_blocks"]
            y = torch.nn.functional.gelu(h @ W[p + "mix.y"].T + W[p + "mix.y.b"], approximate="tanh")
            u = h @ W[p + "mix.x"].T + W[p + "mix.x.b"]
            padded = torch.cat([u.new_zeros(z["conv"] - 1, w), u])
            u = sum(padded[j:j + T] * W[p + "mix.conv"][:, j] for j in range(z["conv"])) + W[p + "mix.conv.b"]
            ub = u.view(T, nb, w // nb)
            r, gi = (torch.sigmoid(torch.einsum("tbi,boi->tbo", ub, W[f"{p}mix.{n}"]) + W[f"{p}mix.{n}.b"]).reshape(T, w) for n in ("ra", "ri"))
            a = torch.exp(-8.0 * r * torch.nn.functional.softplus(W[p + "mix.lam"]))
            drive = torch.sqrt(1.0 - a * a) * gi * u
            s, rows = u.new_zeros(w), []
            for t in range(T):
                s = a[t] * s + drive[t]
                rows.append(s)
            mix = (torch.stack(rows) * y) @ W[p + "mix.o"].T
        else:
            H, KV, hd, mh, md, mv = z["heads"], z["kv"], z["dim"], z["m_heads"], z["m_dim"], z["m_vdim"]
            q = (h @ W[p + "mix.left.q"].T).view(T, H, hd)
            k, v = ((h @ W[f"{p}mix.left.{n}"].T).view(T, KV, hd) for n in "kv")
            at = torch.arange(T, device=dev)
            gone = (at[None, :] > at[:, None]) | (at[None, :] // z["chunk"] != at[:, None] // z["chunk"])
            o = torch.empty(T, H, hd, dtype=torch.float64, device=dev)
            for n in range(H):
                sc = (q[:, n] @ k[:, n * KV // H].T) * hd ** -0.5 - 2.0 ** (-8.0 * (n + 1) / H) * (at[:, None] - at[None, :])
                o[:, n] = torch.softmax(sc.masked_fill(gone, -math.inf), -1) @ v[:, n * KV // H]
            mix = o.reshape(T, H * hd) @ W[p + "mix.left.o"].T
            q, k = ((h @ W[f"{p}mix.right.{n}"].T).view(T, mh, md) for n in "qk")
            q, v = q * md ** -0.5, (h @ W[p + "mix.right.v"].T).view(T, mh, mv)
            li, lf = (z["cap"] * torch.tanh((h @ W[f"{p}mix.right.{n}"].T + W[f"{p}mix.right.{n}.b"]) / z["cap"]) for n in "if")
            lf = torch.nn.functional.logsigmoid(lf)
            # every pair of positions at once: weight of k_j v_j^T in the memory at t is exp(F_t - F_j + li_j - m_t), m_t the running largest
            F = lf.cumsum(0)
            o = torch.empty(T, mh, mv, dtype=torch.float64, device=dev)
            for n in range(mh):
                lw = (F[:, None, n] - F[None, :, n] + li[None, :, n]).masked_fill(at[None, :] > at[:, None], -math.inf)
                m = torch.maximum(lw.max(-1).values, F[:, n])           # the empty memory before the first token has m = 0
                wts = torch.exp(lw - m[:, None]) * (q[:, n] @ k[:, n].T)
                o[:, n] = (wts @ v[:, n]) / (torch.maximum(wts.sum(-1).abs(), torch.exp(-m)) + 1e-6)[:, None]
            o = (o / torch.sqrt(o.pow(2).mean(-1, keepdim=True) + z["eps"])).reshape(T, mh * mv)
            mix = mix + (o * W[p + "mix.right.norm"] * torch.sigmoid(h @ W[p + "mix.right.g"].T)) @ W[p + "mix.right.o"].T
        if mlp == "dense":
            ff = torch.nn.functional.gelu(h @ W[p + "mlp.up"].T) @ W[p + "mlp.down"].T
        else:
            pr = torch.sigmoid(h @ W[p + "mlp.router"].T)
            ff = unit(h, p + "mlp.shared.")
            chosen = pr.topk(z["top"], -1).indices
            for e in range(z["experts"]):
                rows = (chosen == e).any(-1).nonzero()[:, 0]
                ff[rows] += unit(pr[rows, e:e + 1] * h[rows], f"{p}mlp.e{e}.")
        x = x + mix + ff
    return rms(x, 1.0 + W["final.norm"]) @ W["head"].T


def _design_exact(case, seed):
    W = {k: v.double() for k, v in _design_weights(case, seed).items()}
    n = case["decode"]
    full = [_design_forward64(W, t)[-(n + 1):] for t in _tokens(case, seed, n)]
    return {"logits": [torch.stack([f[k] for f in full]) for k in range(n + 1)], "tokens": [None] * (n + 1)}


def _design_work(case):
    z, D, n = _D, case["width"], case["decode"]
    T = case["reqs"] * (case["ctx_lo"] + case["ctx_hi"]) / 2
    att = D * z["dim"] * (2 * z["heads"] + 2 * z["kv"]) + D * z["m_heads"] * (2 * z["m_dim"] + 3 * z["m_vdim"])
    rec = 3 * D * z["r_width"] + 2 * z["r_width"] ** 2 // z["r_blocks"]
    dense, expert, shared, head = 2 * D * z["ff"], 3 * D * z["eff"], 3 * D * z["sff"], z["vocab"] * D
    always = 2 * (att + rec + dense + shared)
    token = always + 2 * z["top"] * expert
    tokens_attn = 2 * T * min(z["chunk"], (case["ctx_lo"] + case["ctx_hi"]) / 2) / 2 * 4 * z["heads"] * z["dim"]
    steps = 2.0 * (always + 2 * z["experts"] * expert + head) + n * 2.0 * (always + head + 2 * expert * min(z["experts"], z["top"] * case["reqs"]))
    return {"bytes": steps + 4.0 * case["reqs"] * (n + 1) * z["vocab"], "flops": 2.0 * (T + n * case["reqs"]) * token + tokens_attn + 2.0 * case["reqs"] * (n + 1) * head}


# ----------------------------------------------------------------------------------------------------------- the interface

def prepare(case, seed):
    return globals()[f"_{case['kind']}_prepare"](case, seed)


def run(state):
    return globals()[f"_{state['case']['kind']}_run"](state)


def exact(case, seed):
    return globals()[f"_{case['kind']}_exact"](case, seed)


def work(case):
    return globals()[f"_{case['kind']}_work"](case)


def tolerance(case):
    # Four times the error that was measured against exact(): one rounding of each stored intermediate to the 16-bit type
    # (2^-9 of it in bfloat16, an eighth of that in float16).  Whole models carry such a rounding through every layer.  A token
    # may differ where two candidates are as good as equal.
    rel = {"attn": 8e-3, "mlp": 2e-2, "qkv": 1.4e-2, "head": 1.2e-2, "step": 4e-2, "design": 6e-2}[case["kind"]]
    if case.get("dtype") == "fp16":
        rel /= 8 if case["kind"] != "attn" else 6
    t = {"rel": rel}
    if case["kind"] in ("head", "step", "design"):
        t["differ"] = 0.15 if case["kind"] == "head" else 0.3
    return t
