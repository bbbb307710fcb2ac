"""Prompt attention with two query tiles per CTA (csrc/attn_pair.cuh) against plain float64 attention: pairs of query tiles, one query
tile with its key tiles shared out, single-token rows beside prompts, ragged ends, group sizes that do not divide a tile, every block size."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

CASES = [   # dtype, heads, kv heads, head size, block, query lengths, tokens cached before them
    ("bf16", 32, 8, 128, 64, [512], [0]),                                       # few long items: one query tile each, split
    ("bf16", 32, 8, 128, 64, [64, 63, 65, 1], [449, 450, 448, 0]),              # ends of 64-key tiles; one key alone
    ("bf16", 32, 8, 128, 32, [1000, 129, 640, 900, 385], [0, 77, 0, 1, 63]),    # pairs
    ("bf16", 4, 4, 128, 16, [1300, 257], [0, 255]),                             # a head of its own per group: 128 tokens a query tile
    ("fp16", 24, 8, 128, 64, [400, 43, 700], [0, 500, 100]),                    # groups of 3: 126 rows of a tile in use
    ("bf16", 64, 2, 64, 8, [333, 5, 1], [0, 800, 1200]),                        # groups of 32: 4 tokens a query tile
    ("bf16", 12, 12, 64, 128, [2048, 1500], [0, 0]),
    ("fp16", 32, 8, 64, 16, [1] * 60 + [700, 130], [37 * i for i in range(60)] + [0, 900]),      # by request, from the last to the first
    ("bf16", 32, 8, 128, 64, [1] * 33 + [300], [5 + 64 * i for i in range(33)] + [0]),
    ("bf16", 128, 1, 128, 64, [1] * 5 + [3], [2000, 0, 63, 64, 65] + [500]),     # groups of 128: a token a query tile
]
# the same over contexts that no small launch has (launch_tc in csrc/attn_tc.cu keeps those for its own kernel)
LONG = [
    ("bf16", 32, 8, 128, 64, [512], [600]),
    ("bf16", 32, 8, 128, 64, [64, 63, 65, 1], [1089, 1090, 1088, 0]),
    ("fp16", 24, 8, 128, 64, [400, 43, 700], [0, 2600, 100]),
    ("bf16", 64, 2, 64, 8, [333, 5, 1], [2300, 800, 1200]),
    ("bf16", 4, 4, 128, 16, [1300, 257], [800, 255]),
    ("bf16", 128, 1, 128, 64, [1] * 5 + [3], [2700, 0, 63, 64, 65] + [500]),
]


def case(kge, dtype, H, KV, hd, bs, q, prior, ramp):
    dt = torch.bfloat16 if dtype == "bf16" else torch.float16
    g = torch.Generator(device="cuda").manual_seed(5)
    ctx = [a + b for a, b in zip(q, prior)]
    B, T, per = len(q), sum(q), [(c + bs - 1) // bs for c in ctx]
    order = torch.randperm(sum(per), generator=g, device="cuda").add(1).to(torch.int32)
    table = torch.zeros(B, max(per), dtype=torch.int32, device="cuda")       # beyond a request's blocks: block 0, which nothing may use
    for b, n in enumerate(per):
        table[b, :n] = order[sum(per[:b]):sum(per[:b + 1])]
    kc, vc = (torch.randn(sum(per) + 1, KV, bs, hd, generator=g, device="cuda").to(dt) for _ in range(2))
    kc[0] = vc[0] = float("nan")
    qkv = torch.randn(T, (H + 2 * KV) * hd, generator=g, device="cuda").to(dt)
    if ramp:        # scores that grow along the context by some 80 powers of two: every tile rescales
        u = torch.nn.functional.normalize(torch.randn(hd, generator=g, device="cuda"), dim=0)
        qkv[:, :H * hd] = (qkv[:, :H * hd].float().view(T, H, hd) + 1.5 * hd ** 0.5 * u).reshape(T, H * hd).to(dt)
        for b, n in enumerate(per):
            pos = torch.arange(n * bs, device="cuda").view(n, 1, bs, 1) / ctx[b]
            rows = table[b, :n].long()
            kc[rows] = (kc[rows].float() + 40.0 * pos * u).to(dt)
    out = torch.full((T, H * hd), float("nan"), dtype=dt, device="cuda")
    lens = torch.tensor(ctx, dtype=torch.int32, device="cuda")
    qsl = torch.tensor(np.concatenate([[0], np.cumsum(q)]), dtype=torch.int32, device="cuda")
    fn = getattr(kge.lib(), "kge_paged_attn" + ("_f16" if dtype == "fp16" else ""))
    rc = fn(out.data_ptr(), qkv.data_ptr(), qkv.shape[1], kc.data_ptr(), vc.data_ptr(), table.data_ptr(), table.shape[1], lens.data_ptr(), qsl.data_ptr(), B, T,
            max(q), max(ctx), H, KV, hd, bs, hd ** -0.5, None, 0, None)
    if rc:
        kge.check(rc, "kge_paged_attn")
    torch.cuda.synchronize()
    at, ref = 0, []
    for b in range(B):
        rows = table[b, :per[b]].long()
        k, v = (x[rows].permute(0, 2, 1, 3).reshape(-1, KV, hd)[:ctx[b]].double().repeat_interleave(H // KV, 1) for x in (kc, vc))
        x = qkv[at:at + q[b], :H * hd].double().view(q[b], H, hd)
        s = torch.einsum("thd,shd->hts", x, k) * hd ** -0.5
        hidden = torch.arange(ctx[b], device="cuda")[None, :] > torch.arange(q[b], device="cuda")[:, None] + prior[b]
        ref.append(torch.einsum("hts,shd->thd", s.masked_fill_(hidden, -np.inf).softmax(-1), v).reshape(q[b], H * hd))
        at += q[b]
    return out.double(), torch.cat(ref), dt


@pytest.mark.parametrize("ramp", [False, True])
@pytest.mark.parametrize("c", CASES + LONG, ids=lambda c: f"{c[0]}-{c[1]}x{c[2]}x{c[3]}-{c[4]}-{max(c[5])}-{max(c[6])}")
def test_against_float64(kge, c, ramp):
    out, ref, dt = case(kge, *c, ramp)
    assert torch.isfinite(out).all()
    # a weight and the result are rounded to the type once each: half an ulp, 2^-8 in bfloat16 and 2^-11 in float16, of either at most
    u = 2.0 ** (-8 if dt == torch.bfloat16 else -11)
    err = (out - ref).reshape(-1, c[3]).norm(dim=1) / ref.reshape(-1, c[3]).norm(dim=1).clamp_min(1e-3)
    assert (out - ref).norm() <= 2 * u * ref.norm()
    # one row of one head: the same bound against the norm of what is summed, |v| of unit variance under weights that sum to one
    assert ((out - ref).abs().amax() <= 2 * u * 6 and err.median() <= 2 * u)
