"""Pages come with what a former owner left in them: prompts over pages whose rows behind each request's last key are not finite give what
they give over clean ones."""
import numpy as np
import pytest
import torch

from oracle import hybrid as oh
from test_attn_pair_gpu import CASES, LONG
from test_hybrid_gpu import check, make_engine, prompt, run_pieces

pytestmark = pytest.mark.gpu


@pytest.fixture(params=[1, 0], ids=["tma", "gather"])
def staging(kge, request):
    kge.check(kge.lib().kge_set_tunable(b"attn_tma", request.param), "tunable")
    yield
    kge.check(kge.lib().kge_set_tunable(b"attn_tma", 1), "tunable")


# prompts of small launches (attn_tc_kernel): a piece of a tile, ends inside and at groups of 16 keys
SMALL = [
    ("bf16", 32, 8, 128, 64, [17], [0]), ("bf16", 8, 8, 64, 16, [64, 50, 3], [0, 30, 77]), ("fp16", 16, 4, 128, 32, [40, 1, 48, 47], [0, 100, 17, 0]),
]


@pytest.mark.parametrize("c", CASES + LONG + SMALL, ids=lambda c: f"{c[0]}-{c[1]}x{c[2]}x{c[3]}-{c[4]}-{max(c[5])}-{max(c[6])}")
def test_prompts(kge, staging, c):
    dtype, H, KV, hd, bs, q, prior = c
    dt = torch.bfloat16 if dtype == "bf16" else torch.float16
    g = torch.Generator(device="cuda").manual_seed(6)
    ctx = [a + b for a, b in zip(q, prior)]
    B, T, per = len(q), sum(q), [(n + bs - 1) // bs for n in ctx]
    table = torch.zeros(B, max(per), dtype=torch.int32, device="cuda")
    for b, n in enumerate(per):
        table[b, :n] = torch.arange(n, device="cuda") + 1 + sum(per[:b])
    clean = [torch.randn(sum(per) + 1, KV, bs, hd, generator=g, device="cuda").to(dt) for _ in range(2)]
    stale = [x.clone() for x in clean]
    for x, bad in zip(stale, (float("nan"), float("inf"))):
        x[0] = bad
        for b in range(B):
            x[table[b, per[b] - 1].item(), :, (ctx[b] - 1) % bs + 1:] = bad
    qkv = torch.randn(T, (H + 2 * KV) * hd, generator=g, device="cuda").to(dt)
    lens = torch.tensor(ctx, dtype=torch.int32, device="cuda")
    qsl = torch.tensor(np.concatenate([[0], np.cumsum(q)]), dtype=torch.int32, device="cuda")
    fn = getattr(kge.lib(), "kge_paged_attn" + ("_f16" if dtype == "fp16" else ""))
    got = []
    for kc, vc in (clean, stale):
        out = torch.full((T, H * hd), float("nan"), dtype=dt, device="cuda")
        kge.check(fn(out.data_ptr(), qkv.data_ptr(), qkv.shape[1], kc.data_ptr(), vc.data_ptr(), table.data_ptr(), table.shape[1], lens.data_ptr(), qsl.data_ptr(), B, T,
                     max(q), max(ctx), H, KV, hd, bs, hd ** -0.5, None, 0, None), "kge_paged_attn")
        got.append(out)
    torch.cuda.synchronize()
    assert torch.isfinite(got[0]).all() and torch.equal(*got)


@pytest.mark.parametrize("hd,chunk", [(128, 1024), (64, 40)])
def test_biased_prompts(kge, tmp_path, staging, hd, chunk):
    """All pages of the pool first hold keys and values of a request whose embeddings are not finite."""
    cfg = oh.make_config(layers=("parallel",), mlps=(None,), right_scale=0.0, chunk=chunk, scale=3.0 / hd ** 0.5, dim=hd, vdim=hd)
    W = oh.make_weights(cfg, seed=31)
    W["embed"][5] = float("inf")
    toks = [t if t != 5 else 6 for t in prompt(cfg, 150)]
    llm = make_engine(kge, tmp_path, cfg, W, "bfloat16", tokens=160, bs=16)
    llm.trace_add(0, [5] * 160)
    assert not np.isfinite(llm.trace_step([(0, 160, [159])])).any()
    llm.trace_end(0)
    got = run_pieces(llm, 1, toks, [99, 50, 1])
    llm.close()
    W["embed"][5] = 0.0
    check(got, oh.forward(cfg, W, toks), "bfloat16")
