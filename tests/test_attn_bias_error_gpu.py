"""Distance-biased prompts in the tcgen05 kernel (csrc/attn_pair.cuh): their error against float64 is that of weights rounded to bfloat16
relative to each row's largest, and no more."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


class Args(C.Structure):      # kge::AttnBiasArgs (csrc/hybrid_ops.h)
    _fields_ = [("q", C.c_void_p), ("ldq", C.c_int), ("out", C.c_void_p), ("ldo", C.c_int)] + [(n, C.c_void_p) for n in ("k_cache", "v_cache", "block_table")] + \
        [("max_blocks", C.c_int)] + [(n, C.c_void_p) for n in ("seq_lens", "qsl", "positions", "token_req")] + \
        [(n, C.c_int) for n in ("B", "T", "H", "G", "dim", "vdim", "block_size", "chunk", "max_q", "num_decode")] + \
        [(n, C.c_float) for n in ("scale", "bias_span", "out_scale", "softcap")] + [("sinks", C.c_void_p)] + [(n, C.c_int) for n in ("window", "keep_first", "pool")] + \
        [(n, C.c_void_p) for n in ("pk_cache", "pv_cache")] + [(n, C.c_int) for n in ("pool_slots", "v_ld", "elt", "max_seq")]


@pytest.mark.parametrize("hd,n,scale", [(64, 300, 0.6), (64, 700, 0.2), (128, 700, 0.6)])
def test_error(kge, hd, n, scale):
    kge.require_cuda()
    H, G, bs, chunk, span = 4, 2, 16, 512, 8.0
    g = torch.Generator(device="cuda").manual_seed(n + hd)
    blocks = -(-n // bs)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()         # noqa: E731
    q, kc, vc, out = r(n, H * hd), r(blocks, G, bs, hd), r(blocks, G, bs, hd), torch.empty(n, H * hd, dtype=torch.bfloat16, device="cuda")
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")              # noqa: E731
    table, lens, qsl, pos, req = i32(range(blocks)), i32([n]), i32([0, n]), i32(range(n)), i32([0] * n)
    a = Args(q=q.data_ptr(), ldq=H * hd, out=out.data_ptr(), ldo=H * hd, k_cache=kc.data_ptr(), v_cache=vc.data_ptr(), block_table=table.data_ptr(), max_blocks=blocks, seq_lens=lens.data_ptr(),
             qsl=qsl.data_ptr(), positions=pos.data_ptr(), token_req=req.data_ptr(), B=1, T=n, H=H, G=G, dim=hd, vdim=hd, block_size=bs, chunk=chunk, max_q=n, scale=scale, bias_span=span,
             out_scale=1.0, max_seq=n)
    fn = kge.lib()["_ZN3kge15attn_bias_chunkERKNS_12AttnBiasArgsEP11CUstream_st"]
    fn.argtypes, fn.restype = [C.c_void_p, C.c_void_p], C.c_int
    assert fn(C.addressof(a), torch.cuda.current_stream().cuda_stream) == 0
    k, v = (x.permute(0, 2, 1, 3).reshape(-1, G, hd)[:n].double().repeat_interleave(H // G, 1) for x in (kc, vc))
    t = torch.arange(n, device="cuda")
    slope = 2.0 ** (-span * (torch.arange(H, device="cuda", dtype=torch.float64) + 1) / H)
    s = torch.einsum("thd,shd->hts", q.double().view(n, H, hd), k) * scale - slope[:, None, None] * (t[:, None] - t[None, :])
    s = s.masked_fill((t[None, :] > t[:, None]) | (t[None, :] < t[:, None] // chunk * chunk), -float("inf"))
    w = (s - s.amax(-1, keepdim=True)).exp()
    of = lambda p: (torch.einsum("hts,shd->thd", p, v) / w.sum(-1).T[..., None]).reshape(n, H * hd)      # noqa: E731
    ref, rounded = of(w), of(w.bfloat16().double()).bfloat16().double()
    err, bound = (out.double() - ref).norm(), (rounded - ref).norm()
    assert err <= 1.03 * bound, (err / ref.norm(), bound / ref.norm())       # measured 0.99 to 1.01; 1.05 and more with a reference that lags behind
