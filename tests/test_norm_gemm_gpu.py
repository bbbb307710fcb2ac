"""LayerNorm, projection and cache write of a few rows in one launch (csrc/gemm_rows.cuh, NORM) against float64."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


class Norm(C.Structure):
    _fields_ = [(n, C.c_void_p) for n in ("res", "add", "res_out", "w", "b")] + [("eps", C.c_float)]


class Kv(C.Structure):
    _fields_ = [(n, C.c_void_p) for n in ("kc", "vc", "slots")] + [(n, C.c_int) for n in ("q_cols", "KV", "hd", "bs")]


# ends of the 64-wide chunks of K and of the 8 warps' shares, one and two tiles of outputs per CTA, an output that fills none
@pytest.mark.parametrize("dtype", ["bf16", "fp16"])
@pytest.mark.parametrize("T,H,KV,hd,K,kv", [(1, 12, 12, 64, 768, True), (8, 12, 12, 64, 768, True), (5, 2, 2, 64, 1024, True), (3, 3, 1, 16, 520, True), (1, 35, 1, 128, 8, False),
                                            (7, 37, 0, 128, 1016, False), (2, 24, 6, 128, 72, True)])
def test_norm_gemm(kge, dtype, T, H, KV, hd, K, kv):
    kge.require_cuda()
    L, dt, u = kge.lib(), *((torch.bfloat16, 2.0 ** -8) if dtype == "bf16" else (torch.float16, 2.0 ** -11))
    L.kge_norm_gemm_ok.restype = C.c_bool
    fn = getattr(L, "kge_norm_gemm" + ("_f16" if dtype == "fp16" else ""))
    fn.argtypes, fn.restype = [C.c_void_p] * 4 + [C.c_int] * 4 + [C.c_void_p] * 2, C.c_int
    N, bs = (H + 2 * KV) * hd, 4
    assert L.kge_norm_gemm_ok(T, N, K)
    g = torch.Generator(device="cuda").manual_seed(T * K)
    r = lambda *s, m=0.0, d=1.0: (torch.randn(*s, generator=g, device="cuda") * d + m).to(dt)         # noqa: E731
    res, add, w, b, W, bias = r(T, K), r(T, K), r(K, m=1.0, d=0.2), r(K, d=0.2), r(N, K, d=K ** -0.5), r(N)
    p = lambda t: t.data_ptr() if t is not None else None                                             # noqa: E731
    slots = torch.arange(T, device="cuda") * 3 + 1
    slots[T // 2] = -1 if T > 1 else slots[0]
    blocks = 3 * T // bs + 2
    for add_t, act in ((add, 0), (None, 1)):
        y, out = torch.full((T, N), float("nan"), dtype=dt, device="cuda"), torch.zeros_like(res)
        kc, vc = (torch.zeros(blocks, max(1, KV), bs, hd, dtype=dt, device="cuda") for _ in range(2))
        nm = Norm(p(res), p(add_t), p(out) if add_t is not None else None, p(w), p(b), 1e-5)
        c = Kv(p(kc), p(vc), p(slots), H * hd, KV, hd, bs) if kv else Kv()
        assert fn(p(y), C.addressof(nm), p(W), p(bias), T, N, K, act, C.addressof(c), None) == 0
        torch.cuda.synchronize()
        s = res if add_t is None else (res.float() + add.float()).to(dt)
        if add_t is not None:
            assert torch.equal(out, s)
        x = torch.nn.functional.layer_norm(s.double(), (K,), w.double(), b.double(), 1e-5)
        ref = x @ W.double().T + bias.double()
        ref = ref.relu() if act else ref
        # the normalised row and the result are rounded once each: u |x| |W| summed in quadrature over K, and u of the result
        bound = u * ((x.abs() ** 2) @ (W.double() ** 2).T).sqrt() * 4 + u * ref.abs() + 1e-3 * u
        assert ((y.double() - ref).abs() <= bound).all()
        if kv:
            kr, vr = torch.zeros_like(kc), torch.zeros_like(vc)
            for t in range(T):
                at = int(slots[t])
                if at >= 0:
                    kr[at // bs, :, at % bs] = y[t, H * hd:(H + KV) * hd].view(KV, hd)
                    vr[at // bs, :, at % bs] = y[t, (H + KV) * hd:].view(KV, hd)
            assert torch.equal(kc, kr) and torch.equal(vc, vr)


def test_sizes_that_are_not_taken(kge):
    L = kge.lib()
    L.kge_norm_gemm_ok.restype = C.c_bool
    assert not any(L.kge_norm_gemm_ok(*s) for s in ((0, 768, 768), (9, 768, 768), (1, 4737, 768), (1, 768, 1032), (1, 768, 12)))
