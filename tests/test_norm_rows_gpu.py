"""Norms of many rows (csrc/elementwise.cu, norm_rows_kernel) against float64: each number of threads per row, rows and pieces that fill no
round of the loop."""
import pytest
import torch

pytestmark = pytest.mark.gpu
HALF_ULP = {"": 2.0 ** -8, "_f16": 2.0 ** -11}        # largest relative error of one rounding: p significant bits (8 and 11), half a step of 2^(1 - p) at 1


def inputs(T, d, kind):
    g = torch.Generator(device="cuda").manual_seed(T + d)
    dt = torch.float16 if kind else torch.bfloat16
    return [(torch.randn(*s, generator=g, device="cuda") * k + m).to(dt) for s, k, m in (((T, d), 1, 0), ((T, d), 2, 0), ((d,), 0.1, 1), ((d,), 0.1, 0))]


def call(kge, name, *a):
    rc = getattr(kge.lib(), name)(*[t.data_ptr() if isinstance(t, torch.Tensor) else t for t in a], None)
    if rc:
        kge.check(rc, name)
    torch.cuda.synchronize()


def close(y, ref, roundings, kind):
    # the sums of a row and the products are in fp32: a few 2^-24 of numbers below 8
    assert ((y.double() - ref).abs() <= roundings * HALF_ULP[kind] * 1.01 * ref.abs() + 2e-5 * HALF_ULP[kind] / HALF_ULP[""] + 4e-6).all()


@pytest.mark.parametrize("kind", ["", "_f16"])
@pytest.mark.parametrize("T,d", [(4096, 768), (4099, 1024), (4097, 1032), (4500, 2048), (4097, 3080), (4098, 8192), (1339, 2048), (489, 4096), (250000, 8)])
def test_rmsnorm(kge, kind, T, d):
    x, res, w, _ = inputs(T, d, kind)
    y = torch.empty_like(x)

    def norm(v):
        return v / torch.sqrt(v.pow(2).mean(-1, keepdim=True) + 1e-5) * w.double()
    call(kge, "kge_rmsnorm" + kind, y, x, w, T, d, 1e-5)
    close(y, norm(x.double()), 2, kind)                    # the normalised number and its product with the weight are rounded
    s = x.float() + res.float()
    call(kge, "kge_add_rmsnorm" + kind, y, res, x, w, T, d, 1e-5)
    assert torch.equal(res, s.to(x.dtype))
    close(y, norm(s.double()), 2, kind)


@pytest.mark.parametrize("kind", ["", "_f16"])
@pytest.mark.parametrize("T,d", [(2605, 768), (1955, 1024), (977, 2056), (489, 4096), (245, 8192), (250003, 8)])
def test_layernorm(kge, kind, T, d):
    add, res, w, b = inputs(T, d, kind)
    y = torch.empty_like(res)
    ln = torch.nn.functional.layer_norm
    call(kge, "kge_layernorm" + kind, y, res, None, w, b, T, d, 1e-5)
    close(y, ln(res.double(), (d,), w.double(), b.double(), 1e-5), 1, kind)
    s = (res.float() + add.float()).to(res.dtype)
    call(kge, "kge_layernorm" + kind, y, res, add, w, b, T, d, 1e-5)
    assert torch.equal(res, s)
    close(y, ln(s.double(), (d,), w.double(), b.double(), 1e-5), 1, kind)
