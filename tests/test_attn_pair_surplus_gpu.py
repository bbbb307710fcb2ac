"""Prompts of models with a key and value head per query head, launched by request with more CTAs than work."""
import pytest
import torch

from test_attn_pair_gpu import case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("c", [
    ("bf16", 12, 12, 64, 16, [2048] + [256] * 12, [0] * 13),
    ("fp16", 8, 8, 128, 32, [1] * 64 + [2048], [10 * i for i in range(64)] + [100]),
    ("bf16", 12, 12, 128, 64, [3000] + [60] * 6, [0] * 7),
], ids=lambda c: f"{c[0]}-{c[1]}x{c[2]}x{c[3]}-{max(c[5])}")
def test_against_float64(kge, c):
    out, ref, dt = case(kge, *c, False)
    u = 2.0 ** (-8 if dt == torch.bfloat16 else -11)          # weights and the result are rounded once each
    assert torch.isfinite(out).all() and (out - ref).norm() <= 2 * u * ref.norm()
