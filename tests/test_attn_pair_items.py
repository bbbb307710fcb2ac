"""Which CTA of a prompt attention launch (csrc/attn_pair.cuh) takes which work, run on the CPU from the kernel's own source: every query
tile of every request is handed out exactly once, and CTAs beyond the work get none."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.join(os.path.dirname(__file__), "..")
SRC = os.path.join(ROOT, "kubernetes-gpu-cluster_b200", "csrc", "attn_pair.cuh")
pytestmark = pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")


@pytest.fixture(scope="module")
def finder(tmp_path_factory):
    d = tmp_path_factory.mktemp("items")
    src = open(SRC).read()
    part = src[src.index("int rank = bz, kvh = bx, b = by;"):]
    (d / "part.inc").write_text(part[:re.search(r"const int tok0 = [^;]*;", part).end()] + "\n")
    exe = str(d / "items")
    subprocess.run(["g++", "-std=c++20", "-O1", "-g", "-fsanitize=undefined", "-fno-sanitize-recover=all", f'-DKERNEL_PART="{d}/part.inc"', os.path.join(ROOT, "tests", "cpp", "pair_items.cc"),
                    "-o", exe, "-lpthread"], check=True)
    return exe


def launch(H, KV, q, max_seq):
    """The grid of launch_pair (attn_pair.cuh) and tc_grid (attn_tc.cu)."""
    TT, B, T = 128 // (H // KV), len(q), sum(q)

    def grid(per):
        tiles = -(-max(q) // (per * TT))
        flat = 2 * (T // (per * TT) + B) < tiles * B
        return flat, (KV * (T // (per * TT) + B),) if flat else (KV, B, tiles)
    per = 2
    flat, g = grid(per)
    n = g[0] if flat else g[0] * g[1] * g[2]
    if n <= 74 or (n <= 148 and max_seq >= 512):
        per = 1
        flat, g = grid(per)
    return per, flat, g + (1, 1) if flat else g


CASES = [  # heads, kv heads, query lengths
    (12, 12, [2048] + [256] * 12), (8, 8, [1] * 64 + [2048]), (12, 12, [3000] + [60] * 6), (32, 32, [1] * 63 + [2048]), (4, 4, [1300, 257]),      # a head per group: 256 tokens an item
    (32, 8, [1] * 60 + [700, 130]), (32, 8, [2048] * 4), (64, 2, [333, 5, 1]), (24, 8, [400, 43, 700]), (32, 8, [1] * 33 + [300]), (128, 1, [1] * 5 + [3]), (8, 8, [17] * 40),
]


@pytest.mark.parametrize("H,KV,q", CASES, ids=str)
def test_every_item_once(finder, H, KV, q):
    per, flat, grid = launch(H, KV, q, max(q))
    qsl = [sum(q[:i]) for i in range(len(q) + 1)]
    ctas = [(x, y, z) for x in range(grid[0]) for y in range(grid[1]) for z in range(grid[2])]
    text = " ".join(map(str, [H, KV, per, int(flat), len(q), *qsl, *[v for c in ctas for v in c]]))
    p = subprocess.run([finder], input=text, capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stderr[-500:]
    got = [tuple(map(int, line.split())) for line in p.stdout.splitlines()]
    assert len(got) == len(ctas)
    TI = per * (128 // (H // KV))
    want = sorted((b, h, t) for b, n in enumerate(q) for h in range(KV) for t in range(0, n, TI))
    assert sorted(g for g in got if g[2] >= 0) == want


def test_a_head_per_group_is_launched_by_request():
    assert all(launch(H, KV, q, max(q))[:2] == (2, True) for H, KV, q in CASES[:4])
