"""How a decode step of the gated recurrence shares a diagonal block's columns out over the blocks of a cluster (csrc/hybrid_ops.h), compiled for
the host: what can be launched for every width that the kernel takes."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.join(os.path.dirname(__file__), "..")
CUDA = "/usr/local/cuda/include"
pytestmark = pytest.mark.skipif(shutil.which("g++") is None or not os.path.isdir(CUDA), reason="needs g++ and CUDA's headers")

MAIN = r"""
#include <algorithm>
#include <cstdio>
#include "hybrid_ops.h"
int main() { for (int bw = -16; bw <= 300; ++bw) printf("%d %d\n", bw, kge::rglru_step_warps(bw)); }
"""


def test_clusters_of_decode_steps_can_be_launched(tmp_path):
    (tmp_path / "m.cc").write_text(MAIN)
    exe = str(tmp_path / "m")
    subprocess.run(["g++", "-std=c++17", "-I" + os.path.join(ROOT, "kubernetes-gpu-cluster_b200", "csrc"), "-I" + os.path.join(ROOT, "include"), "-I" + CUDA, str(tmp_path / "m.cc"),
                    "-o", exe], check=True)
    warps = {int(a): int(b) for a, b in (line.split() for line in subprocess.run([exe], capture_output=True, text=True, check=True).stdout.splitlines())}
    assert {bw for bw, w in warps.items() if w} == {bw for bw in range(16, 257, 16)} - {176, 208}
    for bw, w in warps.items():
        if w:
            parts = bw // (8 * w)
            assert bw == 8 * w * parts and 1 <= parts <= 8, (bw, w)            # a portable cluster
            assert w <= 10, (bw, w)                                            # the kernel's launch bound, 320 threads
            assert (2 * 8 * w + 16) * (bw + 8) * 2 <= (2 * 80 + 16) * (256 + 8) * 2, (bw, w)      # its limit of shared memory
