"""Rules of the kernels that no result shows, read from their sources: distributed shared memory is touched only behind a cluster
barrier, since a block's peers may not have started before it; and barrier waits are bounded in time, in one place."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "kubernetes-gpu-cluster_b200", "csrc")
# what reaches into a peer's shared memory, or signals a barrier there, from a kernel's body
REMOTE = re.compile(r"\b(st_cluster\w*|ld_dsmem_\w+|cluster_reduce|mapa_u32|mbar_arrive_cluster)\(|shared::cluster\.(?!b64)")
BARRIER = re.compile(r"\bcluster_wait\(\)")


def kernels():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        src = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__[^;{]*?(\w+_kernel)\(", src):
            body = src[src.index("{", m.end()):]
            end = re.search(r"\n}\n", body)
            yield os.path.basename(path), m.group(1), body[:end.start() if end else len(body)]


USERS = [(f, k, b) for f, k, b in kernels() if REMOTE.search(b)]


def test_the_kernels_are_found():
    assert {k for _, k, _ in USERS} >= {"sample_kernel", "gemm_tc_kernel", "gemm_wide_kernel", "attn_decode_kernel"}


@pytest.mark.parametrize("file,kernel,body", USERS, ids=[k for _, k, _ in USERS])
def test_a_cluster_barrier_comes_before_the_first_remote_access(file, kernel, body):
    # a lambda that only forms an address is not an access: calls count from where the first one is made
    code = re.sub(r"auto \w+ = \[&\]\([^)]*\) \{[^\n]*\};", "", body)
    first = REMOTE.search(code)
    assert first, (file, kernel)
    wait = BARRIER.search(code)
    assert wait and wait.start() < first.start(), (file, kernel, code[first.start():first.start() + 80])


def test_barrier_waits_are_bounded_by_the_clock():
    """A try on a shared-memory barrier that fails lasts microseconds: counting tries bounds a wait by minutes."""
    users = {os.path.basename(p) for p in glob.glob(os.path.join(CSRC, "*.cu*")) if "try_wait" in re.sub(r"//[^\n]*", "", open(p).read())}
    assert users == {"common.cuh"}
    src = open(os.path.join(CSRC, "common.cuh")).read()
    assert 1e9 <= int(re.search(r"kBarrierCycles = (\d+)ll", src).group(1)) <= 2e10


def test_waits_for_tensor_memory_hold_back_what_reads_it():
    """A load from tensor memory names registers that are filled later: a wait that does not name them holds back no arithmetic on them."""
    waits = 0
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        src = re.sub(r"//[^\n]*", "", open(path).read())
        assert ("tcgen05.wait::ld" in src) == path.endswith("common.cuh"), path
        for call in re.findall(r"tmem_wait_ld\(([^()]*)\);", src):
            assert call, path
            waits += 1
    assert waits >= 8


TENSOR_MEMORY = [(f, k, b) for f, k, b in kernels() if "tcgen05.alloc" in b and "pdl_launch_dependents" in b]


def test_the_kernels_with_tensor_memory_are_found():
    assert {k for _, k, _ in TENSOR_MEMORY} >= {"gemm_tc_kernel", "gemm_wide_kernel", "attn_tc_kernel", "attn_pair_kernel", "rglru_gates_kernel"}


@pytest.mark.parametrize("file,kernel,body", TENSOR_MEMORY, ids=[k for _, k, _ in TENSOR_MEMORY])
def test_tensor_memory_is_allocated_before_the_next_kernel_may_start(file, kernel, body):
    """An allocation waits until columns are free.  Blocks of a later kernel that had taken them would wait for this kernel to end."""
    alloc, start = body.index("tcgen05.alloc"), body.index("pdl_launch_dependents")
    assert alloc < start, (file, kernel)
    assert "__syncthreads()" in body[alloc:start], (file, kernel)      # by one warp: the others may not announce it earlier
