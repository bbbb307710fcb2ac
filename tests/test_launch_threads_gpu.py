"""Launches of one kernel with different amounts of shared memory from two threads of a program (two engines on a device) do not get in
each other's way: what a function may ask for is set once for all sizes, not for the call at hand."""
import ctypes as C
import threading

import pytest
import torch

from test_norm_gemm_gpu import Kv, Norm

pytestmark = pytest.mark.gpu


def test_norm_gemm_of_two_sizes(kge):
    kge.require_cuda()
    fn, K, N, turns = kge.lib().kge_norm_gemm, 1024, 4736, 4000
    fn.argtypes, fn.restype = [C.c_void_p] * 4 + [C.c_int] * 4 + [C.c_void_p] * 2, C.c_int
    failed = []

    def run(T):
        torch.cuda.set_device(0)
        stream = torch.cuda.Stream()
        res, w, b, W, y = (torch.zeros(*s, dtype=torch.bfloat16, device="cuda") for s in ((T, K), (K,), (K,), (N, K), (T, N)))
        nm, kv = Norm(res.data_ptr(), None, None, w.data_ptr(), b.data_ptr(), 1e-5), Kv()
        torch.cuda.synchronize()
        start.wait()
        failed.extend(T for _ in range(turns) if fn(y.data_ptr(), C.addressof(nm), W.data_ptr(), None, T, N, K, 0, C.addressof(kv), stream.cuda_stream) != 0)
        stream.synchronize()
    start = threading.Barrier(2)
    threads = [threading.Thread(target=run, args=(T,)) for T in (1, 8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed
