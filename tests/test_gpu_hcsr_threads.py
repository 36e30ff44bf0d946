"""GPU: HCSR products of several block sizes, whose kernels want different
amounts of shared memory, called from several threads at once: each succeeds
and equals a run on its own.  (The limit on a kernel's shared memory is a
property of the kernel, common to all threads.)"""
import ctypes as C
import threading

import pytest
import torch

import rvvlasparse_b200 as R
from rvvlasparse_b200 import workloads as W

pytestmark = pytest.mark.gpu


def test_block_sizes_in_threads():
    m, n, Rst, Col, Val = W.powerlaw(20000, band=256, seed=4)
    A = R.spMtxCRS.from_host(m, n, Rst, Col, Val, dtype=torch.float64)
    x = torch.as_tensor(W.vector(n, 3)).cuda()

    lib = R.load()

    def mv(d, y, st):
        return lib.rvvla_hcsr_spmv_f64(d, 1.0, x.data_ptr(), 0.0, y.data_ptr(), st)

    cases = []
    for r in (64, 9000, 500, 20000, 4000, 13000):
        H = R.convert(R.spMtxHCSR(), A, R.convertParams(R=r, C=2000))
        y = torch.empty(m, dtype=torch.float64, device="cuda")
        d = H.desc()
        assert mv(C.byref(d), y, torch.cuda.current_stream().cuda_stream) == 0
        cases.append((d, H, y))
    torch.cuda.synchronize()
    bad = []

    def work(d, _, ref):
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            y, dp, st = torch.empty_like(ref), C.byref(d), s.cuda_stream
            for _ in range(6000):
                if mv(dp, y, st):
                    bad.append(lib.rvvla_last_error())
            s.synchronize()
            if not torch.equal(y, ref):
                bad.append("result")

    ts = [threading.Thread(target=work, args=c) for c in cases]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad, (len(bad), bad[0])
