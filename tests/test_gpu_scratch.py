"""GPU: the library's own pool of temporary buffers under several threads and
streams, trimmed in between, and inside a captured graph; every product
against a run on its own (bitwise: the sums run in a fixed order)."""
import threading

import pytest
import torch

import rvvlasparse_b200 as R
from rvvlasparse_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _mv(A, x, y):
    st = R.sparse_mv(R.SPARSE_OPERATION_NON_TRANSPOSE, 1.0, A, R.sparse_matrix_descr(), x, 0.0, y)
    assert st.code == 0, R.load().rvvla_last_error()


def _case(n, seed):
    m, n, Rst, Col, Val = W.powerlaw(n, band=256, seed=seed)
    A = R.spMtxCRS.from_host(m, n, Rst, Col, Val, dtype=torch.float64)
    x = torch.as_tensor(W.vector(n, seed)).cuda()
    y = torch.empty(m, dtype=torch.float64, device="cuda")
    _mv(A, x, y)
    torch.cuda.synchronize()
    return A, x, y.clone()


def test_threads_streams_and_trim():
    cases = [_case(20000 + 7001 * i, 3 + i) for i in range(4)]
    bad = []

    def work(A, x, ref):
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            for it in range(25):
                y = torch.full_like(ref, float("nan"))
                _mv(A, x, y)
                if it % 5 == 0:
                    s.synchronize()
                    if R.load().rvvla_trim_scratch() != 0:
                        bad.append("trim")
                if not torch.equal(y, ref):
                    bad.append(it)

    ts = [threading.Thread(target=work, args=c) for c in cases]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad


def test_captured_product():
    A, x, ref = _case(30011, 9)
    y = torch.full_like(ref, float("nan"))
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        _mv(A, x, y)
    for _ in range(3):
        y.fill_(float("nan"))
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(y, ref)
