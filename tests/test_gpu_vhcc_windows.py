"""GPU: VHCC's register windows of end-of-row vectors and rows: vectors of 32
row ends, vectors without any, windows that run out inside a thread, threads
of one vector, and descriptors that leave the arrays' lengths unset; against
the long-double oracle (the format tests' tolerances)."""
import ctypes as C

import numpy as np
import pytest
import torch

import oracle as O
import rvvlasparse_b200 as R
from helpers import tol_for

pytestmark = pytest.mark.gpu
TDT = {np.float64: torch.float64, np.float32: torch.float32}


def _lengths(kind, rng):
    if kind == "ones":
        return np.ones(5003, int)
    if kind == "long":
        return np.array([3000, 1, 1, 33, 700, 0, 64, 32, 31, 2048])
    if kind == "alternating":
        return np.tile([1] * 31 + [97], 60)
    return rng.geometric(1 / 7.0, 6000) - 1


@pytest.mark.parametrize("dt", [np.float64, np.float32])
@pytest.mark.parametrize("kind", ["ones", "long", "alternating", "geometric"])
@pytest.mark.parametrize("threads", [0, 1, 3, 50])
def test_windows(dt, kind, threads):
    rng = np.random.default_rng(threads + len(kind))
    ln = _lengths(kind, rng)
    m, n = len(ln), 4000
    Rst = np.concatenate([[0], np.cumsum(ln)]).astype(np.int32)
    Col = np.concatenate([np.sort(rng.choice(n, int(k), replace=False)) for k in ln]).astype(np.int32)
    Val = rng.uniform(-1, 1, len(Col)).astype(dt)
    A = R.spMtxCRS.from_host(m, n, Rst, Col, Val, dtype=TDT[dt])
    V = R.convert(R.spMtxVHCC(), A, R.convertParams(num_threads=threads))
    x, y0 = rng.uniform(-1, 1, n).astype(dt), rng.uniform(-1, 1, m).astype(dt)
    xd = torch.as_tensor(x).cuda()
    ref = O.crs_spmv_ld(O.crs(m, n, Rst, Col, Val), 1.5, x, -0.5, y0)
    lib = R.load()
    fn = lib.rvvla_vhcc_spmv_f64 if dt == np.float64 else lib.rvvla_vhcc_spmv_f32
    for unset in (False, True):
        d = V.desc()
        if unset:
            d.n_eor = d.n_rowarr = 0
        y = torch.as_tensor(y0).cuda()
        assert fn(C.byref(d), 1.5, xd.data_ptr(), -0.5, y.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
        assert O.normwise_relerr(y.cpu().numpy(), ref) < tol_for(dt)
