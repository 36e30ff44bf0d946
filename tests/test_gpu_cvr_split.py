"""GPU: CVR ranges shared by several warps, where the shares can go wrong:
ranges of fewer vectors than warps, of one vector more or less than the
shares' multiples, rows that run through several shares, lanes that drain
early, empty rows; against the long-double oracle (the format tests'
tolerances) and bitwise equal when repeated."""
import numpy as np
import pytest
import torch

import oracle as O
import rvvlasparse_b200 as R
from helpers import tol_for

pytestmark = pytest.mark.gpu
TDT = {np.float64: torch.float64, np.float32: torch.float32}


def _rows(kind, rng):
    if kind == "few":  # 32 rows or less: as many vectors as the longest row
        return rng.integers(0, 9, 29)
    if kind == "even":
        return np.full(32 * 17, 16)
    if kind == "long":  # one row runs through every share of its range
        ln = rng.poisson(3, 900)
        ln[[5, 400, 899]] = [4000, 2500, 1777]
        return ln
    return np.where(rng.random(3000) < 0.3, 0, rng.geometric(0.08, 3000))


@pytest.mark.parametrize("dt", [np.float64, np.float32])
@pytest.mark.parametrize("kind", ["few", "even", "long", "mixed"])
@pytest.mark.parametrize("threads", [1, 2, 7, 40])
def test_shares(dt, kind, threads):
    rng = np.random.default_rng(len(kind) + threads)
    ln = _rows(kind, rng)
    m, n = len(ln), 5000
    Rst = np.concatenate([[0], np.cumsum(ln)]).astype(np.int32)
    Col = np.concatenate([np.sort(rng.choice(n, int(k), replace=False)) for k in ln]).astype(np.int32)
    Val = rng.uniform(-1, 1, len(Col)).astype(dt)
    A = R.spMtxCRS.from_host(m, n, Rst, Col, Val, dtype=TDT[dt])
    V = R.convert(R.spMtxCVR(), A, R.convertParams(Nthreads=threads))
    x, y0 = rng.uniform(-1, 1, n).astype(dt), rng.uniform(-1, 1, m).astype(dt)
    outs = []
    for _ in range(3):
        y = torch.as_tensor(y0).cuda()
        st = R.sparse_mv(R.SPARSE_OPERATION_NON_TRANSPOSE, 1.5, V, R.sparse_matrix_descr(),
                         torch.as_tensor(x).cuda(), -0.5, y)
        assert st.code == 0, R.load().rvvla_last_error()
        outs.append(y.cpu().numpy())
    ref = O.crs_spmv_ld(O.crs(m, n, Rst, Col, Val), 1.5, x, -0.5, y0)
    assert O.normwise_relerr(outs[0], ref) < tol_for(dt)
    assert np.array_equal(outs[0], outs[1]) and np.array_equal(outs[0], outs[2])
