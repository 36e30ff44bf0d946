"""GPU: HCSR products of matrices with fewer rows than a block row (the default
block size included), whose accumulator is sized by the matrix; against the
long-double oracle (the format tests' tolerances)."""
import numpy as np
import pytest
import torch

import oracle as O
import rvvlasparse_b200 as R
from helpers import tol_for

pytestmark = pytest.mark.gpu
TDT = {np.float64: torch.float64, np.float32: torch.float32}


@pytest.mark.parametrize("dt", [np.float64, np.float32])
@pytest.mark.parametrize("m", [1, 17, 1009, 1999, 2000, 2001])
@pytest.mark.parametrize("mean", [3, 25])
def test_fewer_rows_than_a_block_row(dt, m, mean):
    rng = np.random.default_rng(m + mean)
    n = 2500
    ln = rng.poisson(mean, m) + (np.arange(m) == m // 2) * 500
    Rst = np.concatenate([[0], np.cumsum(ln)]).astype(np.int32)
    Col = np.concatenate([np.sort(rng.choice(n, int(k), replace=False)) for k in ln]).astype(np.int32)
    Val = rng.uniform(-1, 1, len(Col)).astype(dt)
    A = R.spMtxCRS.from_host(m, n, Rst, Col, Val, dtype=TDT[dt])
    H = R.convert(R.spMtxHCSR(), A, R.convertParams())
    x, y0 = rng.uniform(-1, 1, n).astype(dt), rng.uniform(-1, 1, m).astype(dt)
    y = torch.as_tensor(y0).cuda()
    st = R.sparse_mv(R.SPARSE_OPERATION_NON_TRANSPOSE, 1.5, H, R.sparse_matrix_descr(), torch.as_tensor(x).cuda(), -0.5, y)
    assert st.code == 0, R.load().rvvla_last_error()
    ref = O.crs_spmv_ld(O.crs(m, n, Rst, Col, Val), 1.5, x, -0.5, y0)
    assert O.normwise_relerr(y.cpu().numpy(), ref) < tol_for(dt)
