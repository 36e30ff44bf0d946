"""GPU: CG and the fused product-and-dot at sizes around the vector width and
the block size, against dense solves.  A = tridiag(-1, 4, -1), condition number
below 3: a residual of rtol leaves an error of at most 3 rtol."""
import numpy as np
import pytest
import torch

import rvvlasparse_b200 as R
from rvvlasparse_b200 import solvers as S

pytestmark = pytest.mark.gpu
TDT = {np.float64: torch.float64, np.float32: torch.float32}


def _tridiag(n, dt):
    i = np.arange(n)
    row = np.concatenate([i, i[1:], i[:-1]])
    col = np.concatenate([i, i[1:] - 1, i[:-1] + 1])
    val = np.concatenate([np.full(n, 4.0), np.full(2 * (n - 1), -1.0)])
    o = np.lexsort((col, row))
    Rst = np.concatenate([[0], np.cumsum(np.bincount(row, minlength=n))]).astype(np.int32)
    return R.spMtxCRS.from_host(n, n, Rst, col[o].astype(np.int32), val[o], dtype=TDT[dt])


def _apply(x):
    y = 4.0 * x
    y[1:] -= x[:-1]
    y[:-1] -= x[1:]
    return y


@pytest.mark.parametrize("dt,rtol", [(np.float64, 1e-12), (np.float32, 1e-5)])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 7, 255, 256, 257, 1025, 70001])
def test_cg_and_dot(dt, rtol, n):
    rng = np.random.default_rng(n)
    A = _tridiag(n, dt)
    xt = rng.uniform(-1, 1, n)
    b = _apply(xt).astype(dt)
    eps = np.finfo(dt).eps
    outs = []
    for _ in range(2):
        x, it, res = S.cg(A, torch.as_tensor(b).cuda(), rtol=rtol, max_iter=100, check_every=5)
        assert it < 100 and res <= rtol
        outs.append(x.cpu().numpy())
    assert np.array_equal(outs[0], outs[1])
    err = np.linalg.norm(outs[0].astype(np.float64) - xt) / np.linalg.norm(xt)
    assert err <= 3 * rtol + 30 * eps  # 30 eps: the recurrence's own rounding and b's
    v = rng.uniform(-1, 1, n).astype(dt)
    y, d = S.spmv_dot(A, torch.as_tensor(v).cuda())
    v64 = v.astype(np.float64)
    assert np.allclose(y.cpu().numpy(), _apply(v64), rtol=0, atol=12 * eps)
    # each of at most n terms below 6 in size, at most 64 added in a row in type dt
    assert abs(float(d.item()) - v64 @ _apply(v64)) <= 64 * eps * 6 * max(n, 2)
