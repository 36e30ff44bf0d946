"""GPU: the batched kernels where their splits can go wrong: matrices smaller
than a slice or a tile, empty rows, more and fewer matrices than SMs, rows of
the widths around the steps of four and eight columns, and X / Y that are not
16-byte aligned; every block of Y against the long-double oracle.  The
tolerances are the format tests' (fp64 1e-12, fp32 1e-5 normwise)."""
import numpy as np
import pytest
import torch

import oracle as O
import rvvlasparse_b200 as R
from helpers import tol_for
from rvvlasparse_b200 import batched as B

pytestmark = pytest.mark.gpu
TDT = {np.float64: torch.float64, np.float32: torch.float32}


def _matrix(rng, m, n, widths):
    ln = np.minimum(rng.choice(widths, m), n)
    Rst = np.zeros(m + 1, np.int32)
    Rst[1:] = np.cumsum(ln)
    Col = np.concatenate([np.sort(rng.choice(n, k, replace=False)) for k in ln] or [np.zeros(0)]).astype(np.int32)
    return m, n, Rst, Col, rng.uniform(-1, 1, len(Col))


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("k", [1, 4, 8, 32])
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("shift", [0, 1])
def test_edges(dt, k, mode, shift):
    rng = np.random.default_rng(17 + k)
    sizes = [(1, 1), (1, 300), (31, 7), (32, 64), (33, 40), (257, 100), (700, 33)] + [(40, 50)] * 180
    host = [_matrix(rng, m, n, [0, 1, 3, 4, 5, 7, 8, 9, 15, 16, 17, 33] if i % 3 else [0, 40, 64, 300])
            for i, (m, n) in enumerate(sizes)]
    for part in (host, host[5:6]):
        mats = [R.spMtxCRS.from_host(m, n, r, c, v.astype(dt), dtype=TDT[dt]) for m, n, r, c, v in part]
        batch = B.SpMVBatch(mats, k=k, mode=np.full(len(part), mode), param=np.full(len(part), 4 if mode == 0 else 32))
        X = rng.uniform(-1, 1, batch.x_len + shift).astype(dt)
        Y0 = rng.uniform(-1, 1, batch.y_len + shift).astype(dt)
        Xd, Yd = torch.as_tensor(X).cuda()[shift:], torch.as_tensor(Y0).cuda()
        assert batch.spmv(1.5, Xd, -0.25, Yd[shift:]) == 0, R.load().rvvla_last_error()
        Y = Yd.cpu().numpy()
        assert shift == 0 or Y[0] == Y0[0]
        for i, (m, n, r, c, v) in enumerate(part):
            A = O.crs(m, n, r, c, v.astype(dt))
            xs = X[shift:][batch.x_off[i]:batch.x_off[i + 1]].reshape(n, k)
            ys = Y[shift:][batch.y_off[i]:batch.y_off[i + 1]].reshape(m, k)
            y0 = Y0[shift:][batch.y_off[i]:batch.y_off[i + 1]].reshape(m, k)
            for q in range(k):
                ref = O.crs_spmv_ld(A, 1.5, np.ascontiguousarray(xs[:, q]), -0.25, np.ascontiguousarray(y0[:, q]))
                assert O.normwise_relerr(ys[:, q], ref) < tol_for(dt), (i, q)
