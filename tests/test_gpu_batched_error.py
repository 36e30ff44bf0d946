"""GPU: the rounding error of CSR batches with several right-hand sides, on
long rows among short ones (few lanes per row on average).

The bound is that of eight running sums of n / 8 products, added as a tree.
A rounding of a value v errs by at most u |v| (u half a unit in the last
place), uniformly, 0.41 u |v| in the root mean square over the mantissas.  With
terms of one sign and size, a sum of N of them passes i / N of its end at step
i, so its N roundings make 0.41 u sqrt(N / 3) of it, eight such sums together
sqrt(8) / 8 of that relative to the row, and the tree's three levels
0.41 u sqrt(7 / 4).  Twice the root mean square of both is allowed, as rows and terms
differ."""
import numpy as np
import pytest
import torch

import rvvlasparse_b200 as R
from rvvlasparse_b200 import batched as B

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("k", [4, 8, 32])
@pytest.mark.parametrize("n", [31, 64, 1000, 2000, 3000])  # up to more than a tile stages
def test_long_rows(dt, k, n):
    rng = np.random.default_rng(n + k)
    m, rows = 40000, 200
    ln = np.full(m, 2)
    long = np.sort(rng.choice(m, rows, replace=False))
    ln[long] = n
    Rst = np.concatenate([[0], np.cumsum(ln)]).astype(np.int32)
    Col = rng.integers(0, m, Rst[-1]).astype(np.int32)
    Val = rng.uniform(0.5, 1, Rst[-1]).astype(dt)
    A = R.spMtxCRS.from_host(m, m, Rst, Col, Val, dtype=torch.from_numpy(Val).dtype)
    batch = B.SpMVBatch([A], k=k, mode=np.zeros(1), param=np.full(1, 4))
    X = rng.uniform(0.5, 1, (m, k)).astype(dt)
    Y = torch.zeros(m * k, dtype=A.dtype, device="cuda")
    assert batch.spmv(1.0, torch.as_tensor(X).cuda().reshape(-1), 0.0, Y) == 0
    Y = Y.cpu().numpy().reshape(m, k)
    rel = []
    for r in long:
        s = slice(Rst[r], Rst[r + 1])
        ref = (Val[s, None].astype(np.longdouble) * X[Col[s]].astype(np.longdouble)).sum(0)
        rel.append((Y[r] - ref) / ref)
    u = np.finfo(dt).eps / 2
    bound = 0.41 * u * np.sqrt(n / 8 / 3 / 8 + 7 / 4)
    assert np.sqrt(np.mean(np.square(np.array(rel, np.float64)))) < 2 * bound
