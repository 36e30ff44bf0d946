"""GPU: SELL batches whose work is shared in segments (large matrices, k = 1)
and in parts (small matrices, several right-hand sides), next to CSR matrices
in the same plan, against torch in fp64.  A row has at most 40 nonzeros, so a
sum in fp32 is off by at most 42 units of 2^-24 of the sum of its terms'
magnitudes."""
import numpy as np
import pytest
import torch

import rvvlasparse_b200 as R
from rvvlasparse_b200 import batched as B

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 4, 8, 32])
@pytest.mark.parametrize("rows,count,segments", [(300_000, 1, True), (70_000, 12, True), (32, 700, False), (100, 331, False),
                                                 (1023, 40, False)])
def test_shares(rows, count, segments, k):
    gen = torch.Generator(device="cuda").manual_seed(rows + k)
    mats, parts = [], []
    for i in range(count + 2):
        m = max(1, rows - 7 * (i % 3))
        ln = torch.randint(0, 41, (m,), generator=gen, device="cuda")
        Rst = torch.zeros(m + 1, dtype=torch.int64, device="cuda")
        Rst[1:] = torch.cumsum(ln, 0)
        row = torch.repeat_interleave(torch.arange(m, device="cuda"), ln)
        col = torch.randint(0, m, (row.numel(),), generator=gen, device="cuda")
        val = torch.rand(row.numel(), generator=gen, device="cuda") * 2 - 1
        mats.append(R.spMtxCRS(m, m, row.numel(), Rst.to(torch.int32), col.to(torch.int32), val))
        parts.append((m, row, col, val))
    mode = np.ones(count + 2, np.int32)
    mode[[0, -1]] = 0 if count > 1 else 1
    batch = B.SpMVBatch(mats, k=k, mode=mode, param=np.where(mode == 0, 4, 256))
    h = batch._plan.h
    assert (h.sell_segs > 0) == (segments and k == 1) and (h.sell_parts > 0) != (h.sell_segs > 0)
    X = torch.rand(batch.x_len, generator=gen, device="cuda") * 2 - 1
    Y0 = torch.rand(batch.y_len, generator=gen, device="cuda") * 2 - 1
    Y = Y0.clone()
    assert batch.spmv(1.5, X, -0.25, Y) == 0, R.load().rvvla_last_error()
    for i, (m, row, col, val) in enumerate(parts):
        x = X[batch.x_off[i]:batch.x_off[i + 1]].view(m, k).double()
        y0 = Y0[batch.y_off[i]:batch.y_off[i + 1]].view(m, k).double()
        t = val.double()[:, None] * x[col]
        ref = (-0.25 * y0).index_add_(0, row, 1.5 * t)
        size = (0.25 * y0.abs()).index_add_(0, row, 1.5 * t.abs())
        err = (Y[batch.y_off[i]:batch.y_off[i + 1]].view(m, k).double() - ref).abs()
        assert (err <= 44 * 2.0 ** -24 * size).all(), i
