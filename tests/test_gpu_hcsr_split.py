"""GPU: HCSR products whose block rows are shared by a cluster of CTAs (1 to 8
of them, powers of two and not), and COO streams around the edges of a warp's
turn (64 nonzeros), a round (512) and a CTA's share; every form, against the
long-double oracle (the format tests' tolerances), twice bitwise alike."""
import numpy as np
import pytest
import torch

import oracle as O
import rvvlasparse_b200 as R
from helpers import tol_for

pytestmark = pytest.mark.gpu


def _product(m, n, ln, dt, mixed, **prm):
    rng = np.random.default_rng(m + n)
    Rst = np.concatenate([[0], np.cumsum(ln)]).astype(np.int32)
    Col = np.concatenate([np.sort(rng.choice(n, int(k), replace=False)) for k in ln] + [np.zeros(0, int)]).astype(np.int32)
    Val = rng.uniform(-1, 1, len(Col)).astype(dt)
    H = R.convert(R.spMtxHCSR(), R.spMtxCRS.from_host(m, n, Rst, Col, Val, dtype=torch.from_numpy(Val).dtype),
                  R.convertParams(prm))
    x, y0 = rng.uniform(-1, 1, n).astype(dt), rng.uniform(-1, 1, m).astype(dt)
    fn = R.sparse_mv_mixed if mixed else R.sparse_mv
    out = []
    for _ in range(2):
        y = torch.as_tensor(y0).cuda()
        st = fn(R.SPARSE_OPERATION_NON_TRANSPOSE, 1.5, H, R.sparse_matrix_descr(), torch.as_tensor(x).cuda(), -0.5, y)
        assert st.code == 0, R.load().rvvla_last_error()
        out.append(y.cpu().numpy())
    ref = O.crs_spmv_ld(O.crs(m, n, Rst, Col, Val), 1.5, x, -0.5, y0)
    assert np.array_equal(out[0], out[1])
    assert O.normwise_relerr(out[0], ref) < (1e-6 if mixed else tol_for(dt))


@pytest.mark.parametrize("dt,mixed", [(np.float64, False), (np.float32, False), (np.float32, True)])
@pytest.mark.parametrize("p", [0.01, 2.0, 1e9])  # all CSR blocks, both kinds, all COO
@pytest.mark.parametrize("brows", [1, 74, 85, 119, 148, 198, 296, 297])  # 8, 7, 6, 4, 3, 2, 1, 1 parts
def test_parts_of_a_block_row(brows, p, dt, mixed):
    m, n = brows * 97 - 5, 5003
    rng = np.random.default_rng(brows)
    _product(m, n, rng.integers(0, 400, m), dt, mixed, R=97, C=500, p=p)


@pytest.mark.parametrize("nz", [1, 31, 32, 63, 64, 65, 511, 512, 513, 1025, 4096, 4127, 16384, 16421])
def test_coo_stream_edges(nz):
    """One block row, all COO (blocks of at most 1023 nonzeros), of nz
    nonzeros in all; from 4096 on two or more parts."""
    m, n = 50, 30011
    ln = np.full(m, nz // m)
    ln[: nz % m] += 1
    _product(m, n, ln, np.float64, False, R=64, C=700, p=1e9)


@pytest.mark.parametrize("rows", [1, 2, 3])
def test_rows_that_repeat_across_lanes(rows):
    """Narrow blocks (one or two nonzeros of each row): every lane of a
    sub-step holds one of a few rows."""
    _product(rows, 4000, np.full(rows, 3000), np.float64, False, R=8, C=2, p=1e9)


@pytest.mark.parametrize("brows", [1, 2, 3])
@pytest.mark.parametrize("dt,mixed", [(np.float64, False), (np.float32, True)])
def test_parts_of_a_tall_block_row(brows, dt, mixed):
    """Accumulators too tall for shared memory: one scratch slice per part."""
    m = brows * 60000 - 7
    _product(m, 3001, np.random.default_rng(m).integers(0, 6, m), dt, mixed, R=60000, C=700, p=2.0)
