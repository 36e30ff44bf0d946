"""GPU: VHCC products at the edges of the thread counts that take 40 warps per
SM in fp64 (more than 32 per SM, at most 40), and of a CTA of four warps;
against the long-double oracle (the format tests' tolerances)."""
import numpy as np
import pytest
import torch

import oracle as O
import rvvlasparse_b200 as R
from helpers import tol_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [np.float64, np.float32])
@pytest.mark.parametrize("per_sm,more", [(0, 1), (0, 4), (0, 5), (32, 0), (32, 1), (40, 0), (40, 1)])
def test_thread_counts(dt, per_sm, more):
    threads = per_sm * torch.cuda.get_device_properties(0).multi_processor_count + more
    rng = np.random.default_rng(threads)
    m, n = 20011, 3000
    ln = rng.integers(0, 30, m)
    Rst = np.concatenate([[0], np.cumsum(ln)]).astype(np.int32)
    Col = rng.integers(0, n, int(Rst[-1])).astype(np.int32)
    Val = rng.uniform(-1, 1, len(Col)).astype(dt)
    A = R.spMtxCRS.from_host(m, n, Rst, Col, Val, dtype=torch.from_numpy(Val).dtype)
    V = R.convert(R.spMtxVHCC(), A, R.convertParams(num_threads=threads))
    x, y0 = rng.uniform(-1, 1, n).astype(dt), rng.uniform(-1, 1, m).astype(dt)
    y = torch.as_tensor(y0).cuda()
    st = R.sparse_mv(R.SPARSE_OPERATION_NON_TRANSPOSE, 1.5, V, R.sparse_matrix_descr(), torch.as_tensor(x).cuda(), -0.5, y)
    assert st.code == 0, R.load().rvvla_last_error()
    ref = O.crs_spmv_ld(O.crs(m, n, Rst, Col, Val), 1.5, x, -0.5, y0)
    assert O.normwise_relerr(y.cpu().numpy(), ref) < tol_for(dt)
