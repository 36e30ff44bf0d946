"""GPU: products whose kernels start while the ones before them drain, each
product reading the vector that the one before wrote, without a host
synchronisation in between: bitwise equal to the same products with one after
every call."""
import numpy as np
import pytest
import torch

import rvvlasparse_b200 as R

pytestmark = pytest.mark.gpu
FORMATS = {"crs": None, "csr5": R.spMtxCSR5, "lav": R.spMtxLAV, "vhcc": R.spMtxVHCC, "cvr": R.spMtxCVR,
           "vnec": R.spMtxVNEC, "hcsr": R.spMtxHCSR, "sell": R.spMtxSELL_C_Sigma}


def _matrix(n, empty, rng):
    ln = rng.geometric(0.1, n)
    ln[rng.integers(0, n, 3)] = 900
    if empty:
        ln[rng.random(n) < 0.3] = 0
    Rst = np.concatenate([[0], np.cumsum(ln)]).astype(np.int32)
    Col = np.concatenate([np.sort(rng.choice(n, int(k), replace=False)) for k in ln]).astype(np.int32)
    return n, n, Rst, Col, rng.uniform(-0.3, 0.3, len(Col))


@pytest.mark.parametrize("fmt", list(FORMATS))
@pytest.mark.parametrize("empty", [False, True])
@pytest.mark.parametrize("n", [1009, 20011])
def test_dependent_products(fmt, empty, n):
    rng = np.random.default_rng(n)
    A = R.spMtxCRS.from_host(*_matrix(n, empty, rng), dtype=torch.float64)
    M = A if FORMATS[fmt] is None else R.convert(FORMATS[fmt](), A, R.convertParams())
    x0 = torch.as_tensor(rng.uniform(-1, 1, n)).cuda()

    def run(sync):
        v = [x0.clone(), torch.full_like(x0, 0.5)]
        for it in range(24):
            st = R.sparse_mv(R.SPARSE_OPERATION_NON_TRANSPOSE, 1.0, M, R.sparse_matrix_descr(), v[it % 2], 0.25,
                             v[1 - it % 2])
            assert st.code == 0, R.load().rvvla_last_error()
            if sync:
                torch.cuda.synchronize()
        return v

    ref = run(True)
    for _ in range(5):
        out = run(False)
        assert torch.equal(out[0], ref[0]) and torch.equal(out[1], ref[1])
    assert torch.isfinite(ref[0]).all()
