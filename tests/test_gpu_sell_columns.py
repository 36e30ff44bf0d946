"""GPU: SELL slices whose widths lie around the groups of 4, 8 and 16 columns
and around the width from which a CTA shares a slice, the last slice of fewer
than 32 rows among them; all precisions, against the long-double oracle on the
stored values (fp64 1e-12, fp32 1e-5, mixed 1e-6 normwise, as the format
tests)."""
import numpy as np
import pytest
import torch

import oracle as O
import rvvlasparse_b200 as R

pytestmark = pytest.mark.gpu
PREC = {"f64": (torch.float64, 1e-12), "f32": (torch.float32, 1e-5), "mixed": (torch.float32, 1e-6),
        "bf16": (torch.bfloat16, 1e-6)}
WIDTHS = [0, 1, 3, 4, 5, 7, 8, 9, 15, 16, 17, 63, 64, 65, 66, 127, 128, 129, 200, 511, 1025]


@pytest.mark.parametrize("prec", list(PREC))
@pytest.mark.parametrize("last", [1, 31, 32])
@pytest.mark.parametrize("wide_last", [False, True])
def test_widths(prec, last, wide_last):
    rng = np.random.default_rng(last)
    # one width per slice: rows up to the width, the first as wide as the slice
    order = list(rng.permutation(WIDTHS))
    order = order + [300 if wide_last else 6]
    ln = []
    for i, w in enumerate(order):
        rows = last if i + 1 == len(order) else 32
        ln += [w] + list(rng.integers(0, w + 1, rows - 1))
    ln = np.array(ln)
    m, n = len(ln), 3000
    Rst = np.concatenate([[0], np.cumsum(ln)]).astype(np.int32)
    Col = np.concatenate([np.sort(rng.choice(n, int(k), replace=False)) for k in ln]).astype(np.int32)
    Val = rng.uniform(-1, 1, len(Col))
    dt, tol = PREC[prec]
    A = R.spMtxCRS.from_host(m, n, Rst, Col, Val, dtype=torch.float64 if prec == "f64" else torch.float32)
    M = R.convert(R.spMtxSELL_C_Sigma(), A, R.convertParams(C=32, sigma=1))
    stored = A.Val.to(dt).double().cpu().numpy()
    if prec == "bf16":
        M = M.astype(torch.bfloat16)
    xt = torch.float64 if prec == "f64" else torch.float32
    x = torch.as_tensor(rng.uniform(-1, 1, n)).to(xt).cuda()
    y0 = torch.as_tensor(rng.uniform(-1, 1, m)).to(xt).cuda()
    mv = R.sparse_mv_mixed if prec in ("mixed", "bf16") else R.sparse_mv
    y = y0.clone()
    st = mv(R.SPARSE_OPERATION_NON_TRANSPOSE, 1.5, M, R.sparse_matrix_descr(), x, -0.5, y)
    assert st.code == 0, R.load().rvvla_last_error()
    ref = O.crs_spmv_ld(O.crs(m, n, Rst, Col, stored), 1.5, x.double().cpu().numpy(), -0.5, y0.double().cpu().numpy())
    assert O.normwise_relerr(y.double().cpu().numpy(), ref) < tol
