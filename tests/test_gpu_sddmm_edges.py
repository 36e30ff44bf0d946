"""GPU: dvalues[k] = g[row(k)] * x[Col[k]] where the row lookup can go wrong:
runs of empty rows, rows longer than a bitmap chunk, CTA ranges that start in
the middle of a bitmap word, fewer rows than a CTA.  One rounded product per
nonzero: bitwise equal to numpy's."""
import ctypes as C

import numpy as np
import pytest
import torch

import rvvlasparse_b200 as R

pytestmark = pytest.mark.gpu


def _lengths(kind, rng):
    if kind == "one":
        return np.array([5])
    if kind == "leading_empty":
        return np.concatenate([np.zeros(300, int), rng.poisson(3, 500), np.zeros(400, int), [1]])
    if kind == "long":  # 4096 is the chunk
        ln = rng.poisson(1, 700)
        ln[[0, 255, 256, 500]] = [4095, 4097, 9000, 4096]
        return ln
    return rng.geometric(1 / 19.0, 5001)


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("kind", ["one", "leading_empty", "long", "geometric"])
def test_rows(dt, kind):
    rng = np.random.default_rng(len(kind))
    ln = _lengths(kind, rng)
    m, n = len(ln), 10007
    Rst = np.concatenate([[0], np.cumsum(ln)]).astype(np.int32)
    Col = rng.integers(0, n, Rst[-1]).astype(np.int32)
    g, x = rng.standard_normal(m).astype(dt), rng.standard_normal(n).astype(dt)
    A = R.spMtxCRS.from_host(m, n, Rst, Col, np.zeros(len(Col)), dtype=torch.float64)
    dv = torch.full((len(Col),), float("nan"), dtype=torch.float64 if dt == np.float64 else torch.float32, device="cuda")
    gd, xd = torch.as_tensor(g).cuda(), torch.as_tensor(x).cuda()
    lib = R.load()
    fn = lib.rvvla_sddmm_values_f64 if dt == np.float64 else lib.rvvla_sddmm_values_f32
    d = A.desc()
    assert fn(C.byref(d), gd.data_ptr(), xd.data_ptr(), dv.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    ref = np.repeat(g, ln) * x[Col]
    assert np.array_equal(dv.cpu().numpy(), ref)
