"""GPU: dvalues of patterns whose last rows are empty, a whole CTA's 256 and
more, with every remainder of the nonzeros modulo 32: bitwise equal to numpy's
product, nothing written past the end.  The columns are followed by one valid
word, which no product may use."""
import ctypes as C

import numpy as np
import pytest
import torch

import rvvlasparse_b200 as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("tail", [256, 300, 512, 700])
def test_empty_tail(dt, tail):
    rng = np.random.default_rng(tail)
    td = torch.float64 if dt == np.float64 else torch.float32
    fn = R.load().rvvla_sddmm_values_f64 if dt == np.float64 else R.load().rvvla_sddmm_values_f32
    n = 1009
    for rows in (256, 300):
        for nz in range(96, 128):
            ln = np.bincount(rng.integers(0, rows, nz), minlength=rows + tail)
            m = len(ln)
            Rst = torch.as_tensor(np.concatenate([[0], np.cumsum(ln)]).astype(np.int32)).cuda()
            col = rng.integers(0, n, nz + 1).astype(np.int32)
            g, x = rng.standard_normal(m).astype(dt), rng.standard_normal(n).astype(dt)
            A = R.spMtxCRS(m, n, nz, Rst, torch.as_tensor(col).cuda()[:nz], torch.zeros(nz, dtype=td, device="cuda"))
            dv = torch.full((nz + 64,), -7.0, dtype=td, device="cuda")
            gd, xd = torch.as_tensor(g).cuda(), torch.as_tensor(x).cuda()
            d = A.desc()
            assert fn(C.byref(d), gd.data_ptr(), xd.data_ptr(), dv.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
            out = dv.cpu().numpy()
            assert np.array_equal(out[:nz], np.repeat(g, ln) * x[col[:nz]])
            assert (out[nz:] == -7).all()
