"""GPU: dvalues of a pattern with 2^31 - 1 nonzeros, the most that 32-bit row
pointers hold: every product equal to torch's, compared in pieces."""
import ctypes as C

import pytest
import torch

import rvvlasparse_b200 as R

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _give_back():
    """The memory that the test's tensors took, back from torch's cache: the
    library's builders of later tests allocate outside it."""
    yield
    torch.cuda.synchronize()
    torch.cuda.empty_cache()


def test_largest_pattern():
    nz, m, n = 2 ** 31 - 1, 300_007, 1_000_003
    if torch.cuda.mem_get_info()[0] < 40 << 30:
        pytest.skip("needs 40 GB of device memory")
    gen = torch.Generator(device="cuda").manual_seed(5)
    per = nz // m
    Rst = torch.arange(m + 1, device="cuda", dtype=torch.int64).mul_(per)
    Rst[-1] = nz  # the last row is longer than a chunk
    Rst = Rst.to(torch.int32)
    Col = torch.randint(0, n, (nz,), generator=gen, device="cuda", dtype=torch.int32)
    g, x = (torch.randn(k, generator=gen, device="cuda") for k in (m, n))
    dv = torch.full((nz,), float("nan"), device="cuda")
    A = R.spMtxCRS(m, n, nz, Rst, Col, dv)
    d = A.desc()
    assert R.load().rvvla_sddmm_values_f32(C.byref(d), g.data_ptr(), x.data_ptr(), dv.data_ptr(),
                                           torch.cuda.current_stream().cuda_stream) == 0
    step = 1 << 27
    for a in range(0, nz, step):
        b = min(nz, a + step)
        row = (torch.arange(a, b, device="cuda") // per).clamp_(max=m - 1)
        assert torch.equal(dv[a:b], g[row] * x[Col[a:b].long()])
