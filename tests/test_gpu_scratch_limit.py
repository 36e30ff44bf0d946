"""GPU: a product when little device memory is left.  HCSR with block rows too
tall for shared memory wants a slice of accumulators per part of a block row
and does with one slice where that does not fit.  The memory is taken by one
tensor that leaves a few GB."""
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


def _mv(A, x, y):
    st = R.sparse_mv(R.SPARSE_OPERATION_NON_TRANSPOSE, 1.0, A, R.sparse_matrix_descr(), x, 0.0, y)
    return st.code


def _leave(gb):
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    return torch.empty(max(0, free - int(gb * 2 ** 30)), dtype=torch.uint8, device="cuda")


def test_tall_block_rows_fall_back_to_one_part():
    m, n, nz = 2 ** 27, 1000, 200_000  # 1 GB of accumulators, 8 GB in eight parts
    gen = torch.Generator(device="cuda").manual_seed(2)
    row = torch.sort(torch.randint(0, m, (nz,), generator=gen, device="cuda")).values
    Rst = torch.zeros(m + 1, dtype=torch.int32, device="cuda")
    Rst[1:] = torch.cumsum(torch.bincount(row, minlength=m), 0)
    Col = torch.randint(0, n, (nz,), generator=gen, device="cuda", dtype=torch.int32)
    Val = torch.randint(-8, 9, (nz,), generator=gen, device="cuda").double()  # whole numbers: sums are exact
    x = torch.randint(-8, 9, (n,), generator=gen, device="cuda").double()
    H = R.convert(R.spMtxHCSR(), R.spMtxCRS(m, n, nz, Rst, Col, Val), R.convertParams(R=2 ** 24, C=1000, p=1e9))
    ref = torch.zeros(m, dtype=torch.float64, device="cuda").index_add_(0, row, Val * x[Col.long()])
    y = torch.full((m,), 7.0, dtype=torch.float64, device="cuda")
    assert _mv(H, x, y) == 0 and torch.equal(y, ref)
    y.fill_(7.0)
    hold = _leave(3)
    code = _mv(H, x, y)
    msg = R.load().rvvla_last_error()
    torch.cuda.synchronize()
    del hold
    assert code == 0, msg
    assert torch.equal(y, ref)
