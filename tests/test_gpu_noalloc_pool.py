"""GPU: the allocation-free fp64 CSR5 entry takes nothing from the library's
own pool of temporary buffers either (the device's default pool is watched in
test_zz_no_alloc).  That pool's memory stays mapped after a call until it is
trimmed, so a call that used it leaves less free memory behind; an fp32
product, which does use it, shows that the measure sees it."""
import ctypes as C

import pytest
import torch

import rvvlasparse_b200 as R
from rvvlasparse_b200 import workloads as W

pytestmark = pytest.mark.gpu


def test_library_pool_untouched():
    m, n, Rst, Col, Val = W.powerlaw(1 << 16, seed=5)
    lib = R.load()
    st = torch.cuda.current_stream().cuda_stream

    def call(dtype, name):
        A = R.spMtxCSR5()
        R.convert(A, R.spMtxCRS.from_host(m, n, Rst, Col, Val, dtype=dtype), R.convertParams(omega=32, sigma=16))
        x = torch.ones(n, dtype=dtype, device="cuda")
        y = torch.zeros(m, dtype=dtype, device="cuda")
        d, fn = A.desc(), getattr(lib, name)

        def run():
            assert fn(C.byref(d), 1.0, x.data_ptr(), 0.0, y.data_ptr(), st) == 0, lib.rvvla_last_error()
            torch.cuda.synchronize()

        run()  # modules loaded, nothing left to set up
        assert lib.rvvla_trim_scratch() == 0
        before = torch.cuda.mem_get_info()[0]
        run()
        return before - torch.cuda.mem_get_info()[0]

    assert call(torch.float32, "rvvla_csr5_spmv_f32") > 0
    assert call(torch.float64, "rvvla_csr5_spmv_f64_noalloc") == 0
