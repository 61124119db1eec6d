"""CPU tests of the kernel reports of the C ABI: null objects and unprepared handles are refused."""
import ctypes

import pytest

import benchmark_spmv_using_csr_gb300 as sp
from benchmark_spmv_using_csr_gb300._lib import lib


def test_kernel_reports_reject_null_and_unprepared_objects():
    n = ctypes.byref(ctypes.c_int())
    assert lib().bhsp_plan_kernel(None, n, n) == sp.BHSPARSE_INVALID_ARGUMENT
    assert lib().bhsp_get_kernel(None, n, n) == sp.BHSPARSE_INVALID_ARGUMENT
    assert lib().bhsp_batch_lists(None, n, n, n, n) == sp.BHSPARSE_INVALID_ARGUMENT
    h = sp.BhsparseSpmvCuda(sp.VALUE_F64)
    with pytest.raises(sp.SpmvError):
        h.kernel()
    h.close()
