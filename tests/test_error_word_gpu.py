"""A handle's error word is a word of host memory where the GPU reads and writes that coherently:
a bit set there is reported once, by the next check, and cleared."""
import ctypes

import numpy as np
import pytest

import benchmark_spmv_using_csr_gb300 as sp
from benchmark_spmv_using_csr_gb300 import gen
from benchmark_spmv_using_csr_gb300._lib import lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bit", [1, 8])
def test_a_set_bit_is_reported_once_and_cleared(cuda_ok, bit):
    a = gen.stencil2d(40, 30)
    h = sp.BhsparseSpmvCuda(sp.VALUE_F64)
    y = np.zeros(a.m)
    assert h.prepare_mem(a.m, a.n, a.nnz, a.row_ptr, a.col, a.val, np.ones(a.n), y) == 0
    word_of = lib().bhsp_debug_host_error_word
    word_of.restype, word_of.argtypes = ctypes.c_void_p, [ctypes.c_void_p]
    address = word_of(h._h)
    if not address:
        h.close()
        pytest.skip("the error word is in device memory here")
    word = ctypes.c_uint32.from_address(address)
    assert h.run_benchmark() == 0 and word.value == 0
    word.value |= bit
    assert h.run_benchmark() == sp.BHSPARSE_DEVICE_CHECK_FAILED
    assert f"0x{bit:x}" in h.last_error and word.value == 0
    assert h.check() == 0 and h.run_benchmark() == 0 and h.get_y() == 0
    want = np.bincount(np.repeat(np.arange(a.m), np.diff(a.row_ptr)), a.val, a.m)
    np.testing.assert_allclose(y, want, rtol=0, atol=1e-12)
    h.close()
