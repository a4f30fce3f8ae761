"""The device prefix sum under the table builders, seen through the incidence of
a Map (its offsets are the scan of the targets' counts)."""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# a thread's four items, a chunk of 4096, and 1024 chunks, from which their totals
# are scanned on their own
@pytest.mark.parametrize("ntargets", [1, 3, 4, 5, 1023, 4095, 4096, 4097, 12289, 4096 * 1024 - 2,
                                      4096 * 1024, 4096 * 1024 + 7])
def test_offsets_equal_the_cumulative_counts(backend, ntargets):
    from pyop2_b200._lib import call
    from pyop2_b200 import b200
    rng = np.random.default_rng(ntargets)
    nelem = 60000
    m = rng.integers(0, ntargets, (nelem, 2)).astype(np.int32)
    m[-1] = ntargets - 1
    dm = b200._upload(m)
    h, ptr, lst, deg = C.c_uint64(), C.c_uint64(), C.c_uint64(), C.c_int32()
    call("op2b_incidence_build", dm.ptr, nelem, 2, ntargets, 0, C.byref(h))
    try:
        call("op2b_incidence_arrays", h.value, C.byref(ptr), C.byref(lst), C.byref(deg))
        got = np.empty(ntargets + 1, np.int32)
        call("op2b_memcpy_d2h", got.ctypes.data, ptr.value, got.nbytes, 0)
    finally:
        call("op2b_incidence_free", h.value)
    want = np.zeros(ntargets + 1, np.int32)
    want[1:] = np.cumsum(np.bincount(m.reshape(-1), minlength=ntargets))
    np.testing.assert_array_equal(got, want)
