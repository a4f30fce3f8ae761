"""Mat assembly stubs of every form compile with every kind of READ argument (NVRTC
needs no GPU)."""

import ctypes as C

import numpy as np
import pytest

from pyop2_b200 import backends, codegen
from pyop2_b200 import configuration as cfg


@pytest.fixture
def op2():
    from pyop2_b200 import _lib, op2
    if backends.get_backend() == "pyop2_b200.void":
        backends.set_backend("b200")
    _lib.load()
    cfg.configure(inc_mode="staged", owner_mode="never", staged_min_size=0)
    return op2


def compiles(spec):
    from pyop2_b200 import _lib
    src, _, _ = codegen.generate(spec)
    opts = codegen.nvrtc_options(extra=())
    arr = (C.c_char_p * len(opts))(*[o.encode() for o in opts])
    out, n, log = C.c_void_p(), C.c_uint64(), C.create_string_buffer(1 << 16)
    rc = _lib._lib.op2b_nvrtc_compile(src.encode(), b"stub.cu", arr, len(opts), C.byref(out), C.byref(n), log,
                                      len(log))
    assert rc == 0, _lib.last_error() + "\n" + src
    _lib._lib.op2b_cubin_free(out)


@pytest.mark.parametrize("arity", [2, 6, 8])
@pytest.mark.parametrize("inc_mode", ["staged", "lma", "color"])
def test_globals_read_by_an_assembly(op2, arity, inc_mode):
    """Local blocks of one thread and, from 6 x 6 on, split across warps."""
    from pyop2_b200 import b200
    cfg.configure(inc_mode=inc_mode)
    el, nd = op2.Set(20, 1, "el"), op2.Set(15, 1, "nd")
    m = op2.Map(el, nd, arity, np.zeros((20, arity), np.int32), "m")
    mat = op2.Mat(op2.Sparsity((m, m), "s"), np.float64, "mat")
    g, h = op2.Global(1, 1.0, np.float64, "g"), op2.Global(2, [1, 2], np.int32, "h")
    w = op2.Dat(el, np.zeros(20), np.float64, "w")
    k = op2.Kernel("void k(double A[1][1], double *g, double *w, int *h, int i, int j) "
                   "{ A[0][0] += g[0] * w[0] * h[1] + i + j; }", "k")
    loop = b200.ParLoop(k, el(arity, arity), mat((m[op2.i[0]], m[op2.i[1]]), op2.INC), g(op2.READ),
                        w(op2.IdentityMap, op2.READ), h(op2.READ))
    spec = b200.loop_spec(loop)["spec"]
    assert bool(spec.itspace_split) == (inc_mode == "staged" and arity >= 6)
    compiles(spec)
