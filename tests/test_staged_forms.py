"""Which staged form a loop takes and with how many elements a block, chosen on
the host (no GPU)."""

import numpy as np
import pytest

from pyop2_b200 import backends
from pyop2_b200 import configuration as cfg

KEYS = 16384     # (element, Map row) pairs of a block the partition builder takes


@pytest.fixture
def op2():
    from pyop2_b200 import _lib, op2
    if backends.get_backend() == "pyop2_b200.void":
        backends.set_backend("b200")
    _lib.load()
    cfg.configure(inc_mode="staged", staged_min_size=0, owner_mode="never")
    return op2


def loop_spec(op2, inc, read, dtype=np.float64):
    """INC through every row of a Map of arity ``inc``, READ through one of arity ``read``."""
    from pyop2_b200 import b200
    n = 500
    el, nd, nr = op2.Set(n, 1, "el"), op2.Set(400, 1, "nd"), op2.Set(700, 1, "nr")
    m = op2.Map(el, nd, inc, np.zeros((n, inc), np.int32), "m")
    r = op2.Map(el, nr, read, np.ones((n, read), np.int32), "r")
    y, x = op2.Dat(nd, np.zeros(400), dtype, "y"), op2.Dat(nr, np.zeros(700), dtype, "x")
    k = op2.Kernel("void k(void **y, void **x) { }", "k")
    return b200.loop_spec(b200.ParLoop(k, el, y(m, op2.INC), x(r, op2.READ)))["spec"]


@pytest.mark.parametrize("inc,read,dtype,elems", [
    (2, 3, np.float64, 256), (2, 64, np.float64, 256), (2, 65, np.float64, 128), (2, 81, np.float64, 128),
    (2, 128, np.float64, 128), (2, 129, np.float64, 0), (2, 400, np.float64, 0), (65, 2, np.float32, 128),
    (129, 2, np.int32, 0)])
@pytest.mark.parametrize("part", [0, 40, 300, 1024])
def test_blocks_of_maps_with_many_rows(op2, inc, read, dtype, elems, part):
    """The builder's bound holds whatever the arities: blocks of 256 or 128
    elements that keep it are summed, else the colour form takes blocks that do."""
    cfg.configure(partition_size=part)
    R = loop_spec(op2, inc, read, dtype).region
    assert R["part_size"] * max(inc, read) <= KEYS
    most = KEYS // max(inc, read)
    if part:
        assert R["part_size"] == min(part, most)
    else:
        assert bool(R.get("sums")) == (elems > 0)
        assert R["part_size"] == (elems or min(384, most))


@pytest.mark.parametrize("threads,sums", [(32, True), (96, True), (128, True), (256, True), (100, False),
                                          (1, False), (129, False)])
def test_cta_sizes_of_the_summing_form(op2, threads, sums):
    """Its sums are shared by whole warps: other CTA sizes keep the colour form."""
    cfg.configure(staged_block_size=threads)
    spec = loop_spec(op2, 2, 3)
    assert spec.mode == "staged" and spec.block_size == threads
    assert bool(spec.region.get("sums")) == sums
