"""The staged forms at the edges of their ranges against the sequential oracle."""

import numpy as np
import pytest

from oracle import seq
from pyop2_b200 import configuration as cfg

pytestmark = pytest.mark.gpu


@pytest.fixture
def op2(backend):
    from pyop2_b200 import op2
    cfg.configure(inc_mode="staged", staged_min_size=0)
    return op2


def run(api, n, inc, read, cdim=1, rdim=1, nx=None):
    """y += sums of rows of x, through Maps of arity ``inc`` and ``read``; whole
    numbers, exact in any order."""
    rng = np.random.default_rng(n + inc + read)
    ny, nx = n // 3 + inc, nx or n // 2 + read
    el, nd, nr = api.Set(n, 1, "el"), api.Set(ny, cdim, "nd"), api.Set(nx, rdim, "nr")
    m = api.Map(el, nd, inc, rng.integers(0, ny, (n, inc)).astype(np.int32), "m")
    r = api.Map(el, nr, read, rng.integers(0, nx, (n, read)).astype(np.int32), "r")
    y = api.Dat(nd, rng.integers(1, 9, (ny, cdim)).astype(np.float64), np.float64, "y")
    x = api.Dat(nr, rng.integers(1, 9, (nx, rdim)).astype(np.float64), np.float64, "x")
    k = api.Kernel("void wide(double **y, double **x) { double s = 0; for (int i = 0; i < %d; ++i) "
                   "for (int j = 0; j < %d; ++j) s += (1 + i %% 3) * x[i][j]; "
                   "for (int i = 0; i < %d; ++i) for (int j = 0; j < %d; ++j) y[i][j] += (1 + i + j) * s; }"
                   % (read, rdim, inc, cdim), "wide")
    api.par_loop(k, el, y(m, api.INC), x(r, api.READ))
    return np.array(y.data)


def bound():
    from pyop2_b200 import b200
    return [b for b in b200.ParLoop._bound_cache.values() if b.spec.kernel_name == "wide"][-1]


@pytest.mark.parametrize("inc,read,sums", [(2, 64, True), (2, 65, True), (2, 81, True), (3, 129, False)])
def test_maps_with_many_rows(op2, inc, read, sums):
    got = run(op2, 2003, inc, read)
    assert bound().spec.mode == "staged" and bool(bound().spec.region.get("sums")) == sums
    np.testing.assert_array_equal(got, run(seq, 2003, inc, read))


@pytest.mark.parametrize("threads", [32, 96, 100, 128, 130])
@pytest.mark.parametrize("cdim", [1, 3, 4])
def test_cta_sizes(op2, threads, cdim):
    """CTAs that are not whole warps run the colour form (the summing form's
    shuffles name every lane)."""
    cfg.configure(staged_block_size=threads)
    got = run(op2, 1501, 2, 3, cdim)
    assert bound().spec.mode == "staged"
    assert bool(bound().spec.region.get("sums")) == (threads % 32 == 0)
    np.testing.assert_array_equal(got, run(seq, 1501, 2, 3, cdim))


@pytest.mark.parametrize("read,rdim,mode", [(100, 1, "staged"), (120, 1, "staged"), (120, 2, "atomic")])
def test_rows_that_fill_the_shared_memory(op2, read, rdim, mode):
    """Nearly every element of a block names rows of its own.  What the summing
    form, with its packets, has no room for still runs colour by colour; the
    atomic form takes what neither can."""
    got = run(op2, 2003, 2, read, 1, rdim, nx=400000)
    assert bound().spec.mode == mode and not (bound().spec.region or {}).get("sums")
    np.testing.assert_array_equal(got, run(seq, 2003, 2, read, 1, rdim, nx=400000))
