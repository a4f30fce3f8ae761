"""The summing staged form against the sequential oracle and the colour form."""

import numpy as np
import pytest

from oracle import seq
from pyop2_b200 import configuration as cfg

pytestmark = pytest.mark.gpu


@pytest.fixture
def op2(backend):
    from pyop2_b200 import op2
    return op2


CT = {np.float64: "double", np.float32: "float", np.int32: "int"}


def run(api, n, arity, cdim, dtype, conn, rows, vec=False):
    nn = int(conn.max()) + 1
    el, nd = api.Set(n, 1, "el"), api.Set(nn, cdim, "nd")
    m = api.Map(el, nd, arity, conn, "m")
    rng = np.random.default_rng(n + cdim)
    x = api.Dat(nd, rng.integers(1, 9, (nn, cdim)).astype(dtype), dtype, "x")
    y = api.Dat(nd, rng.integers(1, 9, (nn, cdim)).astype(dtype), dtype, "y")
    w = api.Dat(el, rng.integers(1, 5, n).astype(dtype), dtype, "w")
    g = api.Global(1, 0, dtype, "g")
    t = CT[dtype]
    if vec:
        code = "void k(%s **y, %s **x, %s *w, %s *g) { for (int r = 0; r < %d; ++r) " \
               "for (int j = 0; j < %d; ++j) y[r][j] += w[0] * x[(r + 1) %% %d][j]; g[0] += w[0]; }" % (
                   t, t, t, t, arity, cdim, arity)
        args = [y(m, api.INC), x(m, api.READ)]
    else:
        names = ", ".join("%s *y%d" % (t, r) for r in range(len(rows)))
        code = "void k(%s, %s *x, %s *w, %s *g) { for (int j = 0; j < %d; ++j) { %s } g[0] += w[0]; }" % (
            names, t, t, t, cdim, " ".join("y%d[j] += (%s)%d * w[0] + x[j];" % (r, t, r + 1)
                                           for r in range(len(rows))))
        args = [y(m[r], api.INC) for r in rows] + [x(m[0], api.READ)]
    api.par_loop(api.Kernel(code, "k"), el, *args, w(api.IdentityMap, api.READ), g(api.INC))
    return np.array(y.data_ro if api is not seq else y.data), np.array(g.data)


def form():
    from pyop2_b200 import b200
    bl = [b for b in b200.ParLoop._bound_cache.values() if b.spec.kernel_name == "k"][-1]
    return bl.spec.mode, bool((bl.spec.region or {}).get("sums"))


# all values are small integers: sums in any order are exact in every type
@pytest.mark.parametrize("dtype,cdim", [(np.float64, 1), (np.float64, 2), (np.float64, 3), (np.float64, 4),
                                        (np.float64, 8), (np.float32, 1), (np.float32, 3), (np.float32, 4),
                                        (np.float32, 16), (np.int32, 1), (np.int32, 2)])
@pytest.mark.parametrize("n,arity,vec", [(1, 2, False), (127, 3, False), (256, 2, True), (257, 2, False),
                                         (1031, 3, True), (20011, 1, False), (20011, 2, False)])
def test_sums_match_the_oracle(op2, n, arity, vec, dtype, cdim):
    """Blocks of one element to several CTA waves, full and ragged; elements
    that name one target twice; rows of every width of shared-memory access;
    an argument read at the reordered element and a Global reduction."""
    rng = np.random.default_rng(n)
    conn = rng.integers(0, max(2, n // 3), (n, arity)).astype(np.int32)
    conn[::5, -1] = conn[::5, 0]
    old = (cfg.cfg['inc_mode'], cfg.cfg['staged_min_size'])
    cfg.configure(inc_mode="staged", staged_min_size=0)
    try:
        got = run(op2, n, arity, cdim, dtype, conn, range(arity), vec)
        assert form() == ("staged", True)
        want = run(seq, n, arity, cdim, dtype, conn, range(arity), vec)
        np.testing.assert_array_equal(got[0], want[0])
        np.testing.assert_array_equal(got[1], want[1])
    finally:
        cfg.configure(inc_mode=old[0], staged_min_size=old[1])


@pytest.mark.parametrize("rows,cdim,config", [((0,), 2, {}), ((0, 0), 2, {}), ((0, 1), 64, {}),
                                              ((0, 1), 2, {"staged_pair": 2}), ((1, 0), 2, {}),
                                              ((0, 1), 2, {"staged_tl_regs": True}),
                                              ((0, 1), 2, {"staged_bank_slots": True}),
                                              ((0, 1), 2, {"partition_size": 2048}),
                                              ((0, 1), 2, {"partition_size": 40})])
def test_which_loops_sum(op2, rows, cdim, config):
    """Loops that increment some rows of a Map, or one twice, with rows too wide or
    with an option of the colour form keep that form; the result is the same."""
    n = 3001
    conn = np.random.default_rng(2).integers(0, 900, (n, 2)).astype(np.int32)
    old = {k: cfg.cfg[k] for k in ('inc_mode', 'staged_min_size', 'staged_pair', 'staged_tl_regs',
                                   'staged_bank_slots', 'partition_size')}
    cfg.configure(inc_mode="staged", staged_min_size=0, **config)
    try:
        got = run(op2, n, 2, cdim, np.float64, conn, rows)
        sums = sorted(rows) == [0, 1] and cdim == 2 and (not config or config == {"partition_size": 40})
        assert form()[1] == sums         # (0, 1), 64: too wide for the colour form too
        want = run(seq, n, 2, cdim, np.float64, conn, rows)
        np.testing.assert_array_equal(got[0], want[0])
    finally:
        cfg.configure(**old)
