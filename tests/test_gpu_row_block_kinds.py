"""Row blocks over everything they accept -- types, Maps, what the loop reads --
against element-by-element sums in numpy, and with the form that ran."""

import numpy as np
import pytest

from oracle import seq
from pyop2_b200 import configuration as cfg

pytestmark = pytest.mark.gpu


@pytest.fixture
def op2(backend, monkeypatch):
    """Every assembly runs as row blocks from its first run."""
    from pyop2_b200 import b200, op2
    monkeypatch.setattr(b200, "_ROWBLK_RUNS", 0)
    monkeypatch.setattr(b200, "_ROWBLK_MIN", 0)
    monkeypatch.setattr(b200, "_TRIAL_MIN", 1 << 40)      # whatever is faster
    return op2


def mode(name):
    from pyop2_b200 import b200
    return [b.spec.mode for b in b200.ParLoop._bound_cache.values() if b.spec.kernel_name == name][-1]


def sums(sp, rows, cols, values, start):
    """``start`` with ``values`` [element, row, column] added in that order."""
    rowptr, colidx = np.asarray(sp._rowptr), np.asarray(sp._colidx)
    width = int(colidx.max()) + 1
    keys = np.repeat(np.arange(len(rowptr) - 1), np.diff(rowptr)).astype(np.int64) * width + colidx
    at = np.searchsorted(keys, rows[:, :, None].astype(np.int64) * width + cols[:, None, :])
    out = start.copy()
    np.add.at(out, at.reshape(-1), values.reshape(-1).astype(start.dtype))
    return out


CT = {np.float64: "double", np.float32: "float", np.int32: "int", np.uint32: "unsigned int"}


@pytest.mark.parametrize("types", [(np.float32,), (np.int32,), (np.uint32,), (np.float64, np.float32),
                                   (np.float32, np.float64), (np.int32, np.float64), (np.float32, np.float32),
                                   (np.float64, np.float64, np.float64), (np.float32, np.int32, np.float32)])
@pytest.mark.parametrize("ra,ca", [(3, 3), (2, 4), (4, 1)])
def test_types_and_shapes(op2, types, ra, ca):
    """Mats of several types at once (their contributions lie together), rows and
    columns through different Maps; added to zero, then to what is there."""
    rng = np.random.default_rng(ra * 10 + ca)
    n, nr, nc = 900, 311, 207
    rows, cols = (rng.integers(0, m, (n, a)).astype(np.int32) for m, a in ((nr, ra), (nc, ca)))
    el, R, K = op2.Set(n, 1, "el"), op2.Set(nr, 1, "R"), op2.Set(nc, 1, "K")
    rm, cm = op2.Map(el, R, ra, rows, "rm"), op2.Map(el, K, ca, cols, "cm")
    sp = op2.Sparsity((rm, cm), "s")
    mats = [op2.Mat(sp, t, "m%d" % k) for k, t in enumerate(types)]
    w = rng.integers(1, 1 << 20, n).astype(np.float64)
    if all(t in (np.float32, np.float64) for t in types):
        w /= 1024.0                 # each value exact in 32 bits, their sums not
    name = "kinds_%s" % "_".join(np.dtype(t).name for t in types)
    code = "void %s(%s, double *w, int i, int j) { %s }" % (
        name, ", ".join("%s A%d[1][1]" % (CT[t], k) for k, t in enumerate(types)),
        " ".join("A%d[0][0] += (%s)w[0] * (%s)(1 + i + 2 * j);" % (k, CT[t], CT[t]) for k, t in enumerate(types)))
    d = op2.Dat(el, w, np.float64, "w")
    loop = lambda: op2.par_loop(op2.Kernel(code, name), el(ra, ca),  # noqa: E731
                                *[m((rm[op2.i[0]], cm[op2.i[1]]), op2.INC) for m in mats],
                                d(op2.IdentityMap, op2.READ))
    want = []
    for t in types:
        factor = (1 + np.arange(ra)[:, None] + 2 * np.arange(ca)[None]).astype(t)
        values = w.astype(t)[:, None, None] * factor
        one = sums(sp, rows, cols, values, np.zeros(sp.nz, t))
        want.append((one, sums(sp, rows, cols, values, one)))
    for turn in range(2):
        loop()
        assert mode(name) == "rowblk"
        for m, w2 in zip(mats, want):
            assert m.array.dtype == m.dtype
            np.testing.assert_array_equal(m.array, w2[turn])


@pytest.mark.parametrize("cdims", [(1,), (2,), (3,), (4,), (8,), (16,), (5, 2), (4, 1, 2), (2, 8, 1, 3), (1, 1, 1, 1, 1)])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_what_is_read(op2, cdims, dtype):
    """Dats read through one to four Maps (whole rows of a Map, and single ones),
    rows of every width of a copy, with Globals; more Maps keep the element form."""
    rng = np.random.default_rng(sum(cdims))
    n, nodes = 700, 333
    el, R = op2.Set(n, 1, "el"), op2.Set(nodes, 1, "R")
    elem = rng.integers(0, nodes, (n, 3)).astype(np.int32)
    m = op2.Map(el, R, 3, elem, "m")
    mat = op2.Mat(op2.Sparsity((m, m), "s"), np.float64, "mat")
    t, args, params, terms, value = CT[dtype], [], [], [], np.zeros(n)
    for q, c in enumerate(cdims):
        nd = op2.Set(200 + q, c, "nd%d" % q)
        conn = rng.integers(0, 200 + q, (n, 2 + q)).astype(np.int32)
        x = rng.integers(1, 9, (200 + q, c)).astype(dtype)
        dat, mp = op2.Dat(nd, x, dtype, "x%d" % q), op2.Map(el, nd, 2 + q, conn, "mp%d" % q)
        if q % 2:
            args.append(dat(mp[1], op2.READ))
            params.append("%s *x%d" % (t, q))
            terms += ["x%d[%d]" % (q, k) for k in range(c)]
            value += x[conn[:, 1]].sum(axis=1)
        else:
            args.append(dat(mp, op2.READ))
            params.append("%s **x%d" % (t, q))
            terms += ["x%d[%d][%d]" % (q, r, k) for r in range(2 + q) for k in range(c)]
            value += x[conn].sum(axis=(1, 2))
    g, h = op2.Global(1, 3.0, np.float64, "g"), op2.Global(2, [5, 7], np.int32, "h")
    name = "reads%d" % len(cdims)
    code = "void %s(double A[1][1], %s, double *g, int *h, int i, int j) { A[0][0] += (%s) * (1 + i + 2 * j) + g[0] * h[1]; }" % (
        name, ", ".join(params), " + ".join(terms))
    op2.par_loop(op2.Kernel(code, name), el(3, 3), mat((m[op2.i[0]], m[op2.i[1]]), op2.INC), *args, g(op2.READ),
                 h(op2.READ))
    assert mode(name) == ("rowblk" if len(cdims) <= 4 else "atomic")
    values = value[:, None, None] * (1 + np.arange(3)[:, None] + 2 * np.arange(3)[None]) + 21.0
    np.testing.assert_array_equal(mat.array, sums(mat.sparsity, elem, elem, values, np.zeros(mat.sparsity.nz)))


@pytest.mark.parametrize("arity", [1, 2, 4, 7])
@pytest.mark.parametrize("case", ["random", "few", "repeated", "unused", "spread", "star"])
def test_order_of_the_sums(op2, arity, case):
    """Values whose sums depend on the order: those of the sequential oracle, bit for
    bit, by row blocks; "spread" takes more room than the builder starts with, and a
    row that every element touches leaves the loop in the element form."""
    rng = np.random.default_rng(arity + 31)
    n, nodes = {"few": (300, 9), "spread": (20000, 9000), "star": (40000, 400)}.get(case, (700, 400))
    elem = rng.integers(0, nodes, (n, arity)).astype(np.int32)
    if case == "repeated" and arity > 1:
        elem[::3, 1] = elem[::3, 0]
    if case == "unused":
        elem = elem // 2 * 2
    if case == "star":
        elem[:, 0] = 5
    w = rng.standard_normal(n)
    name = "order_%s%d" % (case, arity)

    def build(api):
        el, R = api.Set(n, 1, "el"), api.Set(nodes, 1, "R")
        m = api.Map(el, R, arity, elem, "m")
        mat = api.Mat(api.Sparsity((m, m), "s"), np.float64, "mat")
        d = api.Dat(el, w, np.float64, "w")
        k = api.Kernel("void %s(double A[1][1], double *w, int i, int j) { A[0][0] += w[0] * (1 + i + 2 * j); }" % name,
                       name)
        for _ in range(2):
            api.par_loop(k, el(arity, arity), mat((m[api.i[0]], m[api.i[1]]), api.INC), d(api.IdentityMap, api.READ))
        return mat
    G, O = build(op2), build(seq)
    assert mode(name) == ("atomic" if case == "star" else "rowblk")
    if case == "star":
        np.testing.assert_allclose(G.array, O.array, rtol=1e-9, atol=1e-9)
    else:
        np.testing.assert_array_equal(G.array, O.array)


@pytest.mark.parametrize("kahan", [False, True])
@pytest.mark.parametrize("arity", [2, 3, 6])
def test_as_the_two_phases(op2, monkeypatch, kahan, arity):
    """inc_mode='lma': the bits of the two-phase form, compensated or not, from zero
    and added to what is there."""
    from pyop2_b200 import b200
    cfg.configure(inc_mode="lma", kahan=kahan)
    rng = np.random.default_rng(arity)
    n, nodes = 2500, 300
    el, R = op2.Set(n, 1, "el"), op2.Set(nodes, 1, "R")
    elem = rng.integers(0, nodes, (n, arity)).astype(np.int32)
    m = op2.Map(el, R, arity, elem, "m")
    sp = op2.Sparsity((m, m), "s")
    w = op2.Dat(el, rng.standard_normal(n) * 10.0 ** rng.integers(-8, 9, n), np.float64, "w")
    k = op2.Kernel("void phases%d(double A[1][1], double *w, int i, int j) { A[0][0] += w[0] / (1 + i + 2 * j); }" % arity,
                   "phases%d" % arity)
    got = []
    for least, form in ((1 << 40, "lma"), (0, "rowblk")):
        monkeypatch.setattr(b200, "_ROWBLK_MIN", least)
        mat = op2.Mat(sp, np.float64, "mat")
        loop = lambda: op2.par_loop(k, el(arity, arity), mat((m[op2.i[0]], m[op2.i[1]]), op2.INC),  # noqa: E731
                                    w(op2.IdentityMap, op2.READ))
        loop()
        first = mat.array
        assert mode("phases%d" % arity) == form
        loop()
        got.append((first, mat.array))
    np.testing.assert_array_equal(got[0][0], got[1][0])
    np.testing.assert_array_equal(got[0][1], got[1][1])
