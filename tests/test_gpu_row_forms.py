"""When an assembly loop takes the row block form, and which one."""

import numpy as np
import pytest

from pyop2_b200 import configuration as cfg
from pyop2_b200.workloads import fem, meshes

pytestmark = pytest.mark.gpu


@pytest.fixture
def op2(backend, monkeypatch):
    """Row blocks at any size, before a capture only."""
    from pyop2_b200 import b200, op2
    monkeypatch.setattr(b200, "_ROWBLK_MIN", 0)
    monkeypatch.setattr(b200, "_ROWBLK_RUNS", 1 << 30)
    return op2


def problem(op2, nx=11, ny=9):
    coords, elem = meshes.rect_p1(nx, ny, 1)
    return fem.build_p1(op2, 0, coords=coords, elem=elem, stiffness=True)


def bound(name, iterset):
    from pyop2_b200 import b200
    return [b for b in b200.ParLoop._bound_cache.values()
            if b.spec.kernel_name == name and b.iterset is iterset]


@pytest.mark.parametrize("other", [{"inc_mode": "color"}, {"inc_mode": "lma", "kahan": True}, {"fmad": True}])
def test_a_capture_leaves_loops_of_another_configuration(op2, other):
    """What ran under other options is not bound again with those of the capture."""
    from pyop2_b200 import b200
    P = problem(op2)
    cfg.configure(inc_mode="staged", kahan=False, fmad=False)
    fem.assemble_p1(op2, P)
    (mass,) = bound("p1_mass", P.elements)
    assert mass.spec.mode == "atomic"
    cfg.configure(**other)
    P.b.zero()
    with b200.capture() as g:
        P.b.zero()
    assert bound("p1_mass", P.elements) == [mass] and mass.spec.mode == "atomic" and mass.row_blocks is None
    cfg.configure(inc_mode="staged", kahan=False, fmad=False)
    with b200.capture() as g:
        P.mat.zero()
        fem.assemble_p1(op2, P)
    (rows,) = bound("p1_mass", P.elements)
    assert rows.spec.mode == "rowblk" and not rows.spec.rowblk["kahan"] and not rows.spec.fmad
    g.launch()
    want = P.mat.array
    P.mat.zero()
    fem.assemble_p1(op2, P)
    np.testing.assert_array_equal(P.mat.array, want)



def test_what_ends_a_build(op2, monkeypatch):
    """Without memory for the tables a loop keeps the element form; any other
    failure of the build is reported."""
    from pyop2_b200 import b200
    from pyop2_b200.exceptions import DeviceError

    def fail(status):
        def of(*args):
            e = DeviceError("op2b_row_blocks_build failed")
            e.status = status
            raise e
        monkeypatch.setattr(b200.RowBlocks, "of", of)
    P = problem(op2, 8, 5)
    fem.assemble_p1(op2, P)
    want = P.mat.array
    fail(1)
    with pytest.raises(DeviceError):
        with b200.capture():
            pass
    P = problem(op2, 8, 5)
    fail(4)
    fem.assemble_p1(op2, P)
    with b200.capture() as g:
        P.mat.zero()
        fem.assemble_p1(op2, P)
    assert [b.spec.mode for b in bound("p1_mass", P.elements)] == ["atomic"]
    g.launch()
    np.testing.assert_allclose(P.mat.array, want, rtol=1e-14)


def test_an_allocation_that_failed_is_over(backend):
    """Its error is the failing call's own: what runs next is not told of it."""
    from pyop2_b200 import b200
    from pyop2_b200._lib import call
    from pyop2_b200.exceptions import DeviceError
    x = b200._upload(np.arange(50.0))
    with pytest.raises(DeviceError) as e:
        b200.DeviceBuffer(1 << 50)
    assert e.value.status == 4
    call("op2b_vec_binop", x.ptr, x.ptr, 0, 2.0, 50, 2, 0, 0)     # checks its launch's error
    got = np.zeros(50)
    x.to_host(got)
    np.testing.assert_array_equal(got, 2 * np.arange(50.0))


@pytest.mark.parametrize("graph", [False, True])
def test_values_written_at_their_address(op2, monkeypatch, graph):
    """Values written through an address taken after the zeroing, or taken again
    after the write, are added to."""
    from pyop2_b200 import b200
    from pyop2_b200._lib import call
    monkeypatch.setattr(b200, "_ROWBLK_RUNS", 0)
    P = problem(op2, 10, 6)
    loop = lambda: fem.assemble_p1_stiffness(op2, P)  # noqa: E731
    loop()
    assert [b.spec.mode for b in bound("p1_stiff", P.elements)] == ["rowblk"]
    one = P.stiff.array
    fives = np.full_like(one, 5.0)

    def write(ptr):
        call("op2b_memcpy_h2d", ptr, fives.ctypes.data, fives.nbytes, 0)
    if graph:
        with b200.capture() as g:
            loop()
        run = g.launch
    else:
        run = loop
    P.stiff.zero()
    write(P.stiff._device_values().ptr)
    run()
    np.testing.assert_allclose(P.stiff.array, one + fives, rtol=1e-14)
    kept = P.stiff._device_values().ptr
    P.stiff.zero()
    write(kept)
    P.stiff._device_values()
    run()
    np.testing.assert_allclose(P.stiff.array, one + fives, rtol=1e-14)


def hexes(n):
    """(points, elem) of n^3 cubes."""
    i, j, k = np.meshgrid(*[np.arange(n)] * 3, indexing="ij")
    at = lambda a, b, c: ((i + a) * (n + 1) + j + b) * (n + 1) + k + c  # noqa: E731
    elem = np.stack([at(a, b, c) for a in (0, 1) for b in (0, 1) for c in (0, 1)], -1).reshape(-1, 8)
    return (n + 1) ** 3, elem.astype(np.int32)


# per entry: whole numbers, exact in any order; the second after a chain of 400
# dependent divisions, and so dearer than anything else in the launch
CHEAP = "A[0][0] += w[0] * (1 + 3 * i + j);"
DEAR = "double s = 1 + w[0] + i * j; for (int q = 0; q < 400; ++q) s = 3.0 / s; " + CHEAP[:-1] + " + (s == 0.0);"


@pytest.mark.parametrize("inc_mode,other", [("staged", "atomic"), ("lma", "lma")])
@pytest.mark.parametrize("cost,code,zeroed", [("cheap", CHEAP, True), ("dear", DEAR, False)])
def test_the_faster_form_runs(backend, monkeypatch, inc_mode, other, cost, code, zeroed):
    """Row blocks evaluate an element of a hexahedral mesh about three times: loops
    whose kernel outweighs the rest keep the form that evaluates it once.  The
    results are those of a loop that never had the choice."""
    from pyop2_b200 import b200, op2
    nodes, elem = hexes(27)
    n = len(elem)
    assert n * 64 >= b200._TRIAL_MIN
    cfg.configure(inc_mode=inc_mode, kahan=False)
    el, nd = op2.Set(n, 1, "el"), op2.Set(nodes, 1, "nd")
    m = op2.Map(el, nd, 8, elem, "m")
    w = op2.Dat(el, np.random.default_rng(3).integers(1, 9, n).astype(np.float64), np.float64, "w")
    g = op2.Global(1, 2.0, np.float64, "g")
    sp = op2.Sparsity((m, m), "s")
    mats = [op2.Mat(sp, np.float64, "m%d" % k) for k in range(2)]
    k = op2.Kernel("void %s(double A[1][1], double *w, double *g, int i, int j) { %s A[0][0] += g[0]; }"
                   % (cost, code), cost)

    def assemble(mat):
        op2.par_loop(k, el(8, 8), mat((m[op2.i[0]], m[op2.i[1]]), op2.INC), w(op2.IdentityMap, op2.READ),
                     g(op2.READ))
    monkeypatch.setattr(b200, "_ROWBLK_MIN", 1 << 40)
    assemble(mats[0])
    assemble(mats[0])
    monkeypatch.setattr(b200, "_ROWBLK_MIN", 1 << 20)
    mat = mats[1]
    assemble(mat)
    with b200.capture() as graph:
        mat.zero()
        assemble(mat)
    assemble(mat)
    np.testing.assert_array_equal(mat.array, mats[0].array)
    graph.launch()
    assemble(mat)
    np.testing.assert_array_equal(mat.array, mats[0].array)
    (bl,) = [b for b in bound(cost, el) if b.mats[0] is mat]
    assert bl.spec.mode == ("rowblk" if zeroed else other)
    assert bl._element is None or bl._element.spec.mode == other


@pytest.mark.parametrize("long,runs", [(1e9, 2 + 6), (0.0, 2)])
def test_long_runs_are_timed_once(op2, monkeypatch, long, runs):
    """Two forms, zeroed and (where row blocks win that) holding values."""
    from pyop2_b200 import b200
    monkeypatch.setattr(b200, "_TRIAL_MIN", 0)
    monkeypatch.setattr(b200, "_TRIAL_LONG", long)
    P = problem(op2)
    fem.assemble_p1(op2, P)
    want = P.mat.array
    made, call = [], b200.call
    monkeypatch.setattr(b200, "call", lambda name, *a: (made.append(name), call(name, *a))[1])
    with b200.capture() as g:
        P.mat.zero()
    n = made.count("op2b_launch")
    assert n in (2 * runs, 3 * runs)
    P.mat.zero()
    fem.assemble_p1(op2, P)
    np.testing.assert_allclose(P.mat.array, want, rtol=1e-14)


def test_row_blocks_within_the_second_phase_run_once(op2, monkeypatch):
    """What the first run shows is not measured again."""
    from pyop2_b200 import b200
    monkeypatch.setattr(b200, "_TRIAL_MIN", 0)
    monkeypatch.setattr(b200, "_LMA_PER_MS", 1e-6)
    monkeypatch.setitem(b200._state, "l2_bytes", 0)
    cfg.configure(inc_mode="lma")
    P = problem(op2)
    made, call = [], b200.call
    monkeypatch.setattr(b200, "call", lambda name, *a: (made.append(name), call(name, *a))[1])
    fem.assemble_p1_stiffness(op2, P)
    assert [b.spec.mode for b in bound("p1_stiff", P.elements)] == ["rowblk"]
    assert made.count("op2b_launch") == 1


@pytest.mark.parametrize("inc_mode", ["staged", "lma"])
@pytest.mark.parametrize("held", [False, True])
@pytest.mark.parametrize("fails", [False, True])
def test_timing_leaves_the_values(op2, monkeypatch, inc_mode, held, fails):
    """Forms are timed into Mats known to be zero, which are zeroed again, but not
    into Mats that hold values; also where the timing ends in an error."""
    from pyop2_b200 import b200
    from pyop2_b200.exceptions import DeviceError
    cfg.configure(inc_mode=inc_mode, kahan=False)
    P = problem(op2)
    monkeypatch.setattr(b200, "_ROWBLK_MIN", 1 << 40)
    fem.assemble_p1_stiffness(op2, P)
    one = P.stiff.array
    P = problem(op2)
    if held:
        fem.assemble_p1_stiffness(op2, P)
    monkeypatch.setattr(b200, "_ROWBLK_MIN", 0)
    monkeypatch.setattr(b200, "_ROWBLK_RUNS", 0)
    monkeypatch.setattr(b200, "_TRIAL_MIN", 0)
    b200.ParLoop._bound_cache.clear()
    time, wrote = b200._BoundLoop._device_ms, []

    def device_ms(self, args, values, *rest, **kw):
        ms = time(self, args, values, *rest, **kw)
        wrote.append(values == [P.stiff._values().ptr])
        if fails:
            raise DeviceError("no memory", 4 if inc_mode == "lma" else 2)
        return ms
    monkeypatch.setattr(b200._BoundLoop, "_device_ms", device_ms)
    if fails and inc_mode == "staged":
        with pytest.raises(DeviceError):
            fem.assemble_p1_stiffness(op2, P)
    fem.assemble_p1_stiffness(op2, P)
    assert wrote and wrote == [not held] * len(wrote)
    np.testing.assert_allclose(P.stiff.array, (2 if held else 1) * one, rtol=1e-14, atol=1e-15 * abs(one).max())


def test_a_pause_keeps_the_stream_busy(backend):
    """About as long as asked (in cycles of 2 GHz); longer ones are refused."""
    from pyop2_b200 import b200
    from pyop2_b200._lib import call
    from pyop2_b200.exceptions import DeviceError
    call("op2b_stream_pause", 1, 0)
    for us in (0, 120, 1000):
        e0 = b200.Event().record()
        call("op2b_stream_pause", us, 0)
        e1 = b200.Event().record()
        e1.synchronize()
        assert 0.9e-3 * us <= e0.elapsed_ms(e1) < 1 + 4e-3 * us
    for us in (-1, 1001):
        with pytest.raises(DeviceError):
            call("op2b_stream_pause", us, 0)
