"""Calls from several host threads: what each keeps for itself is ready in time."""

import ctypes as C
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def in_threads(n, work):
    """work(k) in n threads at once; their results."""
    got, start = [None] * n, threading.Barrier(n)

    def run(k):
        start.wait()
        try:
            got[k] = work(k)
        except Exception as e:      # shown by the comparison
            got[k] = e
    threads = [threading.Thread(target=run, args=(k,)) for k in range(n)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    return got


@pytest.mark.parametrize("size", [1, 257, 300001])
def test_first_dot_of_a_thread(backend, size):
    """A thread's first dot product, while the stream is busy: whole numbers, so
    exact in any order; the scratch is cleared before the kernel counts in it."""
    from pyop2_b200 import b200
    from pyop2_b200._lib import call
    x = np.random.default_rng(size).integers(-9, 10, size).astype(np.float64)
    d = b200._upload(x)
    busy = b200.DeviceBuffer(1 << 28)
    want = float(x @ x)

    def dots(k):
        out = []
        for _ in range(3):
            r = C.c_double(-1.0)
            busy.memset(k)
            call("op2b_vec_dot", d.ptr, d.ptr, size, C.byref(r), 0)
            out.append(r.value)
        return out
    for _ in range(5):
        assert in_threads(6, dots) == [[want] * 3] * 6


def test_small_downloads_of_several_threads(backend):
    """Downloads of at most 256 bytes land in memory of the calling thread."""
    from pyop2_b200 import b200
    rng = np.random.default_rng(2)
    want = [rng.integers(0, 256, 200, dtype=np.uint8) for _ in range(6)]
    bufs = [b200._upload(w) for w in want]

    def down(k):
        out = np.zeros(200, np.uint8)
        for _ in range(50):
            out[:] = 0
            bufs[k].to_host(out)
            if not np.array_equal(out, want[k]):
                return "wrong"
        return "right"
    assert in_threads(6, down) == ["right"] * 6


def test_a_loop_changes_form_while_threads_run_it(backend, monkeypatch):
    """Threads repeat one assembly; one of them binds it as row blocks while the
    others are in the element form.  Whole numbers: exact in any order."""
    from pyop2_b200 import b200, op2
    from pyop2_b200.workloads import meshes
    monkeypatch.setattr(b200, "_ROWBLK_MIN", 0)
    coords, elem = meshes.rect_p1(40, 31, 2)
    n, nodes = len(elem), len(coords)
    el, nd = op2.Set(n, 1, "el"), op2.Set(nodes, 1, "nd")
    m = op2.Map(el, nd, 3, elem, "m")
    k = op2.Kernel("void threads(double A[1][1], double *w, int i, int j) { A[0][0] += w[0] * (1 + 3 * i + j); }",
                   "threads")
    w = op2.Dat(el, np.random.default_rng(1).integers(1, 9, n).astype(np.float64), np.float64, "w")

    def assemble(mat):
        op2.par_loop(k, el(3, 3), mat((m[op2.i[0]], m[op2.i[1]]), op2.INC), w(op2.IdentityMap, op2.READ))
    sp = op2.Sparsity((m, m), "s")
    one = op2.Mat(sp, np.float64, "one")
    assemble(one)
    for _ in range(4):
        monkeypatch.setattr(b200, "_ROWBLK_RUNS", 8)
        mat = op2.Mat(sp, np.float64, "mat")
        assemble(mat)          # bound

        def work(_):
            for _ in range(10):
                assemble(mat)
            return True
        assert in_threads(4, work) == [True] * 4
        forms = [b.spec.mode for b in b200.ParLoop._bound_cache.values() if b.mats == [mat]]
        assert forms == ["rowblk"]
        np.testing.assert_array_equal(mat.array, 41 * one.array)


def test_one_thread_binds_the_row_blocks(backend, monkeypatch):
    """Threads that find at once that a loop has run often enough: one of them builds
    and times, the others go on in the element form."""
    from pyop2_b200 import b200, op2
    from pyop2_b200.workloads import meshes
    monkeypatch.setattr(b200, "_ROWBLK_MIN", 0)
    monkeypatch.setattr(b200, "_ROWBLK_RUNS", 1)
    coords, elem = meshes.rect_p1(40, 31, 2)
    el, nd = op2.Set(len(elem), 1, "el"), op2.Set(len(coords), 1, "nd")
    m = op2.Map(el, nd, 3, elem, "m")
    w = op2.Dat(el, np.ones(len(elem)), np.float64, "w")
    mat = op2.Mat(op2.Sparsity((m, m), "s"), np.float64, "mat")
    k = op2.Kernel("void once(double A[1][1], double *w, int i, int j) { A[0][0] += w[0] * (1 + i + j); }", "once")

    def assemble(_):
        op2.par_loop(k, el(3, 3), mat((m[op2.i[0]], m[op2.i[1]]), op2.INC), w(op2.IdentityMap, op2.READ))
        return True
    assemble(0)
    want = mat.array
    here, timed = threading.Barrier(4), []
    bind, choose = b200._BoundLoop._in_rows, b200._BoundLoop._faster_form

    def together(self, args):
        here.wait(30)
        return bind(self, args)

    def counted(self, rows, loop):
        timed.append(rows)
        return choose(self, rows, loop)
    monkeypatch.setattr(b200._BoundLoop, "_in_rows", together)
    monkeypatch.setattr(b200._BoundLoop, "_faster_form", counted)
    assert in_threads(4, assemble) == [True] * 4
    assert len(timed) == 1
    np.testing.assert_array_equal(mat.array, 5 * want)


@pytest.mark.parametrize("runs", [0, 1 << 30])
def test_threads_add_to_a_mat_just_zeroed(backend, monkeypatch, runs):
    """Loops of several threads into one zeroed Mat (row blocks; or two of them row
    blocks and two the element form): the first write ends what is known of it,
    whoever makes it, so nothing is added to a zero that has gone."""
    from pyop2_b200 import b200, op2
    from pyop2_b200.workloads import meshes
    monkeypatch.setattr(b200, "_ROWBLK_MIN", 0)
    coords, elem = meshes.rect_p1(30, 21, 2)
    el, nd = op2.Set(len(elem), 1, "el"), op2.Set(len(coords), 1, "nd")
    m = op2.Map(el, nd, 3, elem, "m")
    w = op2.Dat(el, np.arange(1.0, 1 + len(elem)), np.float64, "w")
    ks = [op2.Kernel("void adds%d(double A[1][1], double *w, int i, int j) { A[0][0] += %d * w[0]; }" % (k, 10 ** k),
                     "adds%d" % k) for k in range(4)]
    mat = op2.Mat(op2.Sparsity((m, m), "s"), np.float64, "mat")

    def assemble(k):
        op2.par_loop(ks[k], el(3, 3), mat((m[op2.i[0]], m[op2.i[1]]), op2.INC), w(op2.IdentityMap, op2.READ))
        return True
    for k in range(4):
        monkeypatch.setattr(b200, "_ROWBLK_RUNS", 0 if k < 2 else runs)
        assemble(k)
    monkeypatch.setattr(b200, "_ROWBLK_RUNS", 1 << 30)
    want = mat.array
    for _ in range(50):
        mat.zero()
        assert in_threads(4, assemble) == [True] * 4
        np.testing.assert_array_equal(mat.array, want)


def test_threads_run_a_loop_for_the_first_time(backend):
    """One of them prepares it; the others launch what it prepared."""
    from pyop2_b200 import b200, op2
    n = 3000
    s = op2.Set(n, 1, "s")
    k = op2.Kernel("void first(double *x, double *g) { *x += 1; }", "first")
    g = op2.Global(1, 1.0, np.float64, "g")
    for _ in range(40):
        d = op2.Dat(s, np.zeros(n), np.float64, "d")
        b200.ParLoop._bound_cache.clear()
        loop = b200.ParLoop(k, s, d(op2.IdentityMap, op2.RW), g(op2.READ))
        d._to_device(), g._to_device()
        bl = loop._bound()

        def work(_):
            for _ in range(5):
                bl.run(loop)
            return True
        assert in_threads(4, work) == [True] * 4
        np.testing.assert_array_equal(d.data.ravel(), np.full(n, 20.0))
