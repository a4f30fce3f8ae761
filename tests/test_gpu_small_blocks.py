"""Device blocks of Globals: the slab of small blocks and its ends."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture
def op2(backend):
    from pyop2_b200 import op2
    return op2


@pytest.mark.parametrize("nbytes", [1, 16, 248, 256, 264])
def test_small_blocks_do_not_overlap(op2, nbytes):
    """More blocks at once than the slab holds, each with its own bytes; what is
    released is handed out again."""
    from pyop2_b200.b200 import DeviceBuffer
    n = 300
    for turn in range(2):
        bufs = [DeviceBuffer(nbytes) for _ in range(n)]
        ptrs = sorted(b.ptr for b in bufs)
        assert all(b - a >= max(nbytes, 16) for a, b in zip(ptrs, ptrs[1:]))
        want = [np.full(nbytes, (7 * k + turn) % 251, np.uint8) for k in range(n)]
        for b, w in zip(bufs, want):
            b.from_host(w)
        for b, w in zip(bufs, want):
            got = np.empty(nbytes, np.uint8)
            b.to_host(got)
            np.testing.assert_array_equal(got, w)
        if turn == 0:
            first = set(ptrs)
            del bufs[::2], b
    assert first & set(ptrs)


def test_fresh_globals_of_a_repeated_reduction(op2):
    """A new Global per loop call, several alive at once: each its own sum."""
    s = op2.Set(1000, 1, "s")
    d = op2.Dat(s, np.arange(1000.0), np.float64, "d")
    k = op2.Kernel("void add(double *x, double *g) { *g += *x; }", "add")
    kept = []
    for n in range(12):
        g = op2.Global(1, float(n), np.float64, "g")
        op2.par_loop(k, s, d(op2.IdentityMap, op2.READ), g(op2.INC))
        if n % 3 == 0:
            kept.append((n, g))
        else:
            assert g.data[0] == n + 499500.0
    assert [g.data[0] for _, g in kept] == [n + 499500.0 for n, _ in kept]


def test_blocks_released_in_a_capture(op2):
    """What a recorded loop writes is not handed to another Global, even if its own
    Global is dropped before the recording ends."""
    from pyop2_b200 import b200
    s = op2.Set(500, 1, "s")
    d = op2.Dat(s, np.arange(500.0), np.float64, "d")
    k = op2.Kernel("void addup(double *x, double *g) { *g += *x; }", "addup")
    g = op2.Global(1, 0.0, np.float64, "g")
    add = lambda v: op2.par_loop(k, s, d(op2.IdentityMap, op2.READ), v(op2.INC))  # noqa: E731
    add(g)
    ptr = g._device.ptr
    with b200.capture() as graph:
        add(g)
        del g
    more = [b200.DeviceBuffer(8) for _ in range(300)]
    assert ptr not in {b.ptr for b in more}
    zero = np.zeros(1)
    for b in more:
        b.from_host(zero)
    graph.launch()
    graph.launch()
    for b in more:
        b.to_host(zero)
        assert zero[0] == 0.0


def test_what_is_not_a_held_block_is_refused(op2):
    """A small block given back twice, or an address inside one: refused, and the
    slab stays as it was."""
    from pyop2_b200._lib import call
    from pyop2_b200.b200 import DeviceBuffer
    from pyop2_b200.exceptions import DeviceError
    keep = DeviceBuffer(64)
    b = DeviceBuffer(64)
    with pytest.raises(DeviceError):
        call("op2b_free", b.ptr + 16)
    call("op2b_free", b.ptr)
    for _ in range(3):
        with pytest.raises(DeviceError):
            call("op2b_free", b.ptr)
    b.ptr = 0
    ptrs = [keep.ptr]
    more = [DeviceBuffer(64) for _ in range(300)]
    ptrs += [m.ptr for m in more]
    assert len(set(ptrs)) == 301


def test_large_blocks_released_in_a_capture(op2):
    """Memory of the allocator cannot be released while its stream is recorded; the
    refusal is that call's own, and the recording and later launches go on."""
    from pyop2_b200 import b200
    from pyop2_b200._lib import call
    n = 400
    x, big = b200._upload(np.arange(float(n))), b200.DeviceBuffer(1 << 16)
    with b200.capture() as graph:
        del big
        call("op2b_vec_binop", x.ptr, x.ptr, 0, 2.0, n, 2, 0, 0)     # checks its launch's error
    graph.launch()
    call("op2b_vec_binop", x.ptr, x.ptr, 0, 1.0, n, 0, 0, 0)
    got = np.zeros(n)
    x.to_host(got)
    np.testing.assert_array_equal(got, 2 * np.arange(float(n)) + 1)
