"""Host copies of results (op2b_host_copy) against numpy, on the CPU."""

import numpy as np
import pytest

from pyop2_b200 import _lib


@pytest.mark.parametrize("sizes", [(0,), (1,), (1 << 18,), ((1 << 19) - 1,), ((1 << 19) + 1,),
                                   (3, 0, (5 << 20) + 17, 4097), ((33 << 20) + 5, 8)])
def test_copies_equal_their_sources(sizes):
    from pyop2_b200 import b200
    _lib.load()
    rng = np.random.default_rng(3)
    src = {n: rng.integers(0, 256, s, dtype=np.uint8) for n, s in enumerate(sizes)}
    got = b200.copies(src)
    assert list(got) == list(src)
    for n, a in src.items():
        np.testing.assert_array_equal(got[n], a)
        assert got[n].flags.owndata and got[n].flags.writeable and not np.shares_memory(got[n], a)


def test_copies_of_other_layouts():
    from pyop2_b200 import b200
    _lib.load()
    a = np.arange(60.0).reshape(5, 12)
    a.setflags(write=False)
    got = b200.copies({"t": a.T, "s": a[:, ::3], "r": a, "x": 4.0})
    np.testing.assert_array_equal(got["t"], a.T)
    np.testing.assert_array_equal(got["s"], a[:, ::3])
    np.testing.assert_array_equal(got["r"], a)
    assert got["r"].flags.writeable and got["x"] == 4.0


def test_copies_from_several_threads():
    """Callers at once, each with its own arrays (more pieces than threads)."""
    import threading
    from pyop2_b200 import b200
    _lib.load()
    rng = np.random.default_rng(9)
    src = [{"a": rng.integers(0, 256, (2 << 20) + 13 * k, dtype=np.uint8), "b": np.arange(5.0) + k}
           for k in range(6)]
    bad = []

    def run(mine):
        for _ in range(8):
            got = b200.copies(mine)
            if not all(np.array_equal(got[k], mine[k]) for k in mine):
                bad.append(mine)
    threads = [threading.Thread(target=run, args=(s,)) for s in src]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
