"""Scalar Mat assembly by row blocks (op2b_row_blocks_build and the stubs that
walk its tables) against the sequential oracle.

A row's contributions are added in element order to the value before the
loop, with the oracle's arithmetic, so the Mats are equal bit for bit."""

import numpy as np
import pytest

from oracle import seq
from pyop2_b200.workloads import fem, meshes

pytestmark = pytest.mark.gpu


@pytest.fixture
def op2(backend, monkeypatch):
    """Every assembly runs as row blocks from its first run."""
    from pyop2_b200 import b200, op2
    monkeypatch.setattr(b200, "_ROWBLK_RUNS", 0)
    monkeypatch.setattr(b200, "_ROWBLK_MIN", 0)
    return op2


ONES = """
void ones(double A[1][1], double *w, int j, int k) { A[0][0] += (3 * j + k + 1) * w[0]; }
"""


def _general(api, elem, nodes, w, loops=1, zero=False):
    """A Mat over an arbitrary connectivity, incremented ``loops`` times."""
    n, a = elem.shape
    elements, rows = api.Set(n, 1, "elements"), api.Set(nodes, 1, "rows")
    m = api.Map(elements, rows, a, elem, "m")
    mat = api.Mat(api.Sparsity((m, m), "s"), np.float64, "mat")
    d = api.Dat(elements, w, np.float64, "w")
    k = api.Kernel(ONES, "ones")
    for _ in range(loops):
        if zero:
            mat.zero()
        api.par_loop(k, elements(a, a), mat((m[api.i[0]], m[api.i[1]]), api.INC),
                     d(api.IdentityMap, api.READ))
    return mat


def _modes(name):
    from pyop2_b200 import b200
    return [bl.spec.mode for bl in b200.ParLoop._bound_cache.values() if bl.spec.kernel_name == name]


@pytest.mark.parametrize("nx,ny,permute", [(1, 1, False), (7, 5, True), (33, 64, True), (131, 17, False),
                                           (150, 150, True)])
def test_p1_equals_oracle(op2, nx, ny, permute):
    coords, elem = meshes.rect_p1(nx, ny, 3 if permute else None)
    G = fem.build_p1(op2, 0, coords=coords, elem=elem, stiffness=True)
    O = fem.build_p1(seq, 0, coords=coords, elem=elem, stiffness=True)
    for api, P in ((op2, G), (seq, O)):
        fem.assemble_p1(api, P)
        fem.assemble_p1_stiffness(api, P)
    np.testing.assert_array_equal(G.mat.array, O.mat.array)
    np.testing.assert_array_equal(G.stiff.array, O.stiff.array)
    assert "rowblk" in _modes("p1_mass")


@pytest.mark.parametrize("n", [1, 6, 37])
def test_p2_two_mats_equal_oracle(op2, n):
    G, O = fem.build_p2(op2, n, seed=4), fem.build_p2(seq, n, seed=4)
    fem.assemble_p2(op2, G)
    fem.assemble_p2(seq, O)
    np.testing.assert_array_equal(G.K.array, O.K.array)
    np.testing.assert_array_equal(G.M.array, O.M.array)


@pytest.mark.parametrize("arity", [1, 2, 4, 7])
@pytest.mark.parametrize("case", ["random", "few", "repeated", "unused", "star"])
def test_connectivities_equal_oracle(op2, arity, case):
    """Long and empty rows, elements that name one row twice, rows no
    element touches, and a row every element touches (the element form)."""
    rng = np.random.default_rng(arity)
    n, nodes = 700, 400
    if case == "few":
        n, nodes = 300, 9
    elem = rng.integers(0, nodes, size=(n, arity)).astype(np.int32)
    if case == "repeated" and arity > 1:
        elem[::3, 1] = elem[::3, 0]
    if case == "unused":
        elem = elem // 2 * 2
    if case == "star":
        n = 40000
        elem = rng.integers(0, nodes, size=(n, arity)).astype(np.int32)
        elem[:, 0] = 5
    w = rng.integers(1, 9, size=n).astype(np.float64)     # sums exact in any order
    G, O = _general(op2, elem, nodes, w, loops=2), _general(seq, elem, nodes, w, loops=2)
    np.testing.assert_array_equal(G.array, O.array)


def test_known_zero_follows_every_writer(op2):
    """A Mat known to be zero is not read: the knowledge ends with a loop,
    zero_rows, a graph launch and a batched launch, and a zeroing recorded in
    a graph holds inside that graph only."""
    from pyop2_b200 import b200
    from pyop2_b200.batch import BatchLoop, LoopInstance
    coords, elem = meshes.rect_p1(9, 8, 1)
    P = fem.build_p1(op2, 0, coords=coords, elem=elem, stiffness=True)
    loop = lambda: fem.assemble_p1_stiffness(op2, P)  # noqa: E731
    loop()
    one = P.stiff.array.copy()
    loop()
    np.testing.assert_allclose(P.stiff.array, 2 * one, rtol=1e-15)
    P.stiff.zero()
    with b200.capture() as adds:          # recorded while the Mat is zero
        loop()
    with b200.capture() as fresh:
        P.stiff.zero()
        loop()
    adds.launch()
    adds.launch()
    np.testing.assert_allclose(P.stiff.array, 2 * one, rtol=1e-15)
    P.stiff.zero()
    adds.launch()
    loop()
    np.testing.assert_allclose(P.stiff.array, 2 * one, rtol=1e-15)
    fresh.launch()
    loop()
    np.testing.assert_allclose(P.stiff.array, 2 * one, rtol=1e-15)
    rows = (P.elem_node[op2.i[0]], P.elem_node[op2.i[1]])
    batch = BatchLoop([LoopInstance(P.k_stiff, P.elements(3, 3), P.stiff(rows, op2.INC),
                                    P.coords(P.elem_vnode, op2.READ))])
    P.stiff.zero()
    batch.launch(sync_host=False)
    loop()
    np.testing.assert_allclose(P.stiff.array, 2 * one, rtol=1e-15)
    P.stiff.zero()
    P.stiff.zero_rows([0], 3.0)
    loop()
    d = P.stiff.sparsity.rowptr[0] + list(P.stiff.sparsity.colidx[:P.stiff.sparsity.rowptr[1]]).index(0)
    assert P.stiff.array[d] == one[d] + 3.0


def test_row_blocks_are_built_when_a_loop_keeps_running(op2, monkeypatch):
    """The element form first; row blocks after _ROWBLK_RUNS runs, or before a
    capture of a loop that ran just before; small loops keep their form."""
    from pyop2_b200 import b200
    monkeypatch.setattr(b200, "_ROWBLK_RUNS", 3)
    monkeypatch.setattr(b200, "_ROWBLK_MIN", 9 * 2 * 12 * 11)
    coords, elem = meshes.rect_p1(12, 11, 1)
    small_c, small_e = meshes.rect_p1(5, 4, 1)
    P = fem.build_p1(op2, 0, coords=coords, elem=elem, stiffness=True)
    S = fem.build_p1(op2, 0, coords=small_c, elem=small_e)
    mode = lambda name, it: [bl.spec.mode for bl in b200.ParLoop._bound_cache.values()  # noqa: E731
                             if bl.spec.kernel_name == name and bl.iterset is it]
    for n in range(5):
        P.mat.zero()
        fem.assemble_p1(op2, P)
        fem.assemble_p1(op2, S)
        assert mode("p1_mass", P.elements) == ["rowblk" if n >= 3 else "atomic"]
    assert mode("p1_mass", S.elements) == ["atomic"]
    fem.assemble_p1_stiffness(op2, P)
    one = P.stiff.array.copy()
    assert mode("p1_stiff", P.elements) == ["atomic"]
    with b200.capture() as g:
        P.stiff.zero()
        fem.assemble_p1_stiffness(op2, P)
    assert mode("p1_stiff", P.elements) == ["rowblk"]
    g.launch()
    np.testing.assert_allclose(P.stiff.array, one, rtol=1e-14, atol=1e-16)


def test_consts_of_a_form_built_for_a_capture(backend, monkeypatch):
    """A loop bound again as row blocks before a capture has its Consts at once: a
    run of the loop is right although the graph was never launched."""
    from pyop2_b200 import b200, op2
    monkeypatch.setattr(b200, "_ROWBLK_MIN", 0)
    scale = op2.Const(1, 2.5, "rowblk_scale", np.float64)
    try:
        coords, elem = meshes.rect_p1(9, 7, 1)
        P = fem.build_p1(op2, 0, coords=coords, elem=elem)
        k = op2.Kernel("void scaled(double A[1][1], double **x, int i, int j) "
                       "{ A[0][0] += rowblk_scale * (1 + i + 2 * j); }", "scaled")
        m = P.elem_node

        def loop():
            P.mat.zero()
            op2.par_loop(k, P.elements(3, 3), P.mat((m[op2.i[0]], m[op2.i[1]]), op2.INC),
                         P.coords(P.elem_vnode, op2.READ))
        loop()
        want = P.mat.array.copy()
        assert abs(want).max() > 0
        with b200.capture() as g:
            loop()
        forms = [bl.spec.mode for bl in b200.ParLoop._bound_cache.values() if bl.spec.kernel_name == "scaled"]
        assert forms == ["rowblk"]
        loop()
        np.testing.assert_allclose(P.mat.array, want, rtol=1e-14)
        g.launch()
        np.testing.assert_allclose(P.mat.array, want, rtol=1e-14)
    finally:
        scale.remove_from_namespace()
