"""What a batched loop says of itself."""

import pytest

from pyop2_b200.workloads import fem, meshes

pytestmark = pytest.mark.gpu


def test_block_sizes_of_the_coloured_form(backend):
    """Batches of one loop signature share their stub, not their partition."""
    from pyop2_b200 import op2
    from pyop2_b200.batch import BatchLoop, LoopInstance
    coords, elem = meshes.rect_p1(9, 8, 1)
    P = fem.build_p1(op2, 0, coords=coords, elem=elem)
    rows = (P.elem_node[op2.i[0]], P.elem_node[op2.i[1]])
    inst = LoopInstance(P.k_mass, P.elements(3, 3), P.mat(rows, op2.INC), P.coords(P.elem_vnode, op2.READ))
    for ps in (64, 128, 32, 64):
        part = inst.recast("color", ps)
        assert BatchLoop([part], block_size=128).config["part_size"] == ps
