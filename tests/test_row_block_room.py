"""The packet array's size for row blocks, against integers without a width."""

import ctypes as C
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pyop2_b200", "csrc")


@pytest.fixture(scope="module")
def room(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("room")
    src, lib = d / "room.cpp", d / "room.so"
    src.write_text('#include "op2b_rowblk_room.h"\nextern "C" int64_t room(int64_t e, int64_t ra, int64_t ca, int64_t n, '
                   'int64_t nnz, int64_t b, int ids, int ns, const int32_t *a) '
                   '{ return op2b::row_block_room(e, ra, ca, n, nnz, b, ids, ns, a); }\n')
    subprocess.check_call(["g++", "-std=c++17", "-shared", "-fPIC", "-I" + CSRC, str(src), "-o", str(lib)])
    fn = C.CDLL(str(lib)).room
    fn.argtypes = [C.c_int64] * 6 + [C.c_int, C.c_int, C.POINTER(C.c_int32)]
    fn.restype = C.c_int64
    return fn


@pytest.mark.parametrize("nelem,ra,ca,stages", [(1, 1, 1, []), (1000, 3, 3, [3]), (10600000, 6, 6, [6]),
                                                (21200000, 3, 3, [3]), (59000000, 6, 6, [6, 6]),
                                                (238000000, 3, 3, [3, 3, 3, 3]), (2000000000, 1, 1, [8])])
@pytest.mark.parametrize("ids", [0, 1])
def test_room(room, nelem, ra, ca, stages, ids):
    """Up to the 2^31 contributions the build accepts."""
    assert nelem * ra * ca < 2 ** 31
    nrows, nnz, nblocks = 2 * nelem + 1, min(12 * nelem, 2 ** 31 - 1), nelem // 50 + 1
    want = (4 * ids + 2 * ra) * nelem * 17 // 10 + 8 * nnz + nelem * ra * ca // 2
    want += sum(8 * nrows + 2 * a * nelem * 17 // 10 for a in stages)
    want = want // 16 + nblocks * (7 + 2 * len(stages))
    got = room(nelem, ra, ca, nrows, nnz, nblocks, ids, len(stages), (C.c_int32 * 4)(*stages))
    assert got == want
