"""Element offsets of realqm_rb.js fields (csrc/rb_index.h, compiled for the host) at sizes whose fields pass 2^31
elements and whose interiors pass 2^32 cells, against Python's integers."""
import ctypes
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "realmolecule_b200", "csrc")

SRC = r"""
#include "rb_index.h"
extern "C" long long offset(int i, int j, int k, int S) { return rq::rb_offset<long long>(i, j, k, S); }
extern "C" int offset32(int i, int j, int k, int S) { return rq::rb_offset<int>(i, j, k, S); }
extern "C" int fits(int NN) { return rq::rb_offsets_fit_31_bits(NN); }
extern "C" long long interior(long long cell, int NM, int S) { return rq::rb_interior_offset<long long>(cell, NM, S); }
extern "C" unsigned interior32(unsigned cell, int NM, int S) { return rq::rb_interior_offset<unsigned>(cell, NM, S); }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    cc = shutil.which("g++")
    if cc is None:
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("rb")
    (d / "t.cpp").write_text(SRC)
    subprocess.run([cc, "-O2", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(d / "t.cpp"), "-o", str(d / "t.so")], check=True)
    l = ctypes.CDLL(str(d / "t.so"))
    for f in (l.offset, l.interior):
        f.restype = ctypes.c_longlong
    l.interior32.restype, l.interior32.argtypes = ctypes.c_uint, [ctypes.c_uint, ctypes.c_int, ctypes.c_int]
    l.interior.argtypes = [ctypes.c_longlong, ctypes.c_int, ctypes.c_int]
    return l


@pytest.mark.parametrize("NN", [8, 9, 150, 1289, 1290, 1291, 1626, 1627, 1700, 2500])
def test_offsets(lib, NN):
    S, NM = NN + 1, NN - 1
    for i, j, k in ((0, 0, 0), (1, 1, 1), (NN - 1, NN - 1, NN - 1), (NN, NN, NN), (NN - 1, 1, NN - 2)):
        assert lib.offset(i, j, k, S) == (i * S + j) * S + k
        assert not lib.fits(NN) or lib.offset32(i, j, k, S) == (i * S + j) * S + k
    fits = bool(lib.fits(NN))
    assert fits == (S ** 3 < 2 ** 31) and (not fits or NM ** 3 + 2 * 8 * 256 * 128 < 2 ** 32)
    cells = {0, 1, NM - 1, NM, NM * NM - 1, NM * NM, NM ** 3 // 2, NM ** 3 - 1}
    cells |= {c for c in (2 ** 31 - 1, 2 ** 31, 2 ** 32 - 1, 2 ** 32, 2 ** 32 + NM) if c < NM ** 3}
    for c in cells:
        i, j, k = c // (NM * NM), c // NM % NM, c % NM
        assert lib.interior(c, NM, S) == ((i + 1) * S + j + 1) * S + k + 1
        assert not fits or lib.interior32(c, NM, S) == ((i + 1) * S + j + 1) * S + k + 1


def test_kernels_take_their_offsets_from_the_header():
    """No offset of a cell is formed in 32 bits beside the header's functions."""
    text = open(os.path.join(CSRC, "rb_flavor.cu")).read()
    assert "rb_offset<I>(i, j, k, S)" in text and "rb_interior_offset<I>(cell, NM, S)" in text
    assert "int id =" not in text and "unsigned cell" not in text
