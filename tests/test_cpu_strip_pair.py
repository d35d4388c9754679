"""Strip plans of a matrix's two directions for launches that know a solve by one
entry class (strip_plan_both): whatever the numbering, both directions get the
class of the widest row of either, so that one stream orders the backward sweep
after the forward one."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT
from meshorder import boundary_first, radial, rcm, renumber


@pytest.fixture(scope="module")
def pair_lib():
    out = os.path.join(ROOT, "tests", "cpu", "_build")
    os.makedirs(out, exist_ok=True)
    so = os.path.join(out, "libstrip_pair_emul.so")
    srcs = [os.path.join(ROOT, "tests", "cpu", "strip_pair_emul.cpp"),
            os.path.join(ROOT, "delfem_gb300", "csrc", "strip.cpp")]
    inc = [d for d in ("/usr/local/cuda/include",) if os.path.isdir(d)]
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", *[f"-I{d}" for d in inc], "-o", so, *srcs],
                   check=True)
    L = ctypes.CDLL(so)
    P = ctypes.c_void_p
    L.emul_strip_pair.argtypes = [ctypes.c_int] * 3 + [P, P, ctypes.c_int, P]
    return L


def _mesh(name):
    from delfem_gb300 import meshgen as mg
    kind, shape = name.split(":")
    if shape.startswith("del"):
        coords, conn = mg.delaunay_mesh(int(shape[3:]), 2, seed=3)
    else:
        coords, conn = mg.tri_grid(*map(int, shape.split("x")))
    if kind != "nat":
        order = {"bfirst": boundary_first, "blast": lambda c, e: boundary_first(c, e)[::-1], "rcm": rcm,
                 "radial": radial}[kind](coords, conn)
        coords, conn = renumber(coords, conn, order)
    return coords, conn


@pytest.mark.parametrize("elem", [4, 8])
@pytest.mark.parametrize("b", [1, 2])
@pytest.mark.parametrize("name,alone,both", [
    ("nat:40x25", (3, 3), 3), ("bfirst:40x25", (7, 3), 7), ("bfirst:120x80", (7, 3), 7), ("blast:40x25", (3, 7), 7),
    ("radial:60x50", (3, 7), 7), ("rcm:del2000", None, None)])
def test_directions_share_a_class(pair_lib, oracle_lib, name, alone, both, b, elem):
    coords, conn = _mesh(name)
    rowptr, colind = oracle_lib.pattern(coords.shape[0], conn)
    rp, ci = np.ascontiguousarray(rowptr, np.int32), np.ascontiguousarray(colind, np.int32)
    ne = np.zeros(4, np.int32)
    rc = pair_lib.emul_strip_pair(rp.size - 1, b, elem, rp.ctypes.data, ci.ctypes.data, 0, ne.ctypes.data)
    assert rc == 0
    if alone:
        assert tuple(ne[:2]) == alone  # the case is one where the directions differ
        assert tuple(ne[2:]) == (both, both)
    assert ne[2] == ne[3] == max(ne[:2])
