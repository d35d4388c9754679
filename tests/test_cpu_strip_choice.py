"""Which strip plans are taken (k_strip.h): grids, row by row or renumbered by
their boundary, are; numberings whose strips hold a row or two per step are not
a grid's, do not serve, and are refused before their tables are built once their
records grow large.  And the mailbox's limit: a chunk that needs one item more
than it has slots is refused, one that needs them all is not."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT
from meshorder import boundary_first, radial, rcm, renumber


@pytest.fixture(scope="module")
def choice_lib():
    out = os.path.join(ROOT, "tests", "cpu", "_build")
    os.makedirs(out, exist_ok=True)
    so = os.path.join(out, "libstrip_choice_emul.so")
    srcs = [os.path.join(ROOT, "tests", "cpu", f) for f in ("strip_choice_emul.cpp", "strip_emul.cpp")]
    inc = [d for d in ("/usr/local/cuda/include",) if os.path.isdir(d)]
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", *[f"-I{d}" for d in inc], "-o", so, *srcs,
                    os.path.join(ROOT, "delfem_gb300", "csrc", "strip.cpp")], check=True)
    L = ctypes.CDLL(so)
    P = ctypes.c_void_p
    L.emul_strip_choice.argtypes = [ctypes.c_int] * 3 + [P, P] + [ctypes.c_int] * 3 + [P]
    L.emul_strip.argtypes = [ctypes.c_int] * 3 + [P, P, ctypes.c_int, ctypes.c_int, ctypes.c_int, P]
    return L


def _mesh(name):
    from delfem_gb300 import meshgen as mg
    kind, shape, *order = name.split(":")
    if kind == "del":
        coords, conn = mg.delaunay_mesh(*map(int, shape.split("d")), seed=2)
    else:
        d = list(map(int, shape.split("x")))
        coords, conn = mg.tri_grid(*d) if len(d) == 2 else mg.tet_grid(*d)
    if order:
        f = {"bfirst": boundary_first, "radial": radial, "rcm": rcm,
             "xsort": lambda c, e: np.argsort(c[:, 0] + 1e-9 * c[:, 1], kind="stable"),
             "random": lambda c, e: np.random.default_rng(1).permutation(c.shape[0])}[order[0]]
        coords, conn = renumber(coords, conn, f(coords, conn))
    return coords.shape[0], conn


def _choices(L, O, name, suited):
    n, conn = _mesh(name)
    rowptr, colind = O.pattern(n, conn)
    rp, ci = np.ascontiguousarray(rowptr, np.int32), np.ascontiguousarray(colind, np.int32)
    out = []
    for b in (1, conn.shape[1] - 1):
        for elem in (4, 8):
            for forward in (1, 0):
                chain = np.zeros(2, np.int64)
                out.append(L.emul_strip_choice(n, b, elem, rp.ctypes.data, ci.ctypes.data, forward,
                                               int(elem == 8 and b > 1), suited, chain.ctypes.data))
                assert out[-1] < 0 or chain[0] == chain[1]
    return out


@pytest.mark.parametrize("name", [
    "grid:1x1", "grid:24x24", "grid:300x20", "grid:20x300", "grid:2x3000", "grid:301x257", "grid:3x3x3", "grid:8x8x8",
    "grid:44x8x8", "grid:8x44x8", "grid:8x8x44", "grid:8x44x44", "grid:3x30x30", "grid:4x60x60", "grid:56x56x20",
    "grid:128x128:bfirst", "grid:60x50:rcm"])
def test_grids_are_swept_in_strips(choice_lib, oracle_lib, name):
    assert set(_choices(choice_lib, oracle_lib, name, 1)) == {3}


@pytest.mark.parametrize("name", ["grid:100x100:radial", "del:20000d2:xsort", "del:20000d2", "grid:100x100:random",
                                  "grid:20x20x20:random", "del:20000d2:rcm"])
def test_scattered_numberings_are_not_a_grids(choice_lib, oracle_lib, name):
    assert set(_choices(choice_lib, oracle_lib, name, 0)) <= {0, -1, -2}


@pytest.mark.parametrize("name", ["grid:140x140:radial", "del:20000d2:xsort"])
def test_records_far_beyond_the_factor_are_refused(choice_lib, oracle_lib, name):
    assert set(_choices(choice_lib, oracle_lib, name, 1)[:4]) == {-1}  # 1x1: a row or two in 256 places


@pytest.mark.parametrize("deps,want", [(8, 0), (9, -1)])
def test_mailbox_limit(choice_lib, deps, want):
    """A strip of steps of 32 rows, each row needing `deps` rows of other strips that
    no other row needs, and the row of its lane in the step before: a chunk of four
    steps (1x1 FP32, up to 16 entries) needs 128 * deps items, the mailbox has 1,024
    slots."""
    src = 256 * deps
    rows = [[] for _ in range(src)]
    for i in range(256):  # two chunks
        rows.append(list(range(i * deps, (i + 1) * deps)) + ([src + i - 32] if i >= 32 else []))
    rp = np.cumsum([0] + [len(r) for r in rows]).astype(np.int32)
    ci = np.array([c for r in rows for c in r], np.int32)
    for eager in (0, 1):
        info = np.zeros(4, np.int64)
        assert choice_lib.emul_strip(rp.size - 1, 1, 4, rp.ctypes.data, ci.ctypes.data, 1, eager, 0,
                                     info.ctypes.data) == want
