"""Strip-sweep plans (delfem_gb300/csrc/strip.cpp), executed with row numbers in
place of values by tests/cpu/strip_emul.cpp: each row once, every reference to
its dependency's row, no item a step needs held back by the mailbox's flow
control, for meshes at the edges of strips and of the mailbox."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def strip_lib():
    out = os.path.join(ROOT, "tests", "cpu", "_build")
    os.makedirs(out, exist_ok=True)
    so = os.path.join(out, "libstrip_emul.so")
    srcs = [os.path.join(ROOT, "tests", "cpu", "strip_emul.cpp"),
            os.path.join(ROOT, "delfem_gb300", "csrc", "strip.cpp")]
    inc = [d for d in ("/usr/local/cuda/include",) if os.path.isdir(d)]
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", *[f"-I{d}" for d in inc], "-o", so, *srcs],
                   check=True)
    L = ctypes.CDLL(so)
    P = ctypes.c_void_p
    L.emul_strip.argtypes = [ctypes.c_int] * 3 + [P, P, ctypes.c_int, ctypes.c_int, ctypes.c_int, P]
    return L


def _run(L, rowptr, colind, b, elem, forward, eager, split=0):
    info = np.zeros(4, np.int64)
    ci = np.ascontiguousarray(colind if colind.size else np.zeros(1), np.int32)
    rp = np.ascontiguousarray(rowptr, np.int32)
    rc = L.emul_strip(rp.size - 1, b, elem, rp.ctypes.data, ci.ctypes.data, forward, eager, split, info.ctypes.data)
    return rc, info


def _pattern(name):
    from delfem_gb300 import meshgen as mg
    import oracle as O
    if name.startswith("tri"):
        nx, ny = map(int, name[3:].split("x"))
        coords, conn = mg.tri_grid(nx, ny)
    elif name.startswith("tet"):
        coords, conn = mg.tet_grid(*map(int, name[3:].split("x")))
    else:  # a chain, a diagonal, a band of 16 entries, a band reaching 40 rows back
        n = 700
        off = {"chain": [1], "diag": [], "wide": list(range(1, 17)), "far": [1, 40], "older": [1, 300]}[name]
        rows = [sorted([i - o for o in off if i >= o] + [i + o for o in off if i + o < n]) for i in range(n)]
        return (np.cumsum([0] + [len(r) for r in rows]), np.array([c for r in rows for c in r], np.int32))
    return O.pattern(coords.shape[0], conn)


@pytest.mark.parametrize("elem", [4, 8])
@pytest.mark.parametrize("b", [1, 2, 3])
@pytest.mark.parametrize("name", ["tri1x1", "tri31x31", "tri32x33", "tri40x65", "tri3x200", "tri1500x20", "tet5x4x3",
                                  "tet16x15x9", "tet33x32x4", "chain", "diag", "wide", "far", "older"])
def test_strip_plan(strip_lib, oracle_lib, name, b, elem):
    rowptr, colind = _pattern(name)
    for forward in (1, 0):
        for eager in (0, 1):
            for split in (0, 1) if b > 1 and elem == 8 else (0,):
                rc, info = _run(strip_lib, rowptr, colind, b, elem, forward, eager, split)
                assert rc == 0, (rc, info, split)


def test_strip_plan_steps_are_levels_of_a_grid(strip_lib, oracle_lib):
    """32 lines of a triangle grid are one strip whose steps are its levels."""
    rowptr, colind = _pattern("tri60x31")
    rc, info = _run(strip_lib, rowptr, colind, 1, 4, 1, 0)
    assert rc == 0 and tuple(info[:4]) == (1, 61 + 31, 0, 0)


def test_strip_plan_refuses_wide_rows_and_scattered_orders(strip_lib):
    n = 40
    full = np.array([c for i in range(n) for c in range(n) if c != i], np.int32)
    assert _run(strip_lib, np.arange(n + 1) * (n - 1), full, 1, 4, 1, 0)[0] == -1
    rng = np.random.default_rng(0)  # 8 dependencies anywhere: more items per chunk than a mailbox
    n = 20000
    a = np.concatenate([np.repeat(np.arange(n), 8), rng.integers(0, n, 8 * n)])
    c = np.concatenate([a[8 * n:], a[: 8 * n]])
    keep = a != c
    key = np.unique(a[keep].astype(np.int64) * n + c[keep])
    a, c = key // n, key % n
    low = a > c
    # rows of at most 16 lower entries
    cnt = np.bincount(a[low], minlength=n)
    ok = (cnt[a] <= 16) & (cnt[c] <= 16)
    a, c = a[ok], c[ok]
    rc, _ = _run(strip_lib, np.concatenate([[0], np.cumsum(np.bincount(a, minlength=n))]), c.astype(np.int32), 1, 4, 1, 0)
    assert rc in (0, -1)
