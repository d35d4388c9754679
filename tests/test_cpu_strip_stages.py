"""The chunk stages of a strip whose warps give up half-way (k_strip.h,
strip_publishes): no stage is issued again while its copy is in flight, and the
launch waits for every copy that it issued."""
import ctypes
import os
import subprocess

import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def stages_lib():
    out = os.path.join(ROOT, "tests", "cpu", "_build")
    os.makedirs(out, exist_ok=True)
    so = os.path.join(out, "libstrip_stages_emul.so")
    inc = [d for d in ("/usr/local/cuda/include",) if os.path.isdir(d)]
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", *[f"-I{d}" for d in inc], "-o", so,
                    os.path.join(ROOT, "tests", "cpu", "strip_stages_emul.cpp")], check=True)
    return ctypes.CDLL(so)


@pytest.mark.parametrize("slow", [0, 1])
@pytest.mark.parametrize("nch,CH,NS", [(1, 2, 2), (3, 2, 2), (9, 2, 3), (20, 4, 8), (17, 8, 3)])
def test_copies_of_a_strip_that_gives_up(stages_lib, nch, CH, NS, slow):
    for fail in range(nch + 1):
        for seed in range(50):
            assert stages_lib.emul_strip_stages(nch, CH, NS, fail, slow, seed) == 0, (fail, seed)
