"""The one-launch ILU factorisation (k_ilu.cu): levels that end inside a unit
of rows, single-row levels, rows as wide as its shared memory takes and wider
(the launch per level), and fill-in; the factor bit-identical to the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _fan(k):
    """k triangles around a hub, node 0 (or, turned round, the last node): its row
    holds every other node."""
    a = 2.0 * np.pi * np.arange(k) / k
    coords = np.vstack([[0.0, 0.0], np.stack([np.cos(a), np.sin(a)], axis=1)])
    i = np.arange(k)
    return coords, np.stack([np.zeros(k, int), 1 + i, 1 + (i + 1) % k], axis=1).astype(np.int32)


def _problem(name):
    from delfem_gb300 import meshgen as mg
    kind, shape = name.split(":")
    kinds = {"poisson2d": mg.POISSON2D, "solid2d": mg.SOLID2D, "poisson3d": mg.POISSON3D, "solid3d": mg.SOLID3D}
    if shape.startswith("fan"):
        coords, conn = _fan(int(shape[3:].rstrip("r")))
        if shape.endswith("r"):  # the hub last
            n = coords.shape[0]
            coords, conn = coords[::-1].copy(), (n - 1 - conn).astype(np.int32)
    else:
        d = [int(v) for v in shape.split("x")]
        coords, conn = mg.tri_grid(*d, jitter=0.2) if len(d) == 2 else mg.tet_grid(*d)
    return mg.mesh_problem(kinds[kind], coords, conn, seed=4, coef_sigma=0.7)


@pytest.mark.parametrize("name,fill", [
    ("poisson2d:4x3", 0), ("poisson2d:8x31", 0), ("poisson2d:33x9", 2), ("solid2d:2x40", 0), ("solid2d:17x16", 0),
    ("solid2d:13x5", -1), ("poisson3d:5x4x6", 0), ("solid3d:4x5x3", 0), ("solid3d:3x3x4", 1), ("poisson2d:fan40", 0),
    ("solid2d:fan40r", 0), ("solid2d:30x10", -1)])
def test_factor_bits(gpu_ctx, oracle_lib, name, fill):
    from delfem_gb300.solver import FESolve
    p = _problem(name)
    ref = oracle_lib.solve(p, stop_after_ilu=True, fill_level=fill)
    s = FESolve(gpu_ctx, p, fill_level=fill)
    try:
        s.assemble()
        for _ in range(2):  # the second factorisation works in used storage
            assert s.factor()
            fdiag, foffd = s.prec.GetFactor()
            assert np.array_equal(fdiag.view(np.uint64), ref["fdiag"].view(np.uint64))
            assert np.array_equal(foffd.view(np.uint64), ref["foffd"].view(np.uint64))
    finally:
        s.close()
