"""Served requests on meshes that are not numbered row by row, beside natural
grids of the same block sizes: a request's widest lower and widest upper row lie
in different entry classes (boundary first 7 and 3, distance from the centre 3
and 7).  Every sweep kernel evaluates a row in the same order, so the default
choice gives the bits and iteration counts of one CTA per solve."""
import numpy as np
import pytest

from meshorder import boundary_first, radial, rcm, renumber

pytestmark = pytest.mark.gpu


def _problems():
    from delfem_gb300 import meshgen as mg
    out = []
    for kind in (mg.POISSON2D, mg.SOLID2D):
        for order in (None, boundary_first, lambda c, e: boundary_first(c, e)[::-1]):
            coords, conn = mg.tri_grid(90, 70, 1.2, 1.0, 0.2, np.random.default_rng(5))
            if order:
                coords, conn = renumber(coords, conn, order(coords, conn))
            out.append(mg.mesh_problem(kind, coords, conn, seed=2, coef_sigma=0.5))
        coords, conn = mg.tri_grid(40, 33)
        out.append(mg.mesh_problem(kind, *renumber(coords, conn, radial(coords, conn)), seed=3, coef_sigma=0.5))
        coords, conn = mg.delaunay_mesh(2000, 2, seed=3)
        out.append(mg.mesh_problem(kind, *renumber(coords, conn, rcm(coords, conn)), seed=4, coef_sigma=0.5))
    coords, conn = mg.tet_grid(9, 8, 7)
    for order in (None, boundary_first):
        c, e = renumber(coords, conn, order(coords, conn)) if order else (coords, conn)
        out += [mg.mesh_problem(kind, c, e, seed=5, coef_sigma=0.5) for kind in (mg.POISSON3D, mg.SOLID3D)]
    return out


@pytest.mark.parametrize("mode", ["fp64", "fp32f", "mixed"])
def test_served_orders(gpu_ctx, mode):
    from delfem_gb300.serve import Server
    probs = _problems()
    got = []
    for sweeps in (0, 2):
        with Server(gpu_ctx, mode=mode, budget_bytes=2 << 30, sweeps=sweeps) as S:
            ids = [S.submit(p) for p in probs + probs[::-1]]
            got.append([S.wait(i) for i in ids])
    for a, c in zip(*got):
        assert a["status"] == 0 and a["rel_true"] <= 1e-8 and a["iterations"] == c["iterations"]
        assert np.array_equal(a["x"], c["x"])


def test_budget_that_fits_without_strips(gpu_ctx):
    """A request that fits the whole budget only in the kind that needs less memory
    than strips is served by it, with the same bits."""
    import re
    from delfem_gb300 import meshgen as mg
    from delfem_gb300.capi import DFG_OOM_REJECTED
    from delfem_gb300.serve import Server
    coords, conn = mg.tet_grid(14, 13, 12)
    coords, conn = renumber(coords, conn, boundary_first(coords, conn))
    p = mg.mesh_problem(mg.SOLID3D, coords, conn, seed=2, coef_sigma=0.5)
    need = {}
    for sweeps in (0, 2):
        with Server(gpu_ctx, budget_bytes=1 << 20, sweeps=sweeps) as S:
            r = S.wait(S.submit(p))
            assert r["status"] == DFG_OOM_REJECTED
            need[sweeps] = int(re.search(r"needs (\d+) device bytes", r["error"]).group(1))
    assert need[0] <= need[2]
    got = []
    for budget in (need[2], 1 << 30):
        with Server(gpu_ctx, budget_bytes=budget) as S:
            got.append(S.wait(S.submit(p)))
    assert got[0]["status"] == 0 and got[0]["iterations"] == got[1]["iterations"]
    assert np.array_equal(got[0]["x"], got[1]["x"])
