"""Single solves on meshes that are not numbered row by row: whatever kind of sweep
the set-up chooses, per precision, the preconditioner meets the oracle's to 1e-12
and the solves its solution to 1e-6 (the FP32 forms a true residual of 1e-8); and a numbering that strips do not suit takes no more than a small
multiple of the factor's memory (10 times, with both precisions, the older kinds'
included; strips of this mesh would take 600 times)."""
import numpy as np
import pytest

from meshorder import boundary_first, radial, rcm, renumber
from test_zz_memory import _free_bytes

pytestmark = pytest.mark.gpu


def _mesh(dim, n, order):
    from delfem_gb300 import meshgen as mg
    coords, conn = mg.delaunay_mesh(n, dim, seed=4)
    if order == "xsort":
        return renumber(coords, conn, np.argsort(coords[:, 0], kind="stable"))
    if order != "random":
        return renumber(coords, conn, {"bfirst": boundary_first, "radial": radial, "rcm": rcm}[order](coords, conn))
    return coords, conn


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("dim,b,order", [(2, 1, "xsort"), (2, 2, "rcm"), (2, 2, "radial"), (2, 1, "random"),
                                         (3, 1, "rcm"), (3, 3, "xsort"), (2, 2, "bfirst")])
def test_single_solves(gpu_ctx, oracle_lib, dim, b, order, mode):
    from delfem_gb300 import meshgen as mg
    from delfem_gb300.capi import DfgError
    from delfem_gb300.solver import FESolve
    kind = {(2, 1): mg.POISSON2D, (2, 2): mg.SOLID2D, (3, 1): mg.POISSON3D, (3, 3): mg.SOLID3D}[dim, b]
    p = mg.mesh_problem(kind, *_mesh(dim, 1500, order), seed=2, coef_sigma=0.5)
    ref = oracle_lib.solve(p)
    s = FESolve(gpu_ctx, p, sweep_mode=mode)
    try:
        s.assemble()
        assert s.factor()
        rp, ci = s.prec.GetPattern()
        fd, fo = s.prec.GetFactor()
        rhs = np.random.default_rng(3).standard_normal(p.nnode * b)
        s.ls.ReSizeTmpVecSolver(1)
        s.ls.SetVector(0, rhs)
        if mode == 1 and b == 3:  # rows of 37 entries: the ranged kind refuses them, strips as well
            with pytest.raises(DfgError, match="shared memory"):
                s.prec.SolvePrecond(s.ls, 0)
            return
        s.prec.SolvePrecond(s.ls, 0)
        z = oracle_lib.precond(p.nnode, b, rp, ci, oracle_lib.diaind(rp, ci), fd, fo, rhs)
        np.testing.assert_allclose(s.ls.GetVector(0), z, rtol=1e-12, atol=1e-13 * np.abs(z).max())
        for form in ("fp64", "fp32f", "mixed"):
            r = s.run(form, target_true=form != "fp64")
            assert r["converged"]
            if form != "fp64":
                assert s.ls.true_residual() <= 1e-8
            assert np.linalg.norm(s.solution() - ref["x"]) <= 1e-6 * np.linalg.norm(ref["x"])
    finally:
        s.close()


def test_memory_of_an_unsuited_numbering(gpu_ctx):
    from delfem_gb300 import meshgen as mg
    from delfem_gb300.solver import FESolve
    p = mg.mesh_problem(mg.POISSON2D, *_mesh(2, 20000, "xsort"), seed=2)
    FESolve(gpu_ctx, p, sweep_mode=2).close()  # what the first use of the library allocates
    before = _free_bytes()
    s = FESolve(gpu_ctx, p)
    try:
        s.assemble()
        assert s.factor()
        s.solve("fp32f", maxit=2)
        used = before - _free_bytes()
        rp, ci = s.prec.GetPattern()
        assert used <= 10 * 20 * (ci.size + p.nnode) + (64 << 20)  # value in FP64 and FP32, index, position
    finally:
        s.close()
