"""The strip sweeps (k_strip.cu; dfg_precond_set_sweep_mode 1) at the sizes
where their plan can go wrong: one line and one line more than a strip, more
items than a mailbox has slots, more strips than the device has CTAs, and every
entry class.  A row is evaluated in the one-CTA kernel's order, so both kinds
give the same bits, in FP64 and (through a few FP32-factor iterations) in FP32;
the FP64 preconditioner also meets the oracle's to 1e-12.  2x2 and 3x3 blocks in FP64 are
summed by columns: there FP64 agrees to rounding (1e-12 through the oracle, a few
iterations to 1e-10), and the error against sums in a wider type is the one-CTA kernel's,
but for the one rounding more of a row's two halves (its 6 operations or more
make that 1/6 at most, and 1.5 leaves room for chance)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problem(name):
    from delfem_gb300 import meshgen as mg
    kind, grid = name.split(":")
    d = [int(v) for v in grid.split("x")]
    if kind == "solid2d":
        return mg.solid2d_cantilever(*d, seed=5)
    if kind == "poisson2d":
        rng = np.random.default_rng(6)
        coords, conn = mg.tri_grid(*d, d[0] / d[1], 1.0, 0.2, rng)
        bc = (coords[:, 0] == 0.0).astype(np.int32)
        prm = np.zeros(8)
        prm[:2] = 1.0, 1.0
        return mg.Problem(mg.POISSON2D, coords, conn, prm, bc, coef=np.exp(rng.standard_normal(conn.shape[0])))
    return mg.box_problem_3d(mg.SOLID3D if kind == "solid3d" else mg.POISSON3D, *d, seed=7)


@pytest.mark.parametrize("name,fill", [
    ("poisson2d:31x31", 0), ("poisson2d:33x32", 0), ("poisson2d:1500x40", 0), ("poisson2d:2x20000", 0),
    ("poisson2d:50x47", 1), ("solid2d:16x15", 0), ("solid2d:700x33", 0), ("solid2d:30x70", 1), ("solid2d:41x300", 0),
    ("poisson3d:12x31x9", 0), ("poisson3d:9x8x7", 1), ("solid3d:11x9x8", 0), ("solid3d:10x20x3", 0),
    ("solid3d:5x6x4", 1)])
def test_strip_sweeps(gpu_ctx, oracle_lib, name, fill):
    from delfem_gb300 import linsys as L
    from delfem_gb300.solver import FESolve
    p = _problem(name)
    n, b = p.nnode, p.b
    rhs = np.random.default_rng(3).standard_normal(n * b)
    got = {}
    for mode in (1, 3):
        s = FESolve(gpu_ctx, p, fill_level=fill, sweep_mode=mode)
        try:
            s.assemble()
            assert s.factor()
            s.ls.ReSizeTmpVecSolver(1)
            s.ls.SetVector(0, rhs)
            s.prec.SolvePrecond(s.ls, 0)
            z = s.ls.GetVector(0)
            if mode == 1:
                rp, ci = s.prec.GetPattern()
                fd, fo = s.prec.GetFactor()
                zref = oracle_lib.precond(n, b, rp, ci, oracle_lib.diaind(rp, ci), fd, fo, rhs)
                np.testing.assert_allclose(z, zref, rtol=1e-12, atol=1e-13 * np.abs(zref).max())
            L.Solve_PCG_ex(1e-30, 6, s.ls, s.prec, "fp32f", False)
            x32 = s.solution()
            s.assemble()
            L.Solve_PCG(1e-30, 6, s.ls, s.prec)
            got[mode] = (z, x32, s.solution())
        finally:
            s.close()
    if b > 1:
        (z, x32, x64), (z3, y32, y64) = got[1], got[3]
        assert np.array_equal(x32, y32)
        assert np.linalg.norm(x64 - y64) <= 1e-10 * np.linalg.norm(y64)
        np.testing.assert_allclose(z3, zref, rtol=1e-12, atol=1e-13 * np.abs(zref).max())
        return
    for a, c in zip(got[1], got[3]):
        assert np.array_equal(a, c)


def _substitute_wide(rp, ci, fd, fo, rhs):
    n, z = fd.shape[0], rhs.reshape(fd.shape[0], -1).astype(np.longdouble)
    for i in range(n):  # L y = r, D^-1 applied
        for c in range(rp[i], rp[i + 1]):
            if ci[c] < i:
                z[i] -= fo[c].astype(np.longdouble) @ z[ci[c]]
        z[i] = fd[i].astype(np.longdouble) @ z[i]
    for i in range(n - 1, -1, -1):
        for c in range(rp[i], rp[i + 1]):
            if ci[c] > i:
                z[i] -= fo[c].astype(np.longdouble) @ z[ci[c]]
    return z


@pytest.mark.parametrize("name,fill", [("solid2d:45x38", 0), ("solid2d:30x21", 1), ("solid3d:13x10x8", 0),
                                       ("solid3d:5x6x4", 1)])
def test_split_strips_are_as_exact(gpu_ctx, name, fill):
    if np.finfo(np.longdouble).nmant <= 52:
        pytest.skip("no wider type than FP64 here")
    from delfem_gb300.solver import FESolve
    p = _problem(name)
    err = {}
    for mode in (1, 3):
        s = FESolve(gpu_ctx, p, fill_level=fill, sweep_mode=mode)
        try:
            s.assemble()
            assert s.factor()
            rp, ci = s.prec.GetPattern()
            fd, fo = (np.asarray(v).reshape(-1, p.b, p.b) for v in s.prec.GetFactor())
            s.ls.ReSizeTmpVecSolver(1)
            err[mode] = 0.0
            for seed in range(3):
                rhs = np.random.default_rng(seed).standard_normal(p.nnode * p.b)
                s.ls.SetVector(0, rhs)
                s.prec.SolvePrecond(s.ls, 0)
                ref = _substitute_wide(rp, ci, fd, fo, rhs)
                err[mode] += float(np.linalg.norm(s.ls.GetVector(0).reshape(ref.shape) - ref) / np.linalg.norm(ref))
        finally:
            s.close()
    print("error against sums in a wider type: by columns %.3g, in order %.3g" % (err[1] / 3, err[3] / 3))
    assert err[1] <= 1.5 * err[3]


@pytest.mark.parametrize("mode", ["fp64", "fp32f", "mixed"])
def test_served_strips(gpu_ctx, mode):
    """The server's strip sweeps (several solves and strips per launch) against
    its one-CTA sweeps: the same bits and iteration counts."""
    from delfem_gb300.serve import Server
    probs = [_problem(n) for n in ("poisson2d:31x31", "poisson2d:20x150", "solid2d:33x12", "solid2d:40x70",
                                   "poisson3d:12x9x8", "solid3d:7x11x6")]
    got = []
    for sweeps in (0, 2):
        with Server(gpu_ctx, mode=mode, budget_bytes=512 << 20, sweeps=sweeps) as S:
            ids = [S.submit(p) for p in probs]
            got.append([S.wait(i) for i in ids])
    for a, c in zip(*got):
        assert a["status"] == 0 and a["rel_true"] <= 1e-8 and a["iterations"] == c["iterations"]
        assert np.array_equal(a["x"], c["x"])
