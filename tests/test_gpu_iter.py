"""The fused PCG iteration (k_iter.cu) at the sizes where its grid changes:
fewer rows than a warp, the last slice partly filled, the largest system of one
cluster and the smallest of the grid, one row slice more than
eight per SM (blocks of 1024 threads), in all three forms and block sizes,
against the oracle: FP64 iterations within +-2 and the solution to 1e-6, the
FP32 forms to a true residual of 1e-8; the same bits when run again."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problem(name):
    from delfem_gb300 import meshgen as mg
    return {"p3": lambda: mg.poisson2d_square(3, seed=1), "p31": lambda: mg.poisson2d_square(31, seed=2),
            "p77": lambda: mg.poisson2d_square(77, seed=7), "p78": lambda: mg.poisson2d_square(78, seed=8),
            "s20x7": lambda: mg.solid2d_cantilever(20, 7, seed=3), "c5": lambda: mg.solid3d_cube(5, seed=4),
            "p196": lambda: mg.poisson2d_square(196, seed=5), "p198": lambda: mg.poisson2d_square(198, seed=6)}[name]()


@pytest.mark.parametrize("name", ["p3", "p31", "s20x7", "c5", "p77", "p78", "p196", "p198"])
def test_fused_iteration(gpu_ctx, oracle_lib, name):
    from delfem_gb300.solver import FESolve
    p = _problem(name)
    ref = oracle_lib.solve(p)
    s = FESolve(gpu_ctx, p)
    try:
        for mode in ("fp64", "fp32f", "mixed"):
            r = s.run(mode, target_true=mode != "fp64")
            x = s.solution()
            assert r["converged"]
            if mode == "fp64":
                assert abs(r["iter"] - ref["iter"]) <= 2
            else:
                assert s.ls.true_residual() <= 1e-8
            assert np.linalg.norm(x - ref["x"]) <= 1e-6 * np.linalg.norm(ref["x"])
            again = s.run(mode, target_true=mode != "fp64")
            assert again["iter"] == r["iter"] and np.array_equal(s.solution(), x)
    finally:
        s.close()
