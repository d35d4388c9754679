"""FP32 sweeps of 3x3 blocks: the strips and one CTA per sweep are as exact as the
level-scheduled kernel, which adds a row's entries up over its lanes.  After one
iteration from zero the solution is alpha times the preconditioned residual, so its
direction against FP64's is the sweeps' error.  Roundings at the size of the row's
sum (products of one size): the lanes' tree has 2 inside its entries, 3 or 4 above
and the subtraction; four sums of two to four entries have 2.6 to 6.5, 2 above and
the subtraction: up to sqrt(9.5 / 7) = 1.17 of the error, 1.3 leaves room for chance."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,fill", [((13, 10, 8), 0), ((20, 21, 19), 0), ((9, 8, 10), 1)])
def test_fp32_sweeps_of_3x3_blocks(gpu_ctx, shape, fill):
    from delfem_gb300 import linsys as L
    from delfem_gb300 import meshgen as mg
    from delfem_gb300.solver import FESolve
    err = {1: 0.0, 2: 0.0, 3: 0.0}
    for seed in range(3):
        p = mg.box_problem_3d(mg.SOLID3D, *shape, seed=seed)
        for mode in err:
            s = FESolve(gpu_ctx, p, fill_level=fill, sweep_mode=mode)
            try:
                s.assemble()
                assert s.factor()
                L.Solve_PCG(1e-30, 1, s.ls, s.prec)
                x = s.solution()
                s.assemble()
                L.Solve_PCG_ex(1e-30, 1, s.ls, s.prec, "fp32f", False)
                y = s.solution()
            finally:
                s.close()
            err[mode] += float(np.linalg.norm(y - (y @ x) / (x @ x) * x) / np.linalg.norm(x))
    print("FP32 sweep error: strips %.3g, levels %.3g, one CTA %.3g" % (err[1] / 3, err[2] / 3, err[3] / 3))
    assert err[1] <= 1.3 * err[2] and err[3] <= 1.3 * err[2]
