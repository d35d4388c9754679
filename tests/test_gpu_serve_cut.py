"""The server's product and vector kernels cut chunks into runs of rows when few
solves are in flight (k_serve.cu, cut_shift): in eight, in four, or not at all.
The sums keep an uncut chunk's order, so a request gives the same bits with any
number of others; its rows end inside a run and inside a chunk."""
import numpy as np
import pytest

from conftest import bits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["fp64", "fp32f", "mixed"])
def test_cut_chunks_same_bits(gpu_ctx, mode):
    from delfem_gb300 import meshgen as mg
    from delfem_gb300.serve import Server
    for p in (mg.poisson2d_square(220, seed=3), mg.solid2d_cantilever(400, 121, seed=4)):  # 24 chunks of 2,048 rows each
        got = []
        for n in (1, 6, 10):
            with Server(gpu_ctx, mode=mode, tol=1e-4, budget_bytes=4 << 30) as S:
                ids = [S.submit(p) for _ in range(n)]
                got.append([S.wait(i) for i in ids])
        first = got[0][0]
        assert first["status"] == 0
        for r in (r for rs in got for r in rs):
            assert r["status"] == 0 and r["iterations"] == first["iterations"]
            assert np.array_equal(bits(r["x"]), bits(first["x"]))
