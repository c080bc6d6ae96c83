"""The batched correction (k_batch_correct, which marches a row per warp up chunks of eight planes)
on boxes whose rows, columns and planes leave remainders of a warp, of the warps of an item and of
a chunk: every problem against its single-problem solve.  Both end at a residual of 1e-10, which
on these boxes leaves at most 5e-10; the bound is twenty times that."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import peps_mg_gb300 as pmg  # noqa: E402
from peps_mg_gb300.batch import BatchSolver  # noqa: E402
from tests.helpers import from_dev, rel  # noqa: E402


@pytest.mark.parametrize("dims", [[(34, 20, 10), (66, 12, 22), (30, 6, 44), (32, 8, 8)],
                                  [(8, 14, 34), (64, 30, 16), (36, 8, 18)], [(62, 12, 6)]], ids=str)
@pytest.mark.parametrize("omega", [1.0, 1.1])
def test_uneven_rows_and_planes(dims, omega):
    rng = np.random.Generator(np.random.PCG64(sum(map(sum, dims))))
    with BatchSolver(np.array(dims)) as bs:
        rhs, sol = bs.field(), bs.field()
        for p, (nx, ny, nz) in enumerate(dims):
            bs.view(rhs, p)[1:-1, 1:-1, 1:-1] = torch.from_numpy(rng.uniform(-1, 1, (nz, ny, nx))).cuda()
        cycles, ratio, _ = bs.solve(sol, rhs, 2, 1e-10, omega, max_cycles=60)
        assert np.all(ratio < 1e-10)
        for p in range(bs.n):
            with pmg.Multigrid(bs.mesh(p), int(bs.levels[p]), 60, "cgs", precision="mixed") as mg:
                s1 = torch.zeros_like(bs.view(rhs, p))
                r1 = torch.zeros_like(s1)
                mg.solve_vcycle(s1, r1, bs.view(rhs, p).contiguous(), 2, 1e-10, omega)
            assert rel(from_dev(bs.view(sol, p)), from_dev(s1)) < 1e-8
