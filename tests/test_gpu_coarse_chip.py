"""The on-chip RBGS coarsest-level solver (coarse_rbgs_chip in pmg_tail64.cuh) at the edges of
its range: FP64 solves against the oracle, bit for bit, with the oracle's coarsest iteration
counts; mixed solves (whose solver takes the norm from the sweeps) within 1e-8,
twenty times the 5e-10 that a residual of 1e-10 leaves on these boxes."""
import numpy as np
import pytest

import peps_mg_gb300 as pmg
from oracle import oracle as O
from peps_mg_gb300 import geometry as G
from tests.helpers import from_dev, rel, to_dev

pytestmark = pytest.mark.gpu

# coarsest levels: a single cell, one warp, odd and flat boxes, 64 and 65+ cells, several norm
# cells per thread, the largest held on chip (1000 stored values) and one beyond it
COARSEST = [(1, 1, 1), (2, 2, 2), (1, 3, 5), (4, 4, 4), (5, 13, 1), (7, 5, 3), (5, 10, 9), (8, 8, 8), (9, 8, 8)]


def problem(coarsest, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    n = [4 * m for m in coarsest]
    mesh = [G.mesh_from_widths(rng.uniform(0.8, 1.2, m) / max(n)) for m in n]
    rhs = G.field(*n)
    rhs[1:-1, 1:-1, 1:-1] = rng.uniform(-1.0, 1.0, n)
    return n, mesh, np.asfortranarray(rhs)


@pytest.mark.parametrize("omega", [1.0, 1.2])
@pytest.mark.parametrize("coarsest", COARSEST, ids=str)
def test_coarsest_solver(coarsest, omega):
    n, mesh, rhs = problem(coarsest, 40 + sum(coarsest))
    omg = O.OracleMG(mesh, 2, 30, method=0)
    osol, orsd = G.field(*n), G.field(*n)
    ncyc, _, ci = omg.solve(osol, orsd, rhs, 2, 1e-10, omega)
    omg.close()
    for precision in ("fp64", "mixed"):
        sol, rsd, b = to_dev(G.field(*n)), to_dev(G.field(*n)), to_dev(rhs)
        with pmg.Multigrid(mesh, 2, 30, "cgs", precision=precision) as mg:
            rep = mg.solve_vcycle(sol, rsd, b, 2, 1e-10, omega)
        assert rep.converged
        if precision == "fp64":
            assert rep.cycles == ncyc
            assert np.array_equal(rep.coarse_iterations, ci[:ncyc])
            assert np.array_equal(from_dev(sol), osol)
        else:
            assert rel(from_dev(sol), osol) < 1e-8
