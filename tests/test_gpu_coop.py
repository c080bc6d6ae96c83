"""The cooperative launch of the small FP64 levels (pmg_coop64.cu) against the oracle, bit for
bit: whole solves whose finest level is inside it (the norm too), on its limit or above, with
one to three sweeps, stride-1 transfers, stretched meshes and Dirichlet faces; and smoother
calls on boxes beside the limit of the one-launch sweeps, also captured in graphs."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import peps_mg_gb300 as pmg  # noqa: E402
from oracle import oracle as O  # noqa: E402
from peps_mg_gb300 import geometry as G  # noqa: E402
from tests.helpers import from_dev, to_dev  # noqa: E402


def box(n, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    mesh = [G.mesh_from_widths(rng.uniform(0.8, 1.2, m) / max(n)) for m in n]
    rhs, sol = G.field(*n), G.field(*n)
    rhs[1:-1, 1:-1, 1:-1] = rng.uniform(-1.0, 1.0, n)
    sol[:, 0, :], sol[-1, :, :] = 0.25, -0.5
    return mesh, np.asfortranarray(rhs), np.asfortranarray(sol)


# finest level on one CTA, in the grid phases, at the limit of 2^15 cells, above it; the last two
# stop halving an axis
@pytest.mark.parametrize("n,levels", [((16, 8, 8), 2), ((16, 16, 24), 3), ((32, 32, 32), 4), ((40, 32, 32), 4),
                                      ((64, 48, 20), 4), ((28, 12, 44), 2)], ids=str)
@pytest.mark.parametrize("maxit,omega", [(1, 1.0), (2, 1.15), (3, 1.0)])
def test_solve(n, levels, maxit, omega):
    mesh, rhs, sol0 = box(n, 60 + sum(n))
    omg = O.OracleMG(mesh, levels, 25, method=0)
    want, wrsd = sol0.copy(order="F"), G.field(*n)
    ncyc, hist, ci = omg.solve(want, wrsd, rhs, maxit, 1e-9, omega)
    omg.close()
    sol, rsd = to_dev(sol0), to_dev(G.field(*n))
    with pmg.Multigrid(mesh, levels, 25, "cgs") as mg:
        rep = mg.solve_vcycle(sol, rsd, to_dev(rhs), maxit, 1e-9, omega)
    assert rep.cycles == ncyc
    assert np.array_equal(rep.coarse_iterations, ci[:ncyc])
    assert np.array_equal(from_dev(sol), want)
    assert np.array_equal(from_dev(rsd), wrsd)
    assert np.allclose(rep.history, hist[:ncyc], rtol=1e-12, atol=0.0)


@pytest.mark.parametrize("n", [(4, 4, 4), (48, 7, 3), (52, 51, 49), (52, 51, 50)], ids=str)
@pytest.mark.parametrize("iters,omega", [(2, 1.0), (3, 1.4)])
def test_sweeps(n, iters, omega):
    mesh, rhs, sol0 = box(n, 90 + sum(n))
    want = sol0.copy(order="F")
    O.rbgs_iterator(O.matrix_create(mesh), want, rhs, iters, omega)
    x = to_dev(sol0)
    with pmg.Multigrid(mesh, 2, 1) as mg:
        mg.rbgs_iterator(0, x, to_dev(rhs), iters, omega)
        mg.sync()
    assert np.array_equal(from_dev(x), want)


def test_sweeps_captured():
    """Two graphs of a context's sweeps, replayed at once on two streams."""
    n = (32, 24, 16)
    mesh, rhs, sol0 = box(n, 5)
    coeff = O.matrix_create(mesh)
    streams = [torch.cuda.Stream() for _ in range(3)]
    b, xs, wants, graphs = to_dev(rhs), [], [], []
    with pmg.Multigrid(mesh, 2, 1, stream=streams[0].cuda_stream) as mg:
        for iters in (2, 5):
            x, g = to_dev(sol0), torch.cuda.CUDAGraph()
            torch.cuda.synchronize()
            with torch.cuda.graph(g, stream=streams[0]):
                mg.rbgs_iterator(0, x, b, iters, 1.0)
            want = sol0.copy(order="F")
            O.rbgs_iterator(coeff, want, rhs, 3 * iters, 1.0)
            xs, wants, graphs = xs + [x], wants + [want], graphs + [g]
        torch.cuda.synchronize()
        for _ in range(3):
            for g, s in zip(graphs, streams[1:]):
                with torch.cuda.stream(s):
                    g.replay()
        torch.cuda.synchronize()
        mg.sync()
    for x, want in zip(xs, wants):
        assert np.array_equal(from_dev(x), want)
