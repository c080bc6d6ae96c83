"""The host scan of the initial guess, shared out over threads from 8 MB on: a guess that is zero
but for one value (the first, the last, or the neighbours of a thread's share) gives the solution
of the same solve from device arrays, bit for bit, in arrays of one share, of two and of many."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import peps_mg_gb300 as pmg  # noqa: E402
from peps_mg_gb300 import problems  # noqa: E402
from tests.helpers import from_dev, to_dev  # noqa: E402


@pytest.mark.parametrize("n", [64, 112, 160])
@pytest.mark.parametrize("where", [None, 0, 1, 2, -1])
def test_single_nonzero_value(n, where):
    mesh, rhs = problems.gaussian_blobs(n)
    size = (n + 2) ** 3
    threads = max(1, size // (1 << 19))
    share = -(-size // threads)
    at = None if where is None else {0: 0, 1: min(size, share) - 1, 2: share % size, -1: size - 1}[where]
    guess = np.zeros((n + 2,) * 3, order="F")
    if at is not None:
        guess.reshape(-1, order="F")[at] = 1.0
    assert at is None or guess.any()
    with pmg.Multigrid(mesh, 4, 30, "cgs", precision="mixed") as mg:
        sol, rsd = guess.copy(order="F"), np.zeros_like(guess, order="F")
        mg.solve_vcycle(sol, rsd, rhs, 2, 1e-10, 1.0)
        dsol, drsd = to_dev(guess), to_dev(np.zeros_like(guess))
        mg.solve_vcycle(dsol, drsd, to_dev(rhs), 2, 1e-10, 1.0)
    assert np.array_equal(sol, from_dev(dsol))
    assert np.array_equal(rsd, from_dev(drsd))
