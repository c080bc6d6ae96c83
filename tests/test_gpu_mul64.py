"""The FP64 level kernels with products on the integer pipe (pmg_mul64.cuh), bit for bit against
the oracle: coefficients of few bits (whose products tie), of many, and beyond the integer
products' range (plain kernels); values of every kind a double can hold (zeros of both signs,
subnormal, huge, infinite, NaN, significands all ones); boxes odd, flat and larger than one
chunk of planes; omega 1 and not."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import peps_mg_gb300 as pmg  # noqa: E402
from oracle import oracle as O  # noqa: E402
from peps_mg_gb300 import geometry as G  # noqa: E402
from tests.helpers import from_dev, to_dev  # noqa: E402

SPECIAL = np.array([0.0, -0.0, 5e-324, -3e-310, 2.0 ** -1022, 1e-200, 1e-160, 1e160, -1e250, np.inf, -np.inf, np.nan,
                    1.0, -1.0, 2.0 - 2.0 ** -52, 1.0 + 2.0 ** -52, 1.5, -1.0 / 3.0, 2.0 ** -500, 2.0 ** 501])


def meshes(kind, n, rng):
    if kind == "few bits":                 # 9, 25 and 3 times powers of two
        return [G.uniform_axis(m, 0.0, m / float(k)) for m, k in zip(n, (96, 160, 48))]
    if kind == "random":
        return [G.mesh_from_widths(rng.uniform(0.5, 1.5, m) / max(n)) for m in n]
    return [G.mesh_from_widths(rng.uniform(0.5, 1.5, m) * 2.0 ** -220) for m in n]    # out of range


def values(shape, kind, rng):
    a = rng.uniform(-1.0, 1.0, shape) * 2.0 ** rng.integers(-40, 40, shape)
    if kind == "short":                    # few bits: exact ties
        a = np.round(rng.uniform(-1.0, 1.0, shape) * 2.0 ** 51) + 0.5
    if kind == "special":
        put = rng.random(shape) < 0.05
        a[put] = rng.choice(SPECIAL, int(put.sum()))
    return np.asfortranarray(a)


def same(a, b):
    """Equal bits, any NaN equal to any NaN."""
    return np.array_equal(np.isnan(a), np.isnan(b)) and np.array_equal(
        np.where(np.isnan(a), 0.0, a).view(np.uint64), np.where(np.isnan(b), 0.0, b).view(np.uint64))


@pytest.mark.parametrize("value", ["plain", "short", "special"])
@pytest.mark.parametrize("mesh", ["few bits", "random", "out of range"])
@pytest.mark.parametrize("n", [(34, 13, 36), (4, 4, 4), (68, 20, 9), (5, 3, 8)], ids=str)
def test_level_operations(n, mesh, value):
    rng = np.random.Generator(np.random.PCG64(7 + sum(n)))
    axes = meshes(mesh, n, rng)
    coeff = O.matrix_create(axes)
    shape = tuple(m + 2 for m in n)
    x, b = values(shape, value, rng), values(shape, value, rng)
    with pmg.Multigrid(axes, 2, 1) as mg:
        d = [to_dev(x), to_dev(b), torch.zeros(shape[::-1], dtype=torch.float64, device="cuda")]
        inner = (slice(1, -1),) * 3
        mg.mv_mul(0, d[2], d[0])
        assert same(from_dev(d[2])[inner], O.mv_mul(coeff, x)[inner])
        mg.residual(0, d[2], d[0], d[1])
        assert same(from_dev(d[2])[inner], O.residual(coeff, x, b)[inner])
        for omega in (1.0, 1.3):
            want = x.copy(order="F")
            O.rbgs_iterator(coeff, want, b, 2, omega)
            got = to_dev(x)
            mg.rbgs_iterator(0, got, d[1], 2, omega)
            assert same(from_dev(got), want)
        coarsest = mg.coarsest_levels()
        mc, mf = ([mg.level_mesh(l, a) for a in range(3)] for l in (1, 0))
        nc = tuple(m + 2 for m in mg.level_dims(1))
        vc = np.zeros(nc, order="F")
        O.restriction(mc, mf, 0, coarsest, x, vc)
        dc = to_dev(np.zeros(nc))
        mg.restriction(0, dc, d[0])
        assert same(from_dev(dc), vc)
        xc = values(nc, value, rng)
        vf = x.copy(order="F")
        O.prolongation(mc, mf, 0, coarsest, xc, vf)
        got = to_dev(x)
        mg.prolongation(0, got, to_dev(xc))
        assert same(from_dev(got)[inner], vf[inner])
        with np.errstate(all="ignore"):
            want = x[inner] + vf[inner]
        got = to_dev(x)
        mg.prolong_add(0, got, to_dev(xc))
        assert same(from_dev(got)[inner], want)


@pytest.mark.parametrize("nz", [4, 5, 180, 182])
def test_diagonal_of_a_column(nz):
    """The tables of the diagonal where a z axis changes its spacing now and then, within one
    chunk of planes and across two, against the oracle's sweep."""
    n = (96, 80, nz)
    rng = np.random.Generator(np.random.PCG64(nz))
    w = np.repeat(rng.uniform(0.5, 1.5, nz), rng.integers(1, 6, nz))[:nz] / nz
    axes = [G.uniform_axis(n[0], 0.0, 1.0), G.mesh_from_widths(rng.uniform(0.5, 1.5, n[1]) / n[1]),
            G.mesh_from_widths(w)]
    x, b = (np.asfortranarray(rng.uniform(-1.0, 1.0, tuple(m + 2 for m in n))) for _ in range(2))
    want = x.copy(order="F")
    O.rbgs_iterator(O.matrix_create(axes), want, b, 1, 1.0)
    with pmg.Multigrid(axes, 2, 1) as mg:
        got = to_dev(x)
        mg.rbgs_iterator(0, got, to_dev(b), 1, 1.0)
    assert same(from_dev(got), want)


@pytest.mark.parametrize("n", [(20, 12, 8), (64, 48, 40)], ids=str)
def test_without_reciprocals(n, monkeypatch):
    """Contexts whose levels are too large for the table of reciprocals: the same bits."""
    rng = np.random.Generator(np.random.PCG64(3))
    axes = meshes("random", n, rng)
    rhs = G.field(*n)
    rhs[1:-1, 1:-1, 1:-1] = rng.uniform(-1.0, 1.0, n)
    out = []
    for value in ("1", "0"):
        monkeypatch.setenv("PEPS_MG_RECIPROCALS", value)
        with pmg.Multigrid(axes, 2, 20) as mg:
            sol, rsd, x = (to_dev(G.field(*n)) for _ in range(3))
            rep = mg.solve_vcycle(sol, rsd, to_dev(rhs), 2, 1e-9, 1.1)
            mg.rbgs_iterator(0, x, to_dev(rhs), 2, 1.0)
        out.append((from_dev(sol), from_dev(rsd), from_dev(x), rep.cycles, list(rep.coarse_iterations)))
    assert out[0][3:] == out[1][3:]
    for a, b in zip(out[0][:3], out[1][:3]):
        assert same(a, b)
