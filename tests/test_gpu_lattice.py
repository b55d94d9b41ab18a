"""The clustered sweep by box and, on large lattices, by octant, against the exact
build: the fast build's per-step rate tolerance 1e-5 of each field's largest
magnitude.  The spacings put 8 to 125 particles in a cell: whole octants alone
and joined, octants too full, and two passes of staging; the walls, corners, free
surface and probes of a dam break; holes that empty octants; and the lattice left
a little and far."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from aquagpusph_gb300 import case as cases


def run(c, fast, steps=1):
    from aquagpusph_gb300.solver import Solver
    sv = Solver(c.params, capacity=c.N)
    sv.set_precision(fast)
    sv.set_case(c)
    sv.step(steps, graph=True)
    sv.check()
    g = sv.get_case()
    sv.close()
    return g


def state(dx, tank, block, hfac, jitter, hole):
    c = cases.dam_break_3d(dx=dx, tank=tank, block=block, probes_z=(0.02, 0.1), hfac=hfac)
    rng = np.random.default_rng(int(100 * hfac + 10 * jitter))
    fl = np.flatnonzero(c.imove == 1)
    c.u[fl, :3] = rng.normal(0, 0.5, (len(fl), 3))
    c.dudt[fl, :3] = rng.normal(0, 2.0, (len(fl), 3))
    c.rho[fl] *= 1 + 1e-3 * rng.normal(size=len(fl))
    c.r[fl, :3] += (jitter * dx * rng.uniform(-1, 1, (len(fl), 3))).astype(np.float32)
    if hole:
        gone = fl[rng.random(len(fl)) < 0.15]
        c.imove[gone] = -256
        c.r[gone] = np.asarray(c.params.domain_max, np.float32)
    c.dt = c.params.dt_fixed
    return c


def compare(c):
    a, b = run(c, True), run(c, False)
    ia, ib = np.argsort(a.id), np.argsort(b.id)
    act = b.imove[ib] >= -3
    for name in ("u", "dudt", "rho", "drhodt", "shepard"):
        x = np.asarray(getattr(a, name), np.float64)[ia][act]
        y = np.asarray(getattr(b, name), np.float64)[ib][act]
        assert np.abs(x - y).max() <= 1e-5 * np.abs(y).max(), name


@pytest.mark.parametrize("hfac", [1.0, 1.5, 1.6, 2.0, 2.4])
@pytest.mark.parametrize("jitter", [0.0, 0.02, 0.3])
@pytest.mark.parametrize("hole", [False, True])
def test_lattice(hfac, jitter, hole):
    compare(state(0.02, (0.6, 0.4, 0.5), (0.32, 0.4, 0.34), hfac, jitter, hole))


@pytest.mark.parametrize("hfac,jitter,hole", [
    (1.3, 0.0, False), (1.6, 0.0, False), (2.0, 0.0, False), (2.0, 0.0, True), (2.0, 0.3, False),
    (1.6, 0.1, True), (2.4, 0.0, False), (2.0, 0.8, False)])
def test_large_lattice(hfac, jitter, hole):
    """More particles than the smallest number swept by octant, 60 by 55 by 47
    cells and odd rests of them."""
    c = state(0.01, (1.5, 1.07, 0.93), (0.75, 1.07, 0.77), hfac, jitter, hole)
    assert c.N > 600000
    compare(c)
