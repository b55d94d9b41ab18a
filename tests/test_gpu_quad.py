"""The quad sweep at the sizes where its clusters, lists and queues can go
wrong: fewer particles than a cluster, one more than a cluster, a cell whose
neighbourhood fills the list's ring several times, empty lists, values outside
the range of the branch-free quotients, and both cluster sizes.  The exact
build equals the oracle bit for bit (positions to 1e-6: powf in the BIe PST),
the fast build to the per-step rate tolerance 1e-5."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import oracle as O
from aquagpusph_gb300 import case as cases


def cloud(dims, n, spread, seed, walls=0, scale=1.0):
    """n fluid particles in a box of `spread` cells, `walls` boundary elements
    on its floor and one probe; masses and pressures in units of `scale`."""
    rng = np.random.default_rng(seed)
    c0 = (cases.dam_break_2d(dx=0.02, tank=(1.0, 0.8), column=(0.2, 0.2)) if dims == 2 else
          cases.dam_break_3d(dx=0.05, tank=(1.0, 0.6, 0.6), block=(0.2, 0.2, 0.2), probes_z=(0.1,)))
    p = c0.params
    c = cases.Case(p, n + walls + 1)
    L = p.cell_length
    r = rng.uniform(0.05, 0.05 + spread, (c.N, dims)) * L
    c.imove[:] = 1
    c.imove[n:n + walls] = -3
    c.imove[-1] = 0
    r[n:n + walls, dims - 1] = 0.0
    c.normal[n:n + walls, dims - 1] = -1.0
    c.tangent[n:n + walls, 0] = 1.0
    c.r[:, :dims] = r
    c.iset[n:] = 1
    dx = 0.5 * p.h
    c.rho[:] = 998.0 * (1 + 1e-3 * rng.normal(size=c.N))
    c.m[:] = 998.0 * dx ** dims * scale
    c.m[n:n + walls] = dx ** (dims - 1)
    c.m[-1] = 0.0
    c.u[:n, :dims] = rng.normal(0, 0.3, (n, dims))
    c.dudt[:n, :dims] = rng.normal(0, 2.0, (n, dims))
    c.drhodt[:n] = rng.normal(0, 50.0, n)
    c.dt = p.dt_fixed
    return c


SIZES = [(1, 0.2, 0), (3, 0.5, 1), (4, 0.5, 5), (5, 0.5, 9), (7, 0.8, 0), (8, 0.8, 8), (9, 0.8, 7),
         (33, 0.9, 40), (260, 0.9, 300), (1200, 2.9, 200)]


def step(c, fast):
    from aquagpusph_gb300.solver import Solver
    sv = Solver(c.params, capacity=c.N)
    sv.set_precision(fast)
    sv.set_case(c)
    sv.step(1, graph=True)
    sv.check()
    g = sv.get_case()
    sv.close()
    return g


def compare(c, g, st, fast):
    assert np.array_equal(g.id, st["id"])
    fl = np.asarray(st["imove"]) == 1
    for name in ("u", "dudt", "rho", "drhodt", "p", "shepard"):
        a, b = np.asarray(getattr(g, name)), np.asarray(st[name])
        if fast:
            a, b = a[fl].astype(np.float64), b[fl].astype(np.float64)
            assert np.abs(a - b).max() <= 1e-5 * max(np.abs(b).max(), 1e-30), name
        else:
            assert np.array_equal(a, b), name
    b = np.asarray(st["r"], np.float64)
    assert np.abs(np.asarray(g.r, np.float64) - b).max() <= 1e-6 * np.abs(b).max()


@pytest.mark.parametrize("fast", [False, True])
@pytest.mark.parametrize("dims", [2, 3])
@pytest.mark.parametrize("n,spread,walls", SIZES)
def test_cluster_edges(dims, n, spread, walls, fast):
    c = cloud(dims, n, spread, 100 * n + dims, walls)
    g = step(c, fast)
    st = O.OracleState(c)
    O.load_oracle().step(st)
    compare(c, g, st, fast)


@pytest.mark.parametrize("scale", [1e-12, 1.0, 1e14])
@pytest.mark.parametrize("dims", [2, 3])
def test_masses_outside_the_branch_free_range(dims, scale):
    """Masses far off (and a velocity of 1e-25, whose products are tiny) go
    through the general expressions: still bit-exact."""
    c = cloud(dims, 60, 0.9, 7, 20, scale)
    c.u[5, 0] = 1e-25
    c.u[6, :] = 0.0
    g = step(c, False)
    st = O.OracleState(c)
    O.load_oracle().step(st)
    fl = np.asarray(st["imove"]) == 1
    for name in ("dudt", "drhodt", "shepard"):
        a, b = np.asarray(getattr(g, name))[fl], np.asarray(st[name])[fl]
        assert np.all((a == b) | (np.isnan(a) & np.isnan(b))), name


@pytest.mark.parametrize("dims", [2, 3])
def test_both_cluster_sizes_agree(dims):
    """The same fluid alone (clusters of 4) and beside enough far-away buffer
    particles that clusters of 8 are used: identical results by id."""
    c = cloud(dims, 300, 1.8, 11, 60)
    n = 30000
    big = cases.Case(c.params, c.N + n)
    for k, v in c.state_arrays().items():
        if k != "id":
            getattr(big, k)[:c.N] = v
    big.imove[c.N:] = -256
    big.r[c.N:] = np.asarray(c.params.domain_max, np.float32)[:big.vs]
    big.rho[c.N:] = 998.0
    big.dt = c.dt
    # the same bounding box on both sides, so the same cells
    lone = cases.Case(c.params, c.N + 1)
    for k, v in c.state_arrays().items():
        if k != "id":
            getattr(lone, k)[:c.N] = v
    lone.imove[-1] = -256
    lone.r[-1] = big.r[-1]
    lone.rho[-1] = 998.0
    lone.dt = c.dt
    a, b = step(lone, False), step(big, False)
    ia, ib = np.argsort(a.id)[:c.N], np.argsort(b.id)[:c.N]
    for name in ("r", "u", "dudt", "rho", "drhodt"):
        assert np.array_equal(np.asarray(getattr(a, name))[ia], np.asarray(getattr(b, name))[ib]), name
