"""The quad sweep beside the direct sweep of a thread per particle (the same
sums in the same order, by plain expressions): equal bit for bit where values
are not finite or zero."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from test_gpu_quad import cloud


def step(c, variant, blocks):
    from aquagpusph_gb300.solver import Solver
    sv = Solver(c.params, capacity=c.N)
    sv.set_tuning(variant, blocks)
    sv.set_case(c)
    sv.step(1, graph=True)
    g = sv.get_case()
    sv.close()
    return g


def assert_same(c):
    a, b = step(c, 16, 3), step(c, 9, 14)
    for name, x in a.state_arrays().items():
        assert np.array_equal(x, getattr(b, name), equal_nan=x.dtype.kind == "f"), name
    assert np.array_equal(a.shepard, b.shepard, equal_nan=True)


@pytest.mark.parametrize("dims", [2, 3])
@pytest.mark.parametrize("n,spread", [(1, 0.2), (5, 0.5), (60, 0.9)])
@pytest.mark.parametrize("name,value", [
    ("u", np.inf), ("u", -np.inf), ("u", np.nan), ("u", 3e38), ("dudt", np.inf),
    ("rho", np.inf), ("rho", np.nan), ("rho", 0.0), ("m", np.inf), ("m", np.nan), ("m", 0.0)])
def test_values_that_are_not_finite(dims, n, spread, name, value):
    """One fluid particle with such a value, alone (with slots that hold no
    neighbour) and among others."""
    c = cloud(dims, n, spread, 31 * n + dims, 8)
    a = getattr(c, name)
    if a.ndim == 2:
        a[n // 2, 0] = value
    else:
        a[n // 2] = value
    assert_same(c)


@pytest.mark.parametrize("dims", [2, 3])
@pytest.mark.parametrize("scale", [1.0, 1e-3, 1e-6])
@pytest.mark.parametrize("seed", range(4))
def test_pairs_at_the_edge_of_the_support(dims, scale, seed):
    """Neighbours within a few units in the last place of the support, inside,
    on and outside it, and on a lattice whose spacing divides it: the smallest
    kernel factors that there are, in and out of the range of the branch-free
    quotients (by the masses)."""
    n = 200
    c = cloud(dims, n, 0.9, 17 + seed, 8, scale)
    rng = np.random.default_rng(seed)
    reach = np.float64(c.params.SUPPORT * c.params.H)
    d = rng.normal(size=(n, dims))
    d /= np.linalg.norm(d, axis=1)[:, None]
    d[:2 * dims] = np.concatenate([np.eye(dims), -np.eye(dims)])
    r = d * reach * (1.0 + rng.integers(-24, 25, (n, 1)) * 2.0 ** -24)
    r[0] = 0.0
    g = np.stack(np.meshgrid(*[np.arange(-2, 3)] * dims, indexing="ij"), -1).reshape(-1, dims)
    r[1:1 + len(g)] = g[:n - 1] * reach / 4
    c.r[:n, :dims] = r
    assert_same(c)


@pytest.mark.parametrize("dims", [2, 3])
@pytest.mark.parametrize("n", [1023, 1025, 1500, 2200])
def test_cells_of_very_many_particles(dims, n):
    """One cell on both sides of the count from which its particles are cut into
    clusters by position: starting within a block of positions and spanning
    several."""
    c = cloud(dims, n, 0.85, n + dims, 12)
    assert_same(c)


@pytest.mark.parametrize("dims", [2, 3])
@pytest.mark.parametrize("n,spread", [(1, 0.2), (5, 0.5), (60, 0.9), (400, 1.9)])
@pytest.mark.parametrize("name", ["rho", "m", "u"])
def test_fast_sweeps_do_not_drop_a_nan(dims, n, spread, name):
    """The default sweeps of the fast build: where the direct sweep's result is
    NaN because a neighbour's value is, theirs is too."""
    from aquagpusph_gb300.solver import Solver
    c = cloud(dims, n, spread, 31 * n + dims, 8)
    a = getattr(c, name)
    a[(n // 2, 0) if a.ndim == 2 else n // 2] = np.nan
    out = []
    for variant, blocks in ((16, 3), (9, 14)):
        sv = Solver(c.params, capacity=c.N)
        sv.set_precision(True)
        sv.set_tuning(variant, blocks)
        sv.set_case(c)
        sv.step(1, graph=True)
        out.append(sv.get_case())
        sv.close()
    g, direct = out
    fl = direct.imove == 1
    for k in ("dudt", "drhodt", "rho", "shepard"):
        x, y = np.asarray(getattr(g, k)), np.asarray(getattr(direct, k))
        # the particle itself keeps a value that its own NaN does not reach
        bad = fl.reshape((-1,) + (1,) * (x.ndim - 1)) & np.isnan(y) & ~np.isnan(x)
        assert not bad.any(), k


@pytest.mark.parametrize("dims", [2, 3])
@pytest.mark.parametrize("name,value", [
    ("m", np.nan), ("m", np.inf), ("m", -1.0), ("normal", np.nan), ("normal", np.inf),
    ("u", np.inf), ("u", np.nan)])
def test_boundary_elements_that_are_not_ordinary(dims, name, value):
    """One boundary element with such an area, normal or velocity, among fluid
    that lies within a radius of the wall, in and out of its support."""
    c = cloud(dims, 240, 2.6, 5 + dims, 120)
    h = c.params.h
    c.r[:240:2, dims - 1] = np.float32(0.1 * h) * (1 + np.arange(120)) / 120
    a = getattr(c, name)
    if a.ndim == 2:
        a[300, :dims] = value
    else:
        a[300] = value
    assert_same(c)
