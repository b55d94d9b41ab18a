"""BI walls with clusters of 8 (steps of more than 128 particles per SM): the golden
BI cases beside parked particles enough to cross that line.  The parked ones lie
at domain_max, as the cases' own removed particle does, so box, cells and sorted
order of the others stay.  The exact build equals the run with clusters of 4 bit
for bit and the reference kernels' step to 1e-5; the fast build is within 1e-5 of
the exact one after a step and 1e-4 after three (the tolerances of test_gpu_bi)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from aquagpusph_gb300 import case as cases
from test_gpu_bi import close, fixture_case

PARKED = 24000
FIELDS = ("id", "imove", "r", "u", "dudt", "rho", "drhodt", "p", "shepard")


def beside_parked(c):
    big = cases.Case(c.params, c.N + PARKED)
    for k, v in c.state_arrays().items():
        getattr(big, k)[:c.N] = v
    big.id[c.N:] = np.arange(c.N, big.N)
    big.imove[c.N:] = -256
    big.r[c.N:] = np.asarray(c.params.domain_max, np.float32)[:big.vs]
    big.rho[c.N:] = 998.0
    big.t, big.dt, big.iter = c.t, c.dt, c.iter
    return big


def run(c, fast, steps):
    from aquagpusph_gb300.solver import Solver
    sv = Solver(c.params, capacity=c.N)
    sv.set_precision(fast)
    sv.set_case(c)
    sv.step(steps, graph=True)
    sv.check()
    g = sv.get_case()
    sv.close()
    return g


@pytest.mark.parametrize("name", ["bi", "ie"])
@pytest.mark.parametrize("dims", [2, 3])
@pytest.mark.parametrize("steps", [1, 3])
def test_clusters_of_8_and_of_4_agree(dims, name, steps):
    torch = pytest.importorskip("torch")
    c, d = fixture_case(dims, name)
    big = beside_parked(c)
    line = 128 * torch.cuda.get_device_properties(0).multi_processor_count
    assert c.N <= line < big.N
    a, b = run(c, False, steps), run(big, False, steps)
    for k in FIELDS:
        assert np.array_equal(getattr(a, k), getattr(b, k)[:c.N], equal_nan=k != "id"), k
    if steps == 1:
        fl, wl = d["out1_imove"] == 1, d["out1_imove"] == -3
        errs = {"dudt": close(b.dudt[:c.N], d["out1_dudt"], fl),
                "drhodt": close(b.drhodt[:c.N], d["out1_drhodt"], fl),
                "p": close(b.p[:c.N], d["out1_p"], wl),
                "rho": close(b.rho[:c.N], d["out1_rho"], wl | fl)}
        assert max(errs.values()) <= 1e-5, errs


@pytest.mark.parametrize("name", ["bi", "ie"])
@pytest.mark.parametrize("dims", [2, 3])
@pytest.mark.parametrize("steps,tol", [(1, 1e-5), (3, 1e-4)])
def test_fast_clusters_of_8(dims, name, steps, tol):
    c, _ = fixture_case(dims, name)
    a, b = run(c, False, steps), run(beside_parked(c), True, steps)
    ib = np.argsort(b.id)[:c.N]
    ia = np.argsort(a.id)
    fl = a.imove[ia] == 1
    for k in ("r", "u", "rho"):
        assert close(getattr(b, k)[ib], getattr(a, k)[ia], fl) <= tol, k
