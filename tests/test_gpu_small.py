"""The one-launch link-list of small steps against numpy's stable sort, at its
edges: fewer particles than a block's, partial warps and blocks, its largest
size and one above it (the separate kernels), one to 32 cases and 33.  Keys,
permutation, cell counts and boxes are whole numbers or exact minima: equal."""
from types import SimpleNamespace

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from aquagpusph_gb300 import case as cases

SIZES = [(2, 1), (31, 1), (256, 1), (257, 3), (1056, 32), (8193, 5), (8193, 33), (20000, 32),
         (49152, 1), (49152, 32), (49153, 1)]


@pytest.mark.parametrize("dims", [2, 3])
@pytest.mark.parametrize("n,n_cases", SIZES)
def test_small_linklist(dims, n, n_cases):
    from aquagpusph_gb300.solver import Solver
    rng = np.random.default_rng(n + dims)
    p = (cases.dam_break_2d(dx=0.005, tank=(1.0, 0.8), column=(0.2, 0.2)) if dims == 2 else
         cases.dam_break_3d(dx=0.02, tank=(1.0, 0.6, 0.6), block=(0.2, 0.2, 0.2),
                            probes_z=(0.1,))).params
    c = cases.Case(p, n)
    c.imove[:] = 0
    lo = np.asarray(p.domain_min[:dims], np.float64)
    hi = np.asarray(p.domain_max[:dims], np.float64)
    c.r[:, :dims] = lo + rng.uniform(0.1, 0.9, (n, dims)) * (hi - lo)
    c.r[:, 0] -= np.float32(0.5 * (lo[0] + hi[0]))  # both signs
    c.rho[:] = 998.0
    c.dt = p.dt_fixed
    offs = np.linspace(0, n, n_cases + 1).astype(np.uint32)
    sv = Solver(p, capacity=n, ihoc_capacity=n_cases * p.max_cells())
    sv.set_case(c)
    if n_cases > 1:
        sv.set_cases(SimpleNamespace(case=c, offsets=offs, motions=[None] * n_cases))
    r = np.asarray(c.r[:, :dims], np.float32).copy()
    inside = np.all((r >= np.float32(p.domain_min[:dims])) &
                    (r <= np.float32(p.domain_max[:dims])), axis=1)
    r[~inside] = np.float32(p.domain_max[:dims])
    for graph in (False, True):
        sv.set_case(c)
        if n_cases > 1:
            sv.set_cases(SimpleNamespace(case=c, offsets=offs, motions=[None] * n_cases))
        sv.step(1, graph=graph)
        sv.check()
        ex = sv.get_extra()
        L = np.float32(p.cell_length)
        key, base = np.zeros(n, np.int64), 0
        for k in range(n_cases):
            s = slice(int(offs[k]), int(offs[k + 1]))
            mn, mx = r[s].min(0), r[s].max(0)
            nc = ((mx - mn) / L).astype(np.int64) + 6
            a = ((r[s] - mn) * (np.float32(1) / L)).astype(np.int64) + 2
            key[s] = base + a @ np.concatenate([[1], np.cumprod(nc)[:-1]])
            base += int(np.prod(nc))
            if k == 0:
                assert np.array_equal(ex["r_min"][:dims], mn)
                assert np.array_equal(ex["r_max"][:dims], mx)
                assert np.array_equal(ex["n_cells"][:dims], nc)
        perm = np.argsort(key, kind="stable")
        assert np.array_equal(ex["id_unsorted"], perm)
        assert np.array_equal(ex["icell"], key[perm])
    sv.close()
