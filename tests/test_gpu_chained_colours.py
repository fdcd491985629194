"""Colours that start ahead of the end of the colour before them (the sweeps of one call) against sweeps in calls of
their own, whose first colour follows what was on the stream in full: the same bits, at the levels of every
chained kernel, upper faces (whose first lane has no element) and partly empty blocks included."""
import numpy as np
import pytest

import exteriorpoissonrecon_gb300 as epr

pytestmark = pytest.mark.gpu

SWEEPS = 6


def samples(dim, depth):
    pos, fr = epr.samples.make_workload("link" if dim == 3 else "clifford", 3000, seed=depth)
    pu, _ = epr.unit_cube(pos)
    return pu, epr.pack_skew(fr)


def fields(dim, level):
    rng = np.random.default_rng(level)
    return [rng.uniform(-0.5, 0.5, (2 ** level + 1) ** dim) for _ in range(2)]


def same(a, b):
    return all(np.array_equal(u, v) for u, v in zip(a, b))


@pytest.mark.parametrize("precision,dim,level", [(p, d, l) for p in ("fp32", "fp64") for d, l in [(3, 4), (3, 5), (3, 6), (4, 2), (4, 3), (4, 4)]] +
                         [("fp64", 3, 3)])
def test_solve_sweeps(dim, level, precision):
    pu, sk = samples(dim, level)
    x, y = fields(dim, level)
    kw = dict(precision=precision, warm_start=1, min_solve_depth=level)
    r = epr.Reconstructor(dim, level, pu, sk, gs_iters=SWEEPS, **kw)
    r.set_coefficients(level, x, y)
    r.solve()
    together = r.coefficients(level)
    r.close()
    r = epr.Reconstructor(dim, level, pu, sk, gs_iters=1, **kw)
    r.set_coefficients(level, x, y)
    for _ in range(SWEEPS):
        r.solve()
    apart = r.coefficients(level)
    r.close()
    assert same(together, apart)


@pytest.mark.parametrize("dim,level", [(3, 4), (3, 5), (3, 6), (4, 2), (4, 3)])
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("radius", [-1, 1])
def test_callers_sweeps(dim, level, precision, radius):
    pu, sk = samples(dim, level)
    x, y = fields(dim, level)
    r = epr.Reconstructor(dim, level, pu, sk, precision=precision, aRadius=radius)
    together = r.gs(level, x, y, SWEEPS)
    apart = r.gs(level, x, y, 1)
    for _ in range(SWEEPS - 1):
        apart = r.gs(level, iters=1)
    r.close()
    assert same(together, apart)
