"""One paired Gauss-Seidel sweep of the relaxation kernels against the oracle at the sizes where their
splits change: 3D levels on either side of the lane-per-element / two-lanes-per-node rule and the
smallest per-colour ones, 4D levels on either side of the single-block kernel, each with every
boundary node; the reference's separate update; and a field with no variation (the shear factor of
the float kernels has nothing to divide by).  The sweep is a solve's: one level, one sweep, from given
coefficients.

Tolerances, relative L2 of the updated coefficients: float 2e-6 (32 rounding units of 2^-24: about
ten roundings on the longest chain from the corner values to the update, inputs and stencils rounded to
float, and the conditioning of the 2 x 2 step), double 1e-12 as the other sweep tests.

A caller's own sweep in float takes the Gauss rule, whose 2 x 2 step divides by a determinant of the size of
its rounding error at the few nodes whose gradients are nearly parallel; all but one node in a hundred agree
with the oracle to the same 32 units of the field's largest value."""
import numpy as np
import pytest

import exteriorpoissonrecon_gb300 as epr
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def system(dim, depth):
    pos, fr = epr.samples.make_workload("link" if dim == 3 else "clifford", 4000, seed=depth)
    pu, _ = epr.unit_cube(pos)
    return pu, epr.pack_skew(fr)


def smooth(dim, level, rng):
    n = 2 ** level + 1
    ax = np.meshgrid(*[np.linspace(0, 1, n)] * dim, indexing="ij")
    f = sum(0.2 * np.sin(rng.uniform(0, 6) + np.pi * rng.integers(-2, 3) * ax[d]) for d in range(dim))
    return (f + 0.01 * rng.uniform(-1, 1, f.shape)).ravel()


@pytest.mark.parametrize("dim,level", [(3, 1), (3, 2), (3, 3), (3, 4), (3, 5), (3, 6), (4, 1), (4, 2), (4, 3)])
@pytest.mark.parametrize("precision,tol", [("fp32", 2e-6), ("fp64", 1e-12)])
@pytest.mark.parametrize("separate", [0, 1])
def test_sweep_against_oracle(dim, level, precision, tol, separate):
    pu, sk = system(dim, level)
    o = O.Oracle(dim, level, separate=separate)
    o.set_samples(pu, sk)
    o.build()
    r = epr.Reconstructor(dim, level, pu, sk, precision=precision, separate=separate, warm_start=1, min_solve_depth=level, gs_iters=1)
    rng = np.random.default_rng(level)
    x, y = smooth(dim, level, rng), smooth(dim, level, rng)
    for a, b in ((x, y), (np.full_like(x, 0.25), y)):
        r.set_coefficients(level, a, b)
        r.solve()
        gx, gy = r.coefficients(level)
        ox, oy = o.gs(level, a, b, 1)
        n = np.sqrt((ox ** 2).sum() + (oy ** 2).sum())
        assert np.sqrt(((gx - ox) ** 2).sum() + ((gy - oy) ** 2).sum()) <= tol * n
    r.close()


@pytest.mark.parametrize("dim,level", [(3, 4), (3, 5), (3, 6), (4, 3)])
@pytest.mark.parametrize("separate", [0, 1])
def test_callers_float_sweep_against_oracle(dim, level, separate):
    pu, sk = system(dim, level)
    o = O.Oracle(dim, level, separate=separate)
    o.set_samples(pu, sk)
    o.build()
    r = epr.Reconstructor(dim, level, pu, sk, precision="fp32", separate=separate)
    rng = np.random.default_rng(level)
    x, y = smooth(dim, level, rng), smooth(dim, level, rng)
    got, want = r.gs(level, x, y, 1), o.gs(level, x, y, 1)
    off = np.maximum(*[np.abs(g - w) for g, w in zip(got, want)])
    assert np.quantile(off, 0.99) <= 2e-6 * max(np.abs(w).max() for w in want)
    r.close()
