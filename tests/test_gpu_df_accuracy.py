"""Rounding error of sweeps in double-float on 3D levels 0-3, against the oracle's in double (whose own error is
a hundredth of it), over systems of built curves with the fields as they come and after twenty sweeps: random
curves' stencils, nodes with nearly parallel gradients among them.  Single errors scatter over two orders with
the conditioning of the worst node, so the geometric mean over the systems is held: it is at most that of the
12-point Gauss rule on fully normalised pairs (GAUSS_RULE, this function's values for that arithmetic), up
to the standard error of the mean ratio of two such arithmetics (0.014 for 1,200 pairs of sweeps, so 0.03 for 320;
with every sum loose it is 1.25)."""
import numpy as np
import pytest

import exteriorpoissonrecon_gb300 as epr
from oracle import oracle as O

pytestmark = pytest.mark.gpu

GAUSS_RULE = 5.959e-15


def fields(level, rng):
    n = 2 ** level + 1
    ax = np.meshgrid(*[np.linspace(0, 1, n)] * 3, indexing="ij")
    f = sum(0.3 * np.sin(rng.uniform(0, 6) + np.pi * sum(rng.integers(-2, 3) * a for a in ax)) for _ in range(3))
    return (f + 0.02 * rng.uniform(-1, 1, f.shape)).ravel()


def log_errors():
    """log of the relative L2 error of every system's sweeps"""
    shapes = [("knot", 2.0, 3.0), ("helix", 2.5, 0.0), ("link", 0.0, 0.0), ("knot", 3.0, 4.0)]
    o = O.Oracle(3, 3)
    f = epr.Reconstructor(3, 3, build=False)
    d = epr.Reconstructor(3, 3, build=False, precision="fp32", fp64_from=0, fp64_levels=4, band_precision="df")
    out = []
    for seed in range(20):
        name, a, b = shapes[seed % 4]
        r = epr.Reconstructor(3, 5, build=False)
        r.set_generated_samples(epr.sampler(name, a, b, pos_sigma=0.004, angle_deg=4.0, seed=300 + seed), 20000)
        r.build()
        for level in range(4):
            R, B = (r.get(k, level).reshape(-1, 27) for k in ("R", "B"))
            for c in (o, f, d):
                c.set_level_system(level, R, B, 0.0)
            rng = np.random.default_rng(8 * seed + level)
            x, y = fields(level, rng), fields(level, rng)
            for before in (0, 20):
                if before:
                    x, y = f.gs(level, x, y, before)
                for sweeps in (1, 8):
                    want, got = o.gs(level, x, y, sweeps), d.gs(level, x, y, sweeps)
                    off = sum(((g - w) ** 2).sum() for g, w in zip(got, want))
                    out.append(np.log(max(np.sqrt(off / sum((w ** 2).sum() for w in want)), 1e-17)))
        r.close()
    return np.array(out)


def test_double_float_error():
    e = log_errors()
    assert np.exp(e.mean()) <= 1.05 * GAUSS_RULE, np.exp(e.mean())
