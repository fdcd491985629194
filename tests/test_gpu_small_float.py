"""Sweeps of small float levels whose coefficients, or their products, are denormal (a deep schedule's coarse levels end there), against
the oracle.  In that range every product is rounded to a multiple of q = 2^-149, by at most q / 2.  With a Hessian
of about 2 a on the diagonal, the gradient's 53 products come to at most 27 q, 27 q / a in the update; the update's
numerator, formed 16 times as large in three roundings, adds 2 q / (16 a^2).  The neighbours' entries are a hundredth
of the diagonal, so errors of earlier colours add at most half as much again."""
import numpy as np
import pytest

import exteriorpoissonrecon_gb300 as epr
from oracle import oracle as O

pytestmark = pytest.mark.gpu

Q = 2.0 ** -149


@pytest.mark.parametrize("level", [0, 1, 2, 3])
def test_denormal_coefficients(level):
    a = 5e-4
    rng = np.random.default_rng(level)
    r = epr.Reconstructor(3, 3, build=False, precision="fp32", dWeight=0.0)
    o = O.Oracle(3, 3, d_weight=0.0)
    n = r.nodes(level)
    R = 0.01 * a * rng.uniform(-1, 1, (n, 27))
    R[:, 13] = a
    B = 0.01 * a * rng.uniform(-1, 1, (n, 27))
    R, B = (v.astype(np.float32).astype(np.float64) for v in (R, B))
    x, y = (np.round(rng.uniform(-1e-37, 1e-37, n) / Q) * Q for _ in range(2))
    r.set_level_system(level, R, B, 0.0)
    o.set_level_system(level, R, B, 0.0)
    got, want = r.gs(level, x, y, 1), o.gs(level, x, y, 1)
    r.close()
    off = max(np.abs(g - w).max() for g, w in zip(got, want))
    assert 0 < off <= 1.5 * Q * (27 / a + 2 / (16 * a * a)), off / Q
