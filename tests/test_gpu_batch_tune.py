"""The batch's autotuner on levels that have one block shape (levels 3 and 4 in double): timed once, left at the
default, where three runs of the same kernel would be told apart by noise; the levels above them are tuned."""
import pytest

import exteriorpoissonrecon_gb300 as epr

pytestmark = pytest.mark.gpu


def test_one_shape_is_not_tuned():
    recons = []
    for k in range(3):
        r = epr.Reconstructor(3, 5, build=False)
        r.set_generated_samples(epr.sampler("knot", 2.0, 3.0, seed=k), 4000)
        recons.append(r)
    b = epr.LockstepBatch(recons)
    b.run(build=True)
    want = [r.coefficients(5) for r in recons]
    ms = b.tune(reps=2)
    assert ms.shape == (3, 3)  # levels 3, 4, 5
    assert (ms > 0).all() and (ms[:2] == ms[:2, :1]).all()
    assert b.info()["tiles"][3:5] == [1, 1]
    b.run()
    for r, w in zip(recons, want):
        assert all((g == v).all() for g, v in zip(r.coefficients(5), w))
    b.close()
