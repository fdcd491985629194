"""Sweeps of a level that has no system yet: a context that was never built, one whose only system is on
another level, one whose build ran out of memory.  Such a level's stencils are zero, so its sweeps are those of
a level that was given zero stencils explicitly (with no Dirichlet weight), bit for bit."""
import numpy as np
import pytest

import exteriorpoissonrecon_gb300 as epr

pytestmark = pytest.mark.gpu


def fields(dim, level):
    rng = np.random.default_rng(10 * dim + level)
    n = 2 ** level + 1
    ax = np.meshgrid(*[np.linspace(0, 1, n)] * dim, indexing="ij")
    return [(np.sin(sum(rng.uniform(1, 3) * a for a in ax)) + 0.05 * rng.uniform(-1, 1, ax[0].shape)).ravel() for _ in range(2)]


def zero_system(r, level):
    z = np.zeros((r.nodes(level), 3 ** r.dim))
    r.set_level_system(level, z, z, 0.0)


@pytest.mark.parametrize("dim,level", [(3, 3), (3, 4), (3, 5), (3, 6), (4, 1), (4, 2), (4, 3), (4, 4)])
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_level_without_a_system(dim, level, precision):
    x, y = fields(dim, level)
    kw = dict(build=False, precision=precision, dWeight=0.0)
    r = epr.Reconstructor(dim, level, **kw)
    zero_system(r, level)
    want = r.gs(level, x, y, 2)
    r.close()
    assert not np.array_equal(want[0], x)
    r = epr.Reconstructor(dim, level, **kw)
    got = r.gs(level, x, y, 2)
    r.close()
    for g, w in zip(got, want):
        assert np.array_equal(g, w)


def test_system_on_another_level():
    x, y = fields(3, 5)
    kw = dict(build=False, precision="fp32", dWeight=0.0)
    r = epr.Reconstructor(3, 5, **kw)
    zero_system(r, 5)
    want = r.gs(5, x, y, 1)
    r.close()
    r = epr.Reconstructor(3, 6, **kw)
    zero_system(r, 6)
    got = r.gs(5, x, y, 1)
    r.close()
    for g, w in zip(got, want):
        assert np.array_equal(g, w)


def test_sweep_after_a_build_that_ran_out_of_memory(monkeypatch):
    """Whatever array a build fails at, a sweep of the finest level afterwards is an error or a result, and the
    next context works."""
    pos, fr = epr.samples.make_workload("link", 3000, seed=1)
    pu, _ = epr.unit_cube(pos)
    sk = epr.pack_skew(fr)
    x, y = fields(3, 4)
    failed = swept = 0
    for cap in range(4 << 20, 9 << 20, 1 << 18):
        monkeypatch.setenv("EPR_ALLOC_CAP_BYTES", str(cap))
        try:
            r = epr.Reconstructor(3, 4, precision="fp32")
        except epr.EprError:
            continue
        try:
            r.set_samples(pu, sk)
            r.build()
        except epr.EprError as e:
            assert "[-5]" in str(e)
            failed += 1
        try:
            assert all(np.isfinite(v).all() for v in r.gs(4, x, y, 1))
            swept += 1
        except epr.EprError as e:
            assert "[-5]" in str(e)
        r.close()
    assert failed and swept
    monkeypatch.delenv("EPR_ALLOC_CAP_BYTES")
    r = epr.Reconstructor(3, 4, pu, sk, precision="fp32")
    r.solve()
    r.close()


@pytest.mark.parametrize("dim,depth", [(3, 6), (4, 4)])
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_timer_and_solve_without_a_build(dim, depth, precision):
    """The kernel timer on a context that was never built; a solve and a batch of a context with a system on its
    finest level alone, the others' stencils zero."""
    r = epr.Reconstructor(dim, depth, build=False, precision=precision)
    for level in range(depth + 1):
        for kernel in ("gs", "energy", "quadfit", "gn"):
            assert r.time_kernel(kernel, level, 1) > 0
    r.close()
    if dim == 4 and precision == "fp64":
        return
    out = []
    for way in ("solve", "batch", "tuned"):
        r = epr.Reconstructor(dim, depth, build=False, precision=precision, dWeight=0.0)
        rng = np.random.default_rng(5)
        R = 0.02 * rng.uniform(-1, 1, (r.nodes(depth), 3 ** dim))
        R[:, 3 ** dim // 2] = 1.0
        r.set_level_system(depth, R, 0.1 * R, 1.0)
        if way == "solve":
            r.solve()
        elif dim == 3:
            b = epr.LockstepBatch([r])
            if way == "tuned":
                b.tune(reps=1)
            b.run()
            b.close()
        else:
            r.solve()
        out.append(r.coefficients(depth))
        r.close()
    for other in out[1:]:
        assert all(np.array_equal(u, v) for u, v in zip(out[0], other))
