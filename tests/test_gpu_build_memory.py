"""A context and its build within the memory of its lasting arrays and the splats' own scratch (EPR_ALLOC_CAP_BYTES
counts every allocation): the frame sums, the cells' masses and the Galerkin products work in arrays that the
build writes afterwards anyway, the finest B and the finest colour blocks."""
import pytest

import exteriorpoissonrecon_gb300 as epr

pytestmark = pytest.mark.gpu

MIXED = dict(precision="fp32", fp64_from=0, fp64_levels=4, band_precision="df")


@pytest.mark.parametrize("dim,depth,n,megabytes,kw", [(3, 5, 20000, 52.9, {}), (3, 5, 60000, 65.1, MIXED), (4, 3, 60000, 43.3, dict(precision="fp32")),
                                                       (4, 4, 60000, 294.9, {}), (4, 4, 60000, 295.7, dict(precision="fp32"))])
def test_build_within(monkeypatch, dim, depth, n, megabytes, kw):
    pos, fr = epr.samples.make_workload("link" if dim == 3 else "clifford", n, seed=3)
    pu, _ = epr.unit_cube(pos)
    monkeypatch.setenv("EPR_ALLOC_CAP_BYTES", str(int(megabytes * 1e6)))
    r = epr.Reconstructor(dim, depth, pu, epr.pack_skew(fr), **kw)
    r.close()


def test_failed_rebuild_leaves_no_half_system(monkeypatch):
    """A rebuild that fails after it began to write the finest stencils is not solved: the context needs a build."""
    pos, fr = epr.samples.make_workload("link", 3000, seed=2)
    pu, _ = epr.unit_cube(pos)
    sk = epr.pack_skew(fr)
    outcomes = set()
    for cap in range(6 << 20, 40 << 20, 1 << 18):
        monkeypatch.setenv("EPR_ALLOC_CAP_BYTES", str(cap))
        try:
            r = epr.Reconstructor(3, 4, pu, sk, aRadius=1)
            first = r.solve()["fit_energy"]
        except epr.EprError:
            continue
        try:
            r.build()
            outcomes.add("built")
        except epr.EprError as e:
            assert "[-5]" in str(e)
            try:
                assert r.solve()["fit_energy"] == first
                outcomes.add("old system")
            except epr.EprError as e:
                assert "[-3]" in str(e)
                outcomes.add("none")
        r.close()
        if outcomes == {"built", "old system", "none"}:
            break
    assert "none" in outcomes and "old system" in outcomes
