"""A build that runs out of memory (EPR_ALLOC_CAP_BYTES, every 1/40 of what it needs) gives its memory back when the
context is destroyed: the device pool's memory in use is what it was before."""
import ctypes
import gc

import pytest

import exteriorpoissonrecon_gb300 as epr

pytestmark = pytest.mark.gpu

USED_MEM_CURRENT = 7  # CU_MEMPOOL_ATTR_USED_MEM_CURRENT


def used():
    cu = ctypes.CDLL("libcuda.so.1")
    pool, value = ctypes.c_void_p(), ctypes.c_uint64()
    assert cu.cuInit(0) == 0
    assert cu.cuDeviceGetDefaultMemPool(ctypes.byref(pool), 0) == 0
    assert cu.cuMemPoolGetAttribute(pool, USED_MEM_CURRENT, ctypes.byref(value)) == 0
    return value.value


@pytest.mark.parametrize("dim,depth,lo,hi,kw", [(3, 4, 2 << 20, 16 << 20, dict(precision="fp32", aRadius=1)), (3, 5, 16 << 20, 80 << 20, dict()),
                                               (4, 2, 2 << 20, 12 << 20, dict())])
def test_failed_builds(monkeypatch, dim, depth, lo, hi, kw):
    pos, fr = epr.samples.make_workload("link" if dim == 3 else "clifford", 3000, seed=2)
    pu, _ = epr.unit_cube(pos)
    sk = epr.pack_skew(fr)
    r = epr.Reconstructor(dim, depth, pu, sk, **kw)
    r.close()
    gc.collect()  # contexts of other tests
    before, failed = used(), 0
    for k in range(40):
        monkeypatch.setenv("EPR_ALLOC_CAP_BYTES", str(lo + (hi - lo) * k // 40))
        try:
            r = epr.Reconstructor(dim, depth, build=False, **kw)
        except epr.EprError:
            assert used() == before
            continue
        try:
            r.set_samples(pu, sk)
            r.build()
        except epr.EprError as e:
            assert "[-5]" in str(e)
            failed += 1
        r.close()
        assert used() == before, k
    assert failed >= 3
