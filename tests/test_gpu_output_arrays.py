"""Results copied into every kind of output array: fresh (no page behind it), in use, resident in part, starting and
ending in the middle of a page, smaller than a page, large enough for four threads to back it.  The values are
those of an array in use and the bytes around the output stay as they were."""
import ctypes
import mmap

import numpy as np
import pytest

import exteriorpoissonrecon_gb300 as epr

pytestmark = pytest.mark.gpu

P = ctypes.POINTER(ctypes.c_double)


def array(n, start, kind):
    """n doubles at byte `start` of an anonymous mapping, and all its bytes"""
    size = start + 8 * n + 3 * mmap.PAGESIZE
    raw = np.frombuffer(mmap.mmap(-1, size), dtype=np.uint8)
    if kind == "used":
        raw[:] = 0xAB
    elif kind == "part":
        for at in range(0, size, 3 * mmap.PAGESIZE):
            raw[at:at + mmap.PAGESIZE] = 0xAB
    return raw[start:start + 8 * n].view(np.float64), raw


def around(raw, start, n):
    return raw[:start].copy(), raw[start + 8 * n:].copy()


@pytest.mark.parametrize("kind", ["fresh", "used", "part"])
@pytest.mark.parametrize("start", [0, 8, 4096 - 24])
@pytest.mark.parametrize("level", [1, 4, 5, 6])
def test_coefficients(level, kind, start):
    r = epr.Reconstructor(3, 6, build=False)
    n = r.nodes(level)
    rng = np.random.default_rng(level)
    x, y = rng.uniform(-1, 1, n), rng.uniform(-1, 1, n)
    r.set_coefficients(level, x, y)
    out = [array(n, start, kind) for _ in range(2)]
    before = [around(raw, start, n) if kind != "fresh" else None for _, raw in out]
    assert epr.load().epr_get_coefficients(r._h, level, *(v.ctypes.data_as(P) for v, _ in out)) == 0
    r.close()
    assert np.array_equal(out[0][0], x) and np.array_equal(out[1][0], y)
    for (_, raw), b in zip(out, before):
        a = around(raw, start, n)
        if b is None:
            assert not a[0].any() and not a[1].any()
        else:
            assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])


@pytest.mark.parametrize("kind", ["fresh", "part"])
def test_fit_by_four_threads(kind):
    r = epr.Reconstructor(3, 7, build=False, precision="fp32")
    n = r.nodes(7)
    rng = np.random.default_rng(7)
    r.set_coefficients(7, rng.uniform(-1, 1, n), rng.uniform(-1, 1, n))
    want = r.quadfit(7)
    out, raw = array(5 * n, 40, kind)
    assert epr.load().epr_quadfit(r._h, 7, out.ctypes.data_as(P)) == 0
    r.close()
    assert np.array_equal(out.reshape(n, 5), want)
