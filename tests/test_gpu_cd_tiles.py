"""Coordinate descent over the ways its tiles are dealt out: one and two rows a warp, single CTAs and pairs,
windows of several tiles a CTA, images of more tiles than a CTA keeps candidates of in registers, sizes that
no tile divides, and runs of several launches.  All against the oracle, bit for bit, as both compute in the
same float32 operations in the same order.
"""
import numpy as np
import pytest

from conftest import oracle, pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,p,iters", [
    (33, 5, 60),       # one tile
    (200, 24, 1300),   # one row a warp, three launches
    (516, 70, 300),    # two rows a warp, fewer than a warp's worth of CTAs
    (1101, 300, 150),  # pairs of CTAs, odd size
    (1400, 700, 40),   # the window covers the image: several tiles a CTA
    (5121, 24, 25),    # more than 32 tiles a CTA
])
def test_tiles_match_oracle(need_gpu, n, p, iters):
    rng = np.random.default_rng(n)
    psf = (rng.standard_normal((p, p)) * 0.05).astype(np.float32)
    psf[p // 2, p // 2] = 1.0
    x0 = np.zeros((n, n), np.float32)
    k = max(1, n // 16)
    x0[rng.integers(0, n, k), rng.integers(0, n, k)] = rng.random(k).astype(np.float32)
    g0 = (rng.standard_normal((n, n)) * 2).astype(np.float32)
    cd = pkg.FastSerialCD(pkg.Rectangle(0, 0, n, n), psf)
    psf2, amap = cd.maps()
    ox, og, oconv, oit = oracle.deconvolve(x0, g0, amap, psf2, 0.3, 0.2, iters, 1e-7)
    x, g = x0.copy(), g0.copy()
    r = cd.Deconvolve(x, g, 0.3, 0.2, iters, 1e-7)
    assert (r.Converged, r.IterationCount) == (oconv, oit) and oit > 0
    assert x.tobytes() == ox.tobytes()
    assert g.tobytes() == og.tobytes()
    cd.destroy()
