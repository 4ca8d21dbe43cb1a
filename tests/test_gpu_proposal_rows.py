"""Exact sums of the learned proposal over masks whose row (plane form) or quad (byte form)
counts are not whole multiples of a warp's batch.

The sums are integers, so a shortlist that holds every position must give the full scan's
realizations bit for bit; no tolerance. The tiles make the staged counts of their masks end
1 to 31 past a batch of 4 x 32 rows (4 codes) or 8 x 32 quads (6 codes), below one batch, and
on a batch boundary.
"""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cat_ti(shape, seed, ncodes):
    import scipy.ndimage as ndi
    rng = np.random.default_rng(seed)
    f = np.stack([ndi.gaussian_filter(rng.standard_normal(shape), (3, 3, 2), mode="wrap")
                  for _ in range(ncodes)])
    return np.argmax(f, axis=0).astype(np.float32)


def _row_counts(tile, overlap):
    """Rows staged for the raster path's masks (previous neighbours only)."""
    _, ty, tz = tile
    oy, oz = (math.ceil(overlap * t) for t in (ty, tz))
    return {ty * tz, ty * tz - (ty - oy) * tz, ty * tz - ty * (tz - oz),
            ty * tz - (ty - oy) * (tz - oz)}


def test_tiles_cover_partial_batches():
    rests = {n % 128 for t in ((10, 16, 16), (8, 24, 12), (12, 22, 14), (9, 16, 8), (8, 32, 16))
             for n in _row_counts(t, 0.25) if n > 96}
    assert 0 in rests and any(97 - 96 <= r - 96 <= 31 for r in rests) and any(0 < r < 96 for r in rests)


@pytest.mark.parametrize("tile,codes", [((10, 16, 16), 4), ((8, 24, 12), 4), ((12, 22, 14), 3),
                                        ((9, 16, 8), 4), ((8, 32, 16), 4), ((11, 16, 16), 6),
                                        ((13, 20, 10), 6)])
def test_partial_row_batches_equal_full_scan(iq, tile, codes):
    shape = tuple(t + e for t, e in zip(tile, (18, 16, 10)))
    simsize = tuple(2 * t for t in tile)
    ti = _cat_ti(shape, 5, codes)
    kw = dict(overlap=(0.25,) * 3, nreal=2, rng=11, tol=0.05)
    ctx = iq.Context(0)
    try:
        full = iq.iqsim(ti, tile, simsize, ctx=ctx, **kw)
        ctx.lp_init(tile, seed=1)
        ctx.set_option("lp.enable", 1)
        ctx.set_option("lp.k", 1 << 20)
        ctx.set_option("lp.monitor", 1)
        lp = iq.iqsim(ti, tile, simsize, ctx=ctx, **kw)
        st = ctx.lp_stats()
    finally:
        ctx.close()
    assert st["cols_shortlist"] > 0 and st["recall"] == 1.0 and st["fell_back"] == 0
    for a, b in zip(full, lp):
        assert np.array_equal(a, b)
