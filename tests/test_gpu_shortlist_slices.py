"""Shortlists over images whose positions take one pass of a list kernel's CTA (32,768 positions),
just above one, several slices, and a last slice of a few blocks.

A shortlist that holds every position gives the full scan's realizations bit for bit (integer
sums), so a position lost, doubled or out of order between slices would show; no tolerance.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,tile", [
    ((196, 188), (16, 16)),       # 181 x 173 = 31,313: one pass
    ((197, 196), (16, 16)),       # 182 x 181 = 32,942: a second slice of a few blocks
    ((270, 255), (16, 16)),       # 255 x 240 = 61,200: two slices
    ((55, 50, 36), (16, 16, 8)),  # 40 x 35 x 29 = 40,600
])
def test_full_shortlists_equal_full_scan(iq, shape, tile):
    rng = np.random.default_rng(sum(shape))
    ti = np.kron(rng.integers(0, 4, tuple(-(-n // 4) for n in shape)),
                 np.ones((4,) * len(shape)))[tuple(slice(0, n) for n in shape)].astype(np.float32)
    kw = dict(overlap=(0.25,) * len(tile), nreal=3, rng=7, tol=0.05)
    simsize = tuple(2 * t for t in tile)
    ctx = iq.Context(0)
    try:
        full = iq.iqsim(ti, tile, simsize, ctx=ctx, **kw)
        ctx.lp_init(tile, seed=1)
        ctx.set_option("lp.enable", 1)
        ctx.set_option("lp.k", 1 << 20)
        lp = iq.iqsim(ti, tile, simsize, ctx=ctx, **kw)
        st = ctx.lp_stats()
    finally:
        ctx.close()
    assert st["cols_shortlist"] > 0 and st["fell_back"] == 0
    for a, b in zip(full, lp):
        assert np.array_equal(a, b)
