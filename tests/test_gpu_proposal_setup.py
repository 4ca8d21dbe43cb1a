"""The full scan's set-up (FP16 image, A2 maps) beside the learned proposal: left out while every column
comes from a shortlist, made when the first chunk takes the full scan."""
import numpy as np
import pytest

from oracle import iqsim_oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture()
def ctx(iq):
    c = iq.Context(0)
    yield c
    c.close()


def _equal(got, want):
    for x, y in zip(got, want):
        assert np.array_equal(np.asarray(x, float), np.asarray(y, float))


def test_no_set_up_without_a_full_scan(iq, ctx):
    """A call served by shortlists launches as many kernels as with the TF32 engine, whose full scan
    has no set-up."""
    rng = np.random.default_rng(701)
    ti = rng.integers(0, 4, (30, 28, 14)).astype(np.float32)
    tile, size = (8, 8, 6), (26, 24, 12)
    kw = dict(overlap=(0.25,) * 3, nreal=2, rng=5, ctx=ctx)
    ctx.lp_init(tile, seed=1)
    ctx.set_option("lp.enable", 1)
    ctx.set_option("lp.k", 1 << 20)  # every position
    want = O.iqsim(ti, tile, size, overlap=(0.25,) * 3, nreal=2, seed=5)
    counts = []
    for engine in (2, 1):
        ctx.set_option("corr.engine", engine)
        for _ in range(2):  # (the first call makes the window embeddings)
            n = ctx.launches
            got = iq.iqsim(ti, tile, size, **kw)
            n = ctx.launches - n
        _equal(got, want)
        st = ctx.lp_stats()
        assert st["cols_shortlist"] > 0 and st["fell_back"] == 0
        counts.append(n)
    assert counts[0] == counts[1]


@pytest.mark.parametrize("streams", [1, 2])
def test_full_scan_after_overflowing_shortlists(iq, ctx, streams):
    """An image that is constant but for a few voxels: thousands of windows share one embedding, the
    shortlists overflow and their chunks take the full scan."""
    rng = np.random.default_rng(702)
    ti = np.zeros((52, 50, 24), np.float32)
    for _ in range(12):
        ti[tuple(int(rng.integers(0, s)) for s in ti.shape)] = 1.0
    tile, size = (8, 8, 6), (26, 24, 12)
    ctx.set_option("sim.streams", streams)
    ctx.lp_init(tile, seed=1)
    ctx.set_option("lp.enable", 1)
    ctx.set_option("lp.k", 8192)
    got = iq.iqsim(ti, tile, size, overlap=(0.25,) * 3, nreal=3, rng=5, ctx=ctx)
    st = ctx.lp_stats()
    _equal(got, O.iqsim(ti, tile, size, overlap=(0.25,) * 3, nreal=3, seed=5))
    # more columns of the full scan than the first tile's (an empty mask)
    assert st["cols_full"] > 3
