"""Threshold picks of exact maps on both sides of the size from which their positions are collected ahead
of the pick (65,536), with candidate lists the collecting pass keeps whole and ones it overflows (8,192):
realizations and near-tie counts equal the oracle's (integer images: no tolerance)."""
import numpy as np
import pytest

from oracle import iqsim_oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(iq):
    c = iq.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("shape", [(263, 263), (264, 263)])  # 65,280 and 65,536 positions
@pytest.mark.parametrize("codes,tol", [(2, 0.1), (6, 0.05), (2, 1.0)])
def test_exact_maps(iq, ctx, shape, codes, tol):
    rng = np.random.default_rng(801)
    ti = rng.integers(0, codes, shape).astype(np.float32)
    kw = dict(overlap=(0.25, 0.25), tol=tol, nreal=2)
    got = iq.iqsim(ti, (9, 8), (21, 20), rng=3, ctx=ctx, **kw)
    gt = ctx.ties
    ties = []
    want = O.iqsim(ti, (9, 8), (21, 20), seed=3, ties=ties, **kw)
    for x, y in zip(got, want):
        assert np.array_equal(x, y)
    assert gt == sum(ties)
