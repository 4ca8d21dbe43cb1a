"""Selections and ranks of images on a coarse grid (multiples of 1/3, which FP16 halves do not hold
exactly): many positions then have distinct Float64 distances that round to one FP32 value, and whole
clusters of them are raised to their Float64 distance before any order is taken. Realizations and
near-tie counts equal the oracle's bit for bit (the pick decides on Float64 distances; no tolerance).
"""
import numpy as np
import pytest

from oracle import iqsim_oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(iq):
    c = iq.Context(0)
    yield c
    c.close()


def _thirds(rng, shape, most):
    return (rng.integers(0, most, shape) / 3.0).astype(np.float32)


def _run(iq, ctx, ti, tile, out, **kw):
    g = iq.iqsim(ti, tile, out, ctx=ctx, rng=kw["seed"], **{k: v for k, v in kw.items() if k != "seed"})
    gt = ctx.ties
    ties = []
    r = O.iqsim(ti, tile, out, ties=ties, **kw)
    for x, y in zip(g, r):
        assert np.array_equal(np.asarray(x), np.asarray(y))
    assert gt == sum(ties)


# tol 0.9 of 40 x 38 x 22 selects more than 8,192 band positions
@pytest.mark.parametrize("hard,nsoft,tol,shape", [(0, 1, 0.1, (30, 28, 14)), (8, 0, 0.1, (30, 28, 14)),
                                                  (8, 1, 0.1, (30, 28, 14)), (6, 2, 0.3, (26, 23, 11)),
                                                  (6, 1, 0.9, (45, 43, 26))])
@pytest.mark.parametrize("seed", [1, 2, 3])
def test_relaxation_on_coarse_images(iq, ctx, hard, nsoft, tol, shape, seed):
    rng = np.random.default_rng(100 + seed)
    ti = _thirds(rng, shape, 4)
    out = (14, 11, 7)
    soft = [(_thirds(rng, out, 5), _thirds(rng, shape, 5)) for _ in range(nsoft)]
    hd = {tuple(int(rng.integers(0, s)) for s in out): float(_thirds(rng, (1,), 4)[0]) for _ in range(hard)}
    _run(iq, ctx, ti, (6, 6, 4), out, overlap=(0.34,) * 3, tol=tol, nreal=3, seed=seed, soft=soft, hard=hd)


@pytest.mark.parametrize("seed", [1, 2])
def test_threshold_on_coarse_images(iq, ctx, seed):
    rng = np.random.default_rng(200 + seed)
    ti = _thirds(rng, (30, 28, 14), 4)
    _run(iq, ctx, ti, (6, 6, 4), (22, 19, 11), overlap=(0.34,) * 3, tol=0.5, path="random", nreal=3, seed=seed)
