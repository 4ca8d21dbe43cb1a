"""The pick's routes by size, against the Float64 oracle bit for bit with its near-tie counts (the
pick decides on exact distances whatever route it takes; no tolerance):

- relaxation selections listed whole (at most 8192 positions) or tested by a scan of the map;
- candidates ranked from distances made between the pick's phases (at most 4096) or in the pick;
- threshold maps of at least 65,536 positions collected by a pass of their own (up to 8192 kept), smaller
  ones by the pick;
- threshold picks decided by the minimum's interval, or, on images whose distances tie (values on a
  coarse grid that FP16 halves do not hold exactly), by its exact value.
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


def _run(iq, ctx, ti, tile, out, **kw):
    g = iq.iqsim(ti, tile, out, ctx=ctx, rng=kw["seed"], **{k: v for k, v in kw.items() if k != "seed"})
    gt = ctx.ties
    ties = []
    r = O.iqsim(ti, tile, out, ties=ties, **kw)
    for x, y in zip(g, r):
        assert np.array_equal(np.asarray(x), np.asarray(y))
    assert gt == sum(ties)


# positions: 53 x 46 x 39 = 95,082; the first relaxation step takes 0.1 tol of them
@pytest.mark.parametrize("tol,hard,nsoft", [(0.02, 0, 1), (0.3, 6, 1), (0.9, 0, 1), (0.9, 4, 2),
                                            (1.0, 0, 2)])
def test_relaxation_routes(iq, ctx, tol, hard, nsoft):
    rng = np.random.default_rng(91)
    ti = np.exp(rng.normal(size=(60, 53, 44))).astype(np.float32)
    out = (14, 8, 6)
    soft = [(rng.normal(size=out).astype(np.float32), rng.normal(size=ti.shape).astype(np.float32))
            for _ in range(nsoft)]
    hd = {tuple(int(rng.integers(0, s)) for s in out): float(np.exp(rng.normal())) for _ in range(hard)}
    _run(iq, ctx, ti, (8, 8, 6), out, overlap=(0.25,) * 3, tol=tol, nreal=2, seed=4, soft=soft, hard=hd)


@pytest.mark.parametrize("values", ["continuous", "coarse"])
@pytest.mark.parametrize("shape,tile,out,tol", [((70, 66), (9, 8), (22, 20), 0.1),
                                                ((70, 66), (9, 8), (22, 20), 1.0),
                                                ((30, 28, 20), (6, 7, 5), (15, 14, 9), 0.4),
                                                # 82,636 positions: collected ahead of the pick
                                                ((300, 290), (9, 8), (15, 14), 0.1),
                                                ((300, 290), (9, 8), (15, 14), 1.0)])
def test_threshold_routes(iq, ctx, values, shape, tile, out, tol):
    rng = np.random.default_rng(92)
    ti = rng.normal(size=shape) if values == "continuous" else rng.integers(1, 4, shape) / 3.0
    _run(iq, ctx, ti.astype(np.float32), tile, out, overlap=(0.25,) * len(tile), tol=tol,
         path="random", nreal=2, seed=8)
