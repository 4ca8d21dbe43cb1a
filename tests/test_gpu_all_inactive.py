"""Grids whose every voxel is inactive (hard data of NaN only) under tiles without spacing: no tile is
simulated and every voxel comes back inactive, with and without soft data, as from the oracle."""
import itertools

import numpy as np
import pytest

from oracle import iqsim_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("engine", [2, 1, 0])
@pytest.mark.parametrize("nsoft", [0, 1, 2])
@pytest.mark.parametrize("shape,tile", [((30,), (9,)), ((20, 18), (6, 5)), ((12, 11, 9), (5, 4, 2))])
def test_every_voxel_inactive(iq, engine, nsoft, shape, tile):
    rng = np.random.default_rng(1201)
    ti = np.exp(rng.normal(size=shape)).astype(np.float32)
    soft = [(rng.normal(size=tile).astype(np.float32), rng.normal(size=shape).astype(np.float32))
            for _ in range(nsoft)]
    hard = {c: float("nan") for c in itertools.product(*(range(t) for t in tile))}
    kw = dict(overlap=(0.95,) * len(tile), nreal=2, soft=soft, hard=hard)
    ctx = iq.Context(0)
    try:
        ctx.set_option("corr.engine", engine)
        got = iq.iqsim(ti, tile, tile, rng=3, ctx=ctx, **kw)
        for x, y in zip(got, O.iqsim(ti, tile, tile, seed=3, **kw)):
            assert np.array_equal(x, y, equal_nan=True) and np.isnan(x).all()
    finally:
        ctx.close()
