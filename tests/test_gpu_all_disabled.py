"""Training images whose every window covers an inactive voxel: every distance is Inf, every position a
candidate of one rank, as in the reference (`findall(D .<= (1 + tol) * minimum(D))`, src/iqsim.jl:237).
Realizations equal the oracle's."""
import numpy as np
import pytest

from oracle import iqsim_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("engine", [2, 1, 0])
@pytest.mark.parametrize("shape,tile,size", [((51,), (48,), (77,)), ((14, 12), (12, 8), (30, 27)),
                                             ((14, 12, 9), (9, 8, 6), (20, 17, 11))])
@pytest.mark.parametrize("values", ["lognormal", "integer"])
def test_every_window_disabled(iq, engine, shape, tile, size, values):
    rng = np.random.default_rng(1001)
    ti = np.exp(rng.normal(size=shape)) if values == "lognormal" else rng.integers(0, 3, shape).astype(float)
    ti = ti.astype(np.float32)
    ti[tuple(s // 2 for s in shape)] = np.nan
    assert O.finddisabled(ti, tile).all()
    ctx = iq.Context(0)
    try:
        ctx.set_option("corr.engine", engine)
        kw = dict(overlap=(0.2,) * len(tile), nreal=3, path="random")
        got = iq.iqsim(ti, tile, size, rng=4, ctx=ctx, **kw)
        for x, y in zip(got, O.iqsim(ti, tile, size, seed=4, **kw)):
            assert np.array_equal(x, y, equal_nan=True)
    finally:
        ctx.close()
