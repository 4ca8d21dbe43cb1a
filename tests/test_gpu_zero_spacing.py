"""Tiles without spacing along a dimension (an overlap of the whole extent, on a grid of one tile there):
they lie in the same place, so each waits for those before it. Realizations equal the oracle's."""
import numpy as np
import pytest

from oracle import iqsim_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("path", ["raster", "random", "dilation"])
@pytest.mark.parametrize("shape,tile,size,overlap", [((20, 21, 19), (2, 6, 5), (2, 19, 17), (0.57, 0.35, 0.3)),
                                                     ((24, 23), (9, 2), (31, 2), (0.3, 0.6)),
                                                     ((20, 21, 16), (4, 8, 2), (12, 19, 2), (0.3, 0.3, 0.59))])
def test_tiles_in_one_place(iq, path, shape, tile, size, overlap):
    rng = np.random.default_rng(1101)
    ti = rng.integers(-3, 4, shape).astype(np.float32)
    kw = dict(overlap=overlap, nreal=3, path=path, tol=0.3)
    for seed in (1, 2):
        got = iq.iqsim(ti, tile, size, rng=seed, **kw)
        for x, y in zip(got, O.iqsim(ti, tile, size, seed=seed, **kw)):
            assert np.array_equal(x, y)


@pytest.mark.parametrize("inactive", [False, True])
@pytest.mark.parametrize("shape,tile,size,overlap", [((20, 21, 19), (2, 6, 5), (2, 19, 17), (0.57, 0.35, 0.3)),
                                                     ((24, 23), (9, 2), (31, 2), (0.3, 0.6)), ((40,), (2,), (2,), (0.6,))])
def test_hard_data_of_tiles_in_one_place(iq, inactive, shape, tile, size, overlap):
    """Each of them holds the data (and the inactive voxels) of that place."""
    rng = np.random.default_rng(1102)
    ti = rng.integers(-3, 4, shape).astype(np.float32)
    hard = {tuple(int(rng.integers(0, s)) for s in size): float(rng.integers(-3, 4)) for _ in range(6)}
    if inactive:
        hard[tuple(s - 1 for s in size)] = float("nan")
    kw = dict(overlap=overlap, nreal=2, tol=0.3, hard=hard)
    for seed in (1, 2):
        got = iq.iqsim(ti, tile, size, rng=seed, **kw)
        for x, y in zip(got, O.iqsim(ti, tile, size, seed=seed, **kw)):
            assert np.array_equal(x, y, equal_nan=True)
