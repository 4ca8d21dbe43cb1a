"""Distance maps of values that need both FP16 halves, against the SIMT kernel.

The image holds small integers and a lattice of odd 12-bit ones (2049..2055), of which a window sees
one at most: their low halves are not zero, and every product and every sum of the maps is a whole
number below 2^24, so both kernels are exact and the maps must be equal bit for bit, with no
tolerance. The shapes put the form's edges in reach: x extents of every remainder by 8 (the padded
pitch of the halves), one to three 8-offset chunks and more than one row entry per row, odd numbers
of rows and of chunks, images smaller than one block of positions, and the last window of the image.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engines(iq):
    a, b = iq.Context(0), iq.Context(0)
    b.set_option("corr.engine", 0)
    yield a, b
    a.close()
    b.close()


@pytest.mark.parametrize("shape,tile,ntmpl,hole", [
    ((40, 21), (8, 5), 1, False),
    ((41, 33), (9, 4), 3, True),
    ((42, 35), (17, 7), 16, True),
    ((43, 40), (25, 3), 17, False),
    ((300,), (31,), 2, False),
    ((21, 20, 13), (5, 5, 4), 4, True),
    ((30, 19, 12), (24, 6, 5), 33, True),
    ((39, 25, 9), (26, 7, 3), 5, True),
    ((11, 9, 7), (11, 9, 7), 2, False),
])
def test_wide_values_equal_simt(iq, engines, shape, tile, ntmpl, hole):
    rng = np.random.default_rng(sum(shape) + ntmpl)
    ti = rng.integers(0, 4, shape).astype(np.float32)
    at = tuple(slice(t - 1, None, t) for t in tile)
    ti[at] = 2049 + 2 * rng.integers(0, 4, ti[at].shape)
    tm = rng.integers(0, 4, (ntmpl,) + tile).astype(np.float32)
    w = np.ones(tile, np.uint8)
    if hole:
        w[tuple(slice(max(1, t // 4), t) for t in tile)] = 0
    got = iq.fastdistance(ti, tm, w, ctx=engines[0])
    ref = iq.fastdistance(ti, tm, w, ctx=engines[1])
    assert np.array_equal(got, ref)
