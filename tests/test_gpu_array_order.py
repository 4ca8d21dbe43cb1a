"""Training images in row-major, column-major and strided host arrays of every accepted type give the
same call: the library reorders row-major arrays on the device. Distance maps equal bit for bit (the
image values are the same floats), for extents around the 32 x 32 tiles of the reordering."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(40,), (33, 31), (1, 70), (64, 1), (32, 32, 2), (31, 33, 5), (5, 2, 65)])
@pytest.mark.parametrize("dtype", ["float32", "float64", "uint8", ">f4"])
def test_orders_equal(iq, shape, dtype):
    rng = np.random.default_rng(3)
    base = rng.integers(0, 200, shape).astype(dtype)
    tile = tuple(min(s, 2) for s in shape)
    tm = rng.normal(size=tile).astype(np.float32)
    wide = np.zeros(tuple(2 * s for s in shape), dtype)
    wide[tuple(slice(None, None, 2) for _ in shape)] = base
    ref = None
    for ti in (np.asfortranarray(base), np.ascontiguousarray(base), np.ma.masked_array(base),
               wide[tuple(slice(None, None, 2) for _ in shape)], base.tolist()):
        c = iq.Context(0)
        try:
            got = iq.fastdistance(ti, tm, ctx=c)
        finally:
            c.close()
        ref = got if ref is None else ref
        assert np.array_equal(got, ref)
    w = np.lib.stride_tricks.sliding_window_view(base.astype(np.float64), tile)
    d = ((w - tm.astype(np.float64)) ** 2).sum(axis=tuple(range(len(shape), 2 * len(shape))))
    assert np.allclose(ref, d, rtol=1e-4, atol=1e-5 * 200.0 ** 2 * tm.size * 2)
