"""The Toeplitz tensor-core correlation (eight consecutive positions per GEMM row, templates packed
with their eight shifts) against the SIMT kernel.

Integer-valued data: products and FP32 sums are exact in both, so the maps must be equal bit for
bit, with no tolerance. The shapes put the form's edges in reach: tile extents around multiples of
8 (a row of w offsets takes ceil((w + 7) / 8) chunks) and above the 8 chunks of one row entry, x
extents of the image that are and are not multiples of 8, odd template counts, one template,
several groups and launches, maps below and above one 1024-position block, 1-D to 3-D, masks with
an inner box that leaves both ends, one end or nothing of a row, and inactive voxels.

Continuous data: whole simulations are exact in any engine (the pick resolves every decision on
Float64 distances), so the realizations of the tensor-core and the SIMT engines must be equal.
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


def _mask(tile, kind):
    w = np.ones(tile, np.uint8)
    if kind == "low":
        w[tuple(slice(max(1, t // 4), t) for t in tile)] = 0
    elif kind == "high":
        w[tuple(slice(0, t - max(1, t // 4)) for t in tile)] = 0
    elif kind == "inner":
        w[tuple(slice(1, t - 1) if t > 2 else slice(0, t) for t in tile)] = 0
    elif kind == "rows":  # whole rows of the middle leave the mask
        w[(slice(None),) + tuple(slice(1, t - 1) if t > 2 else slice(0, 1) for t in tile[1:])] = 0
    return w


@pytest.mark.parametrize("shape,tile,ntmpl,kind,nan", [
    ((300,), (49,), 3, "full", False),
    ((64,), (1,), 1, "full", False),
    ((2100,), (9,), 2, "inner", False),
    ((97, 61), (16, 9), 5, "low", True),
    ((128, 40), (17, 8), 33, "high", False),
    ((90, 80), (62, 62), 2, "low", False),
    ((150, 33), (97, 12), 1, "inner", False),
    ((40, 33, 21), (8, 8, 5), 16, "rows", False),
    ((48, 30, 19), (24, 12, 6), 40, "low", True),
    ((56, 41, 18), (32, 16, 8), 70, "high", False),
    ((33, 29, 17), (7, 29, 17), 4, "inner", False),
    ((24, 20, 12), (24, 20, 12), 3, "full", False),
])
def test_integer_maps_equal_simt(iq, engines, shape, tile, ntmpl, kind, nan):
    rng = np.random.default_rng(sum(shape) + ntmpl)
    ti = rng.integers(0, 5, shape).astype(np.float32)
    if nan:
        ti[tuple(s // 2 for s in shape)] = np.nan
    tm = rng.integers(-2, 6, (ntmpl,) + tile).astype(np.float32)
    w = _mask(tile, kind)
    got = iq.fastdistance(ti, tm, w, ctx=engines[0])
    ref = iq.fastdistance(ti, tm, w, ctx=engines[1])
    assert np.array_equal(got, ref)


@pytest.mark.parametrize("shape,tile,out,path,nreal", [
    ((70, 61), (18, 23), (80, 75), "random", 5),
    ((41, 38, 19), (13, 9, 7), (50, 41, 22), "random", 3),
    ((40, 36, 20), (16, 12, 8), (44, 40, 24), "raster", 17),
])
def test_continuous_realizations_equal_simt(iq, engines, shape, tile, out, path, nreal):
    rng = np.random.default_rng(7)
    ti = np.exp(rng.normal(size=shape)).astype(np.float32)
    aux = rng.normal(size=out).astype(np.float32)
    auxti = rng.normal(size=shape).astype(np.float32)
    for soft in ([], [(aux, auxti)]):
        kw = dict(overlap=(0.3,) * len(tile), path=path, nreal=nreal, rng=3, soft=soft)
        a = iq.iqsim(ti, tile, out, ctx=engines[0], **kw)
        b = iq.iqsim(ti, tile, out, ctx=engines[1], **kw)
        for x, y in zip(a, b):
            assert np.array_equal(x, y)


@pytest.mark.parametrize("shape,tile,out,path", [
    ((37,), (9,), (60,), "random"), ((50, 44), (12, 10), (70, 66), "random"),
    ((24, 20, 14), (8, 8, 6), (30, 30, 20), "dilation"),
])
def test_draws_of_unconstrained_tiles_equal_oracle(iq, engines, shape, tile, out, path):
    """Tiles without pasted neighbours: every position a candidate of rank 1, drawn on the host."""
    from oracle import iqsim_oracle as O
    rng = np.random.default_rng(12)
    ti = rng.integers(0, 3, shape).astype(np.float32)
    kw = dict(overlap=(0.3,) * len(tile), path=path, nreal=4, tol=0.1)
    a = iq.iqsim(ti, tile, out, ctx=engines[0], rng=21, **kw)
    r = O.iqsim(ti, tile, out, seed=21, **kw)
    for x, y in zip(a, r):
        assert np.array_equal(x, y)
