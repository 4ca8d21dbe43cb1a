"""Calls near the device's memory limit: all but a few GB of the device are held by another owner while
the call runs, and its results equal those of the same call with the device to itself (integer images:
every distance exact, no tolerance)."""
import contextlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 20


@contextlib.contextmanager
def left(nbytes):
    """Hold the device's free memory but `nbytes` of it."""
    torch = pytest.importorskip("torch")
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    if free < nbytes + 64 * MB:
        pytest.skip("not enough free memory")
    hold = torch.empty((free - nbytes) // (2 * MB) * (2 * MB), dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del hold
        torch.cuda.empty_cache()


def _call(iq, ctx, *args, **kw):
    return [np.asarray(x) for x in iq.iqsim(*args, ctx=ctx, **kw)]


def _fresh(iq, *args, **kw):
    ctx = iq.Context(0)
    try:
        return _call(iq, ctx, *args, **kw)
    finally:
        ctx.close()


def test_packed_templates_of_many_realizations(iq):
    """A level's 8,192 columns of 64 x 64 templates (0.6 GB packed at once) beside 1.2 GB of grids and
    lists."""
    rng = np.random.default_rng(301)
    ti = rng.integers(0, 3, (68, 69)).astype(np.float32)
    args = (ti, (64, 64), (430, 430))
    kw = dict(overlap=(0.45, 0.45), path="random", nreal=512, rng=3)
    want = _fresh(iq, *args, **kw)
    with left(1450 * MB):
        got = _fresh(iq, *args, **kw)
    for x, y in zip(got, want):
        assert np.array_equal(x, y)


def _image(values, shape):
    rng = np.random.default_rng(302)
    z = rng.normal(size=shape)
    return ((z > 0).astype(np.float32) if values == "binary" else np.exp(z).astype(np.float32))


# Nine tiles, the first drawn without a map: the Toeplitz form computes eight columns, the other form
# launches of 16. Five A2 maps of 2,017 x 2,017 positions take 81 MB.
ARGS = ((32, 32), (56, 56))
KW = dict(overlap=(0.25, 0.25), rng=4)


@pytest.mark.parametrize("values,mb,padded", [("binary", 800, False), ("binary", 500, True),
                                              ("lognormal", 900, False), ("lognormal", 560, True)])
def test_form_of_the_correlation(iq, values, mb, padded):
    """The Toeplitz form while its maps fit an eighth of the memory, for a first and a repeated call
    alike, and the FP16 form of wider data's kernel where they do not: the same realizations."""
    ti = _image(values, (2048, 2048))
    want = _fresh(iq, ti, *ARGS, **KW)
    ctx = iq.Context(0)
    try:
        ctx.set_ti(ti)
        with left(mb * MB):
            for _ in range(2):
                ctx.profile(True)
                got = _call(iq, ctx, ti, *ARGS, **KW)
                cols = ctx.profile_get("corr.columns")[2]
                assert cols == (8 * 16 if padded else 8)
                for x, y in zip(got, want):
                    assert np.array_equal(x, y)
    finally:
        ctx.close()
