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
