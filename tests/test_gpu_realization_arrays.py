"""Each realization of `iqsim` is an array of its own, whatever its size: keeping one does not keep the
memory of the others."""
import numpy as np
import pytest

from oracle import iqsim_oracle as O

pytestmark = pytest.mark.gpu


def _owner(a):
    while a.base is not None:
        a = a.base
    return a


# 521 x 509 float32 realizations are copied from the device one by one, the small ones all at once
@pytest.mark.parametrize("size,nreal", [((521, 509), 3), ((41, 38), 3), ((41, 38), 1)])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_realizations_own_their_memory(iq, size, nreal, dtype):
    rng = np.random.default_rng(501)
    ti = rng.integers(0, 3, (70, 66)).astype(dtype)
    kw = dict(overlap=(0.2, 0.2), nreal=nreal)
    got = iq.iqsim(ti, (40, 36), size, rng=9, **kw)
    assert len(got) == nreal
    owners = [_owner(x) for x in got]
    assert len({id(o) for o in owners}) == nreal
    for x, o in zip(got, owners):
        assert x.shape == size and x.dtype == dtype and x.flags.f_contiguous and x.flags.writeable
        assert o.nbytes == x.nbytes
    if size[0] < 100:
        for x, y in zip(got, O.iqsim(ti, (40, 36), size, seed=9, **kw)):
            assert np.array_equal(x, y)


def test_both_ways_back_give_the_same(iq, monkeypatch):
    from importlib import import_module
    api = import_module("iqgpu.api")
    rng = np.random.default_rng(502)
    ti = rng.integers(0, 3, (40, 38, 12)).astype(np.float32)
    kw = dict(overlap=(0.25,) * 3, nreal=4, rng=2, debug=True)
    runs = []
    for most in (0, 1 << 40):
        monkeypatch.setattr(api, "OWN_BYTES", most)
        runs.append(iq.iqsim(ti, (9, 8, 5), (30, 26, 11), **kw))
    for a, b in zip(*runs):
        for x, y in zip(a, b):
            assert np.array_equal(x, y)
