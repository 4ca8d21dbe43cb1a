"""The boundary cut's forms against the oracle's exact cut (masks are the canonical minimum cut, so
they must be equal; no tolerance): slabs without and with one interior slice, every cut dimension,
interior sizes around a warp and a flag word, all in shared memory, excesses in global scratch
(4,096 interior nodes), everything in global scratch with 16- and 32-bit heights; capacities from the
table (codes 0..7) and divided one by one (codes above 7, continuous, a mix of both).
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


def _pair(shape, kind, seed):
    rng = np.random.default_rng(seed)
    if kind == "codes":
        return [rng.integers(0, 8, shape).astype(np.float32) for _ in range(2)]
    if kind == "many":
        return [rng.integers(0, 12, shape).astype(np.float32) for _ in range(2)]
    if kind == "mixed":
        a = rng.integers(0, 3, shape).astype(np.float32)
        b = a.copy()
        b.flat[rng.integers(0, b.size)] += 0.5
        return [a, b]
    return [np.exp(rng.normal(size=shape)).astype(np.float32) for _ in range(2)]


@pytest.mark.parametrize("kind", ["codes", "many", "mixed", "continuous"])
@pytest.mark.parametrize("shape,dim", [((1, 9), 0), ((2, 9), 0), ((3, 9), 0), ((9, 3), 1), ((4, 16), 0),
                                       ((6, 33), 0), ((40, 11), 1), ((3, 5, 4), 0), ((7, 5, 6), 1),
                                       ((6, 7, 5), 2), ((8, 32, 16), 0)])
def test_cut_small_and_shared(iq, ctx, shape, dim, kind):
    A, B = _pair(shape, kind, sum(shape) + dim)
    assert np.array_equal(iq.graphcut(A, B, dim, ctx=ctx), O.graphcut(A, B, dim))


@pytest.mark.parametrize("kind", ["codes", "continuous"])
@pytest.mark.parametrize("shape,dim", [((10, 32, 16), 0), ((32, 10, 16), 1), ((14, 32, 20), 0),
                                       ((36, 32, 30), 2)])
def test_cut_in_scratch(iq, ctx, shape, dim, kind):
    A, B = _pair(shape, kind, sum(shape))
    assert np.array_equal(iq.graphcut(A, B, dim, ctx=ctx), O.graphcut(A, B, dim))


@pytest.mark.parametrize("threads,period", [(256, 1), (512, 3), (1024, 48)])
def test_cut_launch_shapes(iq, threads, period):
    A, B = _pair((9, 14, 11), "continuous", 5)
    c = iq.Context(0)
    try:
        c.set_option("graphcut.threads", threads)
        c.set_option("graphcut.gr_period", period)
        got = iq.graphcut(A, B, 0, ctx=c)
    finally:
        c.close()
    assert np.array_equal(got, O.graphcut(A, B, 0))
