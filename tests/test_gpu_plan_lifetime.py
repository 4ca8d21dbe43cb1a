"""The Toeplitz plan of a call (here 0.1 MB of host lists) stays valid until its copy to the device is
done: calls one after the other, each building and dropping a plan, give the SIMT kernel's maps (integer
images: exact, no tolerance)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_plans_outlive_their_copies(iq):
    rng = np.random.default_rng(601)
    ti = rng.integers(0, 4, (75, 70, 20)).astype(np.float32)
    tmpl = rng.integers(0, 4, (3, 64, 60, 16)).astype(np.float32)
    masks = []
    for k in range(4):
        w = np.ones(tmpl.shape[1:], np.uint8)
        w[9 + k:, 7:, 3:] = 0
        masks.append(w)
    simt, tc = iq.Context(0), iq.Context(0)
    simt.set_option("corr.engine", 0)
    try:
        want = [iq.fastdistance(ti, tmpl, w, ctx=simt) for w in masks]
        for _ in range(8):
            for w, x in zip(masks, want):
                assert np.array_equal(iq.fastdistance(ti, tmpl, w, ctx=tc), x)
    finally:
        simt.close()
        tc.close()
