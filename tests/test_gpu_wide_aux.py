"""Wide-range operands beside an image that FP16 halves would hold: their maps come from the TF32 form,
and no FP16 image is made for them (as many launches as with the TF32 engine; realizations equal the
oracle's, decided on Float64 distances)."""
import numpy as np
import pytest

from oracle import iqsim_oracle as O

pytestmark = pytest.mark.gpu


def test_no_fp16_image_for_wide_range_soft_data(iq):
    rng = np.random.default_rng(901)
    ti = np.exp(6.0 * rng.normal(size=(40, 36))).astype(np.float32)      # wide range
    auxti = (1.0 + rng.random(ti.shape)).astype(np.float32)               # within a factor of two
    aux = np.exp(6.0 * rng.normal(size=(30, 28))).astype(np.float32)     # wide range
    kw = dict(overlap=(0.25, 0.25), nreal=2, soft=[(aux, auxti)])
    want = O.iqsim(ti, (8, 7), (30, 28), seed=2, **kw)
    counts = []
    for engine in (2, 1):
        ctx = iq.Context(0)
        try:
            ctx.set_option("corr.engine", engine)
            for x, y in zip(iq.iqsim(ti, (8, 7), (30, 28), rng=2, ctx=ctx, **kw), want):
                assert np.array_equal(x, y)
            counts.append(ctx.launches)
        finally:
            ctx.close()
    assert counts[0] == counts[1]


def test_no_fp16_image_for_wide_range_templates(iq):
    """The same for maps of wide-range templates, TF32 in either engine: the same bits."""
    rng = np.random.default_rng(902)
    ti = (1.0 + rng.random((30, 28, 12))).astype(np.float32)
    tmpl = np.exp(6.0 * rng.normal(size=(3, 8, 7, 4))).astype(np.float32)
    runs, counts = [], []
    for engine in (2, 1):
        ctx = iq.Context(0)
        try:
            ctx.set_option("corr.engine", engine)
            runs.append(iq.fastdistance(ti, tmpl, ctx=ctx))
            counts.append(ctx.launches)
        finally:
            ctx.close()
    assert np.array_equal(*runs) and counts[0] == counts[1]
