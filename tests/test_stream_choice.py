"""The automatic choice of `sim.streams` (-1): a context can return to it, and tuning another knob leaves
it alone."""
import numpy as np
import pytest

from oracle import iqsim_oracle as O


class _Recorder:
    """Stands in for a context: keeps the options set."""

    def __init__(self):
        self.options = {}

    def set_option(self, name, value):
        self.options[name] = value


def _tuned(iq, monkeypatch, knobs):
    from importlib import import_module
    monkeypatch.setattr(import_module("iqgpu.api"), "iqsim", lambda *a, **kw: None)
    ctx = _Recorder()
    best, _, hist = iq.autotune(ctx, np.zeros((4, 4)), (2, 2), knobs=knobs, repeats=1)
    return ctx, best, hist


def test_tuning_another_knob_leaves_the_streams_automatic(iq, monkeypatch):
    ctx, best, hist = _tuned(iq, monkeypatch, {"graphcut.threads": (256, 512)})
    assert ctx.options["sim.streams"] == -1 and best["sim.streams"] == -1
    assert all(s["sim.streams"] == -1 for s, _ in hist)


def test_the_automatic_choice_is_the_first_candidate(iq, monkeypatch):
    _, _, hist = _tuned(iq, monkeypatch, None)
    assert hist[0][0]["sim.streams"] == -1
    assert {s["sim.streams"] for s, _ in hist} == {-1, 1, 2}


def test_given_candidates_are_kept(iq, monkeypatch):
    _, best, hist = _tuned(iq, monkeypatch, {"sim.streams": (1, 2)})
    assert {s["sim.streams"] for s, _ in hist} == {1, 2} and best["sim.streams"] in (1, 2)


@pytest.mark.gpu
def test_a_context_returns_to_the_automatic_choice(iq):
    """Continuous images take two groups (as many correlation launches again), integer ones one."""
    rng = np.random.default_rng(401)
    ctx = iq.Context(0)

    def launches(ti):
        ctx.profile(True)
        got = iq.iqsim(ti, (8, 7), (30, 26), overlap=(0.25, 0.25), nreal=2, rng=6, ctx=ctx)
        want = O.iqsim(ti, (8, 7), (30, 26), overlap=(0.25, 0.25), nreal=2, seed=6)
        for x, y in zip(got, want):
            assert np.array_equal(x, y)
        return ctx.profile_get("corr.columns")[1]

    try:
        for ti in (np.exp(rng.normal(size=(40, 36))).astype(np.float32),
                   rng.integers(0, 3, (40, 36)).astype(np.float32)):
            default = launches(ti)
            counts = []
            for v in (1, 2, -1):
                ctx.set_option("sim.streams", v)
                counts.append(launches(ti))
            assert counts[0] < counts[1] and counts[2] == default
        for bad in (-2, 0, 3):
            with pytest.raises(iq.IQError):
                ctx.set_option("sim.streams", bad)
    finally:
        ctx.close()
