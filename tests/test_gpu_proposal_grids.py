"""The encoder's kernels over the cell grids their work splits depend on (rows of layer 2's output
per item 1, 3, 4, 8; odd extents, whose last taps fall outside; 1-D to 3-D tiles; item counts that
are not multiples of a batch), for integer images (32-bit cell sums) and others (Float64 ones),
against the Float64 oracle.

Tolerances as in test_gpu_proposal.py: embeddings within 1e-2 of their scale (BF16 outputs: 2^-9
each), loss and gradients within 2e-3 (2-norm; FP32 sums of at most a few thousand terms, 2^-24
each, give below 1e-4 even if every rounding pointed the same way).
"""
import numpy as np
import pytest

from oracle import proposal_oracle as Q

pytestmark = pytest.mark.gpu

CASES = [((40,), (7,), (40,), True), ((40, 33), (16, 16), (4, 5), True),
         ((30, 25), (12, 5), (12, 2), False), ((14, 13, 9), (5, 7, 3), (2, 7, 1), True),
         ((14, 13, 9), (3, 3, 3), (1, 1, 1), False), ((20, 19, 12), (9, 6, 2), (3, 2, 1), True),
         ((24, 22, 20), (16, 10, 12), (4, 3, 3), False)]


def _params(flat, tile):
    p, off = {}, 0
    for k, s in Q.param_shapes(tile).items():
        n = int(np.prod(s))
        p[k] = flat[off:off + n].astype(np.float64).reshape(s)
        off += n
    return p


def _bf16(x):
    u = np.asarray(x, np.float32).view(np.uint32).astype(np.uint64)
    return ((u + 0x7FFF + ((u >> 16) & 1)) & 0xFFFF0000).astype(np.uint32).view(np.float32)


def _setup(iq, shape, tile, lo, integer):
    rng = np.random.default_rng(sum(shape) + sum(tile))
    ti = (rng.integers(0, 5, shape) if integer else rng.normal(size=shape)).astype(np.float32)
    ctx = iq.Context(0)
    ctx.set_ti(ti)
    ctx.lp_init(tile, seed=3)
    flat = ctx.lp_params()
    flat = flat + (0.05 * rng.normal(size=flat.size)).astype(np.float32)  # nonzero biases too
    ctx.lp_set_params(tile, flat)
    pad = (0,) * (3 - len(tile))
    box = tuple(min(v, t) for v, t in zip(lo, tile)) + pad + tuple(tile) + tuple(1 for _ in pad)
    m = np.ones(tile, bool)
    m[tuple(slice(a, t) for a, t in zip(lo, tile))] = False
    dist = tuple(T - t + 1 for T, t in zip(shape, tile))

    def feats(q):
        at = np.unravel_index(q, dist, order="F")
        w = ti[tuple(slice(a, a + t) for a, t in zip(at, tile))]
        ext = tile + (1,) * (3 - len(tile))
        return Q.cell_features(w.reshape(ext), m.reshape(ext), ext)

    return ctx, flat, box, dist, feats, rng


@pytest.mark.parametrize("shape,tile,lo,integer", CASES)
def test_embeddings_vs_oracle(iq, shape, tile, lo, integer):
    ctx, flat, box, dist, feats, rng = _setup(iq, shape, tile, lo, integer)
    try:
        pos = rng.integers(0, int(np.prod(dist)), 37)
        got = ctx.lp_embed(pos, box)
    finally:
        ctx.close()
    p = _params(_bf16(flat), tile)
    for i, q in enumerate(pos):
        ref = Q.forward(p, feats(q))[0]
        assert np.allclose(got[i], ref, rtol=1e-2, atol=1e-2 * np.abs(ref).max())


@pytest.mark.parametrize("shape,tile,lo,integer", CASES)
def test_gradients_vs_oracle(iq, shape, tile, lo, integer):
    ctx, flat, box, dist, feats, rng = _setup(iq, shape, tile, lo, integer)
    nA, nneg, temp = 3, 5, 8.0
    P = int(np.prod(dist))
    a, pos, neg = rng.integers(0, P, nA), rng.integers(0, P, nA), rng.integers(0, P, nA * nneg)
    A = np.stack([feats(q) for q in a])
    try:
        loss, grad = ctx.lp_loss_grad(
            np.stack([x.reshape(3, -1, order="F") for x in A]).astype(np.float32), pos, neg, box, temp)
    finally:
        ctx.close()
    N = np.stack([feats(q) for q in neg]).reshape((nA, nneg) + A.shape[1:])
    ref_loss, ref = Q.batch_loss_and_grads(_params(flat, tile), A, np.stack([feats(q) for q in pos]),
                                           N, temp)
    assert abs(loss - ref_loss) <= 2e-3 * max(1.0, abs(ref_loss))
    g = _params(grad, tile)
    for k in ref:
        assert np.linalg.norm(g[k] - ref[k]) <= 2e-3 * np.linalg.norm(ref[k]) + 1e-6, k
