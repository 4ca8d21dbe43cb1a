"""Timed workloads of the image-quilting library, through its public entry points.

Each case is one call a program makes: `iqsim` on 2-D and 3-D training images of every kind the
library distinguishes (binary, categorical and continuous; plain, with hard and soft data, with
inactive voxels; every path), `voxelreuse`, `fastdistance` through the C ABI on device buffers,
and the learned proposal (simulation, window embeddings, loss and gradients). Training images
are seeded Gaussian fields: thresholded (binary), argmax over several (facies codes) or
exponentiated (lognormal).

A case is a dict of plain values; extents are texts such as "128x128x64" in dim-1-first order.
"""
import ctypes
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    """The package directory's name holds a dot, so it is loaded by path."""
    if "iqgpu" not in sys.modules:
        pkg = os.path.join(ROOT, "imagequilting.jl_gb300")
        spec = importlib.util.spec_from_file_location("iqgpu", os.path.join(pkg, "__init__.py"),
                                                      submodule_search_locations=[pkg])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["iqgpu"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["iqgpu"]


def _ext(text):
    return tuple(int(v) for v in text.split("x"))


def _txt(ext):
    return "x".join(str(int(v)) for v in ext)


# ---------------------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------------------
SIM = dict(kind="sim", values="facies", codes=4, dtype="float32", overlap=0.25, tol=0.05,
           path="raster", nreal=1, hard=0, soft=0, inactive=False)


def _sim(name, **kw):
    c = dict(SIM, **kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # choosing a tile size: voxelreuse over ten small realizations, the smallest call
        dict(name="reuse_2d", kind="reuse", values="binary", codes=2, dtype="float64",
             ti="100x100", tile="20x20", overlap=1 / 6, tol=0.1, path="raster", nreal=10),
        # one realization of a binary 2-D image on a larger grid, the reference's plain use:
        # a long chain of small dependent steps
        _sim("sim_2d_binary", values="binary", codes=2, dtype="float64", ti="128x128",
             tile="32x32", out="256x256", overlap=1 / 6, tol=0.1),
        # a 2-D continuous image with large tiles, random path, a handful of realizations
        _sim("sim_2d_continuous", values="lognormal", dtype="float64", ti="250x250",
             tile="62x62", out="250x250", overlap=1 / 6, tol=0.1, path="random", nreal=8),
        # a 2-D categorical image of ragged extents conditioned to wells, an inactive corner in
        # the grid, data-first dilation path, integer type (masked arrays back)
        _sim("sim_2d_wells", codes=3, dtype="uint8", ti="151x133", tile="27x31",
             out="203x187", tol=0.1, path="dilation", nreal=5, hard=40, inactive=True),
        # a 3-D continuous image of odd extents, unconditioned, random path
        _sim("sim_3d_continuous", values="lognormal", ti="91x83x47", tile="21x19x11",
             out="110x97x53", overlap=0.3, tol=0.1, path="random", nreal=3),
        # a 3-D continuous ensemble conditioned to hard data and one soft variable
        _sim("sim_3d_conditioned", values="lognormal", ti="100x100x50", tile="24x24x12",
             out="100x100x50", tol=0.1, nreal=16, hard=60, soft=1),
        # a 3-D facies ensemble, full scan, on a training image of ordinary size
        _sim("sim_3d_facies", ti="128x128x64", tile="32x32x16", out="128x128x64", nreal=8),
        # the same on the largest training image the benchmark uses
        _sim("sim_3d_facies_large", ti="256x256x128", tile="32x32x16", out="96x96x32",
             nreal=16),
        # a 3-D facies ensemble through the learned proposal's shortlists
        dict(name="proposal_sim", kind="lp_sim", codes=4, ti="128x128x64", tile="32x32x16",
             out="192x192x64", overlap=0.25, tol=0.05, nreal=16, k=16384),
        # one training batch of the proposal's encoder: forward, loss and gradients
        dict(name="proposal_train_batch", kind="lp_grad", codes=4, ti="128x128x64",
             tile="32x32x16", overlap=0.25, anchors=128, negatives=32),
        # window embeddings of a set of positions, what a new training image costs per window
        dict(name="proposal_embed", kind="lp_embed", codes=4, ti="128x128x64",
             tile="32x32x16", overlap=0.25, n=20000),
        # distance maps of a batch of templates under an overlap mask, device buffers
        dict(name="distance_3d", kind="dist", values="lognormal", ti="100x100x50",
             tile="24x24x12", overlap=0.25, templates=16, mask="overlap"),
    ]


# (y, z) tile extents the proposal's simulations are drawn from, x extents 16 to 32 (facies
# codes 0..3 and overlap 1/4, the form its benchmark runs)
PROPOSAL_ROWS = ((12, 6), (12, 12), (13, 11), (14, 12), (16, 8), (16, 10), (17, 9), (18, 10),
                 (20, 8), (20, 10), (20, 15), (22, 7), (22, 14), (24, 8), (24, 14), (26, 12),
                 (28, 11), (30, 10), (32, 12), (32, 16))


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def _fits(c, most):
    return work(c)["flops"] <= most


def _most(kind, values=None):
    return max(work(c)["flops"] for c in listed()
               if c["kind"] == kind and (values is None or c["values"] == values))


def draw(rng):
    kind = rng.choice(("reuse", "sim2", "sim2", "sim3c", "sim3f", "sim3f", "lp_sim", "lp_grad",
                       "lp_embed", "dist"))
    ov = round(rng.uniform(0.15, 0.4), 3)
    paths = ("raster", "random", "dilation")
    if kind == "reuse":
        t = [rng.randint(9, 40) for _ in range(2)]
        ti = [v + rng.randint(30, 110) for v in t]
        return dict(kind="reuse", values="binary", codes=2, dtype="float64", ti=_txt(ti),
                    tile=_txt(t), overlap=ov, tol=0.1, path=rng.choice(paths),
                    nreal=rng.randint(2, 12))
    if kind == "sim2":
        while True:
            t = [rng.randint(12, 62) for _ in range(2)]
            ti = [v + _log(rng, 60, 190) for v in t]
            out = [max(v, _log(rng, 64, 260)) for v in t]
            values = rng.choice(("binary", "facies", "lognormal"))
            data = values != "lognormal" and rng.random() < 0.4
            c = _sim(None, values=values, codes=2 if values == "binary" else rng.randint(3, 5),
                     dtype=rng.choice(("float32", "float64")) if values == "lognormal" else
                     rng.choice(("float32", "float64", "uint8")),
                     ti=_txt(ti), tile=_txt(t), out=_txt(out), overlap=ov,
                     tol=rng.choice((0.05, 0.1)), path=rng.choice(paths),
                     nreal=_log(rng, 1, 10), hard=rng.randint(10, 50) if data else 0,
                     inactive=data and rng.random() < 0.5)
            # small tiles on a large grid: no more tiles than the largest listed 2-D case
            if _columns(c) <= 450 and _fits(c, 4 * _most("sim", "binary")):
                return c
    if kind in ("sim3c", "sim3f"):
        cont = kind == "sim3c"
        most = _most("sim", "lognormal" if cont else "facies")
        cols = 1600 if cont else 3000
        while True:
            t = [rng.randint(12, 32), rng.randint(12, 32), rng.randint(7, 16)]
            big = _log(rng, 60, 110 if cont else 250)
            ti = [big, max(40, big - rng.randint(0, 20)), max(30, big // 2)]
            out = [max(v, _log(rng, 48, 128)) for v in t[:2]] + [max(t[2], _log(rng, 20, 64))]
            data = cont and rng.random() < 0.5
            c = _sim(None, values="lognormal" if cont else "facies", codes=rng.randint(2, 6),
                     ti=_txt(ti), tile=_txt(t), out=_txt(out), overlap=ov,
                     tol=rng.choice((0.05, 0.1)), path=rng.choice(paths),
                     nreal=_log(rng, 1, 16), hard=rng.randint(20, 60) if data else 0,
                     soft=1 if data else 0)
            if _columns(c) <= cols and _fits(c, most):
                return c
    if kind == "lp_sim":
        while True:
            t = [rng.randint(16, 32)] + list(rng.choice(PROPOSAL_ROWS))
            big = _log(rng, 80, 128)
            ti = [big, max(64, big - rng.randint(0, 20)), big // 2]
            out = [_log(rng, 64, 192), _log(rng, 64, 192), _log(rng, 32, 64)]
            c = dict(kind="lp_sim", codes=rng.randint(2, 4), ti=_txt(ti), tile=_txt(t),
                     out=_txt(out), overlap=0.25, tol=0.05, nreal=rng.randint(4, 16),
                     k=rng.choice((8192, 16384)))
            if _columns(c) <= 6144 and _fits(c, _most("lp_sim")):
                return c
    ti = [rng.randint(64, 128), rng.randint(64, 128), rng.randint(32, 64)]
    t = [rng.randint(12, 32), rng.randint(12, 32), rng.randint(6, 16)]
    if kind == "lp_grad":
        return dict(kind="lp_grad", codes=rng.choice((3, 4, 6)), ti=_txt(ti), tile=_txt(t),
                    overlap=ov, anchors=_log(rng, 16, 128), negatives=rng.randint(8, 32))
    if kind == "lp_embed":
        return dict(kind="lp_embed", codes=rng.choice((3, 4, 6)), ti=_txt(ti), tile=_txt(t),
                    overlap=ov, n=_log(rng, 1000, 20000))
    while True:
        dims = rng.choice((2, 3))
        t = [rng.randint(12, 62) for _ in range(2)] if dims == 2 else t[:2] + [min(t[2], 12)]
        ti = [v + rng.randint(50, 200) for v in t] if dims == 2 else [100, 90, 47]
        c = dict(kind="dist", values=rng.choice(("lognormal", "facies")), codes=4, ti=_txt(ti),
                 tile=_txt(t), overlap=ov, templates=_log(rng, 1, 32),
                 mask=rng.choice(("overlap", "full", "scattered")))
        if _fits(c, _most("dist")):
            return c


# ---------------------------------------------------------------------------------------
# geometry and algorithmic work
# ---------------------------------------------------------------------------------------
def _overlap(c):
    tile = _ext(c["tile"])
    return [math.ceil(c["overlap"] * t) for t in tile]


def _ntiles(c):
    tile, ov, out = _ext(c["tile"]), _overlap(c), _ext(c["out"])
    return [math.ceil(s / max(t - o, 1)) for s, t, o in zip(out, tile, ov)]


def _live(c):
    """Tiles that start inside the grid."""
    tile, ov, out = _ext(c["tile"]), _overlap(c), _ext(c["out"])
    return [sum(1 for i in range(n) if i * (t - o) < s)
            for n, s, t, o in zip(_ntiles(c), out, tile, ov)]


def _columns(c):
    return int(np.prod(_live(c))) * c["nreal"]


def _positions(c):
    return int(np.prod([a - b + 1 for a, b in zip(_ext(c["ti"]), _ext(c["tile"]))]))


def _overlap_terms(c):
    """Overlap voxels summed over the tiles of one realization: every overlap between
    neighbouring tiles is compared once, whatever the path."""
    tile, ov, n = _ext(c["tile"]), _overlap(c), _live(c)
    total = 0
    for idx in np.ndindex(*n):
        inner = 1
        for i, t, o in zip(idx, tile, ov):
            inner *= t - (o if i > 0 and o > 1 else 0)
        total += int(np.prod(tile)) - inner
    return total


def _cells(c):
    tile = _ext(c["tile"]) + (1,) * (3 - len(_ext(c["tile"])))
    g = (min(tile[0], 8), min(tile[1], 8), min(tile[2], 4))
    g2 = tuple((v + 1) // 2 for v in g)
    g3 = tuple((v + 1) // 2 for v in g2)
    return g, g2, g3


def _encoder_flops(c):
    g, g2, g3 = (int(np.prod(v)) for v in _cells(c))
    return 2.0 * (g * 3 * 32 + g2 * 32 * 32 * 27 + g3 * 32 * 32 * 27 + 32 * g3 * 64)


def work(case):
    """Bytes: inputs read once and outputs written once. FLOPs: the masked distances (two per
    position and offset), or the encoder's multiply-adds."""
    c = case
    nti = int(np.prod(_ext(c["ti"])))
    tile = int(np.prod(_ext(c["tile"])))
    if c["kind"] == "reuse":
        s = dict(c, out=_txt([2 * (t - o) + o if o > 1 else t
                              for t, o in zip(_ext(c["tile"]), _overlap(c))]))
        return {"bytes": 4.0 * nti + 4.0 * c["nreal"] * int(np.prod(_ext(s["out"]))),
                "flops": 2.0 * _positions(s) * _overlap_terms(s) * c["nreal"]}
    if c["kind"] == "sim":
        out = int(np.prod(_ext(c["out"])))
        f = 2.0 * _positions(c) * _overlap_terms(c) * c["nreal"]
        f += 2.0 * _positions(c) * tile * int(np.prod(_live(c))) * c["soft"]
        return {"bytes": 4.0 * (nti * (1 + c["soft"]) + out * (c["nreal"] + c["soft"])),
                "flops": f}
    if c["kind"] == "lp_sim":
        out = int(np.prod(_ext(c["out"])))
        f = _columns(c) * 2.0 * 64 * _positions(c)
        f += 3.0 * c["k"] * _overlap_terms(c) * c["nreal"] + _columns(c) * _encoder_flops(c)
        return {"bytes": 4.0 * (nti + out * c["nreal"]) + 128.0 * _positions(c), "flops": f}
    if c["kind"] == "lp_grad":
        items = c["anchors"] * (2 + c["negatives"])
        return {"bytes": 4.0 * (nti + 12 * c["anchors"] * int(np.prod(_cells(c)[0]))),
                "flops": 3.0 * items * _encoder_flops(c)}
    if c["kind"] == "lp_embed":
        return {"bytes": 4.0 * nti + 264.0 * c["n"], "flops": c["n"] * _encoder_flops(c)}
    k = int(_weights(c).sum())
    return {"bytes": 4.0 * (nti + c["templates"] * (tile + _positions(c))),
            "flops": 2.0 * _positions(c) * k * c["templates"]}


# ---------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------
def _field(shape, gen, sigma):
    """Seeded Gaussian field: white noise smoothed on the torus, zero mean, unit deviation."""
    f = torch.randn(shape, generator=gen, device="cuda", dtype=torch.float64)
    h = torch.fft.fftn(f)
    for d, (n, s) in enumerate(zip(shape, sigma)):
        k = torch.fft.fftfreq(n, device="cuda", dtype=torch.float64)
        e = torch.exp(-2.0 * (math.pi * s * k) ** 2)
        h = h * e.reshape([-1 if i == d else 1 for i in range(len(shape))])
    f = torch.fft.ifftn(h).real
    return (f - f.mean()) / f.std()


def _sigma(shape, c):
    if len(shape) == 2:
        return (8.0, 8.0)
    return (6.0, 6.0, 2.0) if c.get("values") == "lognormal" else (6.0, 6.0, 3.0)


def _values(shape, c, gen):
    sigma = _sigma(shape, c)
    if c.get("values") == "lognormal":
        return torch.exp(_field(shape, gen, sigma))
    if c.get("values") == "binary":
        f = _field(shape, gen, sigma)
        return (f > torch.quantile(f.flatten()[:1 << 20], 0.6)).double()
    f = torch.stack([_field(shape, gen, sigma) for _ in range(c["codes"])])
    return torch.argmax(f, dim=0).double()


def _smooth(a, sigma):
    h = torch.fft.fftn(a)
    for d, n in enumerate(a.shape):
        k = torch.fft.fftfreq(n, device="cuda", dtype=torch.float64)
        e = torch.exp(-2.0 * (math.pi * sigma * k) ** 2)
        h = h * e.reshape([-1 if i == d else 1 for i in range(a.dim())])
    return torch.fft.ifftn(h).real


def _box(c):
    """Mask box of an inner tile of the raster path: overlaps on the low side of every dim."""
    tile = _ext(c["tile"])
    ov = _overlap(c)
    lo = ov + [0] * (3 - len(tile))
    hi = list(tile) + [1] * (3 - len(tile))
    return lo, hi


def _weights(c):
    """Mask of a `dist` case (1: compared), in the tile's shape."""
    tile = _ext(c["tile"])
    w = np.ones(tile, np.uint8)
    if c["mask"] == "overlap":
        w[tuple(slice(o, None) for o in _overlap(c))] = 0
    elif c["mask"] == "scattered":
        w = (np.random.default_rng(5).random(tile) < 0.25).astype(np.uint8)
    return w


def _encoder_params(c, seed):
    """He-initialized parameters in the library's layout (w1 b1 w2 b2 w3 b3 w4 b4)."""
    rng = np.random.default_rng(seed)
    nf = 32 * int(np.prod(_cells(c)[2]))
    parts = []
    for shape in ((32, 3), (32, 32 * 27), (32, 32 * 27), (64, nf)):
        parts.append(rng.normal(size=shape) * math.sqrt(2.0 / shape[1]))
        parts.append(0.02 * rng.normal(size=shape[0]))
    return np.concatenate([p.ravel() for p in parts]).astype(np.float32)


def _features(ti, c, pos):
    """(n, 3, cells) cell inputs (mask fraction, masked mean, masked mean of squares) of the
    windows at linear positions `pos` under the mask of `_box`, Float64."""
    tile = _ext(c["tile"])
    g, _, _ = _cells(c)
    size = [math.ceil(t / n) for t, n in zip(tile, g)]
    dist = [a - b + 1 for a, b in zip(ti.shape, tile)]
    lo, hi = _box(c)
    m = torch.ones(tile, dtype=torch.float64, device="cuda")
    m[lo[0]:hi[0], lo[1]:hi[1], lo[2]:hi[2]] = 0.0
    win = ti.double().unfold(0, tile[0], 1).unfold(1, tile[1], 1).unfold(2, tile[2], 1)
    pos = torch.as_tensor(pos, device="cuda")
    x, y, z = pos % dist[0], (pos // dist[0]) % dist[1], pos // (dist[0] * dist[1])
    padded = [n * s for n, s in zip(g, size)]
    out = torch.empty((pos.numel(), 3) + g, dtype=torch.float64, device="cuda")
    for i in range(0, pos.numel(), 512):
        v = win[x[i:i + 512], y[i:i + 512], z[i:i + 512]]
        for k, q in enumerate((m.expand_as(v), v * m, v * v * m)):
            p = torch.zeros((v.shape[0],) + tuple(padded), dtype=torch.float64, device="cuda")
            p[:, :tile[0], :tile[1], :tile[2]] = q
            p = p.reshape(v.shape[0], g[0], size[0], g[1], size[1], g[2], size[2])
            out[i:i + 512, k] = p.sum(dim=(2, 4, 6)) / float(np.prod(size))
    return out


def _flat_cells(x):
    """(..., gx, gy, gz) to (..., cells) with x fastest."""
    return x.permute(*range(x.dim() - 3), x.dim() - 1, x.dim() - 2, x.dim() - 3).flatten(-3)


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _lp_inputs(c, seed):
    gen = _gen(seed)
    ti = _values(_ext(c["ti"]), dict(c, values="facies"), gen).float()
    params = _encoder_params(c, seed)
    rng = np.random.default_rng(seed + 1)
    P = _positions(c)
    s = dict(ti=ti, params=params, box=_box(c))
    if c["kind"] == "lp_embed":
        s["pos"] = rng.integers(0, P, c["n"])
    elif c["kind"] == "lp_grad":
        s["anchor"] = rng.integers(0, P, c["anchors"])
        # a positive looks like its anchor: a window next to it
        s["pos"] = np.clip(s["anchor"] + rng.integers(-2, 3, c["anchors"]), 0, P - 1)
        s["neg"] = rng.integers(0, P, c["anchors"] * c["negatives"])
        s["feats"] = _flat_cells(_features(ti, c, s["anchor"])).float().cpu().numpy()
    return s


def prepare(case, seed):
    iq = _package()
    c = dict(case, seed=int(seed))
    gen = _gen(seed)
    if c["kind"] in ("sim", "reuse"):
        ti = _values(_ext(c["ti"]), c, gen)
        s = dict(c=c, iq=iq, ti=ti.cpu().numpy().astype(c["dtype"]))
        if c["kind"] == "reuse":
            return s
        out = _ext(c["out"])
        kw = dict(overlap=(c["overlap"],) * len(out), tol=c["tol"], path=c["path"],
                  nreal=c["nreal"], rng=int(seed))
        other = _values(out, c, gen) if c["hard"] or c["soft"] else None
        if c["hard"]:
            # data of another realization of the same field; an inactive corner block on request
            rng = np.random.default_rng(seed)
            ref = other.cpu().numpy()
            pts = np.stack([rng.integers(0, n, c["hard"]) for n in out], axis=1)
            hard = {tuple(int(v) for v in p): float(ref[tuple(p)]) for p in pts}
            if c["inactive"]:
                for p in np.ndindex(*[max(1, n // 5) for n in out]):
                    hard[p] = float("nan")
            kw["hard"] = hard
        if c["soft"]:
            kw["soft"] = [(_smooth(other, 4.0).float().cpu().numpy(),
                           _smooth(ti, 4.0).float().cpu().numpy())]
        s["kw"] = kw
        return s
    if c["kind"] == "dist":
        ctx = iq.Context(0)
        ti = _values(_ext(c["ti"]), c, gen).float()
        tile = _ext(c["tile"])
        # templates are patches of another field, as the overlap of a simulation grid is
        other = _values([2 * t for t in tile], c, gen).float()
        rng = np.random.default_rng(seed)
        tm = []
        for _ in range(c["templates"]):
            o = [int(rng.integers(0, t + 1)) for t in tile]
            p = other[tuple(slice(a, a + t) for a, t in zip(o, tile))]
            tm.append(p.permute(*range(p.dim() - 1, -1, -1)).flatten())
        ctx.set_ti(ti.cpu().numpy())
        w = torch.from_numpy(_weights(c).ravel(order="F").copy()).cuda()
        out = torch.empty((c["templates"], _positions(c)), dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        return dict(c=c, iq=iq, ctx=ctx, ti=ti, tmpl=torch.stack(tm), w=w, out=out)
    s = _lp_inputs(c, int(seed))
    ctx = iq.Context(0)
    tih = s["ti"].cpu().numpy()
    ctx.set_ti(tih)
    ctx.lp_set_params(_ext(c["tile"]), s["params"])
    if c["kind"] == "lp_sim":
        ctx.set_option("lp.enable", 1)
        ctx.set_option("lp.k", c["k"])
        # the encoder is not trained here: its shortlists are kept whatever they recall
        ctx.set_option("lp.fallback", 0)
    s.update(c=c, iq=iq, ctx=ctx, tih=tih)
    return s


def run(state):
    s, c, iq = state, state["c"], state["iq"]
    if c["kind"] == "sim":
        return iq.iqsim(s["ti"], _ext(c["tile"]), _ext(c["out"]), **s["kw"])
    if c["kind"] == "reuse":
        return iq.voxelreuse(s["ti"], _ext(c["tile"]), overlap=(c["overlap"],) * 2,
                             nreal=c["nreal"], tol=c["tol"], path=c["path"], rng=c["seed"])
    if c["kind"] == "dist":
        from iqgpu import _lib
        _lib.check(iq.load().iq_fastdistance(s["ctx"].h, _lib.i64arr(_ext(c["tile"])),
                                             c["templates"], s["tmpl"].data_ptr(),
                                             s["w"].data_ptr(), s["out"].data_ptr()))
        return s["out"]
    if c["kind"] == "lp_sim":
        return iq.iqsim(s["tih"], _ext(c["tile"]), _ext(c["out"]),
                        overlap=(c["overlap"],) * 3, tol=c["tol"], nreal=c["nreal"],
                        rng=c["seed"], ctx=s["ctx"])
    lo, hi = s["box"]
    if c["kind"] == "lp_embed":
        return s["ctx"].lp_embed(s["pos"], lo + hi)
    loss, grad = s["ctx"].lp_loss_grad(s["feats"], s["pos"], s["neg"], lo + hi, 8.0)
    return {"loss": loss, "grad": grad}


# ---------------------------------------------------------------------------------------
# the same in 64 bits, without the library
# ---------------------------------------------------------------------------------------
def _encode(params, c, x):
    """Embeddings (n, 64) of cell inputs x (n, 3, gx, gy, gz)."""
    p, off = [], 0
    g3 = _cells(c)[2]
    nf = 32 * int(np.prod(g3))
    for shape in ((32, 3), (32,), (32, 32, 27), (32,), (32, 32, 27), (32,), (64, nf), (64,)):
        n = int(np.prod(shape))
        p.append(params[off:off + n].reshape(shape))
        off += n
    relu = torch.relu

    def taps(w):  # tap dx + 3 dy + 9 dz
        return w.reshape(32, 32, 3, 3, 3).permute(0, 1, 4, 3, 2)

    h = relu(torch.einsum("ci,nixyz->ncxyz", p[0], x) + p[1][None, :, None, None, None])
    h = relu(torch.nn.functional.conv3d(h, taps(p[2]), p[3], stride=2, padding=1))
    h = relu(torch.nn.functional.conv3d(h, taps(p[4]), p[5], stride=2, padding=1))
    f = _flat_cells(h).transpose(1, 2).flatten(1)  # cell-major, channel fastest
    return f @ p[6].T + p[7]


def exact(case, seed):
    c = dict(case)
    if c["kind"] == "dist":
        s = prepare(c, seed)
        tile = _ext(c["tile"])
        ti = s["ti"].double()
        w = torch.from_numpy(_weights(c)).cuda().double()
        tm = s["tmpl"].double()
        tm = tm.reshape((c["templates"],) + tile[::-1]).permute(0, *range(len(tile), 0, -1))
        conv = torch.nn.functional.conv2d if len(tile) == 2 else torch.nn.functional.conv3d
        out = torch.empty((c["templates"], _positions(c)), dtype=torch.float64, device="cuda")
        with torch.backends.cudnn.flags(enabled=False):
            a2 = conv((ti * ti)[None, None], w[None, None])[0, 0]
            for i in range(c["templates"]):
                d = a2 - 2.0 * conv(ti[None, None], (tm[i] * w)[None, None])[0, 0]
                d = (d + (w * tm[i] * tm[i]).sum()).abs()
                out[i] = d.permute(*range(d.dim() - 1, -1, -1)).flatten()
        return out
    if c["kind"] == "lp_embed":
        s = _lp_inputs(c, int(seed))
        # inference reads BF16 weights (w2, w3, w4 and w1) and Float32 biases
        p = torch.from_numpy(s["params"]).cuda().bfloat16().double()
        return _encode(p, c, _features(s["ti"], c, s["pos"])).cpu().numpy()
    if c["kind"] == "lp_grad":
        s = _lp_inputs(c, int(seed))
        p = torch.from_numpy(s["params"]).cuda().double().requires_grad_()
        nA, nn = c["anchors"], c["negatives"]
        g = _cells(c)[0]
        a = torch.from_numpy(s["feats"]).cuda().double()
        a = a.reshape((nA, 3) + g[::-1]).permute(0, 1, 4, 3, 2)
        w = _features(s["ti"], c, np.concatenate([s["pos"], s["neg"]]))
        with torch.backends.cudnn.flags(enabled=False):
            e = _encode(p, c, torch.cat([a, w]))
            ea = e[:nA]
            ej = torch.cat([e[nA:2 * nA, None], e[2 * nA:].reshape(nA, nn, 64)], dim=1)
            z = -((ea[:, None] - ej) ** 2).sum(-1) / 8.0
            loss = (torch.logsumexp(z, 1) - z[:, 0]).mean()
            loss.backward()
        return {"loss": float(loss.detach()), "grad": p.grad.cpu().numpy()}
    return None
