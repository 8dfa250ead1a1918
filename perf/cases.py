"""What is timed of this framework: deconvolution calls and transforms over the sizes they are used at.

A case names one public call and its sizes.  `listed` gives the standing cases, `draw` more of the same ranges,
`prepare` what a program holds before the call, `run` the call, `work` the bytes and operations it cannot do
without and `exact` its result in 64 bits, from plain torch.

Sizes are (planes, rows, columns), x fastest, as everywhere in the package.  Iteration counts are at the lower end
of what is used (5 to 30; a served request asks for 20 or more): the time of a run is its set-up plus a constant per
iteration, and the set-up counts most in the short runs.
"""
import math

import numpy as np
import torch

import deconwolf_b200 as dw


# ------------------------------------------------------------------ cases

def _case(name, kind, shape, psf=(0, 0, 0), **kw):
    c = {"name": name, "kind": kind, "P": shape[0], "N": shape[1], "M": shape[2], "pP": psf[0], "pN": psf[1],
         "pM": psf[2], "method": "shb", "iters": 0, "bq": 2, "stop": "fixed", "start": "flat", "metric": "idiv",
         "images": 1, "tile": 0, "err": 0.02}
    c.update(kw)
    return c


def listed():
    return [
        # a small crop around one object, tried with a few settings: launches and host work
        _case("crop", "call", (10, 48, 40), (7, 9, 11), iters=10),
        # one focal plane (no z): a 2-D image against a 2-D PSF
        _case("plane", "call", (1, 700, 903), (1, 63, 63), iters=30, method="rl"),
        # a quick look with circular borders at sizes that have no transform of their own
        _case("quick_ragged", "call", (33, 241, 317), (21, 31, 31), iters=15, bq=1, start="identity"),
        # a field from one nucleus' neighbourhood
        _case("field_256", "call", (40, 256, 256), (79, 127, 127), iters=20),
        # frames of one size through a job that stays set up on the device
        _case("frames_512", "job", (40, 512, 512), (79, 181, 181), iters=20, method="rl"),
        # a whole camera field, resident on the device: the headline workload
        _case("camera_2048", "call", (60, 2048, 2048), (119, 181, 181), iters=20),
        # four small channels at once
        _case("channels_256", "batch", (20, 256, 256), (39, 181, 181), iters=20, images=4),
        # host arrays, run until the error settles
        _case("host_stop", "host", (31, 260, 301), (61, 65, 65), iters=40, stop="rel", err=0.001),
        # host arrays, a larger field
        _case("host_1024", "host", (60, 1024, 1024), (119, 181, 181), iters=10),
        # an image in overlapping tiles, from and to host arrays
        _case("tiles", "tiled", (30, 900, 1100), (59, 101, 101), iters=10, tile=512),
        # the transforms by themselves, each direction
        _case("r2c", "r2c", (60, 512, 512)),
        _case("c2r_ragged", "c2r", (45, 375, 630)),
    ]


_RADICES = [r for r in range(2, 17) if all(r % p for p in (11, 13))]


def _lengths(most):
    """Lengths with a transform: products of at most three factors of at most 16 over 2, 3, 5 and 7."""
    out = {a * b * c for a in _RADICES + [1] for b in _RADICES + [1] for c in _RADICES + [1]}
    return sorted(n for n in out if 8 <= n <= most)


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["call", "call", "call", "job", "host", "host", "batch", "tiled", "r2c", "c2r"])
    if kind in ("r2c", "c2r"):
        near = lambda v, even: min((n for n in _lengths(1200) if not even or n % 2 == 0), key=lambda n: abs(n - v))  # noqa: E731
        x = 2 * near(_log(rng, 32, 1024) // 2, False)
        return _case("", kind, (near(_log(rng, 8, 128), False), near(_log(rng, 32, 1024), False), x))
    big = {"call": 1536, "job": 768, "host": 768, "batch": 300, "tiled": 1000}[kind]
    N, M = _log(rng, 400 if kind == "tiled" else 40, big), _log(rng, 400 if kind == "tiled" else 40, big)
    P = 1 if kind == "call" and rng.random() < 0.15 else _log(rng, 8, 30 if kind == "tiled" else 64)
    side = lambda n: 2 * _log(rng, 5, max(6, min(90, n))) + 1  # noqa: E731
    lateral = side(min(N, M) // 2)
    bq = rng.choice([2, 2, 2, 1, 0])
    return _case("", kind, (P, N, M), (1 if P == 1 else min(2 * P - 1, side(P)), lateral, lateral),
                 method=rng.choice(["shb", "shb", "rl"]), iters=_log(rng, 5, 20), bq=bq,
                 stop="rel" if kind == "host" and rng.random() < 0.4 else "fixed",
                 err=rng.choice([0.02, 0.005, 0.001]),
                 start=rng.choice(["flat", "flat", "identity"]), metric=rng.choice(["idiv", "idiv", "mse"]),
                 images=rng.randint(2, 6) if kind == "batch" else 1,
                 tile=rng.randint(150, 399) if kind == "tiled" else 0)


# ------------------------------------------------------------------ inputs

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _psf(size, g):
    """A widefield-like PSF, sum 1: every plane holds the same energy, spread wider away from focus."""
    pP, pN, pM = size
    u = torch.rand(3, generator=g, device="cuda", dtype=torch.float64)
    z = torch.arange(pP, device="cuda", dtype=torch.float64) - (pP - 1) / 2
    y = torch.arange(pN, device="cuda", dtype=torch.float64) - (pN - 1) / 2
    x = torch.arange(pM, device="cuda", dtype=torch.float64) - (pM - 1) / 2
    s = (1.1 + 0.4 * u[0]) * torch.sqrt(1 + (z / (2.5 + u[1])) ** 2)
    s = torch.clamp(s, max=max(1.0, min(pN, pM) / 4))[:, None, None]
    p = torch.exp(-(y[None, :, None] ** 2 + x[None, None, :] ** 2) / (2 * s * s)) / (s * s)
    p = p * torch.exp(-0.5 * (z / max(1.0, 0.6 * pP)) ** 2)[:, None, None]
    return (p / p.sum()).to(torch.float32).contiguous()


def _image(shape, psf, g):
    """Photon counts of point sources and faint blobs seen through the PSF, on a background."""
    obj = (torch.rand(shape, generator=g, device="cuda") < 4e-4).float()
    obj *= 2000 + 4000 * torch.rand(shape, generator=g, device="cuda")
    # blurred as a circular image: what matters is what the counts look like
    k = torch.zeros(shape, device="cuda")
    c = [min(a, b) for a, b in zip(shape, psf.shape)]
    lo = [(b - a) // 2 for a, b in zip(c, psf.shape)]
    k[: c[0], : c[1], : c[2]] = psf[lo[0]: lo[0] + c[0], lo[1]: lo[1] + c[1], lo[2]: lo[2] + c[2]]
    k = torch.roll(k, shifts=[-(a // 2) for a in c], dims=(0, 1, 2))
    blur = torch.fft.irfftn(torch.fft.rfftn(obj) * torch.fft.rfftn(k / k.sum()), s=shape)
    return torch.poisson(torch.clamp(blur, min=0) + 80.0, generator=g).clamp(max=65535).contiguous()


def _inputs(case, seed):
    g = _gen(seed)
    shape = (case["P"], case["N"], case["M"])
    if case["kind"] in ("r2c", "c2r"):
        return torch.randn(shape, generator=g, device="cuda") + 3.0, None
    psf = _psf((case["pP"], case["pN"], case["pM"]), g)
    return [_image(shape, psf, g) for _ in range(case["images"])], psf


def _options(case):
    return dict(method=case["method"], n_iter=case["iters"], maxiter=case["iters"], border_quality=case["bq"],
                iter_type=dw.ITER_REL if case["stop"] == "rel" else dw.ITER_FIXED, err_rel=case["err"],
                start=dw.START_IDENTITY if case["start"] == "identity" else dw.START_FLAT,
                metric=dw.METRIC_MSE if case["metric"] == "mse" else dw.METRIC_IDIV)


def prepare(case, seed):
    data, psf = _inputs(case, seed)
    kind, shape = case["kind"], (case["P"], case["N"], case["M"])
    st = {"kind": kind, "shape": shape, "opts": _options(case), "case": case}
    if kind == "r2c":
        st["in"] = data
        st["out"] = torch.empty(shape[:2] + (shape[2] // 2 + 1, 2), device="cuda")
    elif kind == "c2r":
        st["in"] = torch.view_as_real(torch.fft.rfftn(data)).contiguous()
        st["out"] = torch.empty(shape, device="cuda")
    elif kind in ("host", "tiled"):
        st["in"], st["psf"] = data[0].cpu().numpy(), psf.cpu().numpy()
    else:
        st["in"], st["psf"] = data, psf
        st["out"] = [torch.empty(shape, device="cuda") for _ in data]
        if kind in ("job", "batch"):
            st["jobs"] = [dw.Job(shape, tuple(psf.shape), **st["opts"]) for _ in data]
    torch.cuda.synchronize()
    torch.cuda.empty_cache()  # the engine allocates beside torch
    return st


def run(st):
    kind, shape = st["kind"], st["shape"]
    if kind == "call":
        r = dw.run_method_device(st["in"][0].data_ptr(), st["psf"].data_ptr(), st["out"][0].data_ptr(), shape,
                                 tuple(st["psf"].shape), **st["opts"])
        return [st["out"][0], r.trace]
    if kind == "job":
        j = st["jobs"][0]
        j.setup(st["in"][0].data_ptr(), st["psf"].data_ptr(), on_device=True)
        j.step(st["opts"]["n_iter"])
        return [st["out"][0], j.result(st["out"][0].data_ptr(), on_device=True).trace]
    if kind == "batch":
        for j, im in zip(st["jobs"], st["in"]):
            j.setup(im.data_ptr(), st["psf"].data_ptr(), on_device=True)
        dw.batch_run(st["jobs"])
        return [[o, j.result(o.data_ptr(), on_device=True).trace] for j, o in zip(st["jobs"], st["out"])]
    if kind == "host":
        r = dw.run_method(st["in"], st["psf"], **st["opts"])
        # how many steps the stopping rule let run depends on the image
        return [r.out, np.pad(r.trace, (0, st["opts"]["n_iter"] - r.iterations)), r.iterations]
    if kind == "tiled":
        return [dw.deconvolve_tiled(st["in"], st["psf"], st["case"]["tile"], **st["opts"]).out]
    if kind == "r2c":
        dw.fft_r2c_device(st["in"].data_ptr(), shape, st["out"].data_ptr())
    else:
        dw.fft_c2r_device(st["in"].data_ptr(), shape, st["out"].data_ptr())
    return st["out"]


# ------------------------------------------------------------------ what a pass cannot do without

def _job_size(shape, psf, bq):
    if bq == 2:
        return tuple(s + p - 1 for s, p in zip(shape, psf))
    return tuple(s + (p + 1) // 2 if bq == 1 else max(s, p) for s, p in zip(shape, psf))


def work(case):
    shape, psf = (case["P"], case["N"], case["M"]), (case["pP"], case["pN"], case["pM"])
    v = float(np.prod(shape))
    if case["kind"] in ("r2c", "c2r"):
        return {"bytes": 4 * v + 8 * v / shape[2] * (shape[2] // 2 + 1), "flops": 2.5 * v * math.log2(v)}
    w = float(np.prod(_job_size(shape, psf, case["bq"])))
    # four transforms of the job a step, three at the set-up (OTF and border weights)
    flops = 2.5 * w * math.log2(w) * (4 * case["iters"] + 3)
    return {"bytes": case["images"] * (8 * v + 4 * float(np.prod(psf))), "flops": case["images"] * flops}


# ------------------------------------------------------------------ 64 bits

def _smooth(n):
    while True:
        m = n
        for p in (2, 3, 5, 7):
            while m % p == 0:
                m //= p
        if m == 1:
            return n
        n += 1


def _deconvolve64(im, psf, case):
    """The iteration with every value in 64 bits; the image and the PSF are the 32-bit inputs."""
    g, bq, shb = im.double(), case["bq"], case["method"] == "shb"
    P, N, M = g.shape
    w = _job_size(tuple(g.shape), tuple(psf.shape), bq)
    logical = float(np.prod(w))
    if bq == 2:  # the whole PSF fits beside the image: a larger transform gives the same
        w = tuple(_smooth(n) for n in w)
    bg = max(float(g.min()), 0.01)
    Z = torch.zeros(w, dtype=torch.float64, device=g.device)
    Z[: psf.shape[0], : psf.shape[1], : psf.shape[2]] = psf.double()
    at = np.unravel_index(int(torch.argmax(Z)), w)
    K = torch.fft.rfftn(torch.roll(Z, shifts=[-int(i) for i in at], dims=(0, 1, 2)))
    del Z

    def conv(x, conj):
        s = torch.fft.rfftn(x)
        s *= K.conj() if conj else K
        return torch.fft.irfftn(s, s=w)

    img = (slice(0, P), slice(0, N), slice(0, M))
    W = 1.0
    if bq > 0:
        one = torch.zeros(w, dtype=torch.float64, device=g.device)
        one[img] = 1.0
        one = conv(one, True)
        W = torch.where(one > 0.01, 1.0 / one, torch.zeros_like(one))
        del one
    if case["start"] == "identity":
        x = torch.zeros(w, dtype=torch.float64, device=g.device)
        x[img] = g
    else:
        x = torch.full(w, float(g.sum()) / logical, dtype=torch.float64, device=g.device)
    last, trace = x, []
    error, before = 1.0, 1.0
    k = 0
    while True:
        if case["stop"] == "rel":
            if k < 2:
                before = 2 * error * case["err"]
            if abs(error - before) / error < case["err"]:
                break
        if k >= case["iters"]:
            break
        p = x
        if shb:
            a = min(max((k - 1.0) / (k + 2.0), 0.0), 1.0)
            p = torch.clamp(x + a * (x - last), min=bg)
        y = conv(p, False)[img].contiguous()
        if case["metric"] == "mse":
            e = float(((y - g) ** 2).sum()) / g.numel()
        else:
            ok = (y > 0) & (g > 0)
            yy, gg = torch.where(ok, y, torch.ones_like(y)), torch.where(ok, g, torch.ones_like(g))
            e = float((gg * torch.log(gg / yy) - (gg - yy)).sum()) / g.numel()
        trace.append(e)
        before, error = error, e
        if shb:
            r = torch.zeros(w, dtype=torch.float64, device=g.device)
            r[img] = g / torch.where(y.abs() < 1e-6, torch.copysign(torch.full_like(y, 1e-6), y), y)
        else:
            r = torch.full(w, 1e-6, dtype=torch.float64, device=g.device)
            r[img] = torch.where(y > 0, g / y, torch.full_like(y, bg))
        del y
        r = conv(r, True)
        r *= p
        r *= W
        r.clamp_(min=bg)
        last, x = x, r
        k += 1
    return (last if shb else x)[img].contiguous(), np.array(trace)


def _crop_psf(psf, shape, bq):
    """The PSF of one tile: sum 1, no larger than the tile needs, faint outer planes off, sum 1 again."""
    p = psf.double() / psf.double().sum()
    most = shape if bq == 0 else tuple(2 * s - 1 for s in shape)
    if p.shape[0] >= most[0]:
        cut = [max(0, (a - b) // 2) for a, b in zip(p.shape, most)]
        p = p[cut[0]: p.shape[0] - cut[0], cut[1]: p.shape[1] - cut[1], cut[2]: p.shape[2] - cut[2]]
    if bq > 0:
        s = p.sum(dim=(0, 1))
        f = int(torch.nonzero(s >= 0.001 * s.max())[0])
        if f >= 1 and min(p.shape[1], p.shape[2]) - 2 * f >= 1:
            p = p[:, f: p.shape[1] - f, f: p.shape[2] - f]
    return (p / p.sum()).float().contiguous()


def _tiled64(im, psf, case):
    P, N, M = im.shape
    overlap, offset = 20, 5.0

    def parts(n):
        c = math.ceil(n / case["tile"])
        ends = [math.ceil(np.float32(n) / np.float32(c) * np.float32(i)) for i in range(1, c)] + [n]
        return [(a, b - 1) for a, b in zip([0] + ends[:-1], ends)]

    def weight(n, lo, hi):
        """1 inside [lo, hi], falling off over the overlap."""
        a, d = max(0, lo - overlap), min(n - 1, hi + overlap)
        i = torch.arange(n, device="cuda", dtype=torch.float64)
        w = torch.zeros_like(i)
        w = torch.where((i >= a) & (i <= lo), (i - a + 1) / (lo - a + 1), w)
        w = torch.where((i >= hi) & (i <= d), 1 - (i - hi) / (d - hi + 1), w)
        return torch.where((i >= lo) & (i <= hi), torch.ones_like(w), w), a, d

    tiles = [(weight(M, *m), weight(N, *n)) for m in parts(M) for n in parts(N)]
    planes = [torch.minimum(wn[0][:, None], wm[0][None, :]) for wm, wn in tiles]
    total, out = sum(planes), torch.zeros(im.shape, dtype=torch.float64, device="cuda")
    for (wm, wn), w in zip(tiles, planes):
        at = (slice(None), slice(wn[1], wn[2] + 1), slice(wm[1], wm[2] + 1))
        part = im[at] + offset
        r, _ = _deconvolve64(part, _crop_psf(psf, tuple(part.shape), case["bq"]), case)
        out[at] += torch.clamp(r - offset, min=0) * (w / total)[at[1:]]
    return out


def exact(case, seed):
    data, psf = _inputs(case, seed)
    kind, shape = case["kind"], (case["P"], case["N"], case["M"])
    if kind == "r2c":
        return torch.view_as_real(torch.fft.rfftn(data.double()))
    if kind == "c2r":
        return torch.fft.irfftn(torch.fft.rfftn(data).to(torch.complex128), s=shape, norm="forward")
    if kind == "tiled":
        return [_tiled64(data[0], psf, case)]
    got = [list(_deconvolve64(im, psf, case)) for im in data]
    if kind == "host":
        out, trace = got[0]
        return [out, np.pad(trace, (0, case["iters"] - len(trace))), len(trace)]
    return got if kind == "batch" else got[0]
