"""The calls a program makes of this framework, with the sizes it makes them at.

One reconstruction is a chain of hundreds of HIO iterations, so most of these
cases are whole calls: the drop-in, a plan, a fixed-support HIO, a batch
through the engine.  The rest are the kernel-level entry points that programs
call by themselves (2D transform, blur, forward model).

A reconstruction returns its image whole, with the cycles it took.  HIO is
chaotic: a difference of one rounding grows by two to three times in every
iteration (the support constraint and the division by |G| are
discontinuous), so after a few dozen iterations 64-bit arithmetic is in another place than
32-bit arithmetic, and no two 32-bit implementations agree.  exact() therefore
gives values for the transforms, the blur and the forward model, and None for
reconstructions.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

import imresh_b200 as imr

DEV = "cuda"
CONFIG_SIDES = (128, 192, 256, 384, 512)   # sides of the uneven batch


def listed():
    return [
        # smallest call: one inverse transform of a small field, launch latency
        {"name": "fft_64x48", "kind": "fft", "width": 64, "height": 48, "sign": 1},
        # ordinary forward transform of a detector-sized field
        {"name": "fft_1024", "kind": "fft", "width": 1024, "height": 1024, "sign": -1},
        # support blur of a large magnitude image at the first cycle's width
        {"name": "blur_2048x1536", "kind": "blur", "width": 2048, "height": 1536, "sigma": 3.0},
        # forward model of a rectangular object in host memory
        {"name": "forward_1000x800", "kind": "forward", "width": 1000, "height": 800},
        # the drop-in with the reference's default counts, host buffer in and out
        {"name": "dropin_256", "kind": "dropin", "width": 256, "height": 256, "cycles": 20, "hio": 20},
        # the drop-in at the size of the reference's example (5-smooth sides)
        {"name": "dropin_600x300", "kind": "dropin", "width": 600, "height": 300, "cycles": 20, "hio": 20},
        # the single large reconstruction, some of its cycles
        {"name": "plan_2048", "kind": "plan", "width": 2048, "height": 2048, "cycles": 8, "hio": 20},
        # the largest image
        {"name": "plan_4096", "kind": "plan", "width": 4096, "height": 4096, "cycles": 4, "hio": 20},
        # a detector crop of arbitrary (prime and semiprime) sides
        {"name": "plan_1021x733", "kind": "plan", "width": 1021, "height": 733, "cycles": 8, "hio": 20},
        # known support, random initial phase, error tested after every iteration
        {"name": "hio_512x384", "kind": "hio", "width": 512, "height": 384, "iterations": 120},
        # a batch of uneven images with sides of the batch configuration
        {"name": "engine_uneven", "kind": "engine", "requests": 48, "sides": "config", "lo": 128, "hi": 512,
         "shape_seed": 2, "cycles": 20, "hio": 20},
        # requests as a service sees them: any side, small to large
        {"name": "engine_served", "kind": "engine", "requests": 24, "sides": "any", "lo": 64, "hi": 1024,
         "shape_seed": 4, "cycles": 10, "hio": 20},
    ]


def _log_side(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sides(rng):
    """Width and height of a reconstruction: a configured side, a round one or any other."""
    how = rng.random()
    if how < 0.35:
        return rng.choice((64, *CONFIG_SIDES, 768, 1024, 1536)), rng.choice((64, *CONFIG_SIDES, 768, 1024, 1536))
    if how < 0.65:
        return 20 * rng.randint(4, 64), 20 * rng.randint(4, 64)
    return _log_side(rng, 64, 1400), _log_side(rng, 64, 1400)


def _cycles(rng, width, height, hio, most):
    """Cycles that keep the whole call within `most` pixel iterations."""
    return max(1, min(rng.randint(8, 40), int(most / (width * height * hio))))


def draw(rng):
    kind = rng.choice(("fft", "blur", "forward", "dropin", "dropin", "plan", "plan", "hio", "engine", "engine"))
    case = {"kind": kind}
    if kind == "fft":
        case.update(width=_log_side(rng, 16, 2048), height=_log_side(rng, 16, 2048), sign=rng.choice((-1, 1)))
    elif kind == "blur":
        case.update(width=_log_side(rng, 64, 4096), height=_log_side(rng, 64, 4096),
                    sigma=round(rng.uniform(1.5, 6.0), 3))
    elif kind == "forward":
        case.update(width=_log_side(rng, 64, 2048), height=_log_side(rng, 64, 2048))
    elif kind in ("dropin", "plan"):
        w, h = _sides(rng)
        hio = rng.choice((10, 20, 20, 40))
        case.update(width=w, height=h, cycles=_cycles(rng, w, h, hio, 2.5e8), hio=hio)
    elif kind == "hio":
        w, h = _sides(rng)
        case.update(width=w, height=h, iterations=max(8, min(rng.randint(40, 400), int(2.5e8 / (w * h)))))
    else:
        any_side = rng.random() < 0.5
        case.update(requests=rng.randint(8, 32), sides="any" if any_side else "config", lo=64 if any_side else 128,
                    hi=rng.choice((512, 768, 1024)) if any_side else 512, shape_seed=rng.randint(0, 1 << 20),
                    cycles=rng.randint(4, 10), hio=rng.choice((10, 20)))
    return case


def _shapes(case):
    """Sizes of an engine case's requests: they belong to the case, not to the seed."""
    rng = random.Random(case["shape_seed"])
    if case["sides"] == "config":
        pick = lambda: rng.choice([s for s in CONFIG_SIDES if case["lo"] <= s <= case["hi"]])   # noqa: E731
    else:
        pick = lambda: _log_side(rng, case["lo"], case["hi"])   # noqa: E731
    return [(pick(), pick()) for _ in range(case["requests"])]


# ---- inputs -------------------------------------------------------------------
def _object(width, height, gen):
    """Gaussian blobs in a centred disk, as the benchmark recipes: float64 [H, W]."""
    n = max(8, min(400, width * height // 1000))
    u = lambda lo, hi: lo + (hi - lo) * torch.rand(n, 1, generator=gen, device=DEV, dtype=torch.float64)   # noqa: E731
    r, th = 0.15 * min(width, height) * u(0.0, 1.0).sqrt(), u(0.0, 2.0 * math.pi)
    s, a = u(1.5, 3.0), u(0.3, 1.0)
    x = torch.arange(width, device=DEV, dtype=torch.float64)[None, :] - (width / 2.0 + r * th.cos())
    y = torch.arange(height, device=DEV, dtype=torch.float64)[None, :] - (height / 2.0 + r * th.sin())
    cut = lambda d: torch.exp(-d * d / (2.0 * s * s)) * (d.abs() <= 5.0 * s)   # noqa: E731
    return (a * cut(y)).T @ cut(x)


def _modulus(width, height, gen, photons=1e8):
    """Square root of the blobs' diffraction intensity with photon noise: float32 [H, W]."""
    inten = torch.fft.fft2(_object(width, height, gen)).abs().square()
    scale = photons / inten.sum()
    return (torch.poisson(inten * scale, generator=gen) / scale).sqrt().float().contiguous()


def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _support(width, height):
    """uint8 [H, W], 1 outside a centred disk that holds the object."""
    x = torch.arange(width, device=DEV, dtype=torch.float64)[None, :] - width / 2.0
    y = torch.arange(height, device=DEV, dtype=torch.float64)[:, None] - height / 2.0
    r = 0.15 * min(width, height) + 12.0
    return ((x * x + y * y) > r * r).to(torch.uint8).contiguous()


def _params(case):
    # every cycle runs: the error target is the smallest positive float
    return imr.Params(n_cycles=case["cycles"], target_error=imr.FLT_MIN, n_hio_cycles=case["hio"])


def prepare(case, seed):
    kind, gen = case["kind"], _generator(seed)
    st = dict(case)
    if kind == "engine":
        st["moduli"] = [_modulus(w, h, gen).cpu().numpy() for w, h in _shapes(case)]
        st["params"] = _params(case)
        st["engine"] = imr.Engine()
        return st
    w, h = case["width"], case["height"]
    if kind == "fft":
        st["field"] = torch.randn(h, w, 2, generator=gen, device=DEV).view(torch.complex64).reshape(h, w).contiguous()
        st["work"] = torch.empty_like(st["field"])
    elif kind == "blur":
        st["image"] = _object(w, h, gen).float().contiguous() + 0.01 * torch.rand(h, w, generator=gen, device=DEV)
        st["work"], st["tmp"] = torch.empty_like(st["image"]), torch.empty_like(st["image"])
    elif kind == "forward":
        st["object"] = _object(w, h, gen).float().cpu().numpy()
    elif kind == "dropin":
        st["modulus"] = _modulus(w, h, gen).cpu().numpy()
        st["io"] = np.empty_like(st["modulus"])
    elif kind == "plan":
        st["modulus"] = _modulus(w, h, gen, 1e9)
        st["out"] = torch.empty_like(st["modulus"])
        st["plan"] = imr.Plan(w, h, _params(case))
    else:   # hio
        st["modulus"] = _modulus(w, h, gen)
        st["mask"] = _support(w, h)
        st["out"] = torch.empty_like(st["modulus"])
        st["plan"] = imr.HioPlan(w, h, case["iterations"])
    return st


def run(st):
    kind = st["kind"]
    if kind == "fft":
        st["work"].copy_(st["field"])   # the transform is in place and unnormalised
        imr.fft2d(st["work"], st["width"], st["height"], st["sign"])
        return st["work"]
    if kind == "blur":
        st["work"].copy_(st["image"])
        imr.gaussian_blur(st["work"], st["tmp"], st["width"], st["height"], st["sigma"])
        return st["work"]
    if kind == "forward":
        return imr.diffraction_intensity(st["object"])
    if kind == "dropin":
        np.copyto(st["io"], st["modulus"])   # the call works in place
        rc = imr.cuda_shrink_wrap(st["io"], st["width"], st["height"], n_cycles=st["cycles"],
                                  target_error=imr.FLT_MIN, n_hio_cycles=st["hio"])
        if rc != 0:
            raise imr.ImrError(rc, "cuda_shrink_wrap")
        return st["io"]
    if kind == "plan":
        st["plan"].execute(st["modulus"], st["out"])
        return st["out"]
    if kind == "hio":
        st["plan"].execute(st["modulus"], st["mask"], st["out"])
        return st["out"]
    for tag, m in enumerate(st["moduli"]):
        st["engine"].submit(m, st["params"], tag=tag)
    st["engine"].run()
    done = sorted(st["engine"].poll(), key=lambda r: r["tag"])
    return {"images": [r["out"] for r in done], "cycles": np.array([r["cycles_done"] for r in done]),
            "status": np.array([r["status"] for r in done])}


# ---- what a pass cannot do without ----------------------------------------------
def _iteration_flops(n):
    """One HIO iteration: a 2D transform and its inverse (5 n log2 n each), update and projection."""
    return 10.0 * n * math.log2(n) + 20.0 * n


def work(case):
    kind = case["kind"]
    if kind == "engine":
        px = [w * h for w, h in _shapes(case)]
        return {"bytes": 8.0 * sum(px), "flops": case["cycles"] * case["hio"] * sum(_iteration_flops(n) for n in px)}
    n = float(case["width"] * case["height"])
    if kind == "fft":
        return {"bytes": 16.0 * n, "flops": 5.0 * n * math.log2(n)}
    if kind == "blur":
        taps = 2 * math.ceil(2.884402748387961466 * case["sigma"] - 0.5) + 1
        return {"bytes": 8.0 * n, "flops": 4.0 * taps * n}
    if kind == "forward":
        return {"bytes": 8.0 * n, "flops": 5.0 * n * math.log2(n)}
    if kind == "hio":
        return {"bytes": 9.0 * n, "flops": case["iterations"] * _iteration_flops(n)}
    return {"bytes": 8.0 * n, "flops": case["cycles"] * case["hio"] * _iteration_flops(n)}


# ---- the same in 64 bits ----------------------------------------------------------
def exact(case, seed):
    kind, gen = case["kind"], _generator(seed)
    if kind == "fft":
        z = prepare(case, seed)["field"].to(torch.complex128)
        return torch.fft.fft2(z) if case["sign"] < 0 else torch.fft.ifft2(z) * z.numel()
    if kind == "forward":
        return torch.fft.fft2(_object(case["width"], case["height"], gen).float().double()).abs().cpu().numpy()
    if kind == "blur":
        half = math.ceil(2.884402748387961466 * case["sigma"] - 0.5)
        i = torch.arange(-half, half + 1, device=DEV, dtype=torch.float64)
        k = torch.exp(-i * i / (2.0 * case["sigma"] ** 2))
        k /= k.sum()
        a = prepare(case, seed)["image"].double()
        for axis in (1, 0):   # rows, then columns, the border value repeated
            n = a.shape[axis]
            at = torch.arange(n, device=DEV)
            a = sum(k[j] * a.index_select(axis, (at + j - half).clamp(0, n - 1)) for j in range(2 * half + 1))
        return a
    return None   # reconstructions: see the top of the file
