"""Timed workloads of the renderer through its Python binding.

Each case is one thing a program using grrt_b200 does: a frame of a thin-disk
or volumetric scene in one of the precision forms, a sweep of many cameras in
one launch, or the learned surrogate's inference and training. Sizes and scenes
are those of the library's own benchmark scenes (``config_params``,
``sweep_cameras``) and tests, with a few odd ones.

A case is a dict of plain values; ``prepare`` makes the context, batch or
network a program would keep between frames (the seed moves the observer, the
spin and the disk's noise or the network's weights and inputs), ``run`` renders
or evaluates once.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

import grrt_b200 as g

# network of the surrogate: 4 -> 256 x 4 -> 16 (9 outputs used)
_HIDDEN, _IN, _OUT, _USED = 256, 4, 16, 9


def listed() -> list:
    return [
        # A preview while a scene is set up: the reference call into host memory, latency alone counts.
        dict(name="preview", kind="thin", width=64, height=48, spp=1, form="fp64", metric="kerr", spin=0.998,
             incl=80.0, stars=True, host=True, tonemap=False),
        # The reference program's ordinary picture: Schwarzschild, black sky, default (FP64) form, host buffer.
        dict(name="schwarzschild_256", kind="thin", width=256, height=256, spp=1, form="fp64",
             metric="schwarzschild", spin=0.0, incl=80.0, stars=False, host=True, tonemap=False),
        # The benchmark frame in the reference's own arithmetic.
        dict(name="kerr_1024_4spp_fp64", kind="thin", width=1024, height=1024, spp=4, form="fp64", metric="kerr",
             spin=0.998, incl=80.0, stars=True, host=False, tonemap=False),
        # The benchmark frame in the mixed form.
        dict(name="kerr_1024_4spp_mixed", kind="thin", width=1024, height=1024, spp=4, form="mixed", metric="kerr",
             spin=0.998, incl=80.0, stars=True, host=False, tonemap=False),
        # One frame of an animation at an odd size, mixed form, into pageable host memory.
        dict(name="kerr_1279x719_mixed_host", kind="thin", width=1279, height=719, spp=1, form="mixed",
             metric="kerr", spin=0.9, incl=60.0, stars=True, host=True, tonemap=False),
        # A large picture on a black sky, tone-mapped on the device.
        dict(name="kerr_2048_black_tonemap", kind="thin", width=2048, height=2048, spp=1, form="mixed",
             metric="kerr", spin=0.998, incl=80.0, stars=False, host=False, tonemap=True),
        # The parameter sweep: 4 spins x 16 inclinations in one launch.
        dict(name="sweep_64x256", kind="batch", cameras=64, width=256, height=256, form="mixed"),
        # The benchmark's spectral cube: volumetric disk, 32 bins.
        dict(name="spectral_512_32bins", kind="spectral", width=512, height=512, spp=1, bins=32, form="fp64",
             spin=0.9, incl=80.0, host=False),
        # A small spectral cube at an odd size into host memory, mixed form.
        dict(name="spectral_101x75_16bins", kind="spectral", width=101, height=75, spp=1, bins=16, form="mixed",
             spin=0.9, incl=70.0, host=True),
        # The volumetric disk as a picture, mixed form.
        dict(name="volume_rgb_512", kind="volume", width=512, height=512, spp=1, form="mixed", spin=0.9,
             incl=80.0, stars=False, host=False),
        # Network inference over one large frame's worth of samples (not a whole number of tiles).
        dict(name="network_1m", kind="network", rows=1048576 + 77),
        # A stretch of surrogate training at the benchmark's batch size.
        dict(name="training_16384", kind="training", batch=16384, steps=24),
    ]


def _log_int(rng: random.Random, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_size(rng: random.Random, lo: int, hi: int, rays: int, spp: int) -> tuple:
    w = _log_int(rng, lo, hi)
    h = max(lo * 3 // 4, int(w * rng.choice([1.0, 0.75, 0.5625, rng.uniform(0.5, 1.0)])))
    while w * h * spp > rays:
        w, h = int(w * 0.9), int(h * 0.9)
    return w, h


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["thin"] * 6 + ["batch"] + ["spectral"] * 2 + ["volume"] + ["network", "training"])
    form = rng.choice(["fp64", "mixed"])
    if kind == "thin":
        spp = rng.choice([1, 1, 4, 9])
        w, h = _draw_size(rng, 64, 2048, 1 << 22, spp)
        metric = rng.choice(["kerr", "kerr", "kerr", "schwarzschild"])
        host = rng.random() < 0.5
        return dict(kind=kind, width=w, height=h, spp=spp, form=form, metric=metric,
                    spin=0.0 if metric == "schwarzschild" else rng.choice([0.5, 0.9, 0.998, rng.uniform(0.2, 0.99)]),
                    incl=rng.uniform(10.0, 88.0), stars=rng.random() < 0.6, host=host,
                    tonemap=not host and rng.random() < 0.3)
    if kind == "batch":
        return dict(kind=kind, cameras=rng.choice([4, 8, 12, 16, 32, 64]), width=_log_int(rng, 48, 256),
                    height=_log_int(rng, 48, 256), form=form)
    if kind == "spectral":
        spp = rng.choice([1, 1, 1, 4])
        w, h = _draw_size(rng, 48, 512, 1 << 18, spp)
        return dict(kind=kind, width=w, height=h, spp=spp, bins=rng.choice([3, 8, 16, 17, 24, 32]), form=form,
                    spin=rng.uniform(0.3, 0.95), incl=rng.uniform(30.0, 85.0), host=rng.random() < 0.5)
    if kind == "volume":
        spp = rng.choice([1, 1, 4])
        w, h = _draw_size(rng, 48, 512, 1 << 18, spp)
        return dict(kind=kind, width=w, height=h, spp=spp, form=form, spin=rng.uniform(0.3, 0.95),
                    incl=rng.uniform(30.0, 85.0), stars=rng.random() < 0.4, host=rng.random() < 0.5)
    if kind == "network":
        return dict(kind=kind, rows=_log_int(rng, 100, 1 << 20))
    return dict(kind=kind, batch=128 * _log_int(rng, 8, 128), steps=rng.choice([8, 16, 24]))


def _scene(case: dict, seed: int) -> dict:
    """Scene parameters of a rendering case; the seed moves the observer, the spin and the disk's noise."""
    r = random.Random(seed)
    incl = case["incl"] + r.uniform(-1.5, 1.5)
    common = dict(width=case["width"], height=case["height"], spp=case["spp"], observer_theta=math.radians(incl),
                  observer_phi=r.uniform(0.0, 2.0 * math.pi))
    if case["kind"] == "thin":
        v = g.config_params(1 if case["metric"] == "schwarzschild" else 2, **common)
        if case["metric"] == "kerr":
            v.update(spin=case["spin"] * (1.0 - 0.004 * r.random()))
        v.update(background_type=g.BG_STARS if case["stars"] else g.BG_BLACK)
    else:
        v = g.config_params(3, **common)
        v.update(spin=case["spin"] * (1.0 - 0.004 * r.random()), disk_seed=r.randrange(1, 10000))
        if case.get("stars"):
            v.update(background_type=g.BG_STARS)
    return v


def _form(case: dict) -> int:
    return g.FORM_MIXED if case["form"] == "mixed" else g.FORM_FP64


def _network_params(seed: int) -> np.ndarray:
    """Flat parameters W1, b1, ..., W5, b5 (row-major): uniform with variance 1/fan_in, unused output rows 0."""
    r = np.random.RandomState(seed % (1 << 32))
    parts = []
    for rows, cols, used in [(_HIDDEN, _IN, _HIDDEN)] + [(_HIDDEN, _HIDDEN, _HIDDEN)] * 3 + [(_OUT, _HIDDEN, _USED)]:
        w = r.uniform(-1.0, 1.0, (rows, cols)) * math.sqrt(3.0 / cols)
        w[used:] = 0.0
        b = r.uniform(-0.05, 0.05, rows)
        b[used:] = 0.0
        parts += [w.reshape(-1), b]
    return np.concatenate(parts).astype(np.float32)


def _network_inputs(case: dict, seed: int) -> torch.Tensor:
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return torch.rand((case["rows"], _IN), generator=gen, device="cuda", dtype=torch.float32) * 2.0 - 1.0


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    if kind in ("thin", "volume", "spectral"):
        freqs = g.log_bins(n=case["bins"]) if kind == "spectral" else None
        ctx = g.Renderer(_scene(case, seed), freqs=freqs)
        ctx.set_precision(_form(case))
        state = dict(case=case, ctx=ctx)
        if not case["host"]:
            shape = (case["height"], case["width"], case["bins"] if kind == "spectral" else 4)
            state["out"] = torch.empty(shape, device="cuda",
                                       dtype=torch.float64 if kind == "spectral" else torch.float32)
        return state
    if kind == "batch":
        r = random.Random(seed)
        n = case["cameras"]
        spins = (0.0, 0.5, 0.9, 0.998)
        cams = g.sweep_cameras(width=case["width"], height=case["height"], spins=spins, n_incl=n // len(spins),
                               incl_lo_deg=5.0 + r.uniform(0.0, 3.0), incl_hi_deg=88.0 + r.uniform(0.0, 2.0)) \
            if n // len(spins) > 1 else \
            g.sweep_cameras(width=case["width"], height=case["height"], spins=spins, n_incl=2,
                            incl_lo_deg=60.0 + r.uniform(0.0, 3.0), incl_hi_deg=80.0)[::2]
        b = g.Batch(cams)
        b.set_precision(_form(case))
        out = torch.empty((len(cams), case["height"], case["width"], 4), device="cuda", dtype=torch.float32)
        return dict(case=case, batch=b, out=out)
    if kind == "network":
        net = g.Surrogate(0)
        net.set_params(_network_params(seed))
        x = _network_inputs(case, seed)
        out = torch.empty((case["rows"], _OUT), device="cuda", dtype=torch.float32)
        return dict(case=case, net=net, x=x, out=out)
    net = g.Surrogate(0)
    r = random.Random(seed)
    cams = [g.config_params(2, observer_theta=math.radians(incl + r.uniform(-3.0, 3.0)), spin=spin)
            for spin, incl in ((0.5, 40.0), (0.998, 80.0))]
    net.generate(cams, 128)
    return dict(case=case, net=net, params=_network_params(seed))


def run(state: dict):
    case = state["case"]
    kind = case["kind"]
    if kind == "thin" or kind == "volume":
        if case["host"]:
            return state["ctx"].render()
        stream = torch.cuda.current_stream()
        state["ctx"].render_device(state["out"], stream=stream)
        if case.get("tonemap"):
            g.tonemap_device(state["out"], case["width"], case["height"], stream=stream.cuda_stream)
        return state["out"]
    if kind == "spectral":
        if case["host"]:
            return state["ctx"].render_spectral()
        state["ctx"].render_spectral_device(state["out"], case["width"], case["height"],
                                            stream=torch.cuda.current_stream())
        return state["out"]
    if kind == "batch":
        state["batch"].render_device(state["out"], stream=torch.cuda.current_stream())
        return state["out"]
    if kind == "network":
        state["net"].forward(state["x"], state["out"], case["rows"])
        return state["out"]
    # a stretch of training from given weights: the updated weights and the loss of each step
    state["net"].set_params(state["params"])
    loss = state["net"].train(case["steps"], case["batch"], 1e-3)
    return {"params": state["net"].params(), "loss": loss}


def work(case: dict) -> dict:
    """Bytes and operations a pass cannot do without.

    Rays: the reference's operations, 1500 per Dormand-Prince attempt; attempts per ray are averages of the scenes
    (120 on a thin disk, of which the mixed form has to do about a fifth in FP64 and the rest as FP32 attempts of a
    third the count). Frames are written once; scene tables are small.
    """
    kind = case["kind"]
    weights = _IN * _HIDDEN + 3 * _HIDDEN * _HIDDEN + _HIDDEN * _OUT
    if kind == "network":
        return {"bytes": 4.0 * case["rows"] * (_IN + _OUT) + 4.0 * weights, "flops": 2.0 * weights * case["rows"]}
    if kind == "training":
        rows = case["batch"] * case["steps"]
        return {"bytes": 4.0 * rows * (_IN + 10) + case["steps"] * 4.0 * weights * 6, "flops": 6.0 * weights * rows}
    pixels = case["width"] * case["height"] * case.get("cameras", 1)
    rays = pixels * case.get("spp", 1)
    attempts = 120.0 if case["form"] == "fp64" else 60.0
    flops = rays * attempts * 1500.0
    if kind == "spectral":
        return {"bytes": 8.0 * pixels * case["bins"], "flops": flops}
    return {"bytes": 16.0 * pixels, "flops": flops}


def exact(case: dict, seed: int):
    """The network's outputs in 64 bits. Frames have no such value: the method's own adaptive steps and table lookups
    define the picture, and tracing it in plain 64-bit array code takes minutes; training likewise rounds by design."""
    if case["kind"] != "network":
        return None
    p = torch.from_numpy(_network_params(seed)).to(device="cuda", dtype=torch.float64)
    layers, at = [], 0
    for rows, cols in [(_HIDDEN, _IN)] + [(_HIDDEN, _HIDDEN)] * 3 + [(_OUT, _HIDDEN)]:
        w = p[at:at + rows * cols].view(rows, cols)
        at += rows * cols
        layers.append((w, p[at:at + rows]))
        at += rows
    x = _network_inputs(case, seed)
    outs = []
    for part in x.split(1 << 17):
        h = part.double()
        for k, (w, b) in enumerate(layers):
            h = h @ w.T + b
            if k < len(layers) - 1:
                h = h * torch.sigmoid(h)
        outs.append(h)
    return torch.cat(outs)
