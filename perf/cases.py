"""The workloads this framework is timed on, through its public entry points.

``listed()`` gives the named cases, ``draw(rng)`` one more of the same ranges,
``prepare(case, seed)`` the state a program holds before its call,
``run(state)`` one pass (a frame, a batch of substeps, a gradient),
``work(case)`` the bytes and operations that pass cannot do without, and
``exact(case, seed)`` its outputs in 64-bit arithmetic, independent of the
package.

A module or batch keeps its field between passes, as a running simulation
does: a pass continues from where the last one stopped, and the first one
starts from the uploaded field.
"""
from __future__ import annotations

import math

import numpy as np
import torch
import torch.utils.checkpoint

import life_simulation_b200 as lb
from life_simulation_b200.adjoint import rollout

M32 = 0xFFFFFFFF

# Ring kernels of the multi-kernel form: the peaks, centres, widths and weights
# of the repository's three-kernel workload, and a fourth for the largest count
# that a scene may give.
RINGS = [
    {"mu": 0.156, "sigma": 0.0118, "weight": 0.5, "betas": [1.0]},
    {"mu": 0.193, "sigma": 0.049, "weight": 0.3, "betas": [0.5, 1.0]},
    {"mu": 0.342, "sigma": 0.0891, "weight": 0.2, "betas": [1.0, 0.667, 0.333]},
    {"mu": 0.25, "sigma": 0.035, "weight": 0.4, "betas": [1.0, 0.6]},
]
# The gradient form's two kernels.
GRAD_RINGS = [
    {"mu": 0.15, "sigma": 0.03, "weight": 0.5, "betas": [1.0]},
    {"mu": 0.25, "sigma": 0.05, "weight": 0.5, "betas": [0.5, 1.0]},
]
BATCH_SIZES = [(128, 128), (256, 256), (384, 216), (512, 512)]
# Sizes the gradient form takes (it has transforms for these lengths).
GRAD_WIDTHS = [128, 256, 384, 512, 1024]
GRAD_HEIGHTS = [64, 128, 216, 256, 512]


def _module(name, conv, w, h, radius, kernels=1, substeps=1, mode=1, core="exp", inject=0.0, noise=0.0, jitter=0.0,
            render=False, precision="fp32"):
    return {"name": name, "kind": "module", "conv": conv, "w": w, "h": h, "radius": radius, "kernels": kernels,
            "substeps": substeps, "mode": mode, "core": core, "inject": inject, "noise": noise, "jitter": jitter,
            "render": render, "precision": precision}


def listed():
    return [
        # One frame of the small single-kernel world (256 x 256, R = 13, exponential core): the smallest call,
        # where the launch and its latency are what a caller waits for.
        _module("direct_256_r13", "direct", 256, 256, 13, mode=0),
        # The default scene of the direct path: a full-HD field with R = 13 and the blob injection that the
        # reference's basic preset has on.
        _module("direct_1080p_r13_inject", "direct", 1920, 1080, 13, core="gaussShell", inject=0.22),
        # The largest radius of the direct path, at the size the reference publishes a time for.
        _module("direct_720p_r32", "direct", 1280, 720, 32, core="gaussShell"),
        # A window-sized field of odd width and height, two substeps a frame, with every option of a live set on:
        # noise, mu jitter and injection.
        _module("direct_1001x703_r9_live", "direct", 1001, 703, 9, substeps=2, inject=0.2, noise=0.05, jitter=0.2,
                core="gaussShell"),
        # The multi-kernel spectral path at the size of the reference's multi-kernel preset, one frame at a time.
        _module("fft_1024x512_k3", "fft", 1024, 512, 24, kernels=3, inject=0.2),
        # The headline size: full HD, three kernels, four substeps a frame.
        _module("fft_1080p_k3_x4", "fft", 1920, 1080, 24, kernels=3, substeps=4),
        # A 720p frame with its colour layer, as a program that shows the field calls it: one substep and the texels.
        _module("fft_720p_k3_render", "fft", 1280, 720, 24, kernels=3, render=True),
        # A field fitted to a window: sizes whose factors are 2, 3 and 5 but that are no video format, two kernels.
        _module("fft_810x486_k2_live", "fft", 810, 486, 18, kernels=2, substeps=2, noise=0.05, inject=0.2),
        # The largest field in use, three kernels of the largest radius, in full FP32.
        _module("fft_4096_k3_r32", "fft", 4096, 4096, 32, kernels=3, mode=0),
        # The opt-in split-precision form of the column stages, on a tall strip.
        _module("fft_fp16x3_1024x4096_k3", "fft", 1024, 4096, 32, kernels=3, precision="fp16x3", mode=0),
        # A parameter sweep: worlds of the sweep's four sizes, a radius, mu, sigma and dt each, 60 substeps between
        # two looks at the fields. Growth mode 1 and wide bells: worlds whose fields stay comparable over that many
        # steps, where narrow ones double a rounding every few.
        {"name": "sweep_48_worlds_x60", "kind": "batch", "worlds": 48, "steps": 60},
        # Gradient search over initial fields and parameters: a rollout and its backward pass.
        {"name": "grad_8x512_t16", "kind": "grad", "w": 512, "h": 512, "batch": 8, "radius": 16, "steps": 16,
         "every": 8, "mode": 1},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _smooth(rng, lo, hi, even):
    """A length with factors 2, 3 and 5 only, spread over the logarithm of lo..hi."""
    sizes = []
    a = 1
    while a <= hi:
        b = a
        while b <= hi:
            c = b
            while c <= hi:
                if c >= lo and not (even and c % 2):
                    sizes.append(c)
                c *= 5
            b *= 3
        a *= 2
    target = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(sorted(sizes), key=lambda s: abs(math.log(s / target)))


def draw(rng):
    kind = rng.choice(["direct", "direct", "directMulti", "fft", "fft", "fft", "fftTall", "batch", "grad"])
    if kind in ("direct", "directMulti"):
        kernels = 1 if kind == "direct" else rng.randint(2, 3)
        w, h = _log_uniform(rng, 64, 1920 if kernels == 1 else 960), _log_uniform(rng, 64, 1080 if kernels == 1 else 540)
        live = rng.random() < 0.5
        c = _module("", kind, w, h, rng.randint(3, 32), kernels=kernels, substeps=rng.randint(1, 3), mode=rng.randint(0, 1),
                    core=rng.choice(["exp", "gaussShell"]) if kernels == 1 else "exp",
                    inject=0.2 if live else 0.0, noise=rng.choice([0.0, 0.05]), jitter=0.2 if live and rng.random() < 0.5 else 0.0)
    elif kind == "fft":
        w, h = _smooth(rng, 96, 2560, True), _smooth(rng, 72, 2048, False)
        c = _module("", "fft", w, h, rng.randint(6, 32), kernels=rng.randint(1, 4), substeps=rng.randint(1, 3),
                    mode=rng.randint(0, 1), inject=rng.choice([0.0, 0.2]), render=rng.random() < 0.3)
    elif kind == "fftTall":
        c = _module("", "fft", rng.choice([512, 1024, 2048]), 4096, rng.randint(12, 32), kernels=rng.randint(1, 3),
                    mode=rng.randint(0, 1), precision=rng.choice(["fp16x3", "bf16x3"]))
    elif kind == "batch":
        c = {"name": "", "kind": "batch", "worlds": rng.randint(4, 60), "steps": rng.randint(8, 60)}
    else:
        every = rng.choice([2, 4, 8])
        c = {"name": "", "kind": "grad", "w": rng.choice(GRAD_WIDTHS), "h": rng.choice(GRAD_HEIGHTS),
             "batch": rng.randint(1, 8), "radius": rng.randint(6, 24), "steps": every * rng.randint(1, 2), "every": every,
             "mode": rng.randint(0, 1)}
    del c["name"]
    return c


# ------------------------------------------------------------------ inputs


def _patches(w, h, seed):
    """A field of uniform [0, 1) values in patches on a torus, zeros between them (H x W, float32)."""
    rng = np.random.default_rng(seed)
    a = np.zeros((h, w), np.float32)
    side = max(8, min(w, h) // 6)
    for _ in range(20):
        y0, x0 = int(rng.integers(0, h)), int(rng.integers(0, w))
        ys, xs = (y0 + np.arange(side)) % h, (x0 + np.arange(side)) % w
        a[np.ix_(ys, xs)] = rng.random((side, side), np.float32)
    return a


def _params(c):
    p = {"convMode": c["conv"], "fftAnySize": True, "simWidth": c["w"], "simHeight": c["h"], "radius": c["radius"],
         "kernelCore": c["core"], "growthMode": c["mode"], "growthMu": 0.15, "growthSigma": 0.03, "dt": 0.1,
         "noiseAmount": c["noise"], "muJitter": c["jitter"], "injectAmount": c["inject"], "injectCount": 4}
    if c["conv"] != "direct":
        p["kernels"] = [dict(k, radiusScale=1.0) for k in RINGS[:c["kernels"]]]
    if c["precision"] != "fp32":
        p["fftPrecision"] = c["precision"]
    return p


def _batch_worlds(c, seed):
    rng = np.random.default_rng(seed)
    out = []
    for i in range(c["worlds"]):
        w, h = BATCH_SIZES[i % len(BATCH_SIZES)]
        out.append({"width": w, "height": h, "radius": int(rng.integers(8, 33)), "mu": float(rng.uniform(0.10, 0.35)),
                    "sigma": float(rng.uniform(0.04, 0.08)), "dt": float(rng.uniform(0.05, 0.2)),
                    "growth_mode": 1, "seed": 3 + i})
    return out


def _world_field(w, seed):
    rng = np.random.default_rng([seed, w["seed"]])
    a = np.zeros((w["height"], w["width"]), np.float32)
    side = min(w["width"], w["height"]) // 2
    y0, x0 = (w["height"] - side) // 2, (w["width"] - side) // 2
    a[y0:y0 + side, x0:x0 + side] = rng.random((side, side), np.float32)
    return a


def _grad_inputs(c, seed):
    rng = np.random.default_rng(seed)
    shape = (c["batch"], c["h"], c["w"])
    return rng.random(shape, np.float32), rng.random(shape, np.float32)


def _grad_params():
    """mu, sigma, weight (K), betas (K x 8) and dt as float32 CPU tensors."""
    k = GRAD_RINGS
    betas = torch.zeros(len(k), 8)
    for i, r in enumerate(k):
        betas[i, :len(r["betas"])] = torch.tensor(r["betas"])
    return (torch.tensor([r["mu"] for r in k]), torch.tensor([r["sigma"] for r in k]),
            torch.tensor([r["weight"] for r in k]), betas, torch.tensor(0.1))


class _View:
    """One of a module's device buffers as torch sees it (H x W float32). It
    holds the module, whose end frees the buffer, for as long as the tensor lives."""

    def __init__(self, module, ptr, w, h):
        self.module = module
        self.__cuda_array_interface__ = {"shape": (h, w), "typestr": "<f4", "data": (ptr, False), "version": 2}


def prepare(case, seed):
    c = case
    if c["kind"] == "module":
        m = lb.LeniaModule(_params(c), c["w"], c["h"])
        if m.warning:
            raise RuntimeError(m.warning)
        m.reset(seed & M32)
        m.upload(_patches(c["w"], c["h"], seed))
        s = {"case": c, "module": m, "frame": 0, "views": {}, "rgba": None}
        if c["render"]:
            s["rgba"] = torch.empty((c["h"], c["w"], 4), dtype=torch.float16, device="cuda")
        return s
    if c["kind"] == "batch":
        worlds = _batch_worlds(c, seed)
        b = lb.LeniaBatch([lb.make_world(**w) for w in worlds])
        for i, w in enumerate(worlds):
            b.upload(i, _world_field(w, seed))
        return {"case": c, "batch": b}
    a0, target = _grad_inputs(c, seed)
    eng = lb.LeniaAdjoint(c["w"], c["h"], c["batch"], GRAD_RINGS, c["radius"], c["steps"], checkpoint_every=c["every"],
                          dt=0.1, growth_mode=c["mode"])
    params = [p.requires_grad_(True) for p in _grad_params()]
    return {"case": c, "engine": eng, "a0": torch.from_numpy(a0).cuda().requires_grad_(True),
            "target": torch.from_numpy(target).cuda(), "params": params}


def run(state):
    c = state["case"]
    if c["kind"] == "module":
        m, frame = state["module"], state["frame"]
        state["frame"] = frame + 1
        if c["render"]:
            fp = m.frame_params(frame)
            m.step_render(fp, c["substeps"], state["rgba"].data_ptr(), c["w"], c["h"])
        else:
            m.encode(frame, c["substeps"])
        ptr = m.field_device_ptr()  # one of the module's two buffers
        view = state["views"].get(ptr)
        if view is None:
            view = state["views"][ptr] = torch.as_tensor(_View(m, ptr, c["w"], c["h"]), device="cuda")
        return {"field": view, "rgba": state["rgba"]} if c["render"] else view
    if c["kind"] == "batch":
        b = state["batch"]
        b.step(c["steps"])
        return [b.field(i) for i in range(c["worlds"])]
    out = rollout(state["engine"], state["a0"], *state["params"])
    grad = (out.detach() - state["target"]) * (2.0 / out.numel())  # of the mean squared error
    grads = torch.autograd.grad(out, [state["a0"], *state["params"]], grad)
    return {"fields": out.detach(), "a0": grads[0], "mu": grads[1], "sigma": grads[2], "weight": grads[3],
            "betas": grads[4], "dt": grads[5]}


# -------------------------------------------------------------------- work


def _step_work(npx, kernels):
    """One spectral substep: the field in and out, and the real transforms, products and growth of `kernels` kernels."""
    return 8.0 * npx, npx * ((1 + kernels) * 2.5 * math.log2(npx) + kernels * 10.0)


def work(case):
    c = case
    if c["kind"] == "module":
        npx = c["w"] * c["h"]
        if c["conv"] == "fft":
            b, f = _step_work(npx, c["kernels"])
        else:
            taps = sum(int(np.count_nonzero(_direct_lut(c["radius"], c["core"]))) for _ in range(c["kernels"]))
            b, f = 8.0 * npx, npx * (2.0 * taps + 10.0 * c["kernels"])
        return {"bytes": b * c["substeps"] + (8.0 * npx if c["render"] else 0.0), "flops": f * c["substeps"]}
    if c["kind"] == "batch":
        sizes = [BATCH_SIZES[i % len(BATCH_SIZES)] for i in range(c["worlds"])]
        per = [_step_work(w * h, 1) for w, h in sizes]
        return {"bytes": c["steps"] * sum(p[0] for p in per) + sum(4.0 * w * h for w, h in sizes),
                "flops": c["steps"] * sum(p[1] for p in per)}
    npx = c["w"] * c["h"] * c["batch"]
    b, f = _step_work(c["w"] * c["h"], len(GRAD_RINGS))
    # Forward: field in and out a step. Backward: that field and the gradient in, the gradient out; K transforms to
    # the frequencies, one back, and the field's own for the ring gradients.
    return {"bytes": c["steps"] * c["batch"] * (b + 12.0 * npx / c["batch"]),
            "flops": c["steps"] * c["batch"] * (2.0 * f + npx / c["batch"] * 2.5 * math.log2(npx / c["batch"]))}


# ------------------------------------------------------------------- exact


def _f32(x):
    return float(np.float32(x))


def _pcg(v):
    """PCG output hash of 32-bit values held in int64 (numpy array, torch tensor or int)."""
    state = (v * 747796405 + 2891336453) & M32
    word = (((state >> ((state >> 28) + 4)) ^ state) * 277803737) & M32
    return ((word >> 22) ^ word) & M32


def _rand01(px, py, tag, seed):
    return (_pcg(px ^ _pcg(py ^ _pcg(tag ^ seed))) >> 8) / 16777216.0


def _exp_core(r):
    inside = (r > 0) & (r < 1)
    q = np.where(inside, r, 0.5)
    return np.where(inside, np.exp(4.0 - 1.0 / (q * (1.0 - q))), 0.0)


def _direct_lut(radius, core):
    d = np.arange(-radius, radius + 1, dtype=np.float64)
    r = np.sqrt(d[:, None] ** 2 + d[None, :] ** 2) / max(radius, 1)
    if core == "exp":
        return _exp_core(r)
    shell = np.exp(-0.5 * ((r - 0.5) / _f32(0.15)) ** 2)
    return np.where((r > 0) & (r <= 1), shell, 0.0)


def _ring_image(w, h, radius, betas, core):
    dy, dx = np.arange(h), np.arange(w)
    dy = np.where(dy > h // 2, dy - h, dy).astype(np.float64)
    dx = np.where(dx > w // 2, dx - w, dx).astype(np.float64)
    r = np.sqrt(dx[None, :] ** 2 + dy[:, None] ** 2)
    inside = (r > 0) & (r <= radius)
    u = r / radius * len(betas)
    i = np.minimum(np.floor(u), len(betas) - 1).astype(np.int64)
    b = np.array([_f32(x) for x in betas])[i]
    val = _exp_core(u - i) if core == "exp" else np.exp(-0.5 * ((u - i - 0.5) / (_f32(0.15) * len(betas))) ** 2)
    return np.where(inside, b * val, 0.0)


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to("cuda" if torch.cuda.is_available() else "cpu")


def _spectrum(img):
    return torch.fft.rfft2(_dev(img / img.sum()))


def _lut_on_torus(lut, w, h):
    r = lut.shape[0] // 2
    d = np.arange(-r, r + 1)
    img = np.zeros((h, w))
    np.add.at(img, ((d % h)[:, None], (d % w)[None, :]), lut)
    return img


def _growth(a, spectra, mu, sigma, weight, mode, dt, shift=0.0):
    fa = torch.fft.rfft2(a)
    total = torch.zeros_like(a)
    for k, s in enumerate(spectra):
        u = torch.fft.irfft2(fa * s, s=a.shape[-2:])
        bell = torch.exp(-0.5 * ((u - (mu[k] + shift)) / sigma[k]) ** 2)
        total = total + weight[k] * (bell if mode == 1 else 2.0 * bell - 1.0)
    return a + dt * (total / sum(weight) - a) if mode == 1 else a + dt * total


def _exact_module(c, seed):
    w, h = c["w"], c["h"]
    a = _dev(_patches(w, h, seed).astype(np.float64))
    if c["conv"] == "direct":
        spectra = [_spectrum(_lut_on_torus(_direct_lut(c["radius"], c["core"]), w, h))]
        mu, sigma, weight = [_f32(0.15)], [_f32(0.03)], [1.0]
    else:
        rings = RINGS[:c["kernels"]]
        spectra = [_spectrum(_ring_image(w, h, float(c["radius"]), k["betas"], c["core"])) for k in rings]
        mu, sigma = [_f32(k["mu"]) for k in rings], [_f32(k["sigma"]) for k in rings]
        weight = [_f32(k["weight"]) for k in rings]
    gx = torch.arange(w, device=a.device)[None, :].expand(h, w)
    gy = torch.arange(h, device=a.device)[:, None].expand(h, w)
    base = _pcg((seed & M32) ^ _pcg(0x4C454E31))
    for i in range(c["substeps"]):
        step_seed = _pcg(base ^ i)
        shift = 0.0
        if c["jitter"] > 0:
            shift = (_rand01(gx, gy, 401, step_seed) - 0.5) * _f32(c["jitter"]) * _f32(0.05)
        a2 = _growth(a, spectra, mu, sigma, weight, c["mode"], _f32(0.1), shift)
        if c["noise"] > 0:
            a2 = a2 + (_rand01(gx, gy, 503, step_seed) - 0.5) * _f32(c["noise"]) * _f32(0.03)
        if c["inject"] > 0:
            ux, uy = (gx.double() + 0.5) / w, (gy.double() + 0.5) / h
            blob = c["radius"] * _f32(0.9) / h
            for b in range(4):
                dx, dy = ux - _rand01(b, 0, 811, step_seed), uy - _rand01(0, b, 823, step_seed)
                dx, dy = (dx - torch.round(dx)) * (w / h), dy - torch.round(dy)
                bump = torch.exp(-0.5 * (dx * dx + dy * dy) / (blob * blob))
                a2 = a2 + (_f32(0.6) - a2) * torch.clamp(bump * _f32(c["inject"]), 0.0, 1.0)
        a = torch.clamp(a2, 0.0, 1.0)
    if not c["render"]:
        return a
    rgb = [torch.clamp(0.5 + 0.5 * torch.cos(2.0 * math.pi * (a + d)), min=0.0) for d in (_f32(0.60), _f32(0.45), _f32(0.30))]
    return {"field": a, "rgba": torch.stack([*rgb, a], dim=-1)}


def _exact_batch(c, seed):
    out = []
    for w in _batch_worlds(c, seed):
        a = _dev(_world_field(w, seed).astype(np.float64))
        s = [_spectrum(_lut_on_torus(_direct_lut(w["radius"], "gaussShell"), w["width"], w["height"]))]
        for _ in range(c["steps"]):
            a = torch.clamp(_growth(a, s, [_f32(w["mu"])], [_f32(w["sigma"])], [1.0], 1, _f32(w["dt"])), 0.0, 1.0)
        out.append(a)
    return out


def _exact_grad(c, seed):
    a0, target = _grad_inputs(c, seed)
    a0, target = _dev(a0.astype(np.float64)), _dev(target.astype(np.float64))
    params = [p.double().to(a0.device).requires_grad_(True) for p in _grad_params()]
    mu, sigma, weight, betas, dt = params
    rings = []  # spectra and sums of the single rings of each kernel, peak 1 each
    for k in GRAD_RINGS:
        n = len(k["betas"])
        imgs = [_ring_image(c["w"], c["h"], float(c["radius"]), [1.0 if j == i else 0.0 for j in range(n)], "exp")
                for i in range(n)]
        rings.append([(torch.fft.rfft2(_dev(i)), float(i.sum())) for i in imgs])
    a0.requires_grad_(True)

    def one_step(a):
        spectra = [sum(betas[k, i] * r[0] for i, r in enumerate(rs)) / sum(betas[k, i] * r[1] for i, r in enumerate(rs))
                   for k, rs in enumerate(rings)]
        pre = _growth(a, spectra, mu, sigma, [weight[k] for k in range(len(rings))], c["mode"], dt)
        return torch.clamp(pre, 0.0, 1.0)

    a = a0
    for _ in range(c["steps"]):
        a = torch.utils.checkpoint.checkpoint(one_step, a, use_reentrant=False)
    grad = (a.detach() - target) * (2.0 / a.numel())
    g = torch.autograd.grad(a, [a0, *params], grad)
    return {"fields": a.detach(), "a0": g[0], "mu": g[1], "sigma": g[2], "weight": g[3], "betas": g[4], "dt": g[5]}


def exact(case, seed):
    c = case
    if c["kind"] == "module":
        return _exact_module(c, seed)
    return _exact_batch(c, seed) if c["kind"] == "batch" else _exact_grad(c, seed)
