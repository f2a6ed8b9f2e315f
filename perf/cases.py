"""Performance cases: the work a program has this library do, through its public entry points.

Every case is one of seven kinds of call:

* ``fit``     one iteration of a captured fit (``FitPlan`` + ``GraphStep``): render, loss,
              backward, Adam, clamp, for one image or a batch of mixed sizes;
* ``step``    one captured render forward + backward of an RS field (``RenderPlan``);
* ``eager``   one autograd forward + backward from a training loop of the user's own
              (``render_field`` on conics and radii, or ``render_gaussians`` on the RS field);
* ``view``    a forward-only render of a finished field (``render_gaussians``, no grad);
* ``place``   structure tensor, density, seeded sampling and field initialisation
              (``placement.place_field``);
* ``prune``   the pruning diagnostics of a field: ``gaussian_activity`` and the joint render
              with coverage;
* ``decode``  an SSPL1 container decoded and rendered (``codec.decode_and_render``), from bytes
              in host memory.

The fields follow the distributions of ``structsplat_b200.synthetic``: means uniform over the
image, sigma = exp(N(ln 2, 0.5)) px (around 1 px in a dense field), and for ``stress`` fields
exp(N(ln 2, 1.2)) with 30 % elongated Gaussians of aspect ratio 5 to 50.
"""
from __future__ import annotations

import json
import math
import struct
import zlib

import numpy as np
import torch

from structsplat_b200 import codec, render_field, render_gaussians
from structsplat_b200.batch import Batch, FitPlan, FitSettings, GraphStep
from structsplat_b200.fit import CapturedStep, RenderPlan
from structsplat_b200.placement import place_field
from structsplat_b200.render import gaussian_activity, render_cuda_exact_with_coverage

NAMES = ("means", "log_scales", "rotations", "colors", "opacity_logits")
CUTOFF = 3.0
EPS = 1e-8


# ------------------------------------------------------------------------------- the cases

def _fit(sizes, density, **kw):
    c = {"kind": "fit", "sizes": sizes, "density": density, "loss": "l2", "ssim": 0.0,
         "deterministic": False, "stress": False, "sigma": 2.0, "fade": 0.0, "opacity": True}
    c.update(kw)
    return c


def listed():
    return [
        # one small image, as an interactive or per-image fit has it: launches and latency
        {"name": "fit_small", **_fit("256x256", 0.0625)},
        # the batched fit of a folder of images of mixed sizes, 0.1 Gaussians per pixel
        {"name": "fit_batch", **_fit("256x256,512x512,768x512,1024x1024,512x768,1920x1080,"
                                     "256x256,2048x2048,512x512,1024x1024,1080x1920,768x512,"
                                     "512x512,1024x1024", 0.1)},
        # the fitter's default loss, 0.7 L1 + 0.3 (1 - SSIM), on a photograph of odd sides
        {"name": "fit_ssim", **_fit("1365x2047", 0.08, loss="l1", ssim=0.3)},
        # a dense fit from a placed field (no opacities), about one Gaussian per pixel
        {"name": "fit_dense", **_fit("1080x1920", 0.96, sigma=1.0, opacity=False)},
        # a reproducible fit of a heavy-tailed field: lists of thousands of Gaussians
        {"name": "fit_stress_exactly", **_fit("1024x1024", 0.24, deterministic=True, stress=True)},
        # forward + backward of 100k Gaussians at 1024x1024, the benchmark's own step
        {"name": "step_1024", "kind": "step", "H": 1024, "W": 1024, "n": 100_000,
         "normalize": True, "deterministic": False, "fade": 0.0, "opacity": True, "tile": 32},
        # a small ragged additive step with the support fade, reproducible, at 16-px tiles
        {"name": "step_ragged_exactly", "kind": "step", "H": 389, "W": 517, "n": 20_011,
         "normalize": False, "deterministic": True, "fade": 1.0, "opacity": False, "tile": 16},
        # the drop-in call of a training loop that computes conics and radii itself
        {"name": "eager_field", "kind": "eager", "H": 512, "W": 768, "n": 40_000,
         "call": "render_field", "normalize": True, "fade": 0.0, "opacity": True},
        # a finished field shown at 4K, once
        {"name": "view_4k", "kind": "view", "H": 2160, "W": 3840, "n": 800_000,
         "normalize": True, "fade": 0.0, "opacity": True},
        # placement of two million Gaussians on an HD image, seeded as the reference seeds it
        {"name": "place_hd", "kind": "place", "H": 1080, "W": 1920, "n": 2_000_000,
         "strategy": "aniso_onedge", "numpy_rng": True},
        # the pruning pass of the fitter between two rounds of a fit
        {"name": "prune_1024", "kind": "prune", "H": 1024, "W": 1024, "n": 250_000,
         "stress": False, "fade": 0.0},
        # a stored container shown: inflate, dequantise, render
        {"name": "decode_768", "kind": "decode", "H": 512, "W": 768, "n": 50_000,
         "morton": True, "opacity": True},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fit", "fit", "fit", "step", "step", "eager", "view", "place", "prune",
                       "decode"])
    H, W = _log_uniform(rng, 160, 1600), _log_uniform(rng, 160, 1600)
    density = math.exp(rng.uniform(math.log(0.02), math.log(0.3)))
    n = max(500, int(H * W * density))
    fade = rng.choice([0.0, 0.0, 1.0])
    opacity = rng.random() < 0.7
    if kind == "fit":
        images = rng.choice([1, 1, 2, 5])
        sizes = [f"{H}x{W}"] + [f"{_log_uniform(rng, 128, 900)}x{_log_uniform(rng, 128, 900)}"
                                for _ in range(images - 1)]
        ssim = rng.choice([0.0, 0.0, 0.3])
        stress = H * W <= 1_000_000 and rng.random() < 0.3
        return _fit(",".join(sizes), round(min(density, 0.2), 4), loss=rng.choice(
            ["l1", "l2", "charbonnier"]), ssim=ssim, deterministic=rng.random() < 0.4,
            stress=stress, sigma=rng.choice([1.0, 2.0]), fade=fade, opacity=opacity)
    if kind == "step":
        return {"kind": kind, "H": H, "W": W, "n": n, "normalize": rng.random() < 0.7,
                "deterministic": rng.random() < 0.4, "fade": fade, "opacity": opacity,
                "tile": rng.choice([16, 32, 32])}
    if kind == "eager":
        return {"kind": kind, "H": H, "W": W, "n": n,
                "call": rng.choice(["render_field", "render_gaussians"]),
                "normalize": rng.random() < 0.7, "fade": fade, "opacity": opacity}
    if kind == "view":
        H, W = _log_uniform(rng, 200, 2100), _log_uniform(rng, 200, 3800)
        return {"kind": kind, "H": H, "W": W, "n": max(500, int(H * W * min(density, 0.1))),
                "normalize": rng.random() < 0.7, "fade": fade, "opacity": opacity}
    if kind == "place":
        return {"kind": kind, "H": H, "W": W, "n": max(500, int(H * W * density)),
                "strategy": rng.choice(["aniso_onedge", "iso_blue_noise"]),
                "numpy_rng": rng.random() < 0.7}
    if kind == "prune":
        return {"kind": kind, "H": H, "W": W, "n": max(500, n // 2),
                "stress": H * W <= 1_000_000 and rng.random() < 0.4, "fade": fade}
    return {"kind": "decode", "H": min(H, 1000), "W": min(W, 1000),
            "n": min(n, 200_000), "morton": rng.random() < 0.7, "opacity": opacity}


# ------------------------------------------------------------------------------- the inputs

def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _target(H, W, g):
    """Gratings, filled discs and noise in [0, 1], as the synthetic targets have them."""
    ys = torch.arange(H, device="cuda", dtype=torch.float32)[:, None]
    xs = torch.arange(W, device="cuda", dtype=torch.float32)[None, :]
    r = torch.rand(8 + 12, 7, device="cuda", generator=g).tolist()
    img = torch.full((H, W, 3), 0.5, device="cuda")
    for a in r[:8]:
        th, k = math.pi * a[0], 2 * math.pi / (8.0 + 56.0 * a[1])
        wave = torch.sin((xs * math.cos(th) + ys * math.sin(th)) * k + 6.28 * a[2])
        img += wave[..., None] * torch.tensor([0.25 * v - 0.125 for v in a[3:6]], device="cuda")
    for a in r[8:]:
        rad = (0.04 + 0.2 * a[2]) * min(H, W)
        inside = (xs - a[0] * W) ** 2 + (ys - a[1] * H) ** 2 < rad * rad
        img = torch.where(inside[..., None], torch.tensor(a[3:6], device="cuda"), img)
    img += 0.02 * torch.randn(H, W, 3, device="cuda", generator=g)
    return img.clamp_(0.0, 1.0).contiguous()


def _field(H, W, n, g, stress=False, opacity=True, sigma=2.0):
    def rand(*s):
        return torch.rand(*s, device="cuda", generator=g)

    def randn(*s):
        return torch.randn(*s, device="cuda", generator=g)
    f = {"means": rand(n, 2) * torch.tensor([float(W), float(H)], device="cuda"),
         "rotations": rand(n) * math.pi, "colors": rand(n, 3),
         "opacity_logits": randn(n) if opacity else None}
    if stress:
        ls = (math.log(2.0) + 1.2 * randn(n))[:, None].repeat(1, 2)
        half = 0.5 * torch.log(5.0 + 45.0 * rand(n)) * (rand(n) < 0.3)
        f["log_scales"] = torch.stack([ls[:, 0] + half, ls[:, 1] - half], 1).contiguous()
    else:
        f["log_scales"] = math.log(sigma) + 0.5 * randn(n, 2)
    return f


def _sizes(case):
    return [tuple(int(v) for v in s.split("x")) for s in case["sizes"].split(",")]


def _counts(case):
    return [max(16, int(round(case["density"] * h * w))) for h, w in _sizes(case)]


def _settings(case):
    # the rates of a fit that is under way, a tenth of the ones it starts with
    return FitSettings(lr_means=5e-3, lr_scales=3e-3, lr_rot=1e-3, lr_color=3e-3,
                       lr_opacity=1e-3, pixel_loss=case["loss"], ssim_weight=case["ssim"],
                       deterministic=case["deterministic"], fade_alpha=case["fade"])


def _fit_inputs(case, seed):
    """Fields, targets and the Adam state of a fit that is resumed after STEPS_DONE steps."""
    g = _generator(seed)
    sizes, counts = _sizes(case), _counts(case)
    fields = [_field(h, w, n, g, case["stress"], case["opacity"], case["sigma"])
              for (h, w), n in zip(sizes, counts)]
    targets = [_target(h, w, g) for h, w in sizes]
    params = Batch.concat_fields(fields)
    scale = torch.repeat_interleave(
        torch.tensor([0.3 / (h * w) for h, w in sizes], device="cuda"),
        torch.tensor(counts, device="cuda"))
    m, v = {}, {}
    for k in NAMES:
        if params[k] is None:
            continue
        s = scale.view([-1] + [1] * (params[k].dim() - 1))
        m[k] = 0.3 * s * torch.randn(params[k].shape, device="cuda", generator=g)
        v[k] = s * s * (0.5 + torch.rand(params[k].shape, device="cuda", generator=g))
    return sizes, counts, params, targets, m, v


STEPS_DONE = 100


def _conics32(ls, rot, dilation=0.0):
    sx2, sy2 = torch.exp(ls[:, 0]) ** 2 + dilation, torch.exp(ls[:, 1]) ** 2 + dilation
    c, s = torch.cos(rot), torch.sin(rot)
    return torch.stack([c * c / sx2 + s * s / sy2, c * s * (1 / sx2 - 1 / sy2),
                        s * s / sx2 + c * c / sy2], 1).contiguous()


def _radii32(ls, rot, cutoff=CUTOFF):
    """ceil(cutoff sqrt(var)) per axis in float32, which is how the support is defined."""
    sx2, sy2 = torch.exp(ls[:, 0]) ** 2, torch.exp(ls[:, 1]) ** 2
    c, s = torch.cos(rot), torch.sin(rot)
    cc, ss = c * c, s * s
    var = torch.stack([cc * sx2 + ss * sy2, ss * sx2 + cc * sy2], 1)
    return torch.ceil(cutoff * torch.sqrt(var)).clamp_min(1.0).to(torch.int64).contiguous()


def _container(case, seed):
    """An SSPL1 container of a quantised field, written as the format's encoder writes it."""
    H, W, n = case["H"], case["W"], case["n"]
    f = _field(H, W, n, _generator(seed), opacity=case["opacity"])
    f = {k: None if v is None else v.double().cpu().numpy() for k, v in f.items()}
    bits = [16, 8, 8, 8]
    lo_s, hi_s = f["log_scales"].min(0), f["log_scales"].max(0)
    lo_c, hi_c = f["colors"].min(0), f["colors"].max(0)

    def quant(x, lo, hi, b):
        return np.rint(np.clip((x - lo) / (hi - lo), 0, 1) * (2 ** b - 1)).astype(np.uint32)
    qm = quant(f["means"], np.zeros(2), np.array([W, H], float), bits[0])
    qs, qc = quant(f["log_scales"], lo_s, hi_s, bits[1]), quant(f["colors"], lo_c, hi_c, bits[3])
    qr = np.floor(f["rotations"] / math.pi * 2 ** bits[2]).astype(np.uint32) % 2 ** bits[2]
    qo = None
    if case["opacity"]:
        qo = quant(1 / (1 + np.exp(-f["opacity_logits"])), 0.0, 1.0, 8)
    if case["morton"]:
        code = np.zeros(n, np.uint64)
        for b in range(bits[0]):
            for d in range(2):
                code |= ((qm[:, d].astype(np.uint64) >> np.uint64(b)) & np.uint64(1)) << np.uint64(
                    2 * b + d)
        order = np.argsort(code, kind="stable")
        qm, qs, qr, qc = qm[order], qs[order], qr[order], qc[order]
        qo = None if qo is None else qo[order]

    def delta(q, b):
        return (np.diff(q, axis=0, prepend=np.zeros_like(q[:1])) & np.uint32(2 ** b - 1))
    means = delta(qm, bits[0]) if case["morton"] else qm
    colors = delta(qc, bits[3]) if case["morton"] else qc
    m16 = means.T.astype("<u2").reshape(-1)
    if case["morton"]:  # byte-planar
        m16 = np.concatenate([(m16 & 0xFF).astype(np.uint8), (m16 >> 8).astype(np.uint8)])
    raws = [m16.tobytes(), qs.T.astype(np.uint8).tobytes(), qr.astype(np.uint8).tobytes(),
            colors.T.astype(np.uint8).tobytes()]
    if qo is not None:
        raws.append(qo.astype(np.uint8).tobytes())
    header = {"n": n, "H": H, "W": W, "bits": bits, "morton": case["morton"],
              "color_delta": case["morton"], "means_byte_planar": case["morton"],
              "rot_circular": True, "stream_codec": "zlib",
              "stream_raw_lengths": [len(r) for r in raws], "color_lo": lo_c.tolist(),
              "color_hi": hi_c.tolist(), "scale_lo": lo_s.tolist(), "scale_hi": hi_s.tolist(),
              "means_lo": [0.0, 0.0], "means_hi": [float(W), float(H)],
              "has_opacity": case["opacity"], "bits_opacity": 8, "renderer": "normalized",
              "aa_dilation": 0.0, "sigma_cutoff": CUTOFF, "support_fade": False}
    head = json.dumps(header).encode()
    blob = b"SSPL1" + struct.pack("<I", len(head)) + head
    for r in raws:
        z = zlib.compress(r, 6)
        blob += struct.pack("<I", len(z)) + z
    quantised = {"qm": qm, "qs": qs, "qr": qr, "qc": qc, "qo": qo, "header": header}
    return blob, quantised


def prepare(case, seed):
    kind = case["kind"]
    if kind == "fit":
        sizes, counts, params, targets, m, v = _fit_inputs(case, seed)
        batch = Batch(sizes, counts)
        plan = FitPlan(batch, params, batch.concat_images(targets), _settings(case))
        step = torch.tensor([STEPS_DONE, 0], dtype=torch.int32, device="cuda")
        plan.restore(({}, m, v, step))
        out = {"loss": plan.loss, "gradients": plan.gradients(), "params": params,
               "exp_avg": plan.exp_avg, "exp_avg_sq": plan.exp_avg_sq}
        if case["ssim"] > 0:
            out["ssim"] = plan.ssim
        return {"kind": kind, "plan": plan, "graph": GraphStep(plan), "out": out}
    g = _generator(seed)
    if kind == "step":
        H, W = case["H"], case["W"]
        params = _field(H, W, case["n"], g, opacity=case["opacity"])
        grad = torch.randn(H, W, 3, device="cuda", generator=g) / (3 * H * W)
        plan = RenderPlan.for_field(params, H, W, normalize=case["normalize"],
                                    fade_alpha=case["fade"], tile_size=case["tile"],
                                    deterministic=case["deterministic"])
        graph = CapturedStep(lambda: plan.forward_backward(params, grad))
        return {"kind": kind, "plan": plan, "graph": graph, "keep": (params, grad)}
    if kind == "eager":
        H, W = case["H"], case["W"]
        f = _field(H, W, case["n"], g, opacity=case["opacity"])
        grad = torch.randn(H, W, 3, device="cuda", generator=g) / (3 * H * W)
        if case["call"] == "render_field":
            leaves = [f["means"], _conics32(f["log_scales"], f["rotations"]), f["colors"]]
            if case["opacity"]:
                leaves.append(torch.sigmoid(f["opacity_logits"]))
        else:
            leaves = [f[k] for k in NAMES if f[k] is not None]
        leaves = [t.detach().requires_grad_(True) for t in leaves]
        return {"kind": kind, "case": case, "leaves": leaves, "grad": grad,
                "radii": _radii32(f["log_scales"], f["rotations"])}
    if kind == "view":
        return {"kind": kind, "case": case,
                "f": _field(case["H"], case["W"], case["n"], g, opacity=case["opacity"])}
    if kind == "place":
        return {"kind": kind, "case": case, "seed": seed,
                "image": _target(case["H"], case["W"], g)}
    if kind == "prune":
        f = _field(case["H"], case["W"], case["n"], g, stress=case["stress"])
        return {"kind": kind, "case": case, "means": f["means"], "colors": f["colors"],
                "conics": _conics32(f["log_scales"], f["rotations"]),
                "radii": _radii32(f["log_scales"], f["rotations"]),
                "opacities": torch.sigmoid(f["opacity_logits"])}
    return {"kind": kind, "blob": _container(case, seed)[0]}


# --------------------------------------------------------------------------------- the pass

def run(state):
    kind = state["kind"]
    if kind == "fit":
        state["graph"].replay()
        return state["out"]
    if kind == "step":
        state["graph"].replay()
        plan = state["plan"]
        return {"image": plan.image, "den": plan.den, "gradients": plan.grads()}
    if kind == "eager":
        c, leaves = state["case"], state["leaves"]
        op = leaves[-1] if c["opacity"] else None
        if c["call"] == "render_field":
            image = render_field(leaves[0], leaves[1], leaves[2], state["radii"], c["H"], c["W"],
                                 mode="b200" if c["normalize"] else "b200_additive",
                                 opacities=op, support_fade=c["fade"] > 0)
        else:
            image = render_gaussians(*leaves[:4], c["H"], c["W"], opacity_logits=op,
                                     normalize=c["normalize"], support_fade=c["fade"] > 0)
        return {"image": image,
                "gradients": torch.autograd.grad(image, leaves, state["grad"])}
    if kind == "view":
        c, f = state["case"], state["f"]
        with torch.no_grad():
            return render_gaussians(f["means"], f["log_scales"], f["rotations"], f["colors"],
                                    c["H"], c["W"], opacity_logits=f["opacity_logits"],
                                    normalize=c["normalize"], support_fade=c["fade"] > 0)
    if kind == "place":
        c = state["case"]
        field, tensor, density = place_field(state["image"], c["n"], strategy=c["strategy"],
                                             seed=state["seed"], numpy_rng=c["numpy_rng"])
        return {"field": {k: field[k] for k in NAMES[:4]}, "density": density,
                "energy": tensor.energy, "label": tensor.label}
    if kind == "prune":
        c = state["case"]
        act = gaussian_activity(state["means"], state["conics"], state["radii"], c["H"], c["W"],
                                support_fade=c["fade"] > 0)
        image, cover = render_cuda_exact_with_coverage(
            state["means"], state["conics"], state["colors"], state["radii"], c["H"], c["W"],
            opacities=state["opacities"], support_fade=c["fade"] > 0)
        return {"activity": act, "image": image, "coverage": cover}
    return codec.decode_and_render(state["blob"])


# ----------------------------------------------------------------------------- the least work

def _pairs(H, W, n, stress=False, sigma=2.0):
    """Expected (pixel, Gaussian) pairs inside the clipped support rectangles, from a sample."""
    rng = np.random.default_rng(0)
    m = 20_000
    if stress:
        s = rng.normal(math.log(2.0), 1.2, m)
        half = 0.5 * np.log(rng.uniform(5, 50, m)) * (rng.random(m) < 0.3)
        sx, sy = np.exp(s + half), np.exp(s - half)
    else:
        sx, sy = np.exp(rng.normal(math.log(sigma), 0.5, (2, m)))
    th = rng.uniform(0, math.pi, m)
    rx = np.ceil(CUTOFF * np.hypot(np.cos(th) * sx, np.sin(th) * sy))
    ry = np.ceil(CUTOFF * np.hypot(np.sin(th) * sx, np.cos(th) * sy))
    x, y = rng.uniform(0, W, m), rng.uniform(0, H, m)
    w = np.clip(np.minimum(x + rx, W - 1) - np.maximum(x - rx, 0) + 1, 0, None)
    h = np.clip(np.minimum(y + ry, H - 1) - np.maximum(y - ry, 0) + 1, 0, None)
    return float((w * h).mean()) * n


FWD, BWD = 20.0, 50.0  # operations of one pair (an exponential counted as one)


def work(case):
    kind = case["kind"]
    if kind == "fit":
        sizes, counts = _sizes(case), _counts(case)
        px, n = sum(h * w for h, w in sizes), sum(counts)
        pairs = sum(_pairs(h, w, k, case["stress"], case["sigma"]) for (h, w), k in zip(sizes, counts))
        p = 36.0 if case["opacity"] else 32.0
        # parameters and both moments in and out, gradients out; targets in
        return {"bytes": n * 7 * p + px * 12.0,
                "flops": pairs * (FWD + BWD) + (px * 600.0 if case["ssim"] else 0.0) + n * 150.0}
    H, W = case["H"], case["W"]
    px = H * W
    n = case["n"]
    if kind == "place":
        # the image in, density, energy and label out; 3 uniforms in and the field out per point
        return {"bytes": px * (12.0 + 13.0) + n * (24.0 + 32.0),
                "flops": px * 260.0 + n * 100.0}
    if kind == "decode":
        return {"bytes": px * 12.0 + n * 11.0, "flops": _pairs(H, W, n) * FWD + n * 60.0}
    pairs = _pairs(H, W, n, case.get("stress", False))
    if kind == "prune":
        return {"bytes": n * (8 + 12 + 12 + 16 + 4 + 4.0) + px * 16.0,
                "flops": pairs * (FWD + 10.0)}
    p = 36.0 if case["opacity"] else 32.0
    if kind == "view":
        return {"bytes": n * p + px * 12.0, "flops": pairs * FWD}
    return {"bytes": n * 2 * p + px * (16.0 + 12.0), "flops": pairs * (FWD + BWD)}


# ------------------------------------------------------------------------- the same in 64 bits

MOST_PAIRS = 1.6e9  # beyond this the 64-bit evaluation takes too long


def _rects(means32, radii, H, W):
    c = torch.round(means32).to(torch.int64)
    x0, x1 = (c[:, 0] - radii[:, 0]).clamp_min(0), (c[:, 0] + radii[:, 0]).clamp_max(W - 1) + 1
    y0, y1 = (c[:, 1] - radii[:, 1]).clamp_min(0), (c[:, 1] + radii[:, 1]).clamp_max(H - 1) + 1
    w, h = (x1 - x0).clamp_min(0), (y1 - y0).clamp_min(0)
    return x0, y0, w, w * h


def _chunks(area, most=12_000_000):
    ends = torch.cumsum(area, 0).cpu()
    n, at, done = area.numel(), 0, 0
    while at < n:
        to = int(torch.searchsorted(ends, torch.tensor(done + most), right=True))
        to = min(n, max(to, at + 1))
        yield at, to
        done, at = int(ends[to - 1]), to


def _pair_terms(a, b, rect, means, conics, W):
    x0, y0, w, area = (t[a:b] for t in rect)
    g = torch.repeat_interleave(torch.arange(a, b, device="cuda"), area)
    first = torch.cumsum(area, 0) - area
    k = torch.arange(g.numel(), device="cuda") - first[g - a]
    ww = w[g - a]
    x, y = x0[g - a] + k % ww, y0[g - a] + k // ww
    dx, dy = x.double() - means[g, 0], y.double() - means[g, 1]
    c = conics[g]
    raw = torch.exp(-0.5 * (c[:, 0] * dx * dx + 2 * c[:, 1] * dx * dy + c[:, 2] * dy * dy))
    return g, y * W + x, dx, dy, raw, area, first


def _sum_runs(v, area, first):
    s = torch.cat([torch.zeros(1, dtype=torch.float64, device="cuda"), torch.cumsum(v, 0)])
    return s[first + area] - s[first]


def _render64(rect, means, conics, colors, op, H, W, tail, normalize):
    num = torch.zeros(H * W, 3, dtype=torch.float64, device="cuda")
    den = torch.zeros(H * W, dtype=torch.float64, device="cuda")
    for a, b in _chunks(rect[3]):
        g, p, _, _, raw, _, _ = _pair_terms(a, b, rect, means, conics, W)
        wt = (raw - tail).clamp_min(0) * op[g]
        num.index_add_(0, p, wt[:, None] * colors[g])
        den.index_add_(0, p, wt)
    image = num / (den + EPS)[:, None] if normalize else num
    return image, den


def _grads64(rect, means, conics, colors, op, H, W, tail, normalize, image, den, go):
    """Gradients of sum(image * go) with respect to means, conics, colours and opacities."""
    inv = 1 / (den + EPS) if normalize else torch.ones_like(den)
    gn = go * inv[:, None]
    gd = -(go * image).sum(1) * inv if normalize else torch.zeros_like(den)
    n = means.shape[0]
    out = torch.zeros(9, n, dtype=torch.float64, device="cuda")
    for a, b in _chunks(rect[3]):
        g, p, dx, dy, raw, area, first = _pair_terms(a, b, rect, means, conics, W)
        vis = (raw - tail).clamp_min(0)
        q = gn[p]
        dw = (q * colors[g]).sum(1) + gd[p]
        for k in range(3):
            out[5 + k, a:b] = _sum_runs(vis * q[:, k], area, first) * op[a:b]
        out[8, a:b] = _sum_runs(vis * dw, area, first)
        t = op[g] * raw * dw * (raw > tail)
        c = conics[g]
        out[0, a:b] = _sum_runs(t * (c[:, 0] * dx + c[:, 1] * dy), area, first)
        out[1, a:b] = _sum_runs(t * (c[:, 1] * dx + c[:, 2] * dy), area, first)
        out[2, a:b] = _sum_runs(-0.5 * t * dx * dx, area, first)
        out[3, a:b] = _sum_runs(-t * dx * dy, area, first)
        out[4, a:b] = _sum_runs(-0.5 * t * dy * dy, area, first)
    return (out[:2].T.contiguous(), out[2:5].T.contiguous(), out[5:8].T.contiguous(), out[8])


def _tail(fade):
    return float(np.float32(fade * math.exp(-0.5 * CUTOFF ** 2))) if fade > 0 else 0.0


def _rs64(f, H, W, normalize, fade, grad_of_image=None):
    """Image, den and (given grad_of_image(image)) the gradients of the RS field f."""
    ls = f["log_scales"].double().requires_grad_(True)
    rot = f["rotations"].double().requires_grad_(True)
    conics = _conics32(ls, rot)
    logits = f.get("opacity_logits")
    n = f["means"].shape[0]
    op = torch.ones(n, dtype=torch.float64, device="cuda")
    if logits is not None:
        op = torch.sigmoid(logits.double())
    rect = _rects(f["means"], _radii32(f["log_scales"], f["rotations"]), H, W)
    means, colors, tail = f["means"].double(), f["colors"].double(), _tail(fade)
    con = conics.detach()
    image, den = _render64(rect, means, con, colors, op, H, W, tail, normalize)
    if grad_of_image is None:
        return image, den, None
    go = grad_of_image(image)
    gm, gc, gcol, gop = _grads64(rect, means, con, colors, op, H, W, tail, normalize, image,
                                 den, go)
    gls, grot = torch.autograd.grad(conics, (ls, rot), gc)
    grads = {"means": gm, "log_scales": gls, "rotations": grot, "colors": gcol,
             "opacity_logits": None if logits is None else gop * op * (1 - op)}
    return image, den, grads


def _ssim64(img, tgt):
    """Mean SSIM of (3, H, W) images: 11-tap window, sigma 1.5, zero padding."""
    x = torch.arange(-5, 6, dtype=torch.float64, device="cuda")
    k = torch.exp(-x * x / (2 * 1.5 ** 2))
    k = k / k.sum()

    def win(t):
        t = t[:, None]
        t = torch.nn.functional.conv2d(t, k.view(1, 1, 1, 11), padding=(0, 5))
        return torch.nn.functional.conv2d(t, k.view(1, 1, 11, 1), padding=(5, 0))[:, 0]
    c1, c2 = 0.01 ** 2, 0.03 ** 2
    mp, mt = win(img), win(tgt)
    sp, st, spt = win(img * img) - mp * mp, win(tgt * tgt) - mt * mt, win(img * tgt) - mp * mt
    return (((2 * mp * mt + c1) * (2 * spt + c2))
            / ((mp * mp + mt * mt + c1) * (sp + st + c2))).mean()


def _fit64(case, seed):
    sizes, counts, params, targets, m, v = _fit_inputs(case, seed)
    s = _settings(case)
    loss, ssims, grads, hi, at = [], [], [], [], 0
    for (H, W), n, tgt in zip(sizes, counts, targets):
        f = {k: None if params[k] is None else params[k][at:at + n] for k in NAMES}
        at += n
        t64 = tgt.double().reshape(-1, 3)

        def grad_of_image(image):
            leaf = image.detach().requires_grad_(True)
            d = leaf - t64
            pixel = {"l1": d.abs(), "l2": d * d, "charbonnier": torch.sqrt(
                d * d + s.charbonnier_eps ** 2)}[s.pixel_loss].mean()
            total = pixel
            if s.ssim_weight > 0:
                def chw(t):
                    return t.reshape(H, W, 3).permute(2, 0, 1)
                value = _ssim64(chw(leaf), chw(t64))
                ssims.append(value.detach())
                total = (1 - s.ssim_weight) * pixel + s.ssim_weight * (1 - value)
            loss.append(torch.stack([pixel.detach(), (d * d).mean().detach()]))
            return torch.autograd.grad(total, leaf)[0]
        grads.append(_rs64(f, H, W, True, case["fade"], grad_of_image)[2])
        hi.append(torch.full((n, 1), math.log(max(H, W)), dtype=torch.float64, device="cuda"))
    g = {k: None if params[k] is None else torch.cat([x[k] for x in grads]) for k in NAMES}
    b1, b2 = s.betas
    t = STEPS_DONE + 1
    out = {"loss": torch.stack(loss), "gradients": g, "params": {}, "exp_avg": {},
           "exp_avg_sq": {}}
    for k, lr in zip(NAMES, s.lrs()):
        if params[k] is None:
            out["params"][k] = None
            continue
        mm = b1 * m[k].double() + (1 - b1) * g[k]
        vv = b2 * v[k].double() + (1 - b2) * g[k] * g[k]
        p = params[k].double() - lr / (1 - b1 ** t) * mm / (
            torch.sqrt(vv / (1 - b2 ** t)) + s.adam_eps)
        if k == "log_scales":
            p = torch.minimum(p, torch.cat(hi)).clamp_min(math.log(s.scale_min))
        out["params"][k], out["exp_avg"][k], out["exp_avg_sq"][k] = p, mm, vv
    if s.ssim_weight > 0:
        out["ssim"] = torch.stack(ssims)
    return out


def _energy64(image):
    """lam1 + lam2 of the structure tensor (sigma 1, rho 2, luma, central) in 64 bits."""
    def blur(t, sigma):
        r = int(round(3.0 * sigma))
        x = np.arange(-r, r + 1, dtype=np.float64)
        k = np.exp(-0.5 * (x / sigma) ** 2)
        k = torch.tensor(k / k.sum(), device="cuda")
        t = torch.nn.functional.pad(t[None], (0, 0, r, r), mode="reflect")[0]
        t = torch.nn.functional.conv2d(t[:, None], k.view(1, 1, -1, 1))[:, 0]
        t = torch.nn.functional.pad(t[None], (r, r, 0, 0), mode="reflect")[0]
        return torch.nn.functional.conv2d(t[:, None], k.view(1, 1, 1, -1))[:, 0]
    luma = torch.tensor([0.2126, 0.7152, 0.0722], dtype=torch.float64, device="cuda")
    img = blur((image.double() * luma).sum(2)[None], 1.0)[0]
    iy, ix = torch.gradient(img)
    j = blur(torch.stack([ix * ix, ix * iy, iy * iy]), 2.0)
    half, diff = 0.5 * (j[0] + j[2]), 0.5 * (j[0] - j[2])
    r = torch.sqrt(diff * diff + j[1] * j[1])
    return half + r + (half - r).clamp_min(0)


def _energy_ref(energy):
    e = energy.flatten()
    s = torch.sort(e)[0]
    n = s.numel()
    pos = (n - 1) * 0.99
    lo = int(math.floor(pos))
    p99 = s[lo] + (s[min(lo + 1, n - 1)] - s[lo]) * (pos - lo)
    med = (s[(n - 1) // 2] + s[n // 2]) / 2
    return torch.maximum(p99, 8 * med) + 1e-12


def exact(case, seed):
    kind = case["kind"]
    if kind == "fit":
        pairs = sum(_pairs(h, w, k, case["stress"], case["sigma"])
                    for (h, w), k in zip(_sizes(case), _counts(case)))
        return _fit64(case, seed) if pairs <= MOST_PAIRS else None
    g = _generator(seed)
    H, W = case["H"], case["W"]
    if kind == "place":
        energy = _energy64(_target(H, W, g))
        d = 0.05 + 0.95 * (energy / _energy_ref(energy)).clamp(0, 1)
        # the sampled points sit on either side of a rounding of the density: no exact value
        return {"field": {k: None for k in NAMES[:4]}, "density": d / d.sum(),
                "energy": energy, "label": None}
    n = case["n"]
    if _pairs(H, W, n, case.get("stress", False)) > MOST_PAIRS:
        return None
    if kind == "decode":
        q = _container(case, seed)[1]
        h = q["header"]

        def value(a, lo, hi, b):
            return np.asarray(lo) + a.astype(np.float64) / (2 ** b - 1) * (
                np.asarray(hi) - np.asarray(lo))
        f = {"means": value(q["qm"], h["means_lo"], h["means_hi"], 16),
             "log_scales": value(q["qs"], h["scale_lo"], h["scale_hi"], 8),
             "rotations": q["qr"].astype(np.float64) / 256 * math.pi,
             "colors": value(q["qc"], h["color_lo"], h["color_hi"], 8)}
        if case["opacity"]:
            p = np.clip(q["qo"].astype(np.float64) / 255, 1e-4, 1 - 1e-4)
            f["opacity_logits"] = np.log(p / (1 - p))
        # the decoded field is float32 by the format's definition
        f = {k: torch.tensor(v, device="cuda").float() for k, v in f.items()}
        return _rs64(f, H, W, True, 0.0)[0].reshape(H, W, 3)
    if kind == "prune":
        f = _field(H, W, n, g, stress=case["stress"])
        con = _conics32(f["log_scales"], f["rotations"]).double()
        rect = _rects(f["means"], _radii32(f["log_scales"], f["rotations"]), H, W)
        tail, means = _tail(case["fade"]), f["means"].double()
        act = torch.zeros(n, dtype=torch.float64, device="cuda")
        for a, b in _chunks(rect[3]):
            _, _, _, _, raw, area, first = _pair_terms(a, b, rect, means, con, W)
            act[a:b] = _sum_runs((raw - tail).clamp_min(0), area, first)
        op = torch.sigmoid(f["opacity_logits"]).double()
        image, den = _render64(rect, means, con, f["colors"].double(), op, H, W, tail, True)
        return {"activity": act, "image": image.reshape(H, W, 3), "coverage": den.reshape(H, W)}
    f = _field(H, W, n, g, opacity=case["opacity"])
    if kind == "view":
        return _rs64(f, H, W, case["normalize"], case["fade"])[0].reshape(H, W, 3)
    go = (torch.randn(H, W, 3, device="cuda", generator=g) / (3 * H * W)).double().reshape(-1, 3)
    if kind == "eager" and case["call"] == "render_field":
        con = _conics32(f["log_scales"], f["rotations"]).double()
        rect = _rects(f["means"], _radii32(f["log_scales"], f["rotations"]), H, W)
        op = torch.ones(n, dtype=torch.float64, device="cuda")
        if case["opacity"]:
            op = torch.sigmoid(f["opacity_logits"]).double()
        args = (rect, f["means"].double(), con, f["colors"].double(), op, H, W,
                _tail(case["fade"]), case["normalize"])
        image, den = _render64(*args)
        grads = _grads64(*args, image, den, go)
        return {"image": image.reshape(H, W, 3),
                "gradients": grads if case["opacity"] else grads[:3]}
    image, den, grads = _rs64(f, H, W, case["normalize"], case["fade"], lambda _: go)
    image = image.reshape(H, W, 3)
    if kind == "eager":
        return {"image": image, "gradients": [grads[k] for k in NAMES if grads[k] is not None]}
    return {"image": image, "den": den.reshape(H, W), "gradients": grads}
