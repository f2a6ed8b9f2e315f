"""Deterministic gradients by slots and by runs are bitwise those by sorted entries (render step, fused
pass and fit step), and an index that overflowed is reported."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from gpu_helpers import require_cuda
from structsplat_b200.batch import Batch, FitPlan, FitSettings
from structsplat_b200.fit import RenderPlan
from structsplat_b200.synthetic import make_field, make_stress_field

pytestmark = pytest.mark.gpu
NAMES = ("means", "log_scales", "rotations", "colors", "opacity_logits")


def _params(f):
    return {k: torch.tensor(getattr(f, k), device="cuda") for k in NAMES}


def _field(kind, H, W, n):
    if kind == "stress":  # streamed lists, rectangles of thousands of tiles, underflowed entries
        return _params(make_stress_field(H, W, n, 3, np.full((H, W), 0.3)))
    p = _params(make_field(H, W, n, 3))
    p["means"][: n // 8] += 3.0 * W  # off the image: no entries
    return p


@pytest.mark.parametrize("fused", [False, True])
@pytest.mark.parametrize("kind,H,W,n,ts", [
    ("plain", 33, 31, 1, 32), ("plain", 200, 170, 257, 16), ("plain", 517, 389, 9_000, 32),
    ("stress", 256, 256, 15_000, 32), ("stress", 250, 199, 9_000, 16)])
def test_slots_are_sorted_entries(kind, H, W, n, ts, fused):
    require_cuda()
    p = _field(kind, H, W, n)
    go = torch.randn(H, W, 3, device="cuda", generator=torch.Generator("cuda").manual_seed(0))
    got = []
    for det in (1, 2):
        plan = RenderPlan.for_field(p, H, W, deterministic=True, tile_size=ts, fused=fused)
        assert plan.det == 2
        plan.det = det
        got.append({k: v.clone() for k, v in plan.forward_backward(p, go).items()})
        assert int(plan.status) == 0
    for k in got[0]:
        assert torch.equal(got[0][k].view(torch.int32), got[1][k].view(torch.int32)), k


@pytest.mark.parametrize("fused", [False, True])
def test_fit_steps_agree(fused):
    require_cuda()
    sizes, counts = [(100, 130), (64, 64), (37, 301)], [900, 1, 700]
    out = []
    for det in (1, 2):
        fields = [_params(make_field(h, w, c, seed=7 + c)) for (h, w), c in zip(sizes, counts)]
        params = Batch.concat_fields(fields)
        batch = Batch(sizes, counts)
        target = torch.rand(batch.pixels, 3, device="cuda",
                            generator=torch.Generator("cuda").manual_seed(1))
        plan = FitPlan(batch, params, target, FitSettings(deterministic=True, fused=fused))
        plan.det = det
        for _ in range(3):
            plan.step()
        out.append({**params, **{f"g_{k}": v.clone() for k, v in plan.gradients().items()}})
    for k in out[0]:
        assert torch.equal(out[0][k], out[1][k]), k


def test_overflow_is_reported():
    require_cuda()
    H = W = 128
    p = _field("plain", H, W, 500)
    plan = RenderPlan(500, H, W, capacity=64, deterministic=True)
    grads = plan.forward_backward(p, torch.ones(H, W, 3, device="cuda"))
    assert plan.overflowed() and int(plan.status) & 4
    assert all(bool((g == 0).all()) for g in grads.values())


@pytest.mark.parametrize("fused", [False, True])
@pytest.mark.parametrize("fade", [0.0, 1.0])
@pytest.mark.parametrize("kind,H,W,n,ts", [
    ("plain", 33, 31, 1, 32), ("plain", 200, 170, 257, 16), ("plain", 517, 389, 9_000, 32),
    ("stress", 256, 256, 15_000, 32), ("stress", 600, 900, 9_000, 16), ("wide", 1000, 900, 40, 16),
    ("wide", 1500, 1500, 12, 16)])
def test_runs_are_sorted_entries(kind, H, W, n, ts, fade, fused):
    """Rectangles of 1, 32, 33 and thousands of tiles; runs beyond a warp's and a CTA's buffer."""
    require_cuda()
    p = _field("plain" if kind == "wide" else kind, H, W, n)
    if kind == "wide":
        p["log_scales"][:] = torch.linspace(2.0, 6.0, n, device="cuda")[:, None]
    go = torch.randn(H, W, 3, device="cuda", generator=torch.Generator("cuda").manual_seed(0))
    got = []
    for det in (1, 3):
        plan = RenderPlan.for_field(p, H, W, deterministic=True, tile_size=ts, fused=fused,
                                    fade_alpha=fade)
        plan.det = det
        got.append({k: v.clone() for k, v in plan.forward_backward(p, go).items()})
        assert int(plan.status) == 0
    for k in got[0]:
        assert torch.equal(got[0][k].view(torch.int32), got[1][k].view(torch.int32)), k


def test_runs_in_a_batch():
    require_cuda()
    sizes, counts = [(100, 130), (64, 64), (337, 301)], [900, 1, 700]
    out = []
    for det in (1, 3):
        fields = [_params(make_field(h, w, c, seed=7 + c)) for (h, w), c in zip(sizes, counts)]
        fields[2]["log_scales"][:50] = 4.0
        params = Batch.concat_fields(fields)
        batch = Batch(sizes, counts)
        target = torch.rand(batch.pixels, 3, device="cuda",
                            generator=torch.Generator("cuda").manual_seed(1))
        plan = FitPlan(batch, params, target, FitSettings(deterministic=True, fade_alpha=1.0))
        assert plan.det == 3
        plan.det = det
        for _ in range(3):
            plan.step()
        out.append({**params, **{f"g_{k}": v.clone() for k, v in plan.gradients().items()}})
    for k in out[0]:
        assert torch.equal(out[0][k], out[1][k]), k


def test_the_mode_follows_the_cull():
    require_cuda()
    assert RenderPlan(10, 64, 64, deterministic=True, fade_alpha=1.0).det == 3
    assert RenderPlan(10, 64, 64, deterministic=True, fade_alpha=0.5).det == 2
    assert RenderPlan(10, 64, 64).det == 0
