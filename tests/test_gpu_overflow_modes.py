"""Deterministic fits and renders whose tile lists outgrew their capacity: every mode sums the tiles that
fit, as the sort of the entries does."""
from __future__ import annotations

import pytest
import torch

from gpu_helpers import require_cuda
from structsplat_b200.batch import Batch, FitPlan, FitSettings, PARAM_NAMES
from structsplat_b200.fit import RenderPlan
from structsplat_b200.synthetic import make_field

pytestmark = pytest.mark.gpu


def _params(f):
    return {k: torch.tensor(getattr(f, k), device="cuda") for k in PARAM_NAMES}


# 2,000-odd entries; the first image's tiles end within its rows, at a row's end, in the second image
@pytest.mark.parametrize("fused", [False, True])
@pytest.mark.parametrize("fade,mode", [(0.0, 2), (1.0, 3)])
@pytest.mark.parametrize("tile_size", [16, 32])
@pytest.mark.parametrize("share", [0.0005, 0.1, 0.3, 0.55, 0.7, 0.97])
def test_fit_steps(share, tile_size, fade, mode, fused):
    require_cuda()
    sizes, counts = [(100, 130), (64, 64), (37, 301)], [900, 200, 700]
    out = []
    for det in (1, mode):
        fields = [_params(make_field(h, w, c, seed=7 + c)) for (h, w), c in zip(sizes, counts)]
        params = Batch.concat_fields(fields)
        params["log_scales"][::50] += 2.0  # rectangles of many rows
        batch = Batch(sizes, counts, tile_size=tile_size)
        target = torch.rand(batch.pixels, 3, device="cuda",
                            generator=torch.Generator("cuda").manual_seed(1))
        s = FitSettings(deterministic=True, fused=fused, fade_alpha=fade)
        whole = FitPlan(batch, params, target, s).entries
        plan = FitPlan(batch, params, target, s, capacity=max(int(share * whole), 1))
        assert plan.det == mode
        plan.det = det
        plan.step()
        assert plan.overflowed() and int(plan.status) & 4
        out.append({**params, **{f"g_{k}": v.clone() for k, v in plan.gradients().items()}})
    if share >= 0.3:
        assert any(bool((out[0][f"g_{k}"] != 0).any()) for k in PARAM_NAMES)
    for k in out[0]:
        assert torch.equal(out[0][k], out[1][k]), k


@pytest.mark.parametrize("fused", [False, True])
def test_runs_of_a_render(fused):
    require_cuda()
    H = W = 128
    p = _params(make_field(H, W, 500, 3))
    go = torch.ones(H, W, 3, device="cuda")
    got = []
    for det in (1, 3):
        plan = RenderPlan(500, H, W, capacity=300, deterministic=True, fade_alpha=1.0, fused=fused)
        plan.det = det
        got.append({k: v.clone() for k, v in plan.forward_backward(p, go).items()})
        assert plan.overflowed() and int(plan.status) & 4
    assert any(bool((g != 0).any()) for g in got[0].values())
    for k in got[0]:
        assert torch.equal(got[0][k], got[1][k]), k
