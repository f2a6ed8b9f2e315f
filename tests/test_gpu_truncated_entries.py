"""Deterministic gradients of an index that outgrew its capacity read nothing of the tile that does not
fit: its ids are not in the list and its partials not in the workspace."""
from __future__ import annotations

import pytest
import torch

from gpu_helpers import require_cuda
from structsplat_b200.fit import RenderPlan
from structsplat_b200.synthetic import make_field

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fused", [False, True])
@pytest.mark.parametrize("capacity", [20, 64, 300, 790])
def test_sorted_entries(capacity, fused):
    require_cuda()
    H = W = 128
    f = make_field(H, W, 500, 3)
    p = {k: torch.tensor(getattr(f, k), device="cuda")
         for k in ("means", "log_scales", "rotations", "colors", "opacity_logits")}
    go = torch.ones(H, W, 3, device="cuda")
    got = []
    for stale in (3, 400):
        plan = RenderPlan(500, H, W, capacity=capacity, deterministic=True, fused=fused)
        plan.det = 1
        plan.gids.fill_(stale)  # ids and partials of an earlier step
        plan.bwd_ws.view(torch.float32).fill_(float("nan"))
        got.append({k: v.clone() for k, v in plan.forward_backward(p, go).items()})
        assert plan.overflowed()
    for k in got[0]:
        assert bool(torch.isfinite(got[0][k]).all()) and torch.equal(got[0][k], got[1][k]), k
    assert capacity < 64 or any(bool((g != 0).any()) for g in got[0].values())
