"""The fit update against torch.optim.Adam on the gradients it reports: the one pass of up to 65,536
Gaussians around its CTA of 256, with parameter tensors off a 16-byte boundary, and the two passes
beyond."""
from __future__ import annotations

import math

import pytest
import torch

from gpu_helpers import require_cuda
from structsplat_b200.batch import PARAM_NAMES, Batch, FitPlan, FitSettings
from structsplat_b200.synthetic import make_field

pytestmark = pytest.mark.gpu


def _off(t, floats):
    """A contiguous copy of t that starts `floats` floats into its buffer."""
    buf = torch.empty(t.numel() + floats, device=t.device)
    v = buf[floats:].view(t.shape)
    v.copy_(t)
    return v


# the update repeats torch's order of operations; its square root, division and fused products differ
# from torch's kernels by a few ulp of a step of at most ~lr: 1e-6 of the value plus 1e-5 lr a step
@pytest.mark.parametrize("n,shift,opacity,deterministic", [
    (1, 0, True, False), (255, 0, True, True), (256, 0, False, False), (257, 0, True, False),
    (512, 1, True, False), (777, 2, False, True), (1_024, 0, True, True), (65_536, 0, True, False),
    (65_537, 0, True, True), (65_537, 3, True, False)])
def test_update_is_adam(n, shift, opacity, deterministic):
    require_cuda()
    H, W, steps = 96, 80, 3
    f = make_field(H, W, n, seed=n)
    params = {k: _off(torch.tensor(getattr(f, k), device="cuda"), shift) for k in PARAM_NAMES}
    if not opacity:
        params["opacity_logits"] = None
    params["log_scales"][0] = 9.0  # clamped
    s = FitSettings(deterministic=deterministic)
    target = torch.rand(H * W, 3, device="cuda", generator=torch.Generator("cuda").manual_seed(0))
    plan = FitPlan(Batch([(H, W)], [n]), params, target, s)
    names = [k for k in PARAM_NAMES if params[k] is not None]
    ref = {k: params[k].clone().requires_grad_(True) for k in names}
    lrs = dict(zip(PARAM_NAMES, s.lrs()))
    opt = torch.optim.Adam([{"params": [ref[k]], "lr": lrs[k]} for k in names], betas=s.betas,
                           eps=s.adam_eps)
    for step in range(1, steps + 1):
        plan.step()
        grads = plan.gradients()
        for k in names:
            ref[k].grad = grads[k].clone()
        opt.step()
        with torch.no_grad():
            ref["log_scales"].clamp_(max=math.log(max(H, W))).clamp_(min=math.log(s.scale_min))
        for k in names:
            want = ref[k].detach()
            assert torch.all((params[k] - want).abs() <= 1e-6 * want.abs() + 1e-5 * lrs[k] * step), k
    assert plan.step_state.tolist() == [steps, 0]
    if not deterministic:
        moments = plan.bwd_ws[:9 * n]
        assert bool((moments == 0).all())
