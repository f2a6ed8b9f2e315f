"""The tuner times a fit's backward in the mode that the fit's steps run."""
from __future__ import annotations

import pytest
import torch

from gpu_helpers import require_cuda
from structsplat_b200 import autotune
from structsplat_b200.batch import FitPlan, FitSettings, PARAM_NAMES
from structsplat_b200.synthetic import make_field

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fused", [False, True])
@pytest.mark.parametrize("deterministic,fade,mode", [(False, 0.0, 0), (True, 0.0, 2), (True, 1.0, 3)])
def test_timed_mode(monkeypatch, deterministic, fade, mode, fused):
    require_cuda()
    f = make_field(96, 80, 500, seed=3)
    params = {k: torch.tensor(getattr(f, k), device="cuda") for k in PARAM_NAMES}
    target = torch.rand(96 * 80, 3, device="cuda")
    seen = []
    for name in ("backward", "forward_backward"):
        real = getattr(FitPlan, name)
        monkeypatch.setattr(FitPlan, name, lambda self, det=None, real=real: (
            seen.append(self._det(det)), real(self, det)))
    shapes = autotune.asked_shapes()
    try:
        autotune.tune_fit([(96, 80)], [500], params, target,
                          FitSettings(deterministic=deterministic, fade_alpha=fade, fused=fused),
                          repeats=1, use_cache=False)
    finally:
        autotune.ask_shapes(shapes)
    assert seen and set(seen) == {mode}
