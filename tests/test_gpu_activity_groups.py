"""The per-Gaussian activity of few and of wide Gaussians: each within a bound of its own, the same
whatever the number of Gaussians beside it, and not as slow as many of them."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from gpu_helpers import require_cuda
from structsplat_b200 import render as R

pytestmark = pytest.mark.gpu
H, W = 640, 600


def _inputs(n, seed=0):
    """Rectangles around 32x32 and 90x91 pixels (the largest of eight lanes and of a warp), slivers, and
    ones that cover the image."""
    rng = np.random.default_rng(seed)
    sides = np.array([[1, 1], [15, 16], [16, 15], [45, 44], [45, 45], [3, 200], [250, 2], [700, 700]])
    radii = sides[rng.integers(0, len(sides), n)]
    means = rng.uniform([-5, -5], [W + 5, H + 5], (n, 2))
    s = np.maximum(radii / 3.0, 0.4) * rng.uniform(0.7, 1.4, (n, 2))
    conics = np.stack([1 / s[:, 0] ** 2, 0.3 / (s[:, 0] * s[:, 1]), 1 / s[:, 1] ** 2], 1)
    f32 = dict(dtype=torch.float32, device="cuda")
    return (torch.tensor(means, **f32), torch.tensor(conics, **f32), torch.tensor(radii, device="cuda"))


# A weight is off by its exponent's rounding (5 ulp of t, t exp(-t) <= 0.37: 1.1e-7) and 2^-22 of
# itself; a lane adds at most 640 rows, then 19 columns and 8 partial sums: 2^-24 each of the sum.
# A lost row or column at three sigma is 1e-4 of the sum or more.
@pytest.mark.parametrize("fade", [0.0, 1.0])
@pytest.mark.parametrize("n", [1, 7, 9, 300, 1_183, 1_185, 2_400])
def test_every_gaussian_within_its_own_bound(n, fade):
    require_cuda()
    means, conics, radii = _inputs(n, n)
    got = R.gaussian_activity(means, conics, radii, H, W, support_fade=fade > 0).double()
    tail = R.fade_tail(3.0, fade)
    c = torch.round(means).long()  # half to even, as the support rectangle's centre
    m, k = means.double(), conics.double()
    want, pixels = torch.zeros(n, dtype=torch.float64), torch.zeros(n, dtype=torch.float64)
    box = [torch.stack([(c - radii)[:, d].clamp_min(0),
                        (c + radii)[:, d].clamp_max(s - 1)], 1).tolist()
           for d, s in ((0, W), (1, H))]
    for i in range(n):
        (x0, x1), (y0, y1) = box[0][i], box[1][i]
        if x1 < x0 or y1 < y0:
            continue
        dx = torch.arange(x0, x1 + 1, device="cuda") - m[i, 0]
        dy = (torch.arange(y0, y1 + 1, device="cuda") - m[i, 1])[:, None]
        q = k[i, 0] * dx * dx + 2 * k[i, 1] * dx * dy + k[i, 2] * dy * dy
        want[i] = (torch.exp(-0.5 * q) - tail).clamp_min(0).sum().cpu()
        pixels[i] = q.numel()
    bound = want * (2.0 ** -22 + 667 * 2.0 ** -24) + 1.1e-7 * pixels
    assert bool(((got.cpu() - want).abs() <= bound).all())


def test_the_same_beside_any_number():
    require_cuda()
    n = 310_000  # 256 to a CTA
    means, conics, radii = _inputs(n)
    radii.clamp_(max=60)
    full = R.gaussian_activity(means, conics, radii, H, W)
    for size in (1, 8, 1_200, 3_000, 5_000, 40_000):
        part = R.gaussian_activity(means[:size].contiguous(), conics[:size].contiguous(),
                                   radii[:size].contiguous(), H, W)
        assert torch.equal(part, full[:size]), size


# 32 to a warp and each in turn, 500 took as long as 20,000
def test_few_wide_gaussians_do_not_cost_what_many_do():
    require_cuda()
    times = []
    for n in (500, 20_000):
        g = torch.Generator("cuda").manual_seed(0)
        means = torch.rand(n, 2, device="cuda", generator=g) * 600
        conics = torch.tensor([4e-4, 0.0, 4e-4], device="cuda").expand(n, 3).contiguous()
        radii = torch.full((n, 2), 150, device="cuda", dtype=torch.int64)
        best = float("inf")
        for _ in range(5):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            R.gaussian_activity(means, conics, radii, H, W)
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b))
        times.append(best)
    assert 4 * times[0] < times[1], times
