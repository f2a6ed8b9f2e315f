"""The sampler's guided search finds the pixel the search of the whole cdf finds: a call with many
points (guide) against calls of 100 points each (no guide) on the same uniforms, index by index."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from gpu_helpers import require_cuda
from structsplat_b200 import placement as PL

pytestmark = pytest.mark.gpu


def _densities(H, W):
    rng = np.random.default_rng(H * W)
    spread = rng.random((H, W))
    skewed = spread ** 40
    holes = spread * (rng.random((H, W)) < 0.02)
    one = np.zeros((H, W))
    one[H // 2, W // 3] = 1.0
    bad = spread.copy()
    bad[-1, 0] = np.nan
    return {"spread": spread, "skewed": skewed, "holes": holes, "one": one, "empty": one * 0,
            "nan": bad}


# 2,048 pixels are the fewest with a guide (256 buckets); one fewer has none
@pytest.mark.parametrize("H,W", [(1, 2047), (32, 64), (61, 67), (389, 517)])
@pytest.mark.parametrize("kind", ["spread", "skewed", "holes", "one", "empty", "nan"])
def test_guided_search_is_the_full_search(H, W, kind):
    require_cuda()
    n = 20_000
    d = torch.tensor(_densities(H, W)[kind], device="cuda")
    u = np.random.default_rng(5).random(3 * n)
    u[:256] = np.arange(256) / 256.0  # bucket boundaries, exactly
    u[256:512] = np.nextafter(np.arange(256) / 256.0, 1.0)
    u[512:768] = np.nextafter(np.arange(1, 257) / 256.0, 0.0)
    u[768:772] = [1.0, -0.5, 2.0, np.nan]  # a caller's own uniforms
    u = torch.tensor(u, device="cuda")
    pts, idx = PL.sample_candidates(d, n, uniforms=u, return_index=True)
    for a in range(0, n, n // 10):
        sel = torch.arange(a, min(a + 100, n), device="cuda")
        part = torch.cat([u[sel], u[n:].view(n, 2)[sel].reshape(-1)])
        p, i = PL.sample_candidates(d, sel.numel(), uniforms=part, return_index=True)
        assert torch.equal(i, idx[sel])
        assert torch.equal(p.view(torch.int64), pts[sel].view(torch.int64))
