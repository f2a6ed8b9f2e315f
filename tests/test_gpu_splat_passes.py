"""The per-Gaussian activity around its size classes, from render inputs and from records, and
packing fused with the tile count."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from gpu_helpers import require_cuda
from structsplat_b200 import _native
from structsplat_b200 import render as R
from structsplat_b200.render import _p, _stream

pytestmark = pytest.mark.gpu


def _inputs(n, H, W, seed=0):
    """Rectangles of every size around 32x32 (the largest walked by eight lanes), slivers, ones cut by
    the border, empty ones and some that cover the image."""
    rng = np.random.default_rng(seed)
    means = rng.uniform([-20, -20], [W + 20, H + 20], (n, 2))
    radii = rng.integers(1, 24, (n, 2))
    radii[: n // 4] = rng.integers(14, 18, (n // 4, 2))
    radii[n // 4: n // 4 + 5] = [[400, 0], [0, 400], [500, 500], [15, 16], [16, 15]]
    means[-1] = [np.nan, 1.0]
    s = rng.uniform(0.5, 20.0, (n, 2))
    conics = np.stack([1 / s[:, 0] ** 2, 0.3 / (s[:, 0] * s[:, 1]), 1 / s[:, 1] ** 2], 1)
    f32 = dict(dtype=torch.float32, device="cuda")
    return (torch.tensor(means, **f32), torch.tensor(conics, **f32),
            torch.tensor(radii, device="cuda"))


# float32 sums of up to 160,000 weights in [0, 1], each within 2^-22 plus the rounding of its
# exponent (below 1e-5 of a weight that matters): 2e-5 of the largest term per lane bounds them
@pytest.mark.parametrize("fade", [0.0, 1.0])
@pytest.mark.parametrize("n", [25, 31, 32, 33, 257, 3_000])
def test_activity(n, fade):
    require_cuda()
    H, W = 400, 370
    means, conics, radii = _inputs(n, H, W, n)
    got = R.gaussian_activity(means, conics, radii, H, W, support_fade=fade > 0)
    tail = R.fade_tail(3.0, fade)
    m, c, r = means.double().cpu().numpy(), conics.double().cpu().numpy(), radii.cpu().numpy()
    want = np.zeros(n)
    for i in range(n):
        if not np.isfinite(m[i]).all():
            continue
        cx, cy = np.rint(m[i].astype(np.float32)).astype(int)
        x = np.arange(max(cx - r[i, 0], 0), min(cx + r[i, 0], W - 1) + 1)
        y = np.arange(max(cy - r[i, 1], 0), min(cy + r[i, 1], H - 1) + 1)
        dx, dy = np.meshgrid(x - m[i, 0], y - m[i, 1])
        q = c[i, 0] * dx * dx + 2 * c[i, 1] * dx * dy + c[i, 2] * dy * dy
        want[i] = np.maximum(np.exp(-0.5 * q) - tail, 0).sum()
    assert np.abs(got.cpu().numpy() - want).max() <= 2e-5 * max(want.max(), 1.0)
    rec = R.pack_records(means, conics, conics, radii, None, H, W)
    for lanes in (8, 32):
        other = torch.empty(n, device="cuda")
        _native.call("ss_gaussian_activity", _p(rec), n, float(tail), lanes, _p(other), _stream())
        assert torch.equal(other, got)


@pytest.mark.parametrize("n,ts,cull,opac", [(1, 32, False, True), (256, 16, True, False),
                                            (257, 8, False, True), (5_000, 32, True, True)])
def test_pack_with_count_is_pack_then_count(n, ts, cull, opac):
    require_cuda()
    H, W = 200, 333
    means, conics, radii = _inputs(max(n, 30), H, W, 3)
    means, conics, radii = means[:n].contiguous(), conics[:n].contiguous(), radii[:n].contiguous()
    colors = torch.rand(n, 3, device="cuda")
    op = torch.rand(n, device="cuda") if opac else None
    want = R.pack_records(means, conics, colors, radii, op, H, W)
    index = R.index_from_records(want, n, H, W, ts, cull, exact=True)
    rec, got = R.pack_and_index(means, conics, colors, radii, op, H, W, ts, cull, 3.0, exact=True)
    assert torch.equal(rec.view(torch.int32), want.view(torch.int32))
    assert torch.equal(got.offsets, index.offsets) and torch.equal(got.gids, index.gids)
    assert int(got.status) == 0
