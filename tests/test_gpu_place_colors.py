"""Bilinear colours of placed Gaussians at every pixel of small images (the wide loads' last pixels),
with the image on and off a 16-byte boundary, against NumPy float64."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from gpu_helpers import require_cuda
from structsplat_b200 import _native
from structsplat_b200.render import _p, _stream

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,W", [(2, 2), (2, 3), (3, 5), (7, 4), (16, 17)])
@pytest.mark.parametrize("shift", [0, 1])
def test_colours(H, W, shift):
    require_cuda()
    rng = np.random.default_rng(H * W + shift)
    img = rng.random((H, W, 3)).astype(np.float32)
    ys, xs = np.mgrid[0:H, 0:W]
    pts = np.stack([xs.ravel() + rng.uniform(-0.5, 0.5, H * W),
                    ys.ravel() + rng.uniform(-0.5, 0.5, H * W)], 1)
    n = H * W
    buf = torch.empty(H * W * 3 + shift, device="cuda")
    image = buf[shift:].view(H, W, 3)
    image.copy_(torch.tensor(img))
    f64 = dict(device="cuda", dtype=torch.float64)
    z = torch.zeros(H, W, device="cuda")
    out = [torch.empty(n, k, device="cuda") for k in (2, 2, 1, 3)]
    p = torch.tensor(pts, **f64)
    d = torch.full((H, W), 1.0 / n, **f64)
    _native.call("ss_place_gaussians", _p(p), n, _p(d), _p(z), _p(z), _p(image), H, W, 0, 6.0, 1.0,
                 1.0, n, *(_p(t) for t in out), _stream())
    x, y = np.clip(pts[:, 0], 0, W - 1.001), np.clip(pts[:, 1], 0, H - 1.001)
    x0, y0 = np.floor(x).astype(int), np.floor(y).astype(int)
    fx, fy = (x - x0)[:, None], (y - y0)[:, None]
    i = img.astype(np.float64)
    want = i[y0, x0] * (1 - fx) * (1 - fy)
    want = want + i[y0, x0 + 1] * fx * (1 - fy)
    want = want + i[y0 + 1, x0] * (1 - fx) * fy
    want = want + i[y0 + 1, x0 + 1] * fx * fy
    assert np.array_equal(out[3].cpu().numpy(), want.astype(np.float32))
