"""Projection of Gaussians whose centre and radius are far beyond the image: the record's rectangle is
that of the radii it reports."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from gpu_helpers import require_cuda
from structsplat_b200.field import project
from structsplat_b200.render import pack_records

pytestmark = pytest.mark.gpu


# radius cutoff * exp(ls) of 0.5 to 1.05e12 px (records cap it at 2^40 = 1.0995e12), centre a little
# farther off than it (empty rectangles) or a little nearer
@pytest.mark.parametrize("radius", [1e3, 5e8, 6e8, 9.9e11, 1.02e12, 1.05e12])
def test_rectangles_agree_with_the_radii(radius):
    require_cuda()
    H, W, n = 40, 50, 8
    ls = torch.full((n, 2), float(np.log(radius / 3.0)), device="cuda")
    means = torch.tensor([[f * radius, 20.0] for f in (1.03, 0.97, -1.03, -0.97)]
                         + [[20.0, f * radius] for f in (1.03, 0.97, -1.03, -0.97)], device="cuda")
    rot = torch.zeros(n, device="cuda")
    col = torch.zeros(n, 3, device="cuda")
    rec, conics, radii = project(means, ls, rot, col, None, H, W, want_conics=True)
    want = pack_records(means, conics, col, radii, None, H, W)
    got = rec[: n * 16].view(n, 16)[:, 12:].view(torch.int32)
    assert torch.equal(got, want[: n * 16].view(n, 16)[:, 12:].view(torch.int32))
    empty = (got[:, 2] <= got[:, 0]) | (got[:, 3] <= got[:, 1])
    lo, hi = torch.round(means).long() - radii, torch.round(means).long() + radii
    side = torch.tensor([W, H], device="cuda")
    assert torch.equal(empty, ((hi < 0) | (lo >= side)).any(1)) and bool(empty.any())
