"""The device draw of a numpy PCG64 generator is numpy's own: bitwise the same doubles, and the
generator left in the same state."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from gpu_helpers import require_cuda
from structsplat_b200 import placement as PL

pytestmark = pytest.mark.gpu


# 131,072 is the kernel's thread count: one value per thread, one more, several per thread
@pytest.mark.parametrize("n", [1, 7, 43_690, 43_691, 131_072, 131_073, 500_001])
def test_draw_is_numpys(n):
    require_cuda()
    ours, theirs = np.random.default_rng(n), np.random.default_rng(n)
    for r in (ours, theirs):
        r.integers(0, 2 ** 31, dtype=np.uint32)  # leaves half a word buffered in the generator
    got = PL.draw_uniforms(n, "cuda", rng=ours).cpu().numpy()
    assert np.array_equal(got, np.concatenate([theirs.random(n), theirs.random((n, 2)).ravel()]))
    assert ours.bit_generator.state == theirs.bit_generator.state
    assert ours.random() == theirs.random()


@pytest.mark.parametrize("bits", [np.random.MT19937, np.random.PCG64DXSM, np.random.Philox])
def test_other_generators_draw_on_the_host(bits):
    require_cuda()
    got = PL.draw_uniforms(100, "cuda", rng=np.random.Generator(bits(3))).cpu().numpy()
    r = np.random.Generator(bits(3))
    assert np.array_equal(got, np.concatenate([r.random(100), r.random((100, 2)).ravel()]))


def test_no_points():
    require_cuda()
    r = np.random.default_rng(1)
    assert PL.draw_uniforms(0, "cuda", rng=r).numel() == 0
    assert torch.equal(PL.draw_uniforms(5, "cpu", rng=r),
                       torch.tensor(np.random.default_rng(1).random(15)))
