"""The sampler's uniforms off the GPU are numpy's, for every way of naming the place that Tensor.to()
takes."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from structsplat_b200.placement import draw_uniforms


@pytest.mark.parametrize("device", ["cpu", torch.device("cpu"), None, torch.zeros(1, dtype=torch.float64)])
def test_host_uniforms(device):
    rng, ref = np.random.default_rng(5), np.random.default_rng(5)
    got = draw_uniforms(7, device, rng=rng)
    want = np.concatenate([ref.random(7), ref.random((7, 2)).ravel()])
    assert got.device.type == "cpu" and np.array_equal(got.numpy(), want)
    assert rng.bit_generator.state == ref.bit_generator.state


def test_a_bad_device_is_refused_as_tensor_to_does():
    with pytest.raises(RuntimeError):
        draw_uniforms(7, "nowhere", rng=np.random.default_rng(5))
