"""The workspace size for a known entry total: the binned form's, or the plain form's where lists would
outgrow their bins and nothing cheaper finds them."""
from __future__ import annotations

import ctypes

import pytest

from structsplat_b200 import _native


def _sizes(n, H, W, ts):
    return (_native.size_query("ss_tile_index_workspace_bytes", n, H, W, ts),
            _native.size_query("ss_tile_index_binned_workspace_bytes", n, H, W, ts))


def _size(n, H, W, ts, entries, images=1):
    T = -(-H // ts) * -(-W // ts)
    return _native.size_query("ss_tile_index_entries_workspace_bytes", n, T, images, entries)


# bins of 96 ids: lists of 70 on average stay within three deviations, of 71 do not; from 1,024 on the
# bins are the better form again
@pytest.mark.parametrize("mean,plain", [(0, False), (20, False), (70, False), (71, True), (180, True),
                                        (1_023, True), (1_024, False)])
def test_short_lists_beyond_their_bins(mean, plain):
    n, H, W, ts = 100_000, 1024, 1024, 4
    sizes = _sizes(n, H, W, ts)
    assert _size(n, H, W, ts, mean * 65_536) == sizes[0 if plain else 1]


def test_few_tests_stay_binned():
    n, H, W, ts = 8_192, 512, 512, 16  # 8.4 M records to test if every list outgrew its bin of 288
    assert _size(n, H, W, ts, 300 * 1024) == _sizes(n, H, W, ts)[1]


def test_lists_of_a_good_part_of_the_image_stay_binned():
    n, H, W, ts = 5_000, 1024, 1024, 16  # bins of 96
    plain, binned = _sizes(n, H, W, ts)
    assert _size(n, H, W, ts, 624 * 4096) == plain
    assert _size(n, H, W, ts, 625 * 4096) == binned
    # of ten images, each with a tenth of the Gaussians
    assert _size(n, H, W, ts, 62 * 4096, images=10) == binned
    assert _size(n, H, W, ts, 75 * 4096, images=1) == plain


def test_empty_sets_and_bad_sizes():
    assert _size(0, 64, 64, 16, 5) == _sizes(0, 64, 64, 16)[0]
    assert _size(10, 0, 64, 16, 5) == _sizes(10, 0, 64, 16)[0]
    out = ctypes.c_size_t()
    for args in ((-1, 4, 1, 0), (1, -4, 1, 0), (1, 4, -1, 0), (1, 4, 1, -1)):
        assert _native.lib().ss_tile_index_entries_workspace_bytes(*args, ctypes.byref(out)) != 0
