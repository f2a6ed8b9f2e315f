"""The binned tile index gives exactly the plain index: offsets and lists, for every way a bin is
put into order (bitmap, buckets, windows, rebuilt from the records) and around the sizes where
the way changes."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from gpu_helpers import require_cuda
from structsplat_b200 import _native
from structsplat_b200.batch import Batch
from structsplat_b200.render import _p, _stream, pack_records, tile_grid

pytestmark = pytest.mark.gpu


def _index(records, n, H, W, ts, cull, which, batch=None):
    """(offsets, list) with the workspace of the `which` query ("" or "binned_")."""
    args = (batch.ref,) if batch else (H, W, ts)
    pre = "ss_batch_" if batch else "ss_"
    if batch:
        T = batch.tiles
        size = _native.size_query(f"ss_batch_tile_index_{which}workspace_bytes", batch.ref, n)
    else:
        tx, ty = tile_grid(H, W, ts)
        T = tx * ty
        size = _native.size_query(f"ss_tile_index_{which}workspace_bytes", n, H, W, ts)
    ws = torch.full((size,), 0xAB, dtype=torch.uint8, device="cuda")
    offsets = torch.empty(T + 1, dtype=torch.int32, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    head = args + (_p(records), n) if batch else (_p(records), n) + args
    _native.call(pre + "tile_index_count", *head, int(cull), 3.0, _p(offsets), _p(ws), size,
                 _p(status), _stream())
    total = int(offsets[-1])
    gids = torch.full((total + 1,), -7, dtype=torch.int32, device="cuda")
    _native.call(pre + "tile_index_fill", *head, int(cull), 3.0, _p(offsets), _p(gids), total,
                 _p(ws), size, _p(status), _stream())
    assert int(gids[-1]) == -7 and int(status) == 0
    return offsets, gids[:-1]


def _same(records, n, H, W, ts, cull=False, batch=None):
    a = _index(records, n, H, W, ts, cull, "", batch)
    b = _index(records, n, H, W, ts, cull, "binned_", batch)
    assert torch.equal(a[0], b[0])
    assert torch.equal(a[1], b[1])
    return a


def _records(means, H, W, r=2, conic=(0.5, 0.0, 0.5)):
    n = means.shape[0]
    m = torch.tensor(means, dtype=torch.float32, device="cuda")
    c = torch.tensor(conic, dtype=torch.float32, device="cuda").expand(n, 3).contiguous()
    radii = torch.as_tensor(r, device="cuda").to(torch.int64).reshape(-1, 1)
    return pack_records(m, c, c, radii.expand(n, 2).contiguous(), None, H, W)


def _uniform(n, H, W, seed=0):
    return np.random.default_rng(seed).uniform([0, 0], [W, H], (n, 2))


# 163,840 Gaussians are the most one bitmap holds
@pytest.mark.parametrize("n,H,W,ts", [
    (1, 5, 7, 16), (33, 64, 64, 32), (4_097, 100, 75, 7), (163_840, 256, 256, 32),
    (163_841, 256, 256, 32), (200_000, 512, 500, 16), (400_000, 130, 70, 32)])
def test_uniform_fields(n, H, W, ts):
    require_cuda()
    rng = np.random.default_rng(n)
    r = torch.tensor(rng.integers(1, 12, n))  # rectangles of 1 to ~100 tiles
    _same(_records(_uniform(n, H, W), H, W, r.reshape(-1, 1)), n, H, W, ts)


# 4,096 ids are the most the buckets take
@pytest.mark.parametrize("per_tile", [4_095, 4_096, 4_097, 9_000])
@pytest.mark.parametrize("ordered", [False, True])
def test_list_lengths_around_the_bucket_sort(per_tile, ordered):
    require_cuda()
    H, W, ts = 64, 256, 32  # 16 tiles, rectangles inside their own tile
    n = 16 * per_tile * 3   # over 163,840 Gaussians, a third of them on the image
    n = max(n, 170_000)
    means = np.full((n, 2), -1e6)
    at = np.sort(np.random.default_rng(1).choice(n, 16 * per_tile, replace=False))
    t = np.repeat(np.arange(16), per_tile)
    if not ordered:
        t = np.random.default_rng(2).permutation(t)
    means[at, 0], means[at, 1] = 32 * (t % 8) + 16, 32 * (t // 8) + 16
    off, _ = _same(_records(means, H, W), n, H, W, ts)
    assert torch.all(off[1:] - off[:-1] == per_tile)


def test_clustered_ids():
    require_cuda()
    n, H, W = 300_000, 512, 512
    m = _uniform(n, H, W)
    m = m[np.lexsort((m[:, 0], (m[:, 1] // 32)))]  # a tile's ids lie together
    _same(_records(m, H, W), n, H, W, 32)


@pytest.mark.parametrize("n,H,W,ts,cull", [(200_000, 1024, 1024, 32, False),
                                           (5_000, 2048, 2040, 8, True),
                                           (5_000, 2048, 2048, 8, False)])
def test_overflowing_bins_are_rebuilt(n, H, W, ts, cull):
    require_cuda()
    m = _uniform(n, ts, ts) + 5 * ts  # everything in one tile or two
    m[: n // 10] = _uniform(n // 10, H, W, 3)
    _same(_records(m, H, W, 3, (3.0, 1.0, 2.0)), n, H, W, ts, cull)


@pytest.mark.parametrize("ts", [8, 16, 32])
def test_ellipse_cull(ts):
    require_cuda()
    n, H, W = 3_000, 301, 417
    m = _uniform(n, H, W)
    _same(_records(m, H, W, 40, (0.9, 0.84, 0.8)), n, H, W, ts, True)


def test_rectangles_of_over_a_million_tiles():
    require_cuda()
    n, H, W, ts = 3, 4224, 4224, 4
    off, gids = _same(_records(_uniform(n, H, W), H, W, 10_000), n, H, W, ts)
    assert off.numel() == 1056 * 1056 + 1 and torch.equal(
        gids.view(-1, 3), torch.arange(3, device="cuda", dtype=torch.int32).expand(1056 ** 2, 3))


# 4,095 tiles are scanned by the count, 65,535 by one launch, more by the device scan
@pytest.mark.parametrize("tiles", [2_047, 2_048, 4_095, 4_096, 65_535, 65_536])
def test_tile_counts_around_the_scans(tiles):
    require_cuda()
    H, W, n = 8, 8 * tiles, 20_000
    _same(_records(_uniform(n, H, W), H, W), n, H, W, 8)


def test_batch_of_images_on_both_sides_of_the_bitmap():
    require_cuda()
    sizes, counts = [(200, 300), (40, 33), (512, 512), (0, 5)], [2_000, 1, 170_000, 0]
    batch = Batch(sizes, counts, tile_size=16)
    g = torch.Generator("cuda").manual_seed(0)
    hw = torch.tensor([[w, h] for h, w in sizes], device="cuda", dtype=torch.float32)
    means = torch.rand(batch.n, 2, device="cuda", generator=g) * torch.repeat_interleave(
        hw, torch.tensor(counts, device="cuda"), 0)
    ls = torch.randn(batch.n, 2, device="cuda", generator=g) * 0.5 + 0.5
    rec = torch.empty(batch.n * 16, device="cuda")
    _native.call("ss_batch_project_rs", batch.ref, _p(means), _p(ls), _p(ls[:, 0].contiguous()),
                 _p(torch.zeros(batch.n, 3, device="cuda")), None, batch.n, 0.0, 3.0, _p(rec),
                 _stream())
    _same(rec, batch.n, 0, 0, 16, batch=batch)


def test_bins_of_another_count_are_not_trusted():
    require_cuda()
    n, H, W, ts = 3_000, 200, 200, 16
    rec = _records(_uniform(n, H, W), H, W)
    want = _index(rec, n, H, W, ts, False, "")
    T = want[0].numel() - 1
    small = _native.size_query("ss_tile_index_workspace_bytes", n, H, W, ts)
    size = _native.size_query("ss_tile_index_binned_workspace_bytes", n, H, W, ts)
    assert size > small
    ws = torch.full((size,), 0x11, dtype=torch.uint8, device="cuda")
    offsets = torch.empty(T + 1, dtype=torch.int32, device="cuda")
    gids = torch.empty_like(want[1])
    _native.call("ss_tile_index_count", _p(rec), n, H, W, ts, 0, 3.0, _p(offsets), _p(ws), small,
                 None, _stream())
    _native.call("ss_tile_index_fill", _p(rec), n, H, W, ts, 0, 3.0, _p(offsets), _p(gids),
                 gids.numel(), _p(ws), size, None, _stream())
    assert torch.equal(offsets, want[0]) and torch.equal(gids, want[1])
