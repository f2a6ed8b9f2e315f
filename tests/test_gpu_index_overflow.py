"""Tile lists that outgrow their bins: the index is exactly the plain one, whichever way such a list is
made, and costs no multiple of it."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from gpu_helpers import require_cuda
from structsplat_b200 import _native
from structsplat_b200 import render as R
from structsplat_b200.batch import Batch
from structsplat_b200.fit import RenderPlan
from structsplat_b200.render import _p, _stream, tile_grid
from test_gpu_binned_index import _index, _records, _same, _uniform

pytestmark = pytest.mark.gpu


# bins of 96 and 832 ids; 100k on 4-px tiles: lists from 20 to 240
@pytest.mark.parametrize("n,H,W,ts,r,cull", [
    (100_000, 1024, 1024, 4, 20, False), (100_000, 1024, 1020, 16, 48, False),
    (30_000, 701, 1003, 7, 40, True), (17_000, 1100, 1100, 4, 30, False)])
def test_wide_gaussians(n, H, W, ts, r, cull):
    require_cuda()
    conic = (0.02, 0.018, 0.02) if cull else (0.5, 0.0, 0.5)
    _same(_records(_uniform(n, H, W), H, W, r, conic), n, H, W, ts, cull)


# bins of 3,168, 832, 2,400 and 31,296 ids, lists of up to 10k, 5k and 45k in one part of the image; ids of
# one, two and seven windows
@pytest.mark.parametrize("n,ts,sigma", [(100_000, 32, 40), (100_000, 16, 40), (300_000, 16, 55),
                                        (1_000_000, 32, 60)])
def test_clumps(n, ts, sigma):
    require_cuda()
    m = np.random.default_rng(0).normal(512, sigma, (n, 2))
    _same(_records(m, 1024, 1024, 6), n, 1024, 1024, ts)


# More than 163,840 Gaussians; one tile gets `run` ids in a row, too many for a bucket, in a list that the
# buckets hold (3,000, 4,096) and one that they do not
@pytest.mark.parametrize("n,side,run", [(200_000, 1024, 3_000), (200_000, 1024, 4_096),
                                        (400_000, 2048, 5_000)])
def test_consecutive_ids_in_one_tile(n, side, run):
    require_cuda()
    m = _uniform(n, side, side)
    m[n // 2: n // 2 + run] = 24.0
    off, _ = _same(_records(m, side, side, 2), n, side, side, 16)
    longest = int((off[1:] - off[:-1]).max())
    assert run <= longest < run + 200


def test_rectangles_of_over_a_million_tiles():
    require_cuda()
    n, H, W, ts = 2_000, 4096, 4100, 4  # bins of 64 ids
    m = np.full((n, 2), -1e6)
    m[::20] = 2048.0
    off, _ = _same(_records(m, H, W, 5_000), n, H, W, ts)
    assert bool(torch.all(off[1:] - off[:-1] == 100))


def test_batch():
    require_cuda()
    sizes, counts = [(512, 512), (33, 40), (1024, 1000)], [20_000, 0, 60_000]
    batch = Batch(sizes, counts, tile_size=4)
    g = torch.Generator("cuda").manual_seed(0)
    hw = torch.tensor([[w, h] for h, w in sizes], device="cuda", dtype=torch.float32)
    means = torch.rand(batch.n, 2, device="cuda", generator=g) * 0.4 * torch.repeat_interleave(
        hw, torch.tensor(counts, device="cuda"), 0)
    ls = torch.randn(batch.n, 2, device="cuda", generator=g) * 0.3 + 1.3
    rec = torch.empty(batch.n * 16, device="cuda")
    _native.call("ss_batch_project_rs", batch.ref, _p(means), _p(ls), _p(ls[:, 0].contiguous()),
                 _p(torch.zeros(batch.n, 3, device="cuda")), None, batch.n, 0.0, 3.0, _p(rec),
                 _stream())
    off, _ = _same(rec, batch.n, 0, 0, 4, batch=batch)
    assert int((off[1:] - off[:-1]).max()) > 64  # ids per bin


def _raw(rec, n, H, W, ts, count_size=None, spoil=None, fills=1):
    """(offsets, list, status) of the binned form: counted with another workspace size, with counter
    words spoilt before the fill, or filled more than once."""
    tx, ty = tile_grid(H, W, ts)
    size = _native.size_query("ss_tile_index_binned_workspace_bytes", n, H, W, ts)
    ws = torch.full((size,), 0x11, dtype=torch.uint8, device="cuda")
    offsets = torch.empty(tx * ty + 1, dtype=torch.int32, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    _native.call("ss_tile_index_count", _p(rec), n, H, W, ts, 0, 3.0, _p(offsets), _p(ws),
                 count_size or size, _p(status), _stream())
    total = int(offsets[-1])
    for word, value in (spoil or {}).items():
        ws[4 * word: 4 * word + 4].view(torch.int32).fill_(value)
    for _ in range(fills):
        gids = torch.zeros(total, dtype=torch.int32, device="cuda")
        _native.call("ss_tile_index_fill", _p(rec), n, H, W, ts, 0, 3.0, _p(offsets), _p(gids), total,
                     _p(ws), size, _p(status), _stream())
    return offsets, gids, int(status)


def test_counts_without_bins_and_repeated_fills():
    require_cuda()
    n, H, W, ts = 20_000, 1024, 1024, 16
    rec = _records(_uniform(n, H, W), H, W, 24)
    want = _index(rec, n, H, W, ts, False, "")
    small = _native.size_query("ss_tile_index_workspace_bytes", n, H, W, ts)
    for kw in ({}, {"fills": 2}, {"count_size": small}, {"count_size": small, "fills": 2}):
        offsets, gids, status = _raw(rec, n, H, W, ts, **kw)
        assert torch.equal(offsets, want[0]) and torch.equal(gids, want[1]) and status == 0, kw


def test_a_wait_that_runs_out_is_reported_and_harmless():
    """With the ticket word moved on, no CTA places anything and the others' wait (about a second)
    runs out: they list their tiles from the records and the overflow is reported."""
    require_cuda()
    n, H, W, ts = 10_000, 1024, 1024, 16  # 1,024 CTAs' tiles, 312 CTAs for the pairs
    m = _uniform(n, H, W)
    m[5_000:6_000] = 24.0
    rec = _records(m, H, W, 2)
    want = _index(rec, n, H, W, ts, False, "")
    offsets, gids, status = _raw(rec, n, H, W, ts, spoil={5: 313})
    assert status & 1
    assert torch.equal(offsets, want[0]) and torch.equal(gids, want[1])


def _ms(fn):
    best = float("inf")
    for _ in range(5):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        fn()
        b.record()
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b))
    return best


# one CTA per tile used to test every record: 70 times the plain form
def test_overflow_costs_no_multiple_of_the_plain_form():
    require_cuda()
    n, H, W, ts = 100_000, 1024, 1024, 4
    rec = _records(_uniform(n, H, W), H, W, 20)
    times = {}
    for which in ("", "binned_"):
        _index(rec, n, H, W, ts, False, which)
        times[which] = _ms(lambda: _index(rec, n, H, W, ts, False, which))
    assert times["binned_"] < 8 * times[""], times


def test_plans_take_the_plain_form_for_wide_fields():
    require_cuda()
    n, H, W, ts = 5_000, 1024, 1024, 16  # bins of 96 ids, lists of ~120
    g = torch.Generator("cuda").manual_seed(0)
    p = {"means": torch.rand(n, 2, device="cuda", generator=g) * 1024,
         "log_scales": torch.full((n, 2), 3.18, device="cuda"),
         "rotations": torch.rand(n, device="cuda", generator=g),
         "colors": torch.rand(n, 3, device="cuda", generator=g), "opacity_logits": None}
    plan = RenderPlan.for_field(p, H, W, tile_size=ts)
    plain = _native.size_query("ss_tile_index_workspace_bytes", n, H, W, ts)
    assert plan.idx_ws_bytes == plain
    narrow = dict(p, log_scales=torch.zeros(n, 2, device="cuda"))
    assert RenderPlan.for_field(narrow, H, W, tile_size=ts).idx_ws_bytes > plain
    image = plan.forward(p).clone()

    from structsplat_b200.field import project
    rec, conics, radii = project(p["means"], p["log_scales"], p["rotations"], p["colors"], None, H, W,
                                  want_conics=True)
    want = R.index_from_records(rec, n, H, W, ts, exact=True)
    for _ in range(2):  # the second call knows its entries
        got = R.build_tile_index(p["means"], conics, radii, H, W, ts)
        assert torch.equal(got[0], want.gids) and torch.equal(got[1], want.offsets)
        out, _ = R.render_cuda_exact_with_coverage(p["means"], conics, p["colors"], radii, H, W,
                                                   tile_size=ts)
        assert torch.equal(out, image)


def test_a_plan_keeps_the_workspace_that_fits():
    """Planning takes one index workspace when the measured entries ask for the form it began with."""
    require_cuda()
    from structsplat_b200.batch import FitPlan
    from structsplat_b200.synthetic import make_field
    n, H, W = 5_000, 256, 256
    f = make_field(H, W, n, 3)
    p = {k: torch.tensor(getattr(f, k), device="cuda")
         for k in ("means", "log_scales", "rotations", "colors", "opacity_logits")}
    seen = []
    empty = torch.empty

    def counted(*args, **kw):
        t = empty(*args, **kw)
        seen.append(t.numel() if t.dtype == torch.uint8 else 0)
        return t
    try:
        torch.empty = counted
        plan = FitPlan(Batch([(H, W)], [n]), p, torch.zeros(H * W, 3, device="cuda"))
    finally:
        torch.empty = empty
    assert seen.count(plan.idx_ws_bytes) == 1
