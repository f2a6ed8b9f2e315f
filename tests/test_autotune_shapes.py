"""The tuner leaves the launch shapes that it did not choose as they were asked: unset ones unset."""
from __future__ import annotations

import itertools

import pytest

from structsplat_b200 import _native, autotune

UNSET = {16: (0, 0), 32: (0, 0)}


@pytest.fixture(autouse=True)
def _shapes():
    autotune.ask_shapes(UNSET)
    yield
    autotune.ask_shapes(UNSET)


def _pick(monkeypatch, times, longest=None):
    seq = itertools.chain(times)
    monkeypatch.setattr(autotune, "_time", lambda fn, repeats: next(seq))
    return autotune._pick("key", autotune.CANDIDATES, lambda ts: None, 1, False, longest)


def test_unset_and_asked_are_told_apart():
    lib = _native.lib()
    for ts in (16, 32):
        assert lib.ss_asked_backward_warps(ts) == 0 and lib.ss_asked_forward_chunk(ts) == 0
        assert lib.ss_get_backward_warps(ts) == 8 and lib.ss_get_forward_chunk(ts) == 256
        autotune.ask_shapes({ts: (8, 256)})
        assert lib.ss_asked_backward_warps(ts) == 8 and lib.ss_asked_forward_chunk(ts) == 256
    assert lib.ss_asked_backward_warps(8) == -1 and lib.ss_asked_forward_chunk(8) == -1


@pytest.mark.parametrize("times,want", [((1.0, 2.0, 3.0, 4.0), {16: (4, 0), 32: (0, 0)}),
                                        ((4.0, 3.0, 2.0, 1.0), {16: (0, 0), 32: (16, 0)})])
def test_the_other_tile_size_stays_unset(monkeypatch, times, want):
    _pick(monkeypatch, times)
    assert autotune.asked_shapes() == want


def test_a_failing_candidate_leaves_everything_unset(monkeypatch):
    def fail(fn, repeats):
        raise RuntimeError("candidate")
    monkeypatch.setattr(autotune, "_time", fail)
    with pytest.raises(RuntimeError, match="candidate"):
        autotune._pick("key", autotune.CANDIDATES, lambda ts: None, 1, False)
    assert autotune.asked_shapes() == UNSET


def test_asked_shapes_come_back(monkeypatch):
    autotune.ask_shapes({16: (8, 64), 32: (8, 128)})
    _pick(monkeypatch, (1.0, 2.0, 3.0, 4.0))
    assert autotune.asked_shapes() == {16: (4, 0), 32: (8, 128)}


def test_a_tuned_fit_leaves_the_shapes(monkeypatch):
    from structsplat_b200 import batch

    def fit(*args):
        autotune.ask_shapes({16: (4, 64), 32: (16, 64)})
        return {"tuned": True}
    monkeypatch.setattr(batch, "_fit_batch", fit)
    assert batch.fit_batch([], [], tune=True)["tuned"]
    assert autotune.asked_shapes() == UNSET


@pytest.mark.parametrize("tile,longest,chunks", [(16, 256, []), (16, 257, [64, 128]), (32, 512, []),
                                                 (32, 513, [64, 128, 256])])
def test_chunks_are_timed_from_the_tiles_own_stage_on(monkeypatch, tile, longest, chunks):
    times = (1.0, 2.0, 3.0, 4.0) if tile == 16 else (4.0, 3.0, 1.0, 2.0)
    r = _pick(monkeypatch, times + tuple(range(1, 1 + len(chunks))), longest=lambda ts: longest)
    assert r.tile_size == tile
    assert [k for k in r.times_ms if "/chunk" in k] == [
        f"{tile}x{r.backward_warps}/chunk{c}" for c in chunks]
    assert r.forward_chunk == (chunks[0] if chunks else 0)


def test_cached_shapes_of_other_kernels_are_not_taken():
    key = autotune.workload_key(1, 1, 1, 1, True, False, False, fit=True)
    assert f"k={autotune.KERNELS}" in key.split("|")
