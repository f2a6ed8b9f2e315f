"""The container's streams inflate to the same bytes one after the other and side by side, and the
errors of damaged containers are the same either way."""
from __future__ import annotations

import json
import os
import struct
import threading
import zlib
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

from structsplat_b200 import codec


def _container(raws, cut=None, damage=None):
    head = json.dumps({"n": 1, "has_opacity": True, "stream_codec": "zlib"}).encode()
    blob = b"SSPL1" + struct.pack("<I", len(head)) + head
    for i, r in enumerate(raws):
        z = zlib.compress(r)
        if i == damage:
            z = z[:-3] + b"xyz"
        blob += struct.pack("<I", len(z)) + z
    return blob if cut is None else blob[:cut]


def _raws(size):
    rng = np.random.default_rng(size)
    return [rng.integers(0, 256, size * (i + 1), dtype=np.uint8).tobytes() for i in range(5)]


@pytest.mark.parametrize("size", [0, 100, 8_700, 8_800, 40_000])  # 8,738 a stream is the threshold
def test_streams(size):
    raws = _raws(size)
    assert codec._streams(_container(raws))[1] == raws


@pytest.mark.parametrize("size", [100, 40_000])
def test_errors_come_in_stream_order(size):
    raws = _raws(size)
    whole = _container(raws)
    with pytest.raises(ValueError, match="truncated"):
        codec._streams(whole[:-len(zlib.compress(raws[-1])) - 2])
    with pytest.raises(zlib.error):
        codec._streams(_container(raws, damage=2))
    with pytest.raises(zlib.error):  # the damaged stream comes before the missing frame
        codec._streams(_container(raws[:4], damage=1))
    with pytest.raises(zlib.error):
        codec._streams(whole[:-4])


def test_a_forked_child_decodes():
    raws = _raws(40_000)
    blob = _container(raws)
    assert codec._streams(blob)[1] == raws  # the parent's threads exist
    pid = os.fork()
    if pid == 0:
        ok = False
        try:
            ok = codec._streams(blob)[1] == raws
        finally:
            os._exit(0 if ok else 1)
    assert os.waitstatus_to_exitcode(os.waitpid(pid, 0)[1]) == 0


def test_many_threads_at_once():
    raws = _raws(40_000)
    blob = _container(raws)
    with ThreadPoolExecutor(16) as pool:
        assert all(r[1] == raws for r in pool.map(codec._streams, [blob] * 64))
    assert len([t for t in threading.enumerate() if t.name.startswith("sspl1-inflate")]) <= 4
