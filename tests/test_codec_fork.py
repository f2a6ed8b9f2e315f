"""A process forked while another thread starts the inflating threads decodes all the same."""
from __future__ import annotations

import json
import os
import struct
import threading
import time
import zlib

import numpy as np

from structsplat_b200 import codec


def test_fork_while_the_pool_is_being_made():
    rng = np.random.default_rng(0)
    raws = [rng.integers(0, 255, 60_000, dtype=np.uint8).tobytes() for _ in range(4)]
    head = json.dumps({"n": 1, "stream_raw_lengths": [len(r) for r in raws]}).encode()
    blob = b"SSPL1" + struct.pack("<I", len(head)) + head
    for r in raws:
        z = zlib.compress(r)
        blob += struct.pack("<I", len(z)) + z
    assert len(blob) > codec.THREADED_BYTES
    held, done = threading.Event(), threading.Event()

    def hold():
        with codec._POOL_LOCK:
            held.set()
            done.wait(30)
    holder = threading.Thread(target=hold)
    holder.start()
    held.wait()
    try:
        pid = os.fork()
        if pid == 0:
            ok = False
            try:
                ok = codec._streams(blob)[1] == raws
            finally:
                os._exit(0 if ok else 1)
        for _ in range(200):  # 20 s
            got, status = os.waitpid(pid, os.WNOHANG)
            if got:
                break
            time.sleep(0.1)
        else:
            os.kill(pid, 9)
            os.waitpid(pid, 0)
            raise AssertionError("the child waits for a lock that nobody holds")
        assert os.waitstatus_to_exitcode(status) == 0
    finally:
        done.set()
        holder.join()
