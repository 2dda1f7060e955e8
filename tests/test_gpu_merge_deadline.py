"""The deadline of the database readers' waits: with a timeout of 1 ms, a call whose
decode alone takes a few returns KITE_ERR_TIMEOUT instead of waiting inside a copy;
the device finishes its queue and works on."""
import ctypes as C
import time

import numpy as np
import pytest

from kite_gb300.kitefile import Chunk, KiteImage

pytestmark = pytest.mark.gpu


def test_wait_runs_out(gpu):
    rows = 200_000_000
    n = 12 + 2 * (rows - 1)
    lib = gpu.lib()
    p = lib.kite_gpu_alloc_pinned(n)
    assert p
    try:
        data = np.ctypeslib.as_array((C.c_uint8 * n).from_address(p))
        data[:12] = (0, 0, 0, 0, 0, 0, 0, 0, 1, 0, 0, 0)
        data[12::2] = 100  # key deltas
        data[13::2] = 1    # counts
        ki = KiteImage(data=data, k=21, partitions=2, key_width=64, part_first=[0, 1], part_count=[1, 0],
                       chunks=[Chunk(0, 2, 0, n, n, rows, 0, 100 * (rows - 1))])
        with gpu.Counter(21, False, 2, timeout_ms=1) as c:
            for call in (lambda: c.histo(ki, base=p), lambda: c.query(ki, [0, 100, 101, 300], base=p)):
                with pytest.raises(gpu.KiteGpuError, match="KITE_ERR_TIMEOUT"):
                    call()
                until = time.time() + 60
                while True:  # the queued work ends by itself; the input lives until then
                    try:
                        c.synchronize()
                        break
                    except gpu.KiteGpuError:
                        assert time.time() < until
        with gpu.Counter(21, False, 2) as c:
            assert c.histo(ki, base=p) == {1: rows}
            # keys of partition 0, where the chunk is
            keys = [k for k in range(0, 4000, 50) if (k * 0x9E3779B97F4A7C15 & (2**64 - 1)) >> 63 == 0]
            assert c.query(ki, keys, base=p) == [int(k % 100 == 0) for k in keys]
    finally:
        lib.kite_gpu_free_pinned(p)
