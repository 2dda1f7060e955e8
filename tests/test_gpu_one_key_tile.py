"""Tiles above twice the on-chip capacity (16,384 keys) that hold one key alone, and
those that one more key shares: at that size and beyond, from an even and an odd
place, the other key first, last or amid the copies.  Byte for byte against the
oracle."""
import numpy as np
import pytest

from gpu_helpers import assert_parity
from kite_build import bucket

pytestmark = pytest.mark.gpu
K = 21


def _reads(keys) -> bytes:
    codes = np.array([[(v >> (2 * (K - 1 - i))) & 3 for i in range(K)] for v in keys], dtype=np.uint8)
    rec = np.full((len(codes), 2 * K + 6), ord("I"), dtype=np.uint8)
    rec[:, 0:2] = (ord("@"), 10)
    rec[:, 2:2 + K] = np.frombuffer(b"ACGT", dtype=np.uint8)[codes]
    rec[:, 2 + K:5 + K] = (10, ord("+"), 10)
    rec[:, -1] = 10
    return rec.tobytes()


@pytest.mark.parametrize("before", [0, 1, 2])
@pytest.mark.parametrize("other", [None, 0, 7000, -1])
@pytest.mark.parametrize("n", [16_384, 16_385, 16_386, 40_001])
def test_one_key(gpu, orc, n, other, before):
    a, b = [v for v in range(1000, 1100) if bucket(v, 2, False) == 1][:2]
    low = [v for v in range(1000) if bucket(v, 2, False) == 0][:before]
    keys = [a] * n
    if other is not None:
        keys.insert(other if other >= 0 else n, b)
    st = assert_parity(gpu, orc, _reads(low + keys), K, False, 2, splitter_mode=gpu.SPLIT_SAMPLED)
    assert st["rows"] == before + 1 + (other is not None)
    assert st["big_tiles"] == 1 and st["big_tile_rows"] == st["rows"] - before
