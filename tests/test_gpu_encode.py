"""DVLE encode at its edges: key deltas at every varint length, counts of one to
five bytes, tiles around a round's rows, and the first row of a partition at
every alignment: a database of one or two chunks merged and read back."""
import random

import pytest

from kite_gb300.kitefile import KiteImage
from kite_build import bucket, build_image, dvle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [31, 32, 63, 64])
@pytest.mark.parametrize("n", [1, 2, 31, 127, 128, 129, 255, 256, 257, 511, 512, 513, 1025, 4096, 4097, 9000])
def test_payload_bytes(gpu, k, n):
    wide, P, rng = k > 31, 4, random.Random(1000 * k + n)
    limit = 1 << (2 * k)
    chunks, want = [], {}
    for p in range(P):
        rows, key = [], 0
        for _ in range(n + p):
            bits = rng.choice([1, 6, 7, 8, 13, 14, 15, 20, 21, 27, 28, 29, 34, 35, 36, 41, 42, 43])
            if rng.random() < 0.002:
                bits = rng.choice([48, 49, 50, 55, 56, 57])
            if wide and rng.random() < 0.3:
                bits = min(rng.choice([62, 63, 64, 69, 70, 71, 97, 98, 99, 111, 112, 113]), 2 * k - 8)
            key += rng.getrandbits(bits) | 1 << (bits - 1)
            while bucket(key, P, wide) != p:
                key += 1
            if key >= limit:
                break
            rows.append((key, rng.choice([1, 2, 127, 128, 16_383, 16_384, 2_097_152, 2**28 - 1, 2**28, 2**32 - 1])))
        chunks.append((p, rows, 2))
        want[p] = dvle(rows, wide)
    ki = KiteImage.parse(build_image(k, False, P, chunks))
    with gpu.Counter(k, False, P) as c:
        out = c.merge([ki])
    assert {m["partition_id"]: bytes(b) for m, b in out} == want
