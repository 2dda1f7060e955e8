"""The DVLE decode at its edges: streams whose varint area ends at, just before
and just after an 8 KiB segment, varints of every length across rounds and
segments, one-row streams, counts up to u32::MAX; `kite dump` of the image
against the oracle's, byte for byte."""
import random

import pytest

from kite_gb300.kitefile import KiteImage
from kite_build import build_image, varint

pytestmark = pytest.mark.gpu

U32 = 0xFFFFFFFF


def _rows(rng, k: int, area: int, long_every: int):
    """Rows whose varint area is `area` bytes (0: the head row alone)."""
    key, rows, left, i = rng.getrandbits(8), [], area, 0
    rows.append((key, rng.choice([1, 2, 200, U32])))
    while left > 0:
        i += 1
        bits = 2 * k - 16 if i % long_every == 0 else rng.choice([6, 7, 13, 14, 27, 28, 2 * k - 26])
        delta = 1 + rng.getrandbits(min(bits, 2 * k - 16))
        count = rng.choice([1, 1, 1, 1, 3, 127, 128, 70_000, U32])
        n = len(varint(delta)) + len(varint(count))
        if n > left - 2 and n != left:  # finish exactly: rows of two and three bytes
            delta, count = (1, 1) if left % 2 == 0 else (200, 1)
            n = len(varint(delta)) + len(varint(count))
        key += delta
        if key >= 1 << (2 * k):
            key, delta = rows[-1][0] + 1, 1
            n = 1 + len(varint(count))
        rows.append((key, count))
        left -= n
    return rows


@pytest.mark.parametrize("k", [21, 31, 47, 64])
@pytest.mark.parametrize("area", [0, 2, 511, 512, 8191, 8192, 8193, 8204, 16_384, 40_003])
def test_decode_segment_edges(gpu, orc, k, area):
    rng = random.Random(100 * k + area)
    chunks = []
    for p in range(4):
        # several chunks per partition, so that streams start at any byte
        for j in range(2):
            chunks.append((p, _rows(rng, k, area + 3 * j if area else 0, 50), 2))
    img = build_image(k, False, 4, chunks)
    ki = KiteImage.parse(img)
    with gpu.Counter(k, False, 4) as c:
        assert c.dump(ki) == orc.dump(img)
