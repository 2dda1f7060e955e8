"""Histograms of databases with more tiles than the table merge has CTAs: each CTA
walks several tiles, among them empty ones and tiles listed for the merge paths
without a try, in every order.  Against sums in numpy."""
import numpy as np
import pytest

from kite_gb300.kitefile import KiteImage
from kite_build import build_image

pytestmark = pytest.mark.gpu
K, P = 31, 256


@pytest.mark.parametrize("large", [0, 2, 3, 5])
@pytest.mark.parametrize("full", [2, 3, 5])
def test_listed_and_empty_tiles(gpu, full, large):
    # Every full-th partition has four tiles, the others one and three empty
    # ones.  One row in a tile of every large-th partition has a count that the
    # table does not take, so that about 1 / large of the tiles fail: around the
    # third where the rest is listed untried.
    rng = np.random.default_rng(10 * full + large)
    want, chunks = {}, []
    for p in range(P):
        n = 12_300 if p % full == 0 else 100
        keys = np.unique(rng.integers(0, 1 << 62, n, dtype=np.uint64))
        counts = rng.integers(1, 40, len(keys))
        if large and p % large == 0:
            counts[::1000] = 1 << 19
        chunks.append((p, list(zip(keys.tolist(), counts.tolist())), 2))
        for c, m in zip(*np.unique(counts, return_counts=True)):
            want[int(c)] = want.get(int(c), 0) + int(m)
    ki = KiteImage.parse(build_image(K, False, P, chunks))
    with gpu.Counter(K, False, P) as c:
        for _ in range(3):
            assert c.histo(ki) == want
        assert c.stats()["tiles"] == 4 * P
