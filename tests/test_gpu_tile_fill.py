"""Tiles per partition: as few as the tile load allows, and for loads that bring tiles
above twice the on-chip capacity (sorted through global memory) a multiple of 32;
the same counts for all."""
import numpy as np
import pytest

from kite_gb300 import synth
from gpu_helpers import gpu_count

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,cap", [(31, 8192), (51, 4096)])
def test_tiles_per_partition(gpu, k, cap):
    rng = np.random.default_rng(k)
    fq = synth.reads_fixed(rng, synth.genome_iid(rng, 200_000), 12_000, 150, 0.005)
    first = None
    for fill in (0.85, 1.0, 1.6, 1.9, 2.6, 4.0):
        out, st = gpu_count(gpu, fq, k, True, 4, tile_fill=fill)
        first = first or out
        assert out == first
        # the largest of the four partitions is within 20% of the mean
        per, least, most = st["tiles"] // 4, st["kmers"] / 4 / (fill * cap), 1.2 * st["kmers"] / 4 / (fill * cap) + 1
        if fill > 1.8:
            assert per % 32 == 0 and least <= per < most + 32
        else:
            assert least <= per < most
