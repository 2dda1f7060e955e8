"""The key-range split over many ranges per bucket: the staged-runs scatter of
u64 keys (more than 256 ranges) against the other launch shapes' and the
oracle's results, with ranges around its radix and parts of few keys."""
import pytest

from kite_gb300 import synth
from gpu_helpers import assert_parity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [0, 2])
@pytest.mark.parametrize("k,P,lo,hi", [(31, 4, 257, 1024), (31, 8, 257, 1024), (21, 16, 200, 300), (31, 2, 2048, 2048),
                                       (63, 4, 257, 1024)])
def test_ranges(gpu, orc, k, P, lo, hi, shape):
    fq = synth.small_workload(seed=k + P, n_reads=12_000, genome_len=300_000)
    st = assert_parity(gpu, orc, fq, k, True, P, tile_fill=0.05, scatter_shape=shape)
    if k <= 31:
        assert lo <= st["tiles_per_bucket"] <= hi


def test_one_heavy_range(gpu, orc):
    fq = synth.small_workload(seed=5, n_reads=8_000, genome_len=300_000)
    fq = bytes(fq) + (b"@a\n" + b"A" * 150 + b"\n+\n" + b"I" * 150 + b"\n") * 4_000
    assert_parity(gpu, orc, fq, 31, True, 4, tile_fill=0.05, splitter_mode=gpu.SPLIT_SAMPLED)
