"""Tile cuts at sample quantiles (automatic splitters of skewed keys): exact
counts, and key ranges as even as the learned CDF's where the histogram's are
not, with samples of one to 64 sorted blocks and with heavy single keys."""
import pytest

from kite_gb300 import synth
from gpu_helpers import assert_parity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,n_reads,P", [(63, 12_000, 2), (31, 12_000, 2), (63, 400, 2), (40, 25_000, 4)])
def test_auto_splitters_of_skewed_keys(gpu, orc, k, n_reads, P):
    fq = synth.skewed_workload(seed=n_reads + k, n_reads=n_reads, genome_len=400_000)
    sampled = assert_parity(gpu, orc, fq, k, True, P, splitter_mode=gpu.SPLIT_SAMPLED)
    auto = assert_parity(gpu, orc, fq, k, True, P)
    assert auto["splitter_used"] == gpu.SPLIT_SAMPLED
    assert auto["range_imbalance"] <= sampled["range_imbalance"]
    if n_reads >= 12_000 and sampled["range_imbalance"] > 4:
        # 128 sampled keys per range and more: a few standard deviations
        assert auto["range_imbalance"] < 0.5 * sampled["range_imbalance"]


def test_heavy_keys(gpu, orc):
    # one key is a third of all keys, so several quantiles are equal
    fq = synth.skewed_workload(seed=3, n_reads=8_000, genome_len=100_000)
    fq = bytes(fq) + (b"@a\n" + b"A" * 250 + b"\n+\n" + b"I" * 250 + b"\n") * 4_000
    assert_parity(gpu, orc, fq, 31, True, 2)
    assert_parity(gpu, orc, fq, 63, False, 2)
