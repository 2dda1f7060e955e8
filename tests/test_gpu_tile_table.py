"""The tile sort's tables at their edges, byte for byte against the oracle: one
read per k-mer, all k-mers in partition 0 of 2, so that the partition is one
tile over the whole key range (or a few, above the tile load).  Distinct keys and
copies around the table's and the bins' sizes; keys spread over the range,
clustered in a 4096th of it (homes from a sample of the keys, full bins), or
next to each other (the tile goes on to the binning sort and its LSD passes)."""
import numpy as np
import pytest

from gpu_helpers import assert_parity
from kite_build import bucket

pytestmark = pytest.mark.gpu


def _keys(k: int, n: int, spread: str, seed: int) -> list:
    rng = np.random.default_rng(seed)
    top = 1 << (2 * k)
    out, seen, v = [], set(), 0
    while len(out) < n:
        if spread == "next":
            v += 1
        else:
            v = int.from_bytes(rng.bytes(16), "little") % (top if spread == "range" else top >> 12)
        if v not in seen and bucket(v, 2, k > 31) == 0:
            seen.add(v)
            out.append(v)
    return out


def _fastq(k: int, keys: list, copies: int, seed: int) -> bytes:
    codes = np.array([[(v >> (2 * (k - 1 - i))) & 3 for i in range(k)] for v in keys], dtype=np.uint8)
    codes = np.repeat(codes, copies, axis=0)
    np.random.default_rng(seed).shuffle(codes)
    rec = np.full((len(codes), 2 * k + 6), ord("I"), dtype=np.uint8)
    rec[:, 0:2] = (ord("@"), 10)
    rec[:, 2:2 + k] = np.frombuffer(b"ACGT", dtype=np.uint8)[codes]
    rec[:, 2 + k:5 + k] = (10, ord("+"), 10)
    rec[:, -1] = 10
    return rec.tobytes()


@pytest.mark.parametrize("spread", ["range", "cluster", "next"])
@pytest.mark.parametrize("n,copies", [(1, 1), (2, 1), (255, 1), (256, 2), (448, 1), (3296, 1), (1025, 3), (6500, 1),
                                      (7000, 1), (40, 300)])
def test_tile_u64(gpu, orc, n, copies, spread):
    fq = _fastq(21, _keys(21, n, spread, n), copies, n)
    st = assert_parity(gpu, orc, fq, 21, False, 2)
    assert st["kmers"] == n * copies


@pytest.mark.parametrize("spread", ["range", "cluster", "next"])
@pytest.mark.parametrize("n,copies", [(1, 1), (128, 1), (129, 1), (513, 1), (1024, 3), (1025, 2), (2049, 1), (3400, 1),
                                      (9, 300)])
def test_tile_u128(gpu, orc, n, copies, spread):
    fq = _fastq(41, _keys(41, n, spread, n), copies, n)
    st = assert_parity(gpu, orc, fq, 41, False, 2)
    assert st["kmers"] == n * copies


@pytest.mark.parametrize("k,fill", [(31, 1.0), (31, 2.5), (51, 1.0), (51, 1.6)])
def test_tiles_of_distinct_keys(gpu, orc, k, fill):
    # random reads: every key once, tiles at and above the on-chip capacity
    rng = np.random.default_rng(k)
    seq = np.frombuffer(b"ACGT", dtype=np.uint8)[rng.integers(0, 4, (2500, 120))]
    fq = b"".join(b"@\n" + s.tobytes() + b"\n+\n" + b"I" * 120 + b"\n" for s in seq)
    st = assert_parity(gpu, orc, fq, k, True, 4, tile_fill=fill, splitter_mode=gpu.SPLIT_SAMPLED)
    assert st["rows"] == st["kmers"]
