"""Tile plans of merge, dump, histo and query at their edges: partitions of one
chunk around the tile capacity (4096 rows) and with equal keys across a cut,
partitions with chunks of some inputs only, key ranges above the capacity (the
host's cut with bisection), and queries of partitions far apart in the file."""
import random

import numpy as np
import pytest

from kite_gb300.kitefile import KiteImage
from kite_build import build_image

pytestmark = pytest.mark.gpu


def _rows(rng, n: int, bits: int, base: int = 0):
    keys = sorted(rng.sample(range(1 << bits), n)) if bits < 40 else sorted({rng.getrandbits(bits) for _ in range(n)})
    return [(base + k, rng.choice([1, 1, 2, 5, 1023, 1024, 70_000])) for k in keys]


def _check_one(gpu, orc, img: bytes, k: int):
    ki = KiteImage.parse(img)
    with gpu.Counter(k, False, ki.partitions) as c:
        dump = c.dump(ki)
        histo = c.histo(ki)
    assert dump == orc.dump(img)
    want = {}
    for line in dump.split(b"\n")[:-1]:
        n = int(line.split(b"\t")[1])
        want[n] = want.get(n, 0) + 1
    assert histo == want


@pytest.mark.parametrize("k", [31, 45])
@pytest.mark.parametrize("sizes", [(1, 4095, 4096, 4097), (0, 12_289, 8192, 3), (5000, 0, 0, 0)])
def test_one_chunk_per_partition(gpu, orc, k, sizes):
    rng = random.Random(sum(sizes) + k)
    img = build_image(k, False, 4, [(p, _rows(rng, n, 2 * k), 2) for p, n in enumerate(sizes) if n])
    _check_one(gpu, orc, img, k)


@pytest.mark.parametrize("at,run", [(4095, 2), (4096, 3), (8190, 6)])
def test_equal_keys_across_a_cut(gpu, orc, at, run):
    # a chunk whose rows repeat a key where the plan cuts it: summed all the same
    rng = random.Random(at)
    rows = _rows(rng, 9000, 62)
    rows[at:at + run] = [(rows[at][0], 7)] * run
    _check_one(gpu, orc, build_image(31, False, 2, [(0, rows, 2)]), 31)


@pytest.mark.parametrize("k,bits", [(31, 62), (31, 16), (40, 80), (40, 18)])
def test_chunks_of_some_partitions(gpu, orc, k, bits):
    # up to five chunks per partition, keys over the whole range or in a small
    # part of it (one range above the capacity, cut again by bisection)
    rng = random.Random(k + bits)
    chunks = [(p, _rows(rng, rng.choice([50, 3000, 9000]), bits), 2) for p in range(8) for _ in range(p % 6)]
    _check_one(gpu, orc, build_image(k, False, 8, chunks), k)


@pytest.mark.parametrize("chunks", [1, 3])
def test_query_sparse_partitions(gpu, orc, chunks):
    rng = np.random.default_rng(chunks)
    table, parts = {}, []
    for p in range(16):
        for _ in range(chunks):
            keys = np.unique(rng.integers(0, 1 << 62, 90_000, dtype=np.uint64))
            keys = keys[(keys * np.uint64(0x9E3779B97F4A7C15)) >> np.uint64(60) == p] if p in (3, 15) else keys[:70_000]
            counts = rng.integers(1, 50, len(keys))
            parts.append((p, [(int(a), int(b)) for a, b in zip(keys, counts)], 2))
            if p in (3, 15):
                for a, b in parts[-1][1]:
                    table[a] = table.get(a, 0) + b
    img = build_image(31, False, 16, parts)
    ki = KiteImage.parse(img)
    some = [k for i, k in enumerate(sorted(table)) if i % 97 == 0]
    near = [k + 1 for k in some if ((k + 1) * 0x9E3779B97F4A7C15 & (2**64 - 1)) >> 60 in (3, 15)]
    with gpu.Counter(31, False, 16) as c:
        assert c.query(ki, some) == [table[k] for k in some]
        assert c.query(ki, near) == [table.get(k, 0) for k in near]
