"""The table merge of u64 keys at the edges of its rule: counts of 0 and around
2^19, sums past 32 bits, keys crowded into a small part of a tile's range, a
chunk that repeats a key, filters with one and with several chunks per
partition, and chunks of very uneven sizes.  Against sums in Python."""
import random

import pytest

from kite_gb300.kitefile import KiteImage
from kite_build import bucket, build_image
from test_zz_no_alloc import _dvle_rows

pytestmark = pytest.mark.gpu
K, P = 31, 2


def rows_of(rng, n, counts, spread=62, base=0):
    out = []
    while len(out) < n:
        key = base + rng.getrandbits(spread)
        if bucket(key, P, False) == 1:
            out.append((key, rng.choice(counts)))
    return sorted(dict(out).items())


def summed(chunks):
    t = {}
    for rows in chunks:
        for key, c in rows:
            t[key] = t.get(key, 0) + c
    return t


def image(chunks, lo=None, hi=None):
    return build_image(K, False, P, [(1, r, 2) for r in chunks], lo, hi)


def check(gpu, inputs):
    """inputs: (chunks, min, max) of each database."""
    kis = [KiteImage.parse(image(*i)) for i in inputs]
    total = {}
    for chunks, lo, hi in inputs:
        for key, c in summed(chunks).items():
            if (lo is None or c >= lo) and (hi is None or c <= hi):
                total[key] = total.get(key, 0) + c
    with gpu.Counter(K, False, P) as c:
        if max(total.values(), default=0) < 2**32:
            out = c.merge(kis)
            got = [r for m, p in out for r in _dvle_rows(p, m["row_count"], False)]
            assert got == sorted(total.items())
        chunks, lo, hi = inputs[0]
        one = summed(chunks)
        kept = [v for v in one.values() if (lo is None or v >= lo) and (hi is None or v <= hi)]
        assert c.histo(kis[0]) == {v: kept.count(v) for v in set(kept)}
        lines = [(k, min(v, 2**32 - 1)) for k, v in sorted(one.items())]
        lines = [(k, v) for k, v in lines if (lo is None or v >= lo) and (hi is None or v <= hi)]
        want = b"".join(b"%s\t%d\n" % (bytes(b"ACGT"[(k >> 2 * (K - 1 - i)) & 3] for i in range(K)), v) for k, v in lines)
        assert c.dump(kis[0]) == want


@pytest.mark.parametrize("inputs", [1, 3])
@pytest.mark.parametrize("chunks", [1, 3])
@pytest.mark.parametrize("counts", [[1, 2, 9], [0, 1, 5], [2**19 - 1, 1], [2**19, 1], [2**32 - 1, 1]])
def test_counts(gpu, inputs, chunks, counts):
    rng = random.Random(str((inputs, chunks, counts)))
    shared = rows_of(rng, 3000, counts)
    mk = lambda: sorted(dict(rng.sample(shared, 2000) + rows_of(rng, 2500, counts)).items())  # noqa: E731
    check(gpu, [([mk() for _ in range(chunks)], None, None) for _ in range(inputs)])


@pytest.mark.parametrize("chunks", [1, 2])
@pytest.mark.parametrize("lo,hi", [(2, None), (None, 3), (3, 4), (99, None)])
def test_filters(gpu, chunks, lo, hi):
    rng = random.Random(str((chunks, lo, hi)))
    shared = rows_of(rng, 4000, [1, 2, 3])
    mk = lambda: sorted(rng.sample(shared, 3000))  # noqa: E731
    check(gpu, [([mk() for _ in range(chunks)], lo, hi), ([mk()], None, None), ([mk()], None, 2)])


def test_crowded_keys(gpu):
    # most keys of a tile lie in a small part of its range: probes run too far
    rng = random.Random(5)
    mk = lambda: sorted(dict(rows_of(rng, 1500, [1, 4], 14) + rows_of(rng, 300, [1])).items())  # noqa: E731
    check(gpu, [([mk(), mk()], None, None), ([mk()], 2, None)])


@pytest.mark.parametrize("lo", [None, 3])
def test_repeated_key_in_a_chunk(gpu, lo):
    rng = random.Random(8)
    rows = rows_of(rng, 2000, [1, 2])
    rows[700:704] = [(rows[700][0], 2)] * 4
    check(gpu, [([rows], lo, None), ([rows_of(rng, 1000, [1, 3])], lo, None)])
    check(gpu, [([rows, rows_of(rng, 10, [3])], lo, None)])


def test_many_uneven_chunks(gpu):
    rng = random.Random(9)
    shared = rows_of(rng, 6000, [1, 2])
    chunks = [sorted(rng.sample(shared, rng.choice([1, 3, 40, 900]))) for _ in range(200)]
    check(gpu, [(chunks, None, None), (chunks[:50], None, None)])
