"""Databases whose bytes are damaged: keys above 2^(2k) are merged and written as
they are, a chunk with fewer rows than its index says is refused, as are places
and row counts that no file has, and the context works on."""
import random

import pytest

from kite_gb300.kitefile import KiteImage
from kite_build import build_image

pytestmark = pytest.mark.gpu


def _rows(rng, n, bits, base=0):
    return [(base + key, rng.choice([1, 2, 7])) for key in sorted({rng.getrandbits(bits) for _ in range(n)})]


def _image(k, high, seed=1):
    # two chunks in each of two partitions, several key ranges; the second
    # chunk's keys (its head key's upper bits) are too large by `high`
    rng = random.Random(seed)
    return build_image(k, False, 2, [(p, _rows(rng, 9000, 2 * k, high * c), 2) for p in range(2) for c in range(2)])


def _histo(dump):
    want = {}
    for line in dump.split(b"\n")[:-1]:
        n = int(line.split(b"\t")[1])
        want[n] = want.get(n, 0) + 1
    return want


@pytest.mark.parametrize("k,bit", [(21, 42), (21, 63), (31, 62), (40, 80), (40, 127)])
def test_keys_above_2k_bits(gpu, orc, k, bit):
    img = _image(k, 1 << bit)
    ki = KiteImage.parse(img)
    with gpu.Counter(k, False, 2) as c:
        want = orc.dump(img)
        assert c.dump(ki) == want
        assert c.histo(ki) == _histo(want)
        assert len(c.merge([ki, ki])) == 2
    with gpu.Counter(k, False, 2, splitter_mode=gpu.SPLIT_LEARNED) as c:
        assert len(c.merge([ki, ki])) == 2


@pytest.mark.parametrize("k", [21, 45])
def test_fewer_rows_than_the_index_says(gpu, orc, k):
    good, img = _image(k, 0), _image(k, 0, 2)
    bad = KiteImage.parse(img)
    bad.chunks[1].row_count += 7000
    some = [key for key, _ in _rows(random.Random(3), 50, 2 * k)]
    with gpu.Counter(k, False, 2) as c:
        for call in (lambda: c.merge([KiteImage.parse(good), bad]), lambda: c.dump(bad), lambda: c.histo(bad),
                     lambda: c.query(bad, some)):
            with pytest.raises(gpu.KiteGpuError) as e:
                call()
            assert "KITE_ERR_BAD_INPUT" in str(e.value) and "DVLE delta" in str(e.value)
            assert c.dump(KiteImage.parse(good)) == orc.dump(good)


@pytest.mark.parametrize("k,codec", [(21, 2), (21, 1), (45, 2), (45, 1)])
@pytest.mark.parametrize("rows,offset,length", [
    (1 << 62, None, None), ((1 << 61) + 1, None, None), ((1 << 60) + 1, None, None), (9001, None, None),
    (None, (1 << 64) - 8, 16), (None, 1 << 40, None), (None, None, (1 << 64) - 1)])
def test_index_of_no_file(gpu, orc, k, codec, rows, offset, length):
    rng = random.Random(4)
    img = build_image(k, False, 2, [(p, _rows(rng, 900, 2 * k), codec) for p in range(2)])
    bad = KiteImage.parse(img)
    c1 = bad.chunks[1]
    c1.row_count = c1.row_count if rows is None else rows
    c1.file_offset = c1.file_offset if offset is None else offset
    c1.encoded_bytes = c1.encoded_bytes if length is None else length
    with gpu.Counter(k, False, 2) as c:
        for call in (lambda: c.merge([bad]), lambda: c.dump(bad), lambda: c.histo(bad),
                     lambda: c.query(bad, list(range(1, 65)))):
            with pytest.raises(gpu.KiteGpuError, match="KITE_ERR_BAD_INPUT"):
                call()
        assert c.dump(KiteImage.parse(img)) == orc.dump(img)
