"""kite_gpu_count_rows_noalloc at the edges of its kernels: text at any byte
alignment, lengths around the extraction segments, tiles of every sort (on
chip, above its capacity, one key), against the context path's rows."""
import numpy as np
import pytest

from kite_gb300 import synth
from test_zz_no_alloc import _fn, context_rows, noalloc_rows

pytestmark = pytest.mark.gpu


def reads(seed, n, length, genome=20_000, weights=None):
    rng = np.random.default_rng(seed)
    g = synth.genome_iid(rng, genome)
    if weights is not None:
        g = rng.choice(4, size=genome, p=weights).astype(np.uint8)
    return bytes(synth.reads_fixed(rng, g, n, length, 0.01, n_rate=0.002, revcomp_frac=0.5))


def check(gpu, data, k, canonical, P):
    parts, tot = context_rows(gpu, data, k, canonical, P)
    rc, got, gtot = noalloc_rows(gpu, data, k, canonical, P)
    assert rc == 0 and gtot == tot and got == parts


@pytest.mark.parametrize("k", [13, 31, 32, 33, 64])
@pytest.mark.parametrize("length", [2047, 2048, 2049, 4095, 4096, 4112, 6145])
def test_segment_edges(gpu, k, length):
    # chunks cut at and around the 2 KiB segments, ending inside any line
    check(gpu, reads(length, 40, 90)[:length], k, True, 16)


@pytest.mark.parametrize("skew", [1, 3, 8, 15])
@pytest.mark.parametrize("k", [31, 51])
def test_unaligned_text(gpu, skew, k):
    import ctypes as C

    import torch
    data = reads(skew, 60, 100)
    want, _ = noalloc_rows(gpu, data, k, True, 64)[1:]
    # the text inside other text: bytes before and after it must not count
    around = b"@x\nACGTACGTACGT"[-skew:].rjust(skew, b"\n") + data + b"ACGTACGTACGTACGTACGT" * 4
    d = torch.frombuffer(bytearray(around), dtype=torch.uint8).to("cuda")
    kb = 8 if k <= 31 else 16
    keys = torch.zeros(len(data) * kb, dtype=torch.uint8, device="cuda")
    counts = torch.zeros(len(data), dtype=torch.int32, device="cuda")
    prow = torch.zeros(64, dtype=torch.int32, device="cuda")
    tot = (C.c_uint64 * 4)()
    torch.cuda.synchronize()
    assert _fn(gpu)(0, k, 1, 64, d.data_ptr() + skew, len(data), keys.data_ptr(), counts.data_ptr(), len(data),
                    prow.data_ptr(), tot, None, 0) == 0
    rows = tot[3]
    assert rows == sum(len(v) for v in want.values())
    assert prow.cpu().tolist() == [len(want.get(p, [])) for p in range(64)]
    flat = [r for p in sorted(want) for r in want[p]]
    got = keys.cpu().numpy()[:rows * kb].view(np.uint64).reshape(rows, kb // 8)
    assert [sum(int(x) << (64 * i) for i, x in enumerate(r)) for r in got] == [r[0] for r in flat]
    assert counts.cpu().tolist()[:rows] == [r[1] for r in flat]


@pytest.mark.parametrize("k,P", [(31, 2), (31, 1024), (11, 4), (63, 16), (48, 16384), (3, 2)])
def test_tiles(gpu, k, P):
    check(gpu, reads(k, 1500, 150, 200_000), k, True, P)


@pytest.mark.parametrize("k", [21, 63])
@pytest.mark.parametrize("P", [2, 64])
def test_tiles_above_capacity(gpu, k, P):
    # mostly A: the keys crowd into the lowest ranges, and one poly-A key repeats
    skewed = reads(k, 1200, 150, 60_000, [0.85, 0.05, 0.05, 0.05]) + (b"@a\n" + b"A" * 150 + b"\n+\n" + b"I" * 150 + b"\n") * 300
    check(gpu, skewed, k, False, P)
