"""u128 k-mer extraction where its windows cross words, threads, warps and
16 KiB blocks: reads longer than a block, shifted byte by byte against the
32-byte words by their headers, with N, lower case and short lines between
them; byte for byte against the oracle."""
import numpy as np
import pytest

from gpu_helpers import assert_parity

pytestmark = pytest.mark.gpu


def _fastq(k: int, shift: int) -> bytes:
    rng = np.random.default_rng(1000 * k + shift)
    out = []
    for i, n in enumerate((20_000 + shift, k, k - 1, 0, 500, 16_384, 63, 2 * k)):
        seq = np.frombuffer(b"ACGT", dtype=np.uint8)[rng.integers(0, 4, n)].copy()
        if n > 400:
            seq[rng.integers(0, n, 5)] = ord("N")
            seq[rng.integers(0, n, 50)] |= 0x20
        out.append(b"@" + b"h" * (shift + 7 * i) + b"\n" + seq.tobytes() + b"\n+\n" + b"@" * n + b"\n")
    return b"".join(out)


@pytest.mark.parametrize("shift", [0, 1, 13, 31, 32, 63])
@pytest.mark.parametrize("k,canonical", [(32, True), (33, False), (48, True), (63, True), (64, True), (64, False)])
def test_extract_u128_edges(gpu, orc, k, canonical, shift):
    assert_parity(gpu, orc, _fastq(k, shift), k, canonical, 8, chunk_size=40_000)
