"""The bins and views that splitters take of sampled keys, on the host: of any key,
also of one above 2^(2k) (a damaged database's), they stay inside their tables."""
import random
import subprocess

from kite_gb300.build import CSRC, INCLUDE, _nvcc

DRIVER = r"""
#include <cstdio>
#include "splitters.h"
using namespace kite;
template <class T> void show(T key, uint32_t bits) {
  const uint32_t hbits = bits < 16 ? bits : 16;
  printf("%u %llu\n", sample_bin(key, bits, hbits), (unsigned long long)view48(key, bits));
}
int main() {
  unsigned wide, bits;
  unsigned long long hi, lo;
  while (scanf("%u %u %llu %llu", &wide, &bits, &hi, &lo) == 4) {
    if (wide) show<u128>((u128)hi << 64 | lo, bits);
    else show<uint64_t>(lo, bits);
  }
}
"""


def test_bins_of_any_key(tmp_path):
    src, exe = tmp_path / "bins.cu", tmp_path / "bins"
    src.write_text(DRIVER)
    subprocess.run([_nvcc(), "-std=c++17", "-I", str(INCLUDE), "-I", str(CSRC), str(src), "-o", str(exe)], check=True)
    rng = random.Random(1)
    asked = []
    for k in range(1, 65):
        bits, wide = 2 * k, k > 31
        width = 128 if wide else 64
        keys = [0, (1 << bits) - 1, 1 << min(bits, width - 1), (1 << width) - 1]
        keys += [rng.getrandbits(bits) for _ in range(20)] + [rng.getrandbits(width) for _ in range(20)]
        asked += [(wide, bits, min(x, (1 << width) - 1)) for x in keys]
    text = "".join(f"{int(w)} {b} {x >> 64} {x & (2**64 - 1)}\n" for w, b, x in asked)
    out = subprocess.run([str(exe)], input=text, capture_output=True, text=True, check=True).stdout.splitlines()
    assert len(out) == len(asked)
    for (_, bits, key), line in zip(asked, out):
        got, view = map(int, line.split())
        x = min(key, (1 << bits) - 1)
        assert got == x >> (bits - min(bits, 16))
        assert view == (x >> (bits - 48) if bits >= 48 else x << (48 - bits)) < 1 << 48
