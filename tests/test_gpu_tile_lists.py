"""The binning sort of listed tiles, launched on its own: a tile of a size that its
list cannot have is reported and left without rows, the others are sorted."""
import subprocess

import pytest

from kite_gb300.build import ARCH, CSRC, INCLUDE, LIB, _nvcc

pytestmark = pytest.mark.gpu

DRIVER = r"""
#include <cstdio>
#include <vector>
#include "kite_internal.h"
using namespace kite;

// Tiles of `sizes` keys one after another, all listed, keys falling: the rows of each and the status.
template <class T, int MULT> void show(std::vector<uint32_t> sizes) {
  std::vector<TileDesc> td;
  uint64_t n = 0;
  for (uint32_t z : sizes) {
    td.push_back(TileDesc{n, z, 0});
    n += z;
  }
  std::vector<T> keys(n);
  for (uint64_t i = 0; i < n; ++i) keys[i] = (T)((n - i) * 3);
  std::vector<uint32_t> ids;
  for (uint32_t i = 0; i < sizes.size(); ++i) ids.push_back(i);
  T* dk;
  uint32_t *dc, *di;
  TileDesc* dt;
  TileOut<T>* dout;
  unsigned* dn;
  unsigned long long* df;
  DevStatus* ds;
  cudaMalloc(&dk, (n + 64) * sizeof(T));
  cudaMalloc(&dc, n * 4);
  cudaMalloc(&di, ids.size() * 4);
  cudaMalloc(&dt, td.size() * sizeof(TileDesc));
  cudaMalloc(&dout, td.size() * sizeof(TileOut<T>));
  cudaMalloc(&dn, 4);
  cudaMalloc(&df, 16);
  cudaMalloc(&ds, sizeof(DevStatus));
  cudaMemset(df, 0, 16);
  cudaMemset(ds, 0, sizeof(DevStatus));
  cudaMemset(dout, 0xff, td.size() * sizeof(TileOut<T>));
  const unsigned count = (unsigned)ids.size();
  cudaMemcpy(dk, keys.data(), n * sizeof(T), cudaMemcpyHostToDevice);
  cudaMemcpy(di, ids.data(), count * 4, cudaMemcpyHostToDevice);
  cudaMemcpy(dt, td.data(), count * sizeof(TileDesc), cudaMemcpyHostToDevice);
  cudaMemcpy(dn, &count, 4, cudaMemcpyHostToDevice);
  const TileRanges<T> rg{nullptr, 1, 0, (T)(3 * n), 0};
  if (MULT == 1) launch_tile_sort_listed<T>(dk, dc, dt, di, 4, dn, dout, df, rg, ds, 0);
  else launch_tile_sort_large<T>(dk, dc, dt, di, 4, dn, dout, df, rg, ds, 0);
  std::vector<TileOut<T>> out(count);
  DevStatus st;
  const cudaError_t e = cudaMemcpy(out.data(), dout, count * sizeof(TileOut<T>), cudaMemcpyDeviceToHost);
  cudaMemcpy(&st, ds, sizeof st, cudaMemcpyDeviceToHost);
  printf("%d %u", (int)e, st.code);
  for (auto& o : out) printf(" %u", o.rows);
  printf("\n");
}
int main() {
  constexpr uint32_t c8 = tile_capacity<uint64_t>(), c16 = tile_capacity<u128>();
  show<uint64_t, 1>({5, c8, 1});
  show<uint64_t, 1>({5, c8 + 1, 0, 7});
  show<uint64_t, 2>({2 * c8, 9});
  show<uint64_t, 2>({2 * c8 + 1, 9});
  show<u128, 1>({5, c16, 1});
  show<u128, 1>({c16 + 1, 7});
  show<u128, 2>({2 * c16, 9});
  show<u128, 2>({9, 2 * c16 + 1});
}
"""


def test_sizes_of_listed_tiles(gpu, tmp_path):
    src, exe = tmp_path / "lists.cu", tmp_path / "lists"
    src.write_text(DRIVER)
    subprocess.run([_nvcc(), *ARCH, "-std=c++17", "-cudart", "shared", "-I", str(INCLUDE), "-I", str(CSRC), str(src),
                    "-o", str(exe), f"-L{LIB}", "-lkite_gpu", "-Xlinker", "-rpath", "-Xlinker", str(LIB)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True, timeout=120).stdout.splitlines()
    overflow = 3
    assert [list(map(int, x.split())) for x in out] == [
        [0, 0, 5, 8192, 1], [0, overflow, 5, 0, 0, 7], [0, 0, 16384, 9], [0, overflow, 0, 9],
        [0, 0, 5, 4096, 1], [0, overflow, 0, 7], [0, 0, 8192, 9], [0, overflow, 9, 0]]
