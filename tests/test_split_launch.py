"""The key-range split's scatter, on the host with the CUDA calls recorded: the part
count asks about the occupancy of the kernel that is then launched, and a launch
without a kernel (many digits, none stored) is refused."""
import subprocess

from kite_gb300.build import ARCH, CSRC, INCLUDE, LIB, _nvcc

FAKE = r"""
#include <cstddef>
struct Dim3 { unsigned x, y, z; };
struct Call { const void* f; unsigned nt; size_t smem; };
Call asked, launched;
static size_t allowed;
extern "C" {
int cudaGetDevice(int* d) { *d = 0; return 0; }
int cudaDeviceGetAttribute(int* v, int, int) { *v = 152; return 0; }
int cudaFuncSetAttribute(const void*, int, int v) { allowed = v; return 0; }
int cudaGetLastError() { return 0; }
int cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void* f, int nt, size_t smem, unsigned) {
  asked = Call{f, (unsigned)nt, smem};
  *n = 3;
  return 0;
}
int __cudaGetKernel(const void** kernel, const void* f) { *kernel = f; return 0; }
int __cudaLaunchKernel(const void* f, Dim3, Dim3 b, void**, size_t smem, void*) {
  launched = Call{f, b.x, smem};
  return smem <= allowed ? 0 : 1;
}
}
"""

DRIVER = r"""
#include <cstdio>
#include "kite_internal.h"
using namespace kite;

struct Call { const void* f; unsigned nt; size_t smem; };
extern Call asked, launched;

template <class T> void show() {
  for (int digits = 0; digits < 2; ++digits)
    for (unsigned D : {2u, 4u, 16u, 17u, 256u, 257u, 1024u})
      for (int shape = 0; shape < 4; ++shape) {
        asked = launched = Call{};
        uint16_t dig;
        TileSplitParams<T> p{};
        p.R = p.G = 1;
        p.D = D;
        p.dig = digits ? &dig : nullptr;
        const unsigned slots = split_scatter_slots<T>(D, shape, digits);
        const cudaError_t e = launch_split_scatter<T>(p, shape, 0);
        const bool same = asked.f == launched.f && asked.nt == launched.nt && asked.smem == launched.smem;
        printf("%d %u %d %d %d %u\n", digits, D, (int)e, launched.f != nullptr, same, slots);
      }
}
int main() {
  show<uint64_t>();
  show<u128>();
}
"""


def test_scatter_of_the_part_count_is_the_one_launched(built, tmp_path):
    src, fake, exe = tmp_path / "split.cu", tmp_path / "fake.cpp", tmp_path / "split"
    src.write_text(DRIVER)
    fake.write_text(FAKE)
    subprocess.run([_nvcc(), *ARCH, "-std=c++17", "-cudart", "shared", "-Xcompiler", "-rdynamic", "-I", str(INCLUDE),
                    "-I", str(CSRC), str(src), str(fake), "-o", str(exe), f"-L{LIB}", "-lkite_gpu", "-Xlinker", "-rpath",
                    "-Xlinker", str(LIB)], check=True)
    lines = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.splitlines()
    assert len(lines) == 2 * 2 * 7 * 4
    for line in lines:
        digits, D, err, launched, same, slots = map(int, line.split())
        if digits or D <= 16:
            assert (err, launched, same, slots) == (0, 1, 1, 3 * 152), line
        else:
            assert err != 0 and not launched, line
