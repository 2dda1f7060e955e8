// FASTQ text as 32-byte words: 2-bit codes, line and base masks, and the runs
// of k bases in them.  Shared by the extraction kernels.
#pragma once

#include "kite_common.cuh"

namespace kite {

struct Word32 {
  uint64_t code;   // 2-bit codes, byte 0 in bits 63..62
  uint64_t rcode;  // complement codes in reverse byte order (byte 31 in bits 63..62)
  uint32_t nl;     // bit i: byte i is '\n'
  uint32_t vb;     // bit i: byte i is A/C/G/T in either case
};

// one bit per byte from a byte-wise 0x00/0xFF mask (byte j -> bit j)
__device__ __forceinline__ uint32_t byte_bits(uint32_t m) { return ((m & 0x01010101u) * 0x10204080u) >> 28; }

__device__ __forceinline__ Word32 encode_word(const uint4 a, const uint4 b) {
  const uint32_t x[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
  Word32 w;
  w.code = 0;
  w.nl = 0;
  w.vb = 0;
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const uint32_t v = x[q];
    // A/a=0 C/c=1 G/g=2 T/t=3 from ASCII bits 1 and 2
    const uint32_t c4 = ((v >> 1) ^ (v >> 2)) & 0x03030303u;
    // a byte is a base when, case folded, it is the letter its code stands
    // for: a byte permute of "ACGT" with the codes as selectors
    const uint32_t x = c4 | (c4 >> 4);
    const uint32_t y = x & 0x00FF00FFu;
    const uint32_t valid = __vcmpeq4(v & 0xDFDFDFDFu, __byte_perm(0x54474341u, 0u, (y | (y >> 8)) & 0xFFFFu));
    const uint32_t p8 = (c4 * 0x40100401u) >> 24;  // byte 0's code in bits 7..6
    w.code |= (uint64_t)p8 << (56 - 8 * q);
    w.nl |= byte_bits(__vcmpeq4(v, 0x0a0a0a0au)) << (4 * q);
    w.vb |= byte_bits(valid) << (4 * q);
  }
  uint64_t r = __brevll(~w.code);
  w.rcode = ((r >> 1) & 0x5555555555555555ull) | ((r & 0x5555555555555555ull) << 1);
  return w;
}

// Sequence-line bytes of a word given the line phase at its first byte;
// advances the phase past the word.
__device__ __forceinline__ uint32_t seq_mask(uint32_t nl, unsigned& ph) {
  uint32_t seq = 0, m = nl;
  unsigned start = 0, p = ph;
  while (m) {
    const unsigned q = __ffs(m) - 1;
    if (p == 1) seq |= (uint32_t)((1ull << q) - (1ull << start));
    p = (p + 1) & 3u;
    start = q + 1;
    m &= m - 1;
  }
  if (p == 1) seq |= (uint32_t)((1ull << 32) - (1ull << start));
  ph = p;
  return seq;
}

// bit j set iff bits j .. j+k-1 of a are all set
__device__ __forceinline__ uint64_t runs_of(uint64_t a, uint32_t k) {
  uint64_t r = a;
  uint32_t len = 1;
  while (2 * len <= k) {
    r &= r >> len;
    len *= 2;
  }
  if (len < k) r &= r >> (k - len);
  return r;
}

// bit j set iff bits j .. j+k-1 of a are all set
__device__ __forceinline__ u128 runs_of128(u128 a, uint32_t k) {
  u128 r = a;
  uint32_t len = 1;
  while (2 * len <= k) {
    r &= r >> len;
    len *= 2;
  }
  if (len < k) r &= r >> (k - len);
  return r;
}

}  // namespace kite
