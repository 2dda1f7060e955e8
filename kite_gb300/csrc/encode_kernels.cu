// DVLE encoding of every hash bucket's rows into one payload per partition
// (encode_dvle_u64 / encode_dvle_u128, src/format/run_block.rs:70-95:
// first key raw LE + count u32 LE, then LEB128(key delta) + LEB128(count)).
//
// Tiles of a bucket are in key order, so a bucket's payload is the
// concatenation of its tiles' encodings; only the first row of each tile needs
// the previous tile's last key.
#include "kite_internal.h"

namespace kite {

// One warp per bucket: walks the bucket's S tiles 32 at a time, links each
// non-empty tile to the last key of the previous non-empty tile, and computes
// tile byte offsets, row totals and the bucket's min/max key.
template <class T>
__global__ void k_tile_link(const TileOut<T>* __restrict__ tout, uint32_t P, uint32_t S,
                            const uint32_t* __restrict__ tile_first, unsigned long long* __restrict__ tile_boff,
                            T* __restrict__ tile_prev, BucketMeta* __restrict__ meta) {
  const int lane = threadIdx.x & 31;
  const uint32_t b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (b >= P) return;
  // tiles of bucket b: [t0, t0 + S) (fixed S) or [tile_first[b], tile_first[b+1])
  const size_t t0 = tile_first ? tile_first[b] : (size_t)b * S;
  if (tile_first) S = tile_first[b + 1] - tile_first[b];
  bool have_prev = false;
  T prev = T(0), kmin = T(0);
  unsigned long long boff = 0, rows = 0;
  const unsigned lt = (1u << lane) - 1u;
  for (uint32_t j0 = 0; j0 < S; j0 += 32) {
    const uint32_t j = j0 + lane;
    TileOut<T> o;
    o.first_key = o.last_key = T(0);
    o.rows = 0;
    o.first_count = 0;
    o.rest_bytes = 0;
    if (j < S) o = tout[t0 + j];
    const bool ne = o.rows > 0;
    const unsigned ball = __ballot_sync(0xffffffffu, ne);
    // previous non-empty lane's last key
    const unsigned below = ball & lt;
    const int src_lane = below ? 31 - __clz(below) : 0;
    const T lk = o.last_key;
    const T from_lane = shfl_key(lk, src_lane);
    const bool has_p = below ? true : have_prev;
    const T p = below ? from_lane : prev;
    unsigned long long bytes = 0;
    if (ne) {
      const int first = has_p ? varint_len((T)(o.first_key - p)) + varint_len((uint64_t)o.first_count)
                              : KeyTraits<T>::kEntry;
      bytes = (unsigned long long)first + o.rest_bytes;
    }
    // warp inclusive scan of bytes and rows
    unsigned long long inc = bytes, rinc = ne ? o.rows : 0;
    for (int d = 1; d < 32; d <<= 1) {
      const unsigned long long y = __shfl_up_sync(0xffffffffu, inc, d);
      const unsigned long long ry = __shfl_up_sync(0xffffffffu, rinc, d);
      if (lane >= d) {
        inc += y;
        rinc += ry;
      }
    }
    if (j < S) {
      tile_boff[t0 + j] = boff + inc - bytes;
      tile_prev[t0 + j] = p;
    }
    // first non-empty tile overall gives kmin
    if (!have_prev && ball) {
      const int fl = __ffs(ball) - 1;
      kmin = shfl_key(o.first_key, fl);
    }
    if (ball) {
      const int ll = 31 - __clz(ball);
      prev = shfl_key(lk, ll);
      have_prev = true;
    }
    boff += __shfl_sync(0xffffffffu, inc, 31);
    rows += __shfl_sync(0xffffffffu, rinc, 31);
  }
  if (lane == 0) {
    BucketMeta m;
    m.rows = rows;
    m.bytes = boff;
    m.byte_off = 0;
    m.kmin_lo = (unsigned long long)kmin;
    m.kmin_hi = hi64(kmin);
    m.kmax_lo = (unsigned long long)prev;
    m.kmax_hi = hi64(prev);
    meta[b] = m;
  }
}

template <class T>
void launch_tile_link(const TileOut<T>* tout, uint32_t P, uint32_t S, unsigned long long* tile_boff, T* tile_prev,
                      BucketMeta* meta, cudaStream_t s) {
  const unsigned threads = 256;
  const unsigned blocks = (unsigned)(((size_t)P * 32 + threads - 1) / threads);
  k_tile_link<T><<<blocks, threads, 0, s>>>(tout, P, S, nullptr, tile_boff, tile_prev, meta);
}

template <class T>
void launch_tile_link_ranges(const TileOut<T>* tout, uint32_t P, const uint32_t* tile_first,
                             unsigned long long* tile_boff, T* tile_prev, BucketMeta* meta, cudaStream_t s) {
  const unsigned threads = 256;
  const unsigned blocks = (unsigned)(((size_t)P * 32 + threads - 1) / threads);
  k_tile_link<T><<<blocks, threads, 0, s>>>(tout, P, 0, tile_first, tile_boff, tile_prev, meta);
}
template void launch_tile_link_ranges<uint64_t>(const TileOut<uint64_t>*, uint32_t, const uint32_t*,
                                                unsigned long long*, uint64_t*, BucketMeta*, cudaStream_t);
template void launch_tile_link_ranges<u128>(const TileOut<u128>*, uint32_t, const uint32_t*, unsigned long long*,
                                            u128*, BucketMeta*, cudaStream_t);
template void launch_tile_link<uint64_t>(const TileOut<uint64_t>*, uint32_t, uint32_t, unsigned long long*,
                                         uint64_t*, BucketMeta*, cudaStream_t);
template void launch_tile_link<u128>(const TileOut<u128>*, uint32_t, uint32_t, unsigned long long*, u128*,
                                     BucketMeta*, cudaStream_t);

// Exclusive scan of bucket byte sizes into byte_off (single CTA; P <= 1<<16).
// With a mirror (pinned host memory mapped into the device's address space),
// the finished records are also written there, so the host reads them when
// the kernel has completed without a copy that would queue on a copy engine.
__global__ void __launch_bounds__(1024) k_bucket_offsets(BucketMeta* meta, uint32_t P, BucketMeta* mirror) {
  __shared__ unsigned long long sm[34];
  unsigned long long carry = 0;
  for (uint32_t b0 = 0; b0 < P; b0 += 1024) {
    const uint32_t b = b0 + threadIdx.x;
    const unsigned long long v = b < P ? meta[b].bytes : 0;
    unsigned long long tot;
    const unsigned long long ex = block_exclusive_scan<1024, unsigned long long>(v, sm, &tot);
    if (b < P) {
      meta[b].byte_off = carry + ex;
      if (mirror) mirror[b] = meta[b];
    }
    carry += tot;
  }
}

void launch_bucket_offsets(BucketMeta* meta, uint32_t P, BucketMeta* host_mirror, cudaStream_t s) {
  k_bucket_offsets<<<1, 1024, 0, s>>>(meta, P, host_mirror);
}

// Four 7-bit groups (28 bits of x) as the low bits of four bytes.
__device__ __forceinline__ uint32_t spread28(uint32_t x) {
  x = (x & 0x3fffu) | ((x << 2) & 0x3fff0000u);
  return (x & 0x007f007fu) | ((x << 1) & 0x7f007f00u);
}
// Word j of the continuation bits of an n-byte varint.
__device__ __forceinline__ uint32_t more_bits(int n, int j) {
  return __funnelshift_rc(0x80808080u, 0u, (unsigned)max(0, 32 - 8 * (n - 1 - 4 * j)));
}
// An n-byte varint as little-endian words.
template <class T>
struct VarintWords {
  static constexpr int N = ((KeyTraits<T>::kBits + 6) / 7 + 3) / 4;
  uint32_t w[N];
  __device__ __forceinline__ VarintWords(T v, int n) {
#pragma unroll
    for (int j = 0; j < N; ++j) w[j] = spread28((uint32_t)(uint64_t)(v >> (28 * j))) | more_bits(n, j);
  }
};
// Words w at byte offset o of a zeroed buffer; words next to each other are
// shared with other rows.
template <int N>
__device__ __forceinline__ void put_words(uint32_t* buf, uint32_t o, const uint32_t (&w)[N]) {
  uint32_t* b = buf + (o >> 2);
  const uint32_t sh = (o & 3u) * 8;
  uint32_t below = 0;
#pragma unroll
  for (int j = 0; j <= N; ++j) {
    const uint32_t x = __funnelshift_l(below, j < N ? w[j] : 0u, sh);
    if (x) atomicOr(b + j, x);
    if (j < N) below = w[j];
  }
}

// One CTA per tile, ROUND rows at a time, a lane per row (128 consecutive rows
// per warp, so that loads are coalesced and a row's previous key is the lane
// below's).  The four rows' sizes of a lane go through one packed warp scan;
// a row's varints are spread from 28 bits to four bytes at a time and ORed into
// zeroed shared memory that lies as the output does modulo 4, so that it leaves
// as whole words.  A byte loop per varint, byte stores and four byte loads per
// output word took 84% of the issue slots; with those gone it is the latency of
// a round's loads, scan and barriers, so that small CTAs (a tile takes a few
// rounds of one) are best.  325M u64 rows of 10M reads 2.0 -> 1.7 ms (256 threads
// 1.9, 512 2.3), 95M u128 rows at k = 63 1.7 -> 0.8 (128 threads 0.83, 256 0.91).
template <class T>
struct EncShape {
  static constexpr int NT = sizeof(T) == 8 ? 128 : 64, ROWS = 4, ROUND = NT * ROWS, PER_SM = sizeof(T) == 8 ? 14 : 18;
};
template <class T>
__global__ void __launch_bounds__(EncShape<T>::NT, EncShape<T>::PER_SM) k_encode(const T* __restrict__ keys, const uint32_t* __restrict__ counts,
                                                        const TileDesc* __restrict__ tiles,
                                                        const TileOut<T>* __restrict__ tout,
                                                        const unsigned long long* __restrict__ tile_boff,
                                                        const T* __restrict__ tile_prev,
                                                        const BucketMeta* __restrict__ meta, uint8_t* __restrict__ out,
                                                        unsigned long long out_cap, DevStatus* st) {
  constexpr int NT = EncShape<T>::NT, ROWS = EncShape<T>::ROWS, ROUND = EncShape<T>::ROUND;
  // largest row: LEB128 of a key delta plus LEB128 of a u32 count, or the raw first row
  constexpr int kRowMax = (KeyTraits<T>::kBits + 6) / 7 + 5;
  static_assert(kRowMax * 32 < 65536, "packed sizes");
  __shared__ __align__(16) uint32_t chunk[(ROUND * kRowMax + 3) / 4 + 5];
  __shared__ unsigned edge[NT / 32];
  const uint32_t t = blockIdx.x;
  const TileOut<T> o = tout[t];
  if (o.rows == 0) return;
  const TileDesc td = tiles[t];
  const unsigned long long base = meta[td.bucket].byte_off + tile_boff[t];
  const bool first_in_bucket = tile_boff[t] == 0;
  const T tprev = tile_prev[t];
  const T* k = keys + td.start;
  const uint32_t* c = counts + td.start;
  const unsigned lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (unsigned i = threadIdx.x; i < (min(o.rows, (uint32_t)ROUND) * kRowMax + 3) / 16 + 1; i += NT)
    reinterpret_cast<uint4*>(chunk)[i] = make_uint4(0, 0, 0, 0);
  unsigned long long run = 0;
  for (uint32_t r0 = 0; r0 < o.rows; r0 += ROUND) {
    const uint32_t rb = r0 + wid * 128;  // the warp's first row
    T key[ROWS];
    uint32_t cnt[ROWS];
#pragma unroll
    for (int i = 0; i < ROWS; ++i) {
      const uint32_t r = rb + i * 32 + lane;
      key[i] = r < o.rows ? k[r] : T(0);
      cnt[i] = r < o.rows ? c[r] : 0u;
    }
    T below = rb == 0 ? tprev : rb < o.rows ? k[rb - 1] : T(0);
    const T raw = key[0];
    int n1[ROWS];
    unsigned long long packed = 0;  // the rows' sizes, 16 bits each
#pragma unroll
    for (int i = 0; i < ROWS; ++i) {
      const uint32_t r = rb + i * 32 + lane;
      T prev = shfl_up_key(key[i], 1);
      if (lane == 0) prev = below;
      below = shfl_key(key[i], 31);
      key[i] -= prev;
      n1[i] = varint_len(key[i]);
      const unsigned sz = r >= o.rows ? 0u : r == 0 && first_in_bucket ? (unsigned)KeyTraits<T>::kEntry
                                                                       : (unsigned)(n1[i] + varint_len32(cnt[i]));
      packed |= (unsigned long long)sz << (16 * i);
    }
    unsigned long long inc = packed;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const unsigned long long y = __shfl_up_sync(0xffffffffu, inc, d);
      if (lane >= (unsigned)d) inc += y;
    }
    const unsigned long long all = __shfl_sync(0xffffffffu, inc, 31);
    const unsigned mine = (unsigned)(all & 0xffff) + (unsigned)(all >> 16 & 0xffff) + (unsigned)(all >> 32 & 0xffff) +
                          (unsigned)(all >> 48);
    if (lane == 0) edge[wid] = mine;
    __syncthreads();  // the totals are there, and the chunk is zeroed
    unsigned at0 = 0, tot = 0;
#pragma unroll
    for (int w = 0; w < NT / 32; ++w) {
      const unsigned x = edge[w];
      at0 += (unsigned)w < wid ? x : 0u;
      tot += x;
    }
    const unsigned long long at = base + run;
    const unsigned skew = (unsigned)((uintptr_t)(out + at) & 3u);
    at0 += skew;
    const unsigned long long ex = inc - packed;
#pragma unroll
    for (int i = 0; i < ROWS; ++i) {
      const uint32_t r = rb + i * 32 + lane;
      const unsigned w = at0 + (unsigned)(ex >> (16 * i) & 0xffff);
      at0 += (unsigned)(all >> (16 * i) & 0xffff);
      if (r >= o.rows) continue;
      if (r == 0 && first_in_bucket) {
        uint32_t v[sizeof(T) / 4 + 1];
#pragma unroll
        for (int j = 0; j < (int)sizeof(T) / 4; ++j) v[j] = (uint32_t)(uint64_t)(raw >> (32 * j));
        v[sizeof(T) / 4] = cnt[i];
        put_words(chunk, w, v);
        continue;
      }
      if constexpr (sizeof(T) == 8) {
        if (n1[i] < 8 && cnt[i] < 128) {
          // nearly all rows: both varints in eight bytes
          const unsigned long long v =
              ((unsigned long long)spread28((uint32_t)(key[i] >> 28)) << 32 | spread28((uint32_t)key[i])) |
              0x0080808080808080ull >> (8 * (8 - n1[i])) | (unsigned long long)cnt[i] << (8 * n1[i]);
          const uint32_t lo = (uint32_t)v, hi = (uint32_t)(v >> 32), sh = (w & 3u) * 8;
          uint32_t* b = chunk + (w >> 2);
          atomicOr(b, lo << sh);
          const uint32_t x1 = __funnelshift_l(lo, hi, sh), x2 = __funnelshift_l(hi, 0u, sh);
          if (x1) atomicOr(b + 1, x1);
          if (x2) atomicOr(b + 2, x2);
          continue;
        }
      }
      put_words(chunk, w, VarintWords<T>(key[i], n1[i]).w);
      const unsigned wc = w + n1[i];
      if (cnt[i] < 128) {
        if (cnt[i]) atomicOr(chunk + (wc >> 2), cnt[i] << ((wc & 3u) * 8));
      } else {
        put_words(chunk, wc, VarintWords<uint64_t>(cnt[i], varint_len32(cnt[i])).w);
      }
    }
    __syncthreads();
    if (at + tot > out_cap) {
      if (threadIdx.x == 0) dev_fail(st, KITE_DEV_ENCODE_OVERFLOW, t, r0, 0);
      return;
    }
    // whole words, and the bytes of the first and the last one that are this round's
    uint32_t* dw = reinterpret_cast<uint32_t*>(out + at - skew);
    const unsigned end = skew + tot, whole = end >> 2;
    for (unsigned i = threadIdx.x + (skew != 0); i < whole; i += NT) {
      dw[i] = chunk[i];
      chunk[i] = 0;
    }
    if (threadIdx.x >= NT - 2) {
      const unsigned i = threadIdx.x & 1u ? whole : 0u;
      const bool part = threadIdx.x & 1u ? whole != 0 && (end & 3u) != 0 : skew != 0 || whole == 0;
      if (part) {
        const uint32_t v = chunk[i];
        chunk[i] = 0;
        for (unsigned j = 4 * i; j < 4 * i + 4; ++j)
          if (j >= skew && j < end) reinterpret_cast<uint8_t*>(dw)[j] = (uint8_t)(v >> (8 * (j & 3u)));
      }
    }
    run += tot;
    __syncthreads();  // the chunk is refilled, and the totals change, next round
  }
}

template <class T>
void launch_encode(const T* keys, const uint32_t* counts, const TileDesc* tiles, const TileOut<T>* tout,
                   const unsigned long long* tile_boff, const T* tile_prev, const BucketMeta* meta, uint32_t ntiles,
                   uint8_t* out, unsigned long long out_cap, DevStatus* st, cudaStream_t s) {
  if (ntiles)
    k_encode<T><<<ntiles, EncShape<T>::NT, 0, s>>>(keys, counts, tiles, tout, tile_boff, tile_prev, meta, out, out_cap,
                                                st);
}
template void launch_encode<uint64_t>(const uint64_t*, const uint32_t*, const TileDesc*, const TileOut<uint64_t>*,
                                      const unsigned long long*, const uint64_t*, const BucketMeta*, uint32_t,
                                      uint8_t*, unsigned long long, DevStatus*, cudaStream_t);
template void launch_encode<u128>(const u128*, const uint32_t*, const TileDesc*, const TileOut<u128>*,
                                  const unsigned long long*, const u128*, const BucketMeta*, uint32_t, uint8_t*,
                                  unsigned long long, DevStatus*, cudaStream_t);

}  // namespace kite
