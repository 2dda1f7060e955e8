// Keys in shared-memory tables: homes in key order, clusters put in order, and
// the rows of a tile written.  Shared by the tile sort and the merge.
#pragma once

#include "kite_internal.h"

namespace kite {

// A key at home in slot h is in [h, h + kProbeLimit): tables have that many
// slots behind their last home.
constexpr unsigned kProbeLimit = 32;

// A key's place in the tile's key range [lo, hi]: the 32 bits of its distance
// from lo that start at hi's top bit (a monotone map of the range).
template <class T>
struct RangeMap {
  T lo;
  int lz;
  __device__ __forceinline__ RangeMap(T mn, T mx) : lo(mn), lz(mx == mn ? 0 : clz_key(T(mx - mn))) {}
  __device__ __forceinline__ uint32_t at(T key) const {
    const T v = key - lo;
    if constexpr (sizeof(T) == 8) {
      return (uint32_t)((v << lz) >> 32);
    } else {
      const uint64_t vh = hi64(v), vl = (uint64_t)v;
      const uint64_t h = lz < 64 ? vh : vl, l = lz < 64 ? vl : 0ull;
      const uint32_t a = (lz & 32) ? (uint32_t)h : (uint32_t)(h >> 32), b = (lz & 32) ? (uint32_t)(l >> 32) : (uint32_t)h;
      return __funnelshift_l(b, a, lz & 31);
    }
  }
};

// width * 2^32 / gap, rounded down a little, so that the places x < gap of an
// interval are spread over `width` slots by __umulhi(x, scale).
__device__ __forceinline__ uint32_t home_scale(uint32_t width, uint32_t gap) {
  const float f = __fdividef((float)width * 4294967296.f, (float)gap) * 0.999999f;
  return gap == 0 ? 0u : f < 4294960000.f ? (uint32_t)f : 0xffffffffu;
}

// Home slot of a key: its place in the range scaled to the homes.
template <class T>
struct HomeLinear {
  RangeMap<T> map;
  uint32_t scale, last;
  __device__ __forceinline__ HomeLinear(const RangeMap<T>& m, T mx, uint32_t homes)
      : map(m), scale(home_scale(homes, m.at(mx))), last(homes - 1) {}
  __device__ __forceinline__ uint32_t operator()(T key) const {
    const uint32_t b = __umulhi(map.at(key), scale);
    return b < last ? b : last;  // a key outside the range cannot leave the table
  }
};

template <class T>
__device__ __forceinline__ void empty_tile(TileOut<T>* out) {
  TileOut<T> o;
  o.first_key = o.last_key = T(0);
  o.rows = 0;
  o.first_count = 0;
  o.rest_bytes = 0;
  *out = o;
}

__device__ __forceinline__ unsigned warp_inclusive(unsigned v, unsigned lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned y = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= (unsigned)o) v += y;
  }
  return v;
}

// The U rows of a sorted tile (row(u, &key, &count)) to global memory, and the
// tile's record; size(u, key - previous key, count) is row u's part of its bytes.  Each warp takes consecutive rows; a lane's previous key comes
// from the lane below, and from the round before for the first lane.  `rest`
// is a zeroed counter, zeroed again; one barrier inside, after the last row has
// been read.
template <int NT, class T, class F, class S>
__device__ __forceinline__ void write_rows(unsigned U, T* g, uint32_t* gc, unsigned* rest_sum, TileOut<T>* out, F&& row,
                                           S&& size) {
  const unsigned lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const unsigned per = (U + NT - 1) / NT * 32;  // rows per warp
  const unsigned ub = wid * per, ue = min(U, ub + per);
  unsigned rest = 0;
  if (ub < ue) {
    T below = T(0);  // the key before the round's first row
    uint32_t x;
    if (ub) row(ub - 1, &below, &x);
    for (unsigned u0 = ub; u0 < ue; u0 += 32) {
      const unsigned u = u0 + lane;
      T key = T(0);
      uint32_t c = 0;
      if (u < ue) row(u, &key, &c);
      T prev = shfl_up_key(key, 1);
      if (lane == 0) prev = below;
      below = shfl_key(key, 31);
      if (u < ue) {
        g[u] = key;
        gc[u] = c;
        rest += size(u, T(key - prev), c);
      }
    }
  }
  rest = __reduce_add_sync(0xffffffffu, rest);
  if (lane == 0 && rest) atomicAdd(rest_sum, rest);
  TileOut<T> o;
  if (threadIdx.x == 0) {
    uint32_t x;
    row(0, &o.first_key, &o.first_count);
    row(U - 1, &o.last_key, &x);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    o.rows = U;
    o.rest_bytes = *rest_sum;
    *out = o;
    *rest_sum = 0;
  }
}

// DVLE bytes of a tile's row after the first, for write_rows.
template <class T>
__device__ __forceinline__ unsigned dvle_size(unsigned u, T delta, uint32_t count) {
  return u ? varint_len(delta) + varint_len32(count) : 0u;
}

// Puts the cluster of occupied slots that starts at `first` in key order (an
// insertion sort by one thread; homes in key order leave it nearly so).
__device__ __forceinline__ void order_cluster(unsigned long long* tab, unsigned* cnt, uint32_t first, uint32_t slots) {
  unsigned long long last = tab[first];
  for (uint32_t e = first + 1; e < slots; ++e) {
    const unsigned long long v = tab[e];
    if (v == ~0ull) break;
    if (v > last) {
      last = v;
      continue;
    }
    const unsigned c = cnt[e];
    uint32_t q = e;
    do {
      tab[q] = tab[q - 1];
      cnt[q] = cnt[q - 1];
      --q;
    } while (q > first && tab[q - 1] > v);
    tab[q] = v;
    cnt[q] = c;
  }
}

}  // namespace kite
