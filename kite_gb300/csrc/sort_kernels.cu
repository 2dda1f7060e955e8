// On-chip tile sort + run-length reduction (the sort/RLE of a flushed bucket:
// radix_sort_u64_kmer / radix_sort_u128_kmer src/count/sorter.rs:67-93,
// :388-437, then rle_compress_typed :514-530 with u32 saturation).
//
// A tile is a key range of one hash bucket, sorted by one CTA.  Tiles whose keys
// repeat (reads at some depth) are counted in a table of distinct keys; the
// others are ordered by a 16384-bin counting pass over their key span (bins
// holding several distinct keys are finished by a thread or a warp, rare
// pathological ones by LSD passes).  Either way unique (key, count) rows come
// out in place, with the tile's DVLE size for every row but the first.
#include <algorithm>

#include "key_table.cuh"
#include "kite_internal.h"

namespace kite {

template <class T>
__device__ __forceinline__ T warp_min(T v) {
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    const T w = shfl_xor_key(v, o);
    v = w < v ? w : v;
  }
  return v;
}
template <class T>
__device__ __forceinline__ T warp_max(T v) {
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    const T w = shfl_xor_key(v, o);
    v = w > v ? w : v;
  }
  return v;
}

// Block-wide min and max of the thread values (smem needs 2*NW keys).
template <int NT, class T>
__device__ __forceinline__ void block_minmax(T& mn, T& mx, T* red) {
  constexpr int NW = NT / 32;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  mn = warp_min(mn);
  mx = warp_max(mx);
  if (lane == 0) {
    red[wid] = mn;
    red[NW + wid] = mx;
  }
  __syncthreads();
  mn = red[0];
  mx = red[NW];
  for (int w = 1; w < NW; ++w) {
    mn = red[w] < mn ? red[w] : mn;
    mx = red[NW + w] > mx ? red[NW + w] : mx;
  }
  __syncthreads();
}

template <class T>
__device__ __forceinline__ int varying_bits(T mn, T mx) {
  const T x = mn ^ mx;
  return x == T(0) ? 0 : KeyTraits<T>::kBits - clz_key(x);
}

template <class T>
struct TileSmem {
  static constexpr int NT = kTileThreads;
  static constexpr int ITEMS = tile_items<T>();
  static constexpr int CAP = NT * ITEMS;
  static constexpr int NW = NT / 32;
  static constexpr size_t buf_bytes = (size_t)CAP * sizeof(T);
  static constexpr size_t hist_bytes = (size_t)256 * NW * 4;
  static constexpr size_t head_bytes = ((size_t)(CAP + 1) * 2 + 15) & ~(size_t)15;
  static constexpr size_t misc_bytes = 64 * 8 + 2 * NW * sizeof(T) + 256 * 8;
  static constexpr size_t total = buf_bytes + hist_bytes + head_bytes + misc_bytes;
};

// Stable LSD passes over bits [lo_bit, nbits) of the n keys in buf (shared
// memory), 8-bit digits.
template <class T, int NT, int ITEMS>
__device__ __forceinline__ void smem_radix_sort(T* buf, unsigned n, int nbits, unsigned* warp_hist,
                                                unsigned* scan_sm, int lo_bit = 0) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  // spread the n keys over every warp: `items` rounds of 32 per warp
  const int items = (int)((n + NT - 1) / NT);
  const unsigned pos0 = (unsigned)wid * 32u * (unsigned)items + lane;
  for (int shift = lo_bit; shift < nbits; shift += 8) {
    T key[ITEMS];
    unsigned dig[ITEMS], dest[ITEMS];
    bool valid[ITEMS];
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
      const unsigned pos = pos0 + r * 32u;
      valid[r] = r < items && pos < n;
      key[r] = valid[r] ? buf[pos] : T(0);
      dig[r] = digit_of(key[r], shift);
    }
    block_rank<NT, ITEMS, 256>(dig, valid, dest, warp_hist, scan_sm, nullptr, nullptr, items);
#pragma unroll
    for (int r = 0; r < ITEMS; ++r)
      if (valid[r]) buf[dest[r]] = key[r];
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Tile sort by binning.  One CTA per tile of n <= CAP keys:
//  1. load the tile into shared memory (one bulk copy), then count the keys per bin:
//     bin = (key - lo) >> s with 16384 bins spanning the tile's key range
//     [lo, hi] (its splitters);
//  2. an exclusive scan of the bin counts; then the keys themselves are
//     scattered into bin order (every thread first takes its keys from the
//     staged tile into registers, so none is overwritten before it is read).
//     Bins are key-ordered; order inside a bin is arbitrary, so every later
//     pass reads shared memory directly;
//  3. a bin holding more than one distinct key is found where two different
//     neighbours share it, and marked (a shared bit per bin);
//  4. a marked bin of at most kSmallBin keys (typically two colliding
//     k-mers) is insertion-sorted by the thread owning its bit; a larger one
//     (typically a repeated k-mer and a colliding one) by the warp owning its
//     bit word.  Up to 32 keys sit one per lane: lanes with equal keys find
//     each other by a match, and each key's new position is the copies of
//     the smaller distinct keys plus its equal predecessors.  A larger bin
//     has its distinct keys extracted in ascending order with their counts
//     and is rewritten with them (equal keys are interchangeable).  A bin of
//     more than kMaxDistinct distinct keys is ranked by counting when it
//     holds at most kMaxMixed keys and otherwise sends the tile to LSD passes;
//  5. run-length reduction over the sorted keys: head flags by warp ballots,
//     rows written to global memory over the tile's keys (u32 counts; a tile
//     holds fewer than 2^32 keys, so no count saturates here).
// ---------------------------------------------------------------------------
// 16384 bins with 16-bit counters packed two to a word (a tile holds at most
// 16384 keys, so no half carries into the other)
constexpr int kBinBits = 14, kBins = 1 << kBinBits;
constexpr unsigned kSmallBin = 16;     // marked bins a single thread sorts
constexpr unsigned kMaxMixed = 256;    // largest bin ranked by counting when it has many distinct keys
constexpr unsigned kMaxDistinct = 32;  // distinct keys a warp extracts from one large bin

// MULT = 1: the regular tile (8192 u64 / 4096 u128 keys, two CTAs per SM);
// MULT = 2: twice that, with twice the threads, for the oversized tiles (one
// CTA per SM).
template <class T, int MULT>
struct BinSmem {
  static constexpr int NT = kTileThreads * MULT;
  static constexpr int ITEMS = tile_items<T>();
  static constexpr int CAP = NT * ITEMS;
  static constexpr int NW = NT / 32;
  // the keys, plus 16 bytes: the bulk copy of a tile starts at the 16-byte
  // boundary at or below its first key
  static constexpr size_t buf_bytes = (size_t)CAP * sizeof(T) + 16;
  // bin counters; later the u16 run heads (CAP + 1 entries), or the LSD
  // fallback's per-warp digit histograms (256 * NW counters)
  static constexpr size_t head_need = ((size_t)(CAP + 1) * 2 + 15) & ~(size_t)15;
  static constexpr size_t bin_bytes = ((size_t)kBins * 2 > head_need ? (size_t)kBins * 2 : head_need) + 16;
  static constexpr size_t fbit_bytes = kBins / 8;
  static constexpr unsigned MAXLARGE = CAP / (kSmallBin + 1) + 1;  // marked bins above kSmallBin keys
  static constexpr size_t misc_bytes = 64 * 8 + 16 + ((MAXLARGE * 2 + 15) & ~(size_t)15) + 16;  // + mbarrier
  static constexpr size_t total = buf_bytes + bin_bytes + fbit_bytes + misc_bytes;
  static_assert((size_t)(CAP + 1) * 2 <= bin_bytes, "run heads must fit the bin area");
  static_assert((size_t)256 * NW * 4 <= bin_bytes, "LSD histograms must fit the bin area");
  static_assert(kBins / 2 % (4 * NT) == 0, "bin scan takes whole uint4 groups");
  static_assert(CAP <= 65535, "bin offsets fit 16 bits");
  static_assert(kBins % (32 * NW) == 0, "every warp owns whole words of bin marks");
  static_assert(kBins % NT == 0 && kBins / NT <= 32 && 32 % (kBins / NT) == 0, "every thread owns bin marks in one word");
};

template <class T>
__device__ __forceinline__ unsigned bin_of(T key, T mn, int s) {
  return (unsigned)(uint64_t)((key - mn) >> s);
}

// Packed 16-bit bin counters: bin b is half (b & 1) of word b >> 1.
__device__ __forceinline__ unsigned bin_add(unsigned* bins, unsigned b) {
  const unsigned sh = (b & 1u) << 4;
  return (atomicAdd(&bins[b >> 1], 1u << sh) >> sh) & 0xffffu;
}
__device__ __forceinline__ unsigned bin_get(const unsigned* bins, unsigned b) {
  return (bins[b >> 1] >> ((b & 1u) << 4)) & 0xffffu;
}

template <class T>
__device__ __forceinline__ unsigned match_key(T v) {
  unsigned eq = __match_any_sync(0xffffffffu, (unsigned long long)(uint64_t)v);
  if (sizeof(T) > 8) eq &= __match_any_sync(0xffffffffu, (unsigned long long)hi64(v));
  return eq;
}

// One warp orders buf[a, a + m), m <= 32, one key per lane: a key's new
// position is the copies of the smaller distinct keys (one shuffle per
// distinct key, from its lowest lane) plus its equal predecessors.
template <class T>
__device__ __forceinline__ void warp_match_sort(T* buf, unsigned a, unsigned m, unsigned lane) {
  const bool act = lane < m;
  const T mine = act ? buf[a + lane] : T(0);
  const unsigned amask = m >= 32 ? 0xffffffffu : ((1u << m) - 1u);
  const unsigned eq = match_key(mine) & amask;
  const unsigned leaders = __ballot_sync(0xffffffffu, act && (unsigned)(__ffs(eq) - 1) == lane);
  const unsigned cnt = __popc(eq);
  unsigned less = 0;
  for (unsigned L = leaders; L; L &= L - 1) {
    const int l = __ffs(L) - 1;
    const T kl = shfl_key(mine, l);
    const unsigned cl = __shfl_sync(0xffffffffu, cnt, l);
    less += kl < mine ? cl : 0u;
  }
  const unsigned pos = a + less + __popc(eq & ((1u << lane) - 1u));
  __syncwarp();
  if (act) buf[pos] = mine;
  __syncwarp();
}

// One warp orders buf[a, a + m), m <= kMaxMixed, by counting: each key's new
// position is the number of smaller keys plus the equal keys before it.
template <class T>
__device__ __forceinline__ void warp_count_sort(T* buf, unsigned a, unsigned m, unsigned lane) {
  constexpr int R = kMaxMixed / 32;
  T key[R];
  unsigned rk[R];
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const unsigned q = lane + 32u * i;
    key[i] = q < m ? buf[a + q] : T(0);
    rk[i] = 0;
  }
  for (unsigned t = 0; t < m; ++t) {
    const T v = buf[a + t];
#pragma unroll
    for (int i = 0; i < R; ++i) rk[i] += (unsigned)(v < key[i]) | ((unsigned)(v == key[i]) & (unsigned)(t < lane + 32u * i));
  }
  __syncwarp();
#pragma unroll
  for (int i = 0; i < R; ++i)
    if (lane + 32u * i < m) buf[a + rk[i]] = key[i];
  __syncwarp();
}

// One warp orders buf[a, a + m) by extracting its distinct keys in ascending
// order with their counts and rewriting the range with them.  False (range
// untouched) when the range holds more than kMaxDistinct distinct keys.
template <class T>
__device__ __forceinline__ bool warp_distinct_sort(T* buf, unsigned a, unsigned m, unsigned lane) {
  const unsigned e = a + m;
  T myv = T(0), cur = T(0);
  unsigned myc = 0, U = 0;
  bool have = false;
  for (;;) {
    // smallest key above `cur` in the range, and its number of copies
    T best = T(0);
    unsigned cnt = 0;
    for (unsigned j = a + lane; j < e; j += 32) {
      const T v = buf[j];
      if (have && !(cur < v)) continue;
      if (cnt == 0 || v < best) {
        best = v;
        cnt = 1;
      } else if (v == best) {
        ++cnt;
      }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      const T ob = shfl_xor_key(best, o);
      const unsigned oc = __shfl_xor_sync(0xffffffffu, cnt, o);
      if (oc && (cnt == 0 || ob < best)) {
        best = ob;
        cnt = oc;
      } else if (oc && ob == best) {
        cnt += oc;
      }
    }
    if (cnt == 0) break;
    if (U == kMaxDistinct) return false;
    if (lane == U) {
      myv = best;
      myc = cnt;
    }
    ++U;
    cur = best;
    have = true;
  }
  __syncwarp();
  unsigned off = a;
  for (unsigned u = 0; u < U; ++u) {
    const T v = shfl_key(myv, (int)u);
    const unsigned c = __shfl_sync(0xffffffffu, myc, (int)u);
    for (unsigned t = lane; t < c; t += 32) buf[off + t] = v;
    off += c;
  }
  __syncwarp();
  return true;
}

// ---- bulk (TMA) copy of a tile's keys into shared memory, completed on an
// mbarrier (PTX cp.async.bulk / mbarrier) ----
__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t* bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(bar)) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  // earlier generic-proxy accesses to the destination come before the copy
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(smem_addr(dst)), "l"(src), "r"(bytes), "r"(smem_addr(bar))
               : "memory");
}
// Waits for phase `parity` of the barrier, giving up after `limit` polls
// (each a try_wait, which may suspend the thread for a while); limit 1 is a
// single non-blocking test.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, uint32_t limit) {
  if (limit == 1) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(done)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return done != 0;
  }
  for (uint32_t it = 0; it < limit; ++it) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(done)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}
constexpr uint32_t kBulkWaitPolls = 1u << 18;                // a bulk copy from device memory ends long before
constexpr uint32_t kBulkDrainPolls = 1u << 26;               // after a timeout: the copy must leave shared memory
constexpr unsigned long long kBulkTimeoutFlag = 1ull << 40;  // added to the sort statistics on a timeout

template <class T, int MULT>
__device__ __forceinline__ void sort_tile(uint32_t tid, T* __restrict__ keys, uint32_t* __restrict__ counts,
                                          const TileDesc* __restrict__ tiles, TileOut<T>* __restrict__ tout,
                                          unsigned long long* fallbacks, const TileRanges<T>& rg, DevStatus* st) {
  using L = BinSmem<T, MULT>;
  constexpr int NT = L::NT, NW = L::NW, ITEMS = L::ITEMS;
  extern __shared__ __align__(16) uint8_t sm[];
  T* buf = reinterpret_cast<T*>(sm);
  unsigned* bins = reinterpret_cast<unsigned*>(sm + L::buf_bytes);
  unsigned* fbits = reinterpret_cast<unsigned*>(sm + L::buf_bytes + L::bin_bytes);
  unsigned long long* scan64 = reinterpret_cast<unsigned long long*>(sm + L::buf_bytes + L::bin_bytes + L::fbit_bytes);
  unsigned* scan_sm = reinterpret_cast<unsigned*>(scan64);
  unsigned* misc = reinterpret_cast<unsigned*>(scan64 + 64);  // [0] LSD fallback, [1] large bins
  unsigned short* large = reinterpret_cast<unsigned short*>(misc + 4);
  uint64_t* bar = reinterpret_cast<uint64_t*>(sm + L::total - 16);

  const TileDesc td = tiles[tid];
  const unsigned n = td.len;
  if (n == 0 || n > (unsigned)L::CAP) {  // the lists have no such tile
    if (threadIdx.x == 0) {
      empty_tile(&tout[tid]);
      dev_fail(st, KITE_DEV_TILE_OVERFLOW, tid, n, L::CAP);
    }
    return;
  }
  T* g = keys + td.start;
  uint32_t* gc = counts + td.start;
  // the tile's key range from its splitters
  const uint32_t tl = rg.S > 1 ? (rg.tile0 + tid) % rg.S : 0u;
  const T mn = tl > 0 ? rg.spl[tl - 1] : T(0);
  T mx = rg.kmax;
  if (tl + 1 < rg.S) {
    const T e = rg.spl[tl];
    mx = e > mn ? T(e - T(1)) : mn;
  }
  const int rb = mx == mn ? 0 : KeyTraits<T>::kBits - clz_key(T(mx - mn));
  const int s = rb > kBinBits ? rb - kBinBits : 0;
  auto bin_at = [&](T key) -> unsigned {  // clamped: a key outside the range cannot leave the table
    const unsigned b = key < mn ? 0u : bin_of(key, mn, s);
    return b < (unsigned)kBins ? b : (unsigned)kBins - 1u;
  };

  // ---- 1. bulk load with the bin histogram; 2. scan, key scatter into bin order ----
  // The tile's keys arrive by one bulk copy of the 16-byte aligned span that
  // holds them (key buffers are allocated with slack past their end), while
  // the threads clear the bins.
  const uintptr_t ga = reinterpret_cast<uintptr_t>(g);
  const uintptr_t s0 = ga & ~(uintptr_t)15, s1 = (ga + (uintptr_t)n * sizeof(T) + 15) & ~(uintptr_t)15;
  const T* tk = reinterpret_cast<const T*>(sm + (ga - s0));  // the tile's keys in shared memory
  if (threadIdx.x == 0) mbar_init(bar);
  for (int b = threadIdx.x; b < kBins / 2; b += NT) bins[b] = 0;
  for (int b = threadIdx.x; b < kBins / 32; b += NT) fbits[b] = 0;
  if (threadIdx.x < 4) misc[threadIdx.x] = 0;
  __syncthreads();
  if (threadIdx.x == 0) bulk_load(sm, reinterpret_cast<const void*>(s0), (uint32_t)(s1 - s0), bar);
  const bool arrived = mbar_wait(bar, 0, rg.wait_polls ? rg.wait_polls : kBulkWaitPolls);
  if (__syncthreads_or(!arrived)) {
    // the wait gave up: report, wait (with a far larger bound) until the copy
    // has landed so that no write to this CTA's shared memory is still in
    // flight when it moves on, and leave the tile empty (the count fails)
    if (threadIdx.x == 0) {
      mbar_wait(bar, 0, kBulkDrainPolls);
      if (fallbacks) atomicAdd(fallbacks, kBulkTimeoutFlag);
      empty_tile(&tout[tid]);  // for the link and encode kernels that follow
    }
    __syncthreads();
    return;
  }
  for (unsigned i = threadIdx.x; i < n; i += NT) bin_add(bins, bin_at(tk[i]));
  __syncthreads();
  {
    constexpr int G = kBins / 2 / (4 * NT);  // uint4 groups (8 bins each) per thread
    uint4* b4 = reinterpret_cast<uint4*>(bins) + threadIdx.x * G;
    uint4 x[G];
    unsigned sum = 0;
#pragma unroll
    for (int j = 0; j < G; ++j) {
      x[j] = b4[j];
      const unsigned w2 = x[j].x + x[j].y + x[j].z + x[j].w;  // both halves, no carry across
      sum += (w2 & 0xffffu) + (w2 >> 16);
    }
    unsigned tot;
    unsigned pre = block_exclusive_scan<NT, unsigned>(sum, scan_sm, &tot);
    // each word becomes (start of its even bin) | (start of its odd bin) << 16
    auto put = [&](unsigned w) {
      const unsigned r = pre | ((pre + (w & 0xffffu)) << 16);
      pre += (w & 0xffffu) + (w >> 16);
      return r;
    };
#pragma unroll
    for (int j = 0; j < G; ++j) {
      uint4 y;
      y.x = put(x[j].x);
      y.y = put(x[j].y);
      y.z = put(x[j].z);
      y.w = put(x[j].w);
      b4[j] = y;
    }
  }
  __syncthreads();
  {
    // every thread takes its keys from the staged tile before any is
    // overwritten, then scatters them into bin order
    T v[ITEMS];
#pragma unroll
    for (int u = 0; u < ITEMS; ++u) {
      const unsigned i = threadIdx.x + u * NT;
      v[u] = i < n ? tk[i] : T(0);
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < ITEMS; ++u)
      if (threadIdx.x + u * NT < n) buf[bin_add(bins, bin_at(v[u]))] = v[u];
  }
  __syncthreads();
  // bin_get(b) is now the end of bin b; its start is the end of bin b - 1 (0 for b = 0)

  // ---- 3. mark the bins holding more than one distinct key ----
  for (unsigned p = threadIdx.x + 1; p < n; p += NT) {
    const T a = buf[p], b = buf[p - 1];
    if (a != b) {
      const unsigned ba = bin_at(a);
      if (bin_at(b) == ba) {
        const unsigned bit = 1u << (ba & 31);
        if (!(atomicOr(&fbits[ba >> 5], bit) & bit)) {
          const unsigned m = bin_get(bins, ba) - (ba ? bin_get(bins, ba - 1) : 0u);
          if (m > kSmallBin) large[atomicAdd(&misc[1], 1u)] = (unsigned short)ba;
        }
      }
    }
  }
  __syncthreads();

  // ---- 4. order the marked bins: small ones by the thread owning their
  // bits, the listed larger ones by the warps in turn ----
  {
    constexpr int BPT = kBins / NT;
    const unsigned lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const unsigned b0 = threadIdx.x * BPT;
    for (unsigned bits = (fbits[b0 >> 5] >> (b0 & 31)) & (BPT == 32 ? 0xffffffffu : ((1u << BPT) - 1u)); bits;
         bits &= bits - 1) {
      const unsigned bb = b0 + (__ffs(bits) - 1);
      const unsigned a = bb ? bin_get(bins, bb - 1) : 0u, e = bin_get(bins, bb);
      if (e - a > kSmallBin) continue;
      for (unsigned j = a + 1; j < e; ++j) {
        const T v = buf[j];
        unsigned q = j;
        while (q > a) {
          const T w = buf[q - 1];
          if (!(v < w)) break;
          buf[q] = w;
          --q;
        }
        buf[q] = v;
      }
    }
    const unsigned nlarge = misc[1];
    for (unsigned li = wid; li < nlarge; li += NW) {
      const unsigned bb = large[li];
      const unsigned a = bb ? bin_get(bins, bb - 1) : 0u, m = bin_get(bins, bb) - a;
      if (m <= 32) warp_match_sort(buf, a, m, lane);
      else if (!warp_distinct_sort(buf, a, m, lane)) {
        if (m <= kMaxMixed) warp_count_sort(buf, a, m, lane);
        else if (lane == 0) misc[0] = 1;
      }
    }
  }
  __syncthreads();
  if (misc[0]) {
    // a large bin of many distinct keys: full LSD over the varying bits, in place
    if (threadIdx.x == 0 && fallbacks) atomicAdd(fallbacks, 1ull);
    smem_radix_sort<T, NT, ITEMS>(buf, n, varying_bits(mn, mx), bins, scan_sm, 0);
  }

  // ---- 5. run-length reduction over the sorted keys ----
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const unsigned rounds = (n + NT - 1) / NT;
  const unsigned w0 = (unsigned)wid * 32u * rounds;
  unsigned hmask = 0, cnt = 0;
  for (unsigned r = 0; r < rounds; ++r) {
    const unsigned p = w0 + r * 32u + lane;
    bool h = false;
    if (p < n) h = p == 0 || buf[p] != buf[p - 1];
    hmask |= (unsigned)h << r;
    cnt += __popc(__ballot_sync(0xffffffffu, h));
  }
  unsigned U;
  unsigned u = block_exclusive_scan<NT, unsigned>(lane == 0 ? cnt : 0u, scan_sm, &U);
  u = __shfl_sync(0xffffffffu, u, 0);
  unsigned short* head = reinterpret_cast<unsigned short*>(bins);
  const unsigned lt = (1u << lane) - 1u;
  for (unsigned r = 0; r < rounds; ++r) {
    const bool h = (hmask >> r) & 1u;
    const unsigned bal = __ballot_sync(0xffffffffu, h);
    if (h) head[u + __popc(bal & lt)] = (unsigned short)(w0 + r * 32u + lane);
    u += __popc(bal);
  }
  if (threadIdx.x == 0) head[U] = (unsigned short)n;
  __syncthreads();
  unsigned long long rest = 0;
  // a warp takes 32 consecutive rows: the next row's start and the previous
  // row's key come from the neighbouring lanes (the warp's ends read them)
  for (unsigned v0 = threadIdx.x - (unsigned)lane; v0 < U; v0 += NT) {
    const unsigned v = v0 + (unsigned)lane;
    const bool act = v < U;
    const unsigned i = act ? (unsigned)head[v] : 0u;
    const T key = act ? buf[i] : T(0);
    unsigned nxt = __shfl_down_sync(0xffffffffu, i, 1);
    if (lane == 31 || v + 1 >= U) nxt = act ? (unsigned)head[v + 1] : 0u;
    T prev = shfl_up_key(key, 1);
    if (lane == 0 && act && v > 0) prev = buf[head[v - 1]];
    if (act) {
      const unsigned c = nxt - i;
      g[v] = key;
      gc[v] = c;
      if (v > 0) rest += (unsigned long long)(varint_len(T(key - prev)) + varint_len((uint64_t)c));
    }
  }
  unsigned long long rest_total;
  block_exclusive_scan<NT, unsigned long long>(rest, scan64, &rest_total);
  if (threadIdx.x == 0) {
    if (MULT > 1 && fallbacks) atomicAdd(&fallbacks[1], (unsigned long long)U);  // rows of tiles above capacity
    TileOut<T> o;
    o.first_key = buf[head[0]];
    o.first_count = (unsigned)head[1] - head[0];
    o.last_key = buf[head[U - 1]];
    o.rows = U;
    o.rest_bytes = rest_total;
    tout[tid] = o;
  }
}

// ---------------------------------------------------------------------------
// Tile sort by an order-preserving hash table.  The keys of a tile are counted
// in a shared-memory table of distinct keys whose home slots grow with the
// key, so that reading the table out is already almost sorted:
//  1. a key's home slot is its place in the tile's key range [lo, hi] (its
//     splitters), scaled to the table; a key that finds another one there takes
//     the next free slot (linear probing, no wrap-around).  Every slot from a
//     key's home to its place is then occupied, so the keys of one run of
//     occupied slots (a cluster) all lie below those of the next run;
//  2. the clusters of two and more are put in order, one lane each (insertion;
//     typically two keys), and the occupied slots are listed in order;
//  3. the listed keys and counts go out as rows over the tile's keys in global
//     memory, with the DVLE size of every row but the first.
// Copies of a key never move: a duplicate costs one compare-and-swap that finds
// it and one counter add.  The binning sort moves every key twice and then
// finishes the bins that hold several keys, 6.5 warp instructions per key in
// all; the table takes 4.9 on the same tiles and is bound by instruction issue
// (about 55%) and shared-memory wavefronts (about 55%) alike, with the latency
// of both between its five barriers.
// Measured (150 bp reads, k = 31, 30-fold, one distinct key in 3.6): 10M reads
// 12.4 -> 7.9 ms, 1M reads 1.58 -> 0.96 ms.
// Two CTAs per SM walk the tiles; a tile's descriptor, key range and first keys
// are fetched while the one before it is worked on.
// A key that would land kProbeLimit slots or more from home (keys clustered in
// a small part of the range, or too many distinct keys for the table) has the
// tile counted again with hashed homes, where only too many distinct keys fail:
// its distinct keys are then binned and ranked.  A tile that fails there too
// goes to the binning sort, through a list; data that often does so is listed
// without the try (choose_next).
//
// The keys (u64, k <= 31) sit in the table themselves, claimed by a 64-bit
// compare-and-swap on an all-ones slot, which no key of at most 62 bits is;
// they stream through registers, so a tile may hold any number of keys.
// ---------------------------------------------------------------------------
constexpr unsigned kHashProbes = 96;   // with hashed homes
constexpr unsigned kMaxRanked = 512;   // distinct keys of a bin ranked by counting
constexpr unsigned kHashAny = 1024;  // u128 tiles of at most so many keys always suit the table

struct TableSmem {
  static constexpr int NT = 512, NW = NT / 32, SLOTS = 7168, HSLOTS = 6144, BINS = 4096;
  static constexpr size_t o_tab = 0;                              // keys
  static constexpr size_t o_cnt = o_tab + (size_t)SLOTS * 8;      // their counts (u32)
  static constexpr size_t o_ord = o_cnt + (size_t)SLOTS * 4;      // the occupied slots in order (u16)
  // hashed homes: fewer slots, and behind them the slots in bin order (u16)
  static constexpr size_t o_hcnt = o_tab + (size_t)HSLOTS * 8;
  static constexpr size_t o_tmp = o_hcnt + (size_t)HSLOTS * 4;
  static_assert(o_tmp + (size_t)HSLOTS * 2 <= o_ord, "the hashed layout fits the other's table and counts");
  // per warp: 64 keys that probe on, or 256 clusters (u16); hashed homes: 4096 bins (u16)
  static constexpr size_t o_queue = o_ord + (size_t)SLOTS * 2;
  static constexpr size_t o_edge = o_queue + (size_t)NW * 512;    // the warps' totals
  static constexpr size_t o_misc = o_edge + (size_t)NW * 4;
  static constexpr size_t total = o_misc + 32;
};

// A tile as the sort meets it: its keys and its key range.
template <class T>
struct TileIn {
  uint64_t start;
  uint32_t n;
  T mn, mx;
};
template <class T>
__device__ __forceinline__ TileIn<T> tile_in(const TileDesc* tiles, uint32_t i, uint32_t ntiles, const TileRanges<T>& rg) {
  TileIn<T> t;
  t.start = 0;
  t.n = 0;
  t.mn = T(0);
  t.mx = rg.kmax;
  if (i >= ntiles) return t;
  const TileDesc td = tiles[i];
  t.start = td.start;
  t.n = td.len;
  const uint32_t tl = rg.tile0 + i - td.bucket * rg.S;  // the tile's range in its bucket
  if (tl > 0) t.mn = rg.spl[tl - 1];
  if (tl + 1 < rg.S) {
    const T e = rg.spl[tl];
    t.mx = e > t.mn ? T(e - T(1)) : t.mn;
  }
  return t;
}

// The CTA's next tile, chosen by thread 0 while the one before it is worked
// on: next[0] = the tile, next[1] = 1 when it is the first of 32 taken at once,
// of which list_others leaves the others to the binning sort.  That is so while
// the tables have met 16 tiles and more than a quarter of them were better
// binned; one tile in 32 (and, of the CTAs' first ones, one CTA in 32) still
// tries.  (1M random 150 bp reads, every key once:
// 1.68 ms binned, 6.9 ms when every tile tried the u64 table first, 1.64-1.72 ms so.)
__device__ __forceinline__ bool mostly_binned(const TileRetry& r) {
  const unsigned a = *(volatile unsigned*)&r.met[0], f = *(volatile unsigned*)&r.met[1];
  return a >= 16 && 4 * f > a;
}
__device__ __forceinline__ void choose_next(const TileRetry& r, unsigned* next) {
  const bool many = mostly_binned(r);
  next[0] = gridDim.x + atomicAdd(r.taken, many ? 32u : 1u);
  next[1] = many;
}
template <class T>
__device__ __forceinline__ void list_others(const TileRetry& r, const unsigned* next, const TileDesc* tiles,
                                            uint32_t ntiles, TileOut<T>* tout) {
  if (threadIdx.x == 0 || threadIdx.x >= 32 || !next[1] || next[0] + threadIdx.x >= ntiles) return;
  const uint32_t i = next[0] + threadIdx.x, n = tiles[i].len;
  if (n) r.add(i, n);
  else empty_tile(&tout[i]);
}

// Whether a tile holds one key alone (a partition of reads of one base): seen by
// reading its keys, where counting them would be an atomic on one slot for each
// (200,000 reads of G, 24M copies: the tile sort 28.8 -> 8.2 ms, most of it now the
// empty tiles).  `other` is a zeroed flag, zeroed again.  Not inlined: its
// registers in the loop over the tiles took 1.3% of the tile sort's time.
__device__ __noinline__ bool one_key(const uint64_t* keys, uint64_t start, uint32_t n, volatile unsigned* other) {
  constexpr int NT = TableSmem::NT, UN = 4;
  const uint32_t lane = threadIdx.x & 31, head = (uint32_t)(start & 1u), pairs = (head + n + 1) >> 1;
  const uint4* p4 = reinterpret_cast<const uint4*>(keys + (start & ~1ull));
  const unsigned long long key = keys[start];
  for (uint32_t p0 = threadIdx.x; p0 - lane < pairs; p0 += UN * NT) {
    uint4 x[UN];
#pragma unroll
    for (int q = 0; q < UN; ++q) x[q] = p0 + q * NT < pairs ? p4[p0 + q * NT] : make_uint4(0, 0, 0, 0);
    bool differs = false;
#pragma unroll
    for (int q = 0; q < UN; ++q) {
      const uint32_t i0 = 2 * (p0 + q * NT) - head;  // wraps for the key before the tile
      differs |= i0 < n && ((unsigned long long)x[q].y << 32 | x[q].x) != key;
      differs |= i0 + 1 < n && ((unsigned long long)x[q].w << 32 | x[q].z) != key;
    }
    if (differs) *other = 1;
    if (__any_sync(0xffffffffu, differs || *other)) break;
  }
  __syncthreads();
  const bool one = *other == 0;
  __syncthreads();
  if (threadIdx.x == 0) *other = 0;
  return one;
}

__global__ void __launch_bounds__(TableSmem::NT, 2)
    k_tile_table(uint64_t* __restrict__ keys, uint32_t* __restrict__ counts, const TileDesc* __restrict__ tiles,
                 uint32_t ntiles, TileOut<uint64_t>* __restrict__ tout, unsigned long long* fallbacks,
                 TileRanges<uint64_t> rg, TileRetry retry) {
  using L = TableSmem;
  constexpr int NT = L::NT, NW = L::NW;
  constexpr unsigned long long kFree = ~0ull;
  extern __shared__ __align__(16) uint8_t sm[];
  unsigned long long* tab = reinterpret_cast<unsigned long long*>(sm + L::o_tab);
  uint16_t* ord = reinterpret_cast<uint16_t*>(sm + L::o_ord);
  unsigned* edge = reinterpret_cast<unsigned*>(sm + L::o_edge);
  // [0] probe limit, [1] another key, [2 + parity] rest, [4], [5] the next tile
  unsigned* misc = reinterpret_cast<unsigned*>(sm + L::o_misc);
  const unsigned lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1u;
  unsigned long long* queue = reinterpret_cast<unsigned long long*>(sm + L::o_queue) + wid * 64;
  // the thread's next two keys, a pair of the tile's 16-byte aligned span
  uint4 ka = make_uint4(0, 0, 0, 0);
  auto fetch = [&](const TileIn<uint64_t>& t, uint32_t p) {
    if (p < ((uint32_t)(t.start & 1u) + t.n + 1) >> 1) ka = reinterpret_cast<const uint4*>(keys + (t.start & ~1ull))[p];
  };
  if (threadIdx.x < 8) misc[threadIdx.x] = threadIdx.x == 6 && (blockIdx.x & 31u) && mostly_binned(retry);
  __syncthreads();
  bool skip = misc[6] || rg.wait_polls;  // a bound on the binning sort's wait (tests of its timeout): every tile goes there
  TileIn<uint64_t> t = tile_in(tiles, blockIdx.x, ntiles, rg);
  fetch(t, threadIdx.x);
  uint32_t clustered = 0;  // tiles in a row that went to hashed homes
  for (uint32_t i = blockIdx.x, par = 0; i < ntiles; par ^= 1) {
    const uint32_t n = t.n;
    if (threadIdx.x == 0) choose_next(retry, &misc[4]);
    const bool one = n > 2u * tile_capacity<uint64_t>() && !skip && one_key(keys, t.start, n, &misc[1]);
    if (n == 0 || skip || one) {
      if (threadIdx.x == 0) {
        if (n == 0) empty_tile(&tout[i]);
        else if (one) {
          counts[t.start] = n;  // the key is in place
          tout[i] = TileOut<uint64_t>{keys[t.start], keys[t.start], 1u, n, 0ull};
          if (fallbacks) atomicAdd(&fallbacks[1], 1ull);
        } else retry.add(i, n);
      }
      skip = rg.wait_polls;
      __syncthreads();
      i = misc[4];
      list_others(retry, &misc[4], tiles, ntiles, tout);
      t = tile_in(tiles, i, ntiles, rg);
      fetch(t, threadIdx.x);
      __syncthreads();
      continue;
    }
    // Keys clustered in a small part of the range (an AT-rich genome) go to
    // hashed homes and are binned afterwards.  After two such tiles in a row
    // the CTA's next ones start there; every eighth tries the order again.
    bool hashed = clustered >= 2 && (clustered & 7u);
    unsigned* cnt = reinterpret_cast<unsigned*>(sm + (hashed ? L::o_hcnt : L::o_cnt));
    // slots: twice the keys, in whole threads' shares
    uint32_t slots = n < (uint32_t)L::SLOTS / 2 - 288 ? (2 * n + 64 + 511) & ~511u : (uint32_t)L::SLOTS;
    auto clear = [&]() {
      if (hashed && slots > (uint32_t)L::HSLOTS) slots = L::HSLOTS;
      uint4* t4 = reinterpret_cast<uint4*>(tab);
      for (uint32_t j = threadIdx.x; j < slots / 2; j += NT) t4[j] = make_uint4(~0u, ~0u, ~0u, ~0u);
      uint4* c4 = reinterpret_cast<uint4*>(cnt);
      for (uint32_t j = threadIdx.x; j < slots / 4; j += NT) c4[j] = make_uint4(0, 0, 0, 0);
    };
    clear();
    __syncthreads();
    const uint32_t ni = misc[4];
    list_others(retry, &misc[4], tiles, ntiles, tout);
    const TileIn<uint64_t> next = tile_in(tiles, ni, ntiles, rg);
    // ---- the keys, counted.  A key whose home holds another one is queued;
    // the warp probes on for 32 such keys at a time, so that the others do not
    // wait for the few ----
    auto count_keys = [&](auto home, uint32_t limit) {
      bool far = false;
      uint32_t nq = 0;
      auto probe = [&](uint32_t m) {  // the last m queued keys
        __syncwarp();
        nq -= m;
        if (lane < m) {
          const unsigned long long v = queue[nq + lane];
          uint32_t s = home(v);
          const uint32_t end = s + limit;
          for (;;) {
            if (++s == end) {
              far = true;
              break;
            }
            const unsigned long long x = atomicCAS(&tab[s], kFree, v);
            if (x == kFree || x == v) {
              atomicAdd(&cnt[s], 1u);
              break;
            }
          }
        }
        __syncwarp();
      };
      const uint32_t head = (uint32_t)(t.start & 1u);
      for (uint32_t p = threadIdx.x; p - lane < (head + n + 1) >> 1; p += NT) {
        const unsigned long long v[2] = {(unsigned long long)ka.y << 32 | ka.x, (unsigned long long)ka.w << 32 | ka.z};
        fetch(t, p + NT);
        const uint32_t i0 = 2 * p - head;
        unsigned long long old[2];
        uint32_t h[2];
        bool in[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          in[q] = i0 + q < n;
          h[q] = home(v[q]);
          old[q] = in[q] ? atomicCAS(&tab[h[q]], kFree, v[q]) : kFree;
        }
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const bool hit = old[q] == kFree || old[q] == v[q];
          if (hit && in[q]) atomicAdd(&cnt[h[q]], 1u);
          const unsigned miss = __ballot_sync(0xffffffffu, !hit);
          if (miss) {
            if (!hit) queue[nq + __popc(miss & lt)] = v[q];
            nq += __popc(miss);
            if (nq >= 32) probe(32);
          }
        }
        if (__any_sync(0xffffffffu, far || *(volatile unsigned*)&misc[0])) break;
      }
      if (nq) probe(nq);
      if (far) misc[0] = 1;
    };
    const RangeMap<uint64_t> map(t.mn, t.mx);
    if (!hashed) {
      count_keys(HomeLinear<uint64_t>(map, t.mx, slots - 2 * kProbeLimit), kProbeLimit);  // probes end inside the table
      __syncthreads();
      hashed = misc[0] != 0;
      if (hashed) {
        __syncthreads();
        if (threadIdx.x == 0) misc[0] = 0;
        cnt = reinterpret_cast<unsigned*>(sm + L::o_hcnt);
        clear();
        fetch(t, threadIdx.x);
        __syncthreads();
      } else {
        clustered = 0;
      }
    }
    if (hashed) {
      const uint32_t homes = slots - kHashProbes;
      count_keys([homes](uint64_t v) { return __umulhi((uint32_t)((v * 0xD6E8FEB86659FD93ull) >> 32), homes); },
                 kHashProbes);
      __syncthreads();
      ++clustered;
    }
    fetch(next, threadIdx.x);
    if (misc[0]) {
      __syncthreads();
      if (threadIdx.x == 0) {
        retry.add(i, n);
        retry.met_tile(true);
        misc[0] = 0;
      }
      i = ni;
      t = next;
      continue;
    }
    // ---- the thread's 16 slots, listed; clusters in order ----
    unsigned U;
    {
      // a slot is in use when its count is not zero
      const uint32_t a = threadIdx.x * 16;
      uint32_t mine = 0, before = 0, after = 0;
      if (a < slots) {
        const uint4* c4 = reinterpret_cast<const uint4*>(cnt + a);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint4 x = c4[j];
          mine |= (x.x ? 1u << (4 * j) : 0u) | (x.y ? 2u << (4 * j) : 0u) | (x.z ? 4u << (4 * j) : 0u) |
                  (x.w ? 8u << (4 * j) : 0u);
        }
        before = a && cnt[a - 1];
        after = a + 16 < slots && cnt[a + 16];
      }
      // occupied slots, and clusters of at least two that start here
      const uint32_t multi = hashed ? 0u : mine & ~((mine << 1) | before) & ((mine >> 1) | (after << 15));
      const unsigned both = __popc(mine) | (__popc(multi) << 16);
      const unsigned inc = warp_inclusive(both, lane), ex = inc - both;
      const unsigned tot = __shfl_sync(0xffffffffu, inc, 31), nc = tot >> 16;
      if (lane == 0) edge[wid] = tot & 0xffffu;
      // the warp's clusters (first slots), one lane each
      uint16_t* list = reinterpret_cast<uint16_t*>(queue);
      unsigned p = ex >> 16;
      for (uint32_t m = multi; m; m &= m - 1) list[p++] = (uint16_t)(a + __ffs(m) - 1);
      __syncthreads();  // every warp has read the counts, and the totals are there
      const unsigned wt = lane < (unsigned)NW ? edge[lane] : 0u;
      const unsigned wi = warp_inclusive(wt, lane);
      U = __shfl_sync(0xffffffffu, wi, NW - 1);
      unsigned u = __shfl_sync(0xffffffffu, wi - wt, wid) + (ex & 0xffffu);
      for (uint32_t m = mine; m; m &= m - 1) ord[u++] = (uint16_t)(a + __ffs(m) - 1);
      for (unsigned j = lane; j < nc; j += 32) {
        const uint32_t first = list[j];
        order_cluster(tab, cnt, first, slots);
      }
    }
    __syncthreads();
    if (hashed) {
      // the slots hold the distinct keys in no order: into bins by their place
      // in the range, then ranked inside their bin by counting
      unsigned* bins = reinterpret_cast<unsigned*>(sm + L::o_queue);
      uint16_t* tmp = reinterpret_cast<uint16_t*>(sm + L::o_tmp);
      const HomeLinear<uint64_t> place(map, t.mx, L::BINS);
      for (uint32_t j = threadIdx.x; j < L::BINS / 2; j += NT) bins[j] = 0;
      __syncthreads();
      for (uint32_t j = threadIdx.x; j < U; j += NT) bin_add(bins, place(tab[ord[j]]));
      __syncthreads();
      {
        static_assert(L::BINS / 2 == 4 * NT, "four words of bins per thread");
        const uint4 x = reinterpret_cast<const uint4*>(bins)[threadIdx.x];
        const unsigned w[4] = {x.x, x.y, x.z, x.w};
        unsigned sum = 0;
        bool full = false;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          full |= (w[j] & 0xffffu) > kMaxRanked || (w[j] >> 16) > kMaxRanked;
          sum += (w[j] & 0xffffu) + (w[j] >> 16);
        }
        if (full) misc[0] = 1;
        const unsigned inc = warp_inclusive(sum, lane);
        if (lane == 31) edge[wid] = inc;
        __syncthreads();
        const unsigned wt = lane < (unsigned)NW ? edge[lane] : 0u;
        const unsigned wi = warp_inclusive(wt, lane);
        unsigned o = __shfl_sync(0xffffffffu, wi - wt, wid) + inc - sum;
        unsigned y[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          y[j] = o | ((o + (w[j] & 0xffffu)) << 16);
          o += (w[j] & 0xffffu) + (w[j] >> 16);
        }
        reinterpret_cast<uint4*>(bins)[threadIdx.x] = make_uint4(y[0], y[1], y[2], y[3]);
      }
      __syncthreads();
      if (misc[0]) {
        __syncthreads();
        if (threadIdx.x == 0) {
          retry.add(i, n);
          retry.met_tile(true);
          misc[0] = 0;
        }
        i = ni;
        t = next;
        continue;
      }
      for (uint32_t j = threadIdx.x; j < U; j += NT) {
        const uint16_t s = ord[j];
        tmp[bin_add(bins, place(tab[s]))] = s;
      }
      __syncthreads();
      for (uint32_t j = threadIdx.x; j < U; j += NT) {
        const uint16_t s = tmp[j];
        const unsigned long long v = tab[s];
        const uint32_t b = place(v);
        const uint32_t a = b ? bin_get(bins, b - 1) : 0u, z = bin_get(bins, b);
        uint32_t r = a;
        if (z - a > 1)
          for (uint32_t q = a; q < z; ++q) r += tab[tmp[q]] < v ? 1u : 0u;
        ord[r] = s;
      }
      __syncthreads();
      if (threadIdx.x == 0 && fallbacks) atomicAdd(fallbacks, 1ull);
    }
    write_rows<NT>(
        U, keys + t.start, counts + t.start, &misc[2 + par], &tout[i],
        [&](unsigned u, uint64_t* key, uint32_t* c) {
          const uint32_t s = ord[u];
          *key = tab[s];
          *c = cnt[s];
        },
        dvle_size<uint64_t>);
    if (threadIdx.x == 0) {
      retry.met_tile(hashed && 2 * U > n);  // mostly distinct keys: the binning sort is the faster one
      if (n > tile_capacity<uint64_t>() && fallbacks) atomicAdd(&fallbacks[1], (unsigned long long)U);
    }
    i = ni;
    t = next;
  }
}

// ---------------------------------------------------------------------------
// Tile sort of u128 keys (32 <= k <= 64).  Long k-mers come in clumps: the reads
// that cover one place of the genome give a k-mer and its copies with an error,
// and those with the error in the second half agree in their first 64 bits and
// more, so no linear map of the range keeps them apart (a table with homes in
// key order probed 7 slots per key on 250 bp reads at k = 63).  Here the keys
// are counted in a table of hashed homes, where clumps do not matter, and only
// the distinct ones (half of the keys there, a quarter at k = 31) are sorted:
// binned by their place in the range, then ranked inside their bin by counting.
// Measured on 1M x 250 bp reads of an AT-rich genome at k = 63 (188M keys):
// 11.8 -> 3.5 ms; half of its tiles had needed LSD passes or many-key bins.
// ---------------------------------------------------------------------------
struct HashSmem {
  static constexpr int NT = 512, NW = NT / 32, CAP = kTileThreads * tile_items<u128>(), SLOTS = 2 * CAP, BINS = CAP;
  static constexpr size_t o_buf = 0;                              // the tile's keys
  static constexpr size_t o_tab = o_buf + (size_t)CAP * 16;       // 6 bits of hash | index + 1 | count
  static constexpr size_t o_bin = o_tab;                          // after the counting: bins, and the keys in bin order
  static constexpr size_t o_ord = o_bin + (size_t)BINS * 4;
  static constexpr size_t o_list = o_tab + (size_t)SLOTS * 4;     // the distinct keys: count << 16 | index
  static constexpr size_t o_edge = o_list + (size_t)CAP * 4;
  static constexpr size_t o_misc = o_edge + (size_t)NW * 4;
  static constexpr size_t o_bar = o_misc + 32;
  static constexpr size_t total = o_bar + 16;
  static_assert(CAP <= 4096, "13-bit indices and counts");
};

__global__ void __launch_bounds__(HashSmem::NT, 2)
    k_tile_hash(u128* __restrict__ keys, uint32_t* __restrict__ counts, const TileDesc* __restrict__ tiles,
                uint32_t ntiles, TileOut<u128>* __restrict__ tout, unsigned long long* fallbacks,
                TileRanges<u128> rg, TileRetry retry) {
  using L = HashSmem;
  constexpr int NT = L::NT, NW = L::NW;
  extern __shared__ __align__(16) uint8_t sm[];
  const u128* buf = reinterpret_cast<const u128*>(sm + L::o_buf);
  unsigned* tab = reinterpret_cast<unsigned*>(sm + L::o_tab);
  unsigned* bin = reinterpret_cast<unsigned*>(sm + L::o_bin);
  unsigned* ord = reinterpret_cast<unsigned*>(sm + L::o_ord);
  unsigned* list = reinterpret_cast<unsigned*>(sm + L::o_list);
  unsigned* edge = reinterpret_cast<unsigned*>(sm + L::o_edge);
  // [0] full bin, [1] copy timeout, [2 + parity] rest, [4], [5] the next tile
  unsigned* misc = reinterpret_cast<unsigned*>(sm + L::o_misc);
  uint64_t* bar = reinterpret_cast<uint64_t*>(sm + L::o_bar);
  const unsigned lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  uint32_t used = 0;  // completed uses of the tile buffer
  auto taken = [&](const TileIn<u128>& t) { return t.n && t.n <= (uint32_t)L::CAP && !rg.wait_polls; };
  auto load = [&](const TileIn<u128>& t) {
    if (threadIdx.x == 0 && taken(t)) bulk_load(sm + L::o_buf, keys + t.start, t.n * 16, bar);
  };
  // exclusive prefix of v over the threads and the total; one barrier inside
  auto scan = [&](unsigned v, unsigned* total) {
    const unsigned inc = warp_inclusive(v, lane);
    if (lane == 31) edge[wid] = inc;
    __syncthreads();
    const unsigned wt = lane < (unsigned)NW ? edge[lane] : 0u;
    const unsigned wi = warp_inclusive(wt, lane);
    *total = __shfl_sync(0xffffffffu, wi, NW - 1);
    return __shfl_sync(0xffffffffu, wi - wt, wid) + inc - v;
  };
  if (threadIdx.x == 0) mbar_init(bar);
  if (threadIdx.x < 8) misc[threadIdx.x] = threadIdx.x == 6 && (blockIdx.x & 31u) && mostly_binned(retry);
  __syncthreads();
  bool skip = misc[6];
  TileIn<u128> t = tile_in(tiles, blockIdx.x, ntiles, rg);
  if (!skip) load(t);
  for (uint32_t i = blockIdx.x, par = 0; i < ntiles; par ^= 1) {
    const uint32_t n = t.n;
    if (threadIdx.x == 0) choose_next(retry, &misc[4]);
    if (skip || !taken(t)) {
      skip = false;
      // larger tiles, and (a bound on the binning sort's wait: tests of its timeout) every tile
      if (threadIdx.x == 0) {
        if (n == 0) empty_tile(&tout[i]);
        else retry.add(i, n);
      }
      __syncthreads();
      i = misc[4];
      list_others(retry, &misc[4], tiles, ntiles, tout);
      t = tile_in(tiles, i, ntiles, rg);
      load(t);
      __syncthreads();
      continue;
    }
    // a power of two of at least twice the keys
    const uint32_t slots = n <= 128 ? 256u : 1u << (33 - __clz((int)(n - 1)));
    for (uint32_t j = threadIdx.x; j < slots / 4; j += NT) reinterpret_cast<uint4*>(tab)[j] = make_uint4(0, 0, 0, 0);
    __syncthreads();
    const uint32_t ni = misc[4];
    list_others(retry, &misc[4], tiles, ntiles, tout);
    const TileIn<u128> next = tile_in(tiles, ni, ntiles, rg);
    if (!mbar_wait(bar, used & 1u, kBulkWaitPolls)) {
      misc[1] = 1;
      mbar_wait(bar, used & 1u, kBulkDrainPolls);
    }
    ++used;
    // ---- the keys, counted: the table has more slots than the tile keys, so
    // every probe ends ----
    for (uint32_t j = threadIdx.x; j < n; j += NT) {
      const u128 v = buf[j];
      const uint64_t m = ((uint64_t)v ^ (hi64(v) * 0x9E3779B97F4A7C15ull)) * 0xD6E8FEB86659FD93ull;
      const uint32_t h = (uint32_t)(m >> 32);
      const unsigned word = (h & 0xFC000000u) | ((j + 1) << 13) | 1u;
      for (uint32_t s = h & (slots - 1);; s = (s + 1) & (slots - 1)) {
        const unsigned x = atomicCAS(&tab[s], 0u, word);
        if (x == 0) break;
        if (((x ^ word) >> 26) == 0 && buf[((x >> 13) & 0x1fffu) - 1] == v) {
          atomicAdd(&tab[s], 1u);
          break;
        }
      }
    }
    __syncthreads();
    // ---- the distinct keys, listed ----
    unsigned U;
    {
      unsigned c = 0;
      for (uint32_t j = threadIdx.x; j < slots; j += NT) c += tab[j] != 0;
      unsigned o = scan(c, &U);
      for (uint32_t j = threadIdx.x; j < slots; j += NT) {
        const unsigned x = tab[j];
        if (x) list[o++] = ((x & 0x1fffu) << 16) | (((x >> 13) & 0x1fffu) - 1);
      }
    }
    __syncthreads();
    // ---- their bins ----
    const uint32_t bins = U <= 1024 ? 2048u : (uint32_t)L::BINS;
    const RangeMap<u128> map(t.mn, t.mx);
    const HomeLinear<u128> bin_of_key(map, t.mx, bins);
    for (uint32_t j = threadIdx.x; j < bins / 4; j += NT) reinterpret_cast<uint4*>(bin)[j] = make_uint4(0, 0, 0, 0);
    __syncthreads();
    for (uint32_t j = threadIdx.x; j < U; j += NT) atomicAdd(&bin[bin_of_key(buf[list[j] & 0xffffu])], 1u);
    __syncthreads();
    {
      const uint32_t per = bins / NT;  // 4 or 8 consecutive bins per thread
      unsigned v[8], sum = 0;
      bool full = false;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        v[j] = (uint32_t)j < per ? bin[threadIdx.x * per + j] : 0u;
        full |= v[j] > kMaxRanked;
        sum += v[j];
      }
      if (full) misc[0] = 1;
      unsigned tot;
      unsigned o = scan(sum, &tot);
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if ((uint32_t)j < per) {
          bin[threadIdx.x * per + j] = o;
          o += v[j];
        }
    }
    __syncthreads();
    if (misc[0] || misc[1]) {
      __syncthreads();
      if (threadIdx.x == 0) {
        if (misc[1]) {
          if (fallbacks) atomicAdd(fallbacks, kBulkTimeoutFlag);
          empty_tile(&tout[i]);
        } else {
          retry.add(i, n);
          retry.met_tile(true);
        }
        misc[0] = misc[1] = 0;
      }
      load(next);
      i = ni;
      t = next;
      continue;
    }
    for (uint32_t j = threadIdx.x; j < U; j += NT) {
      const unsigned e = list[j];
      ord[atomicAdd(&bin[bin_of_key(buf[e & 0xffffu])], 1u)] = e;
    }
    __syncthreads();
    // bin[b] is now the end of bin b; a key's place among its bin's by counting
    for (uint32_t j = threadIdx.x; j < U; j += NT) {
      const unsigned e = ord[j];
      const u128 v = buf[e & 0xffffu];
      const uint32_t b = bin_of_key(v);
      const uint32_t a = b ? bin[b - 1] : 0u, z = bin[b];
      uint32_t r = a;
      if (z - a > 1)
        for (uint32_t q = a; q < z; ++q) r += buf[ord[q] & 0xffffu] < v ? 1u : 0u;
      list[r] = e;
    }
    __syncthreads();
    write_rows<NT>(U, keys + t.start, counts + t.start, &misc[2 + par], &tout[i],
                   [&](unsigned u, u128* key, uint32_t* c) {
                     const unsigned e = list[u];
                     *key = buf[e & 0xffffu];
                     *c = e >> 16;
                   },
                   dvle_size<u128>);
    // mostly distinct keys: the binning sort is the faster one
    if (threadIdx.x == 0) retry.met_tile(n > kHashAny && 4 * U > 3 * n);
    load(next);
    i = ni;
    t = next;
  }
}

// CTAs walk the tiles ids[0 .. *nids) in turn.
template <class T, int MULT>
__global__ void __launch_bounds__(kTileThreads * MULT, MULT == 1 ? 2 : 1)
    k_tile_sort(T* __restrict__ keys, uint32_t* __restrict__ counts, const TileDesc* __restrict__ tiles,
                const uint32_t* __restrict__ ids, const unsigned* __restrict__ nids, TileOut<T>* __restrict__ tout,
                unsigned long long* fallbacks, TileRanges<T> rg, DevStatus* st) {
  const unsigned cnt = *nids;
  for (unsigned i = blockIdx.x; i < cnt; i += gridDim.x) {
    sort_tile<T, MULT>(ids[i], keys, counts, tiles, tout, fallbacks, rg, st);
    __syncthreads();  // shared memory is reused by the next tile
  }
}

template <class T, int MULT>
static void tile_sort_with(T* keys, uint32_t* counts, const TileDesc* tiles, const uint32_t* ids,
                           const unsigned* nids, uint32_t grid, TileOut<T>* out, unsigned long long* fallbacks,
                           TileRanges<T> rg, DevStatus* st, cudaStream_t s) {
  const size_t smem = BinSmem<T, MULT>::total;
  cudaFuncSetAttribute(k_tile_sort<T, MULT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  cudaFuncSetAttribute(k_tile_sort<T, MULT>, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
  k_tile_sort<T, MULT><<<grid, BinSmem<T, MULT>::NT, smem, s>>>(keys, counts, tiles, ids, nids, out, fallbacks, rg, st);
}

template <class T>
void launch_tile_sort(T* keys, uint32_t* counts, const TileDesc* tiles, uint32_t ntiles, TileOut<T>* out,
                      unsigned long long* fallbacks, TileRanges<T> rg, TileRetry retry, cudaStream_t s) {
  int dev = 0, sms = 1;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const uint32_t grid = std::min<uint32_t>(ntiles, 2 * (uint32_t)sms);
  if (!ntiles) return;
  auto go = [&](auto kern, size_t smem, int nt) {
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    kern<<<grid, nt, smem, s>>>(keys, counts, tiles, ntiles, out, fallbacks, rg, retry);
  };
  if constexpr (sizeof(T) == 8) go(k_tile_table, TableSmem::total, TableSmem::NT);
  else go(k_tile_hash, HashSmem::total, HashSmem::NT);
}
template <class T>
void launch_tile_sort_listed(T* keys, uint32_t* counts, const TileDesc* tiles, const uint32_t* ids, uint32_t grid,
                             const unsigned* nids, TileOut<T>* out, unsigned long long* fallbacks,
                             TileRanges<T> rg, DevStatus* st, cudaStream_t s) {
  tile_sort_with<T, 1>(keys, counts, tiles, ids, nids, 2 * grid, out, fallbacks, rg, st, s);
}
template <class T>
void launch_tile_sort_large(T* keys, uint32_t* counts, const TileDesc* tiles, const uint32_t* ids, uint32_t grid,
                            const unsigned* nids, TileOut<T>* out, unsigned long long* fallbacks,
                            TileRanges<T> rg, DevStatus* st, cudaStream_t s) {
  tile_sort_with<T, 2>(keys, counts, tiles, ids, nids, grid, out, fallbacks, rg, st, s);
}
template void launch_tile_sort<uint64_t>(uint64_t*, uint32_t*, const TileDesc*, uint32_t, TileOut<uint64_t>*,
                                         unsigned long long*, TileRanges<uint64_t>, TileRetry, cudaStream_t);
template void launch_tile_sort<u128>(u128*, uint32_t*, const TileDesc*, uint32_t, TileOut<u128>*, unsigned long long*,
                                     TileRanges<u128>, TileRetry, cudaStream_t);
template void launch_tile_sort_listed<uint64_t>(uint64_t*, uint32_t*, const TileDesc*, const uint32_t*, uint32_t,
                                                const unsigned*, TileOut<uint64_t>*, unsigned long long*,
                                                TileRanges<uint64_t>, DevStatus*, cudaStream_t);
template void launch_tile_sort_listed<u128>(u128*, uint32_t*, const TileDesc*, const uint32_t*, uint32_t,
                                            const unsigned*, TileOut<u128>*, unsigned long long*, TileRanges<u128>,
                                            DevStatus*, cudaStream_t);
template void launch_tile_sort_large<uint64_t>(uint64_t*, uint32_t*, const TileDesc*, const uint32_t*, uint32_t,
                                               const unsigned*, TileOut<uint64_t>*, unsigned long long*,
                                               TileRanges<uint64_t>, DevStatus*, cudaStream_t);
template void launch_tile_sort_large<u128>(u128*, uint32_t*, const TileDesc*, const uint32_t*, uint32_t,
                                           const unsigned*, TileOut<u128>*, unsigned long long*, TileRanges<u128>,
                                            DevStatus*, cudaStream_t);

// ---------------------------------------------------------------------------
// Oversized tiles: one CTA, LSD passes through global memory.  Each pass
// histograms the digit, then walks the tile in CAP-key chunks, ranks each
// chunk stably on chip and appends every digit group at its running offset.
// Then a chunked run-length reduction with carries between chunks.
// ---------------------------------------------------------------------------
template <class T>
__device__ __forceinline__ void big_sort_tile(uint32_t tid, T* __restrict__ keys, uint32_t* __restrict__ counts,
                                              T* __restrict__ scratch, const TileDesc* __restrict__ tiles,
                                              TileOut<T>* __restrict__ tout, unsigned long long* sstats) {
  using L = TileSmem<T>;
  constexpr int NT = L::NT, ITEMS = L::ITEMS, CAP = L::CAP;
  extern __shared__ __align__(16) uint8_t sm[];
  unsigned* warp_hist = reinterpret_cast<unsigned*>(sm + L::buf_bytes);
  unsigned long long* scan64 = reinterpret_cast<unsigned long long*>(sm + L::buf_bytes + L::hist_bytes + L::head_bytes);
  unsigned* scan_sm = reinterpret_cast<unsigned*>(scan64);
  T* red = reinterpret_cast<T*>(scan64 + 64);
  unsigned long long* run_off = reinterpret_cast<unsigned long long*>(red + 2 * L::NW);  // 256
  unsigned* dtot = reinterpret_cast<unsigned*>(sm + L::buf_bytes + L::hist_bytes);        // 256 (head area)
  unsigned* dstart = dtot + 256;                                                          // 256

  const TileDesc td = tiles[tid];
  const unsigned long long n = td.len;
  T* src = keys + td.start;
  T* dst = scratch + td.start;

  T mn = ~T(0), mx = T(0);
  for (unsigned long long i = threadIdx.x; i < n; i += NT) {
    const T v = src[i];
    mn = v < mn ? v : mn;
    mx = v > mx ? v : mx;
  }
  block_minmax<NT>(mn, mx, red);
  if (mn == mx) {  // one key fills the tile: a single row
    if (threadIdx.x == 0) {
      if (sstats) atomicAdd(&sstats[1], 1ull);
      keys[td.start] = mn;
      counts[td.start] = n > 0xffffffffull ? 0xffffffffu : (uint32_t)n;
      TileOut<T> o;
      o.first_key = o.last_key = mn;
      o.rows = 1;
      o.first_count = counts[td.start];
      o.rest_bytes = 0;
      tout[tid] = o;
    }
    return;
  }
  const int nbits = varying_bits(mn, mx);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const unsigned pos0 = (unsigned)wid * 32u * ITEMS + lane;
  for (int shift = 0; shift < nbits; shift += 8) {
    // digit histogram
    for (int d = threadIdx.x; d < 256; d += NT) warp_hist[d] = 0;
    __syncthreads();
    for (unsigned long long i = threadIdx.x; i < n; i += NT) atomicAdd(&warp_hist[digit_of(src[i], shift)], 1u);
    __syncthreads();
    if (threadIdx.x == 0) {
      unsigned long long acc = 0;
      for (int d = 0; d < 256; ++d) {
        run_off[d] = acc;
        acc += warp_hist[d];
      }
    }
    __syncthreads();
    for (unsigned long long c0 = 0; c0 < n; c0 += CAP) {
      const unsigned cn = (unsigned)((n - c0) < (unsigned long long)CAP ? (n - c0) : CAP);
      T key[ITEMS];
      unsigned dig[ITEMS], dest[ITEMS];
      bool valid[ITEMS];
#pragma unroll
      for (int r = 0; r < ITEMS; ++r) {
        const unsigned pos = pos0 + r * 32u;
        valid[r] = pos < cn;
        key[r] = valid[r] ? src[c0 + pos] : T(0);
        dig[r] = digit_of(key[r], shift);
      }
      block_rank<NT, ITEMS, 256>(dig, valid, dest, warp_hist, scan_sm, dtot, dstart);
#pragma unroll
      for (int r = 0; r < ITEMS; ++r)
        if (valid[r]) dst[run_off[dig[r]] + (dest[r] - dstart[dig[r]])] = key[r];
      __syncthreads();
      for (int d = threadIdx.x; d < 256; d += NT) run_off[d] += dtot[d];
      __syncthreads();
    }
    T* t = src;
    src = dst;
    dst = t;
  }
  // Run-length reduction of the sorted keys in src (keys or scratch).
  // Pass A: unique keys to keys[start+u], head positions to counts[start+u].
  T* ok = keys + td.start;
  uint32_t* oc = counts + td.start;
  unsigned long long U = 0;
  for (unsigned long long c0 = 0; c0 < n; c0 += CAP) {
    const unsigned cn = (unsigned)((n - c0) < (unsigned long long)CAP ? (n - c0) : CAP);
    const unsigned b0 = threadIdx.x * ITEMS;
    T kv[ITEMS];
    bool hd[ITEMS];
    unsigned nh = 0;
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
      const unsigned i = b0 + r;
      hd[r] = false;
      if (i < cn) {
        const unsigned long long gi = c0 + i;
        kv[r] = src[gi];
        hd[r] = gi == 0 || kv[r] != src[gi - 1];
        nh += hd[r];
      }
    }
    unsigned tot;
    unsigned long long u = U + block_exclusive_scan<NT, unsigned>(nh, scan_sm, &tot);
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ITEMS; ++r)
      if (hd[r]) {
        ok[u] = kv[r];
        oc[u] = (uint32_t)(c0 + b0 + r);
        u++;
      }
    U += tot;
    __syncthreads();
  }
  // Pass B: head positions -> counts (saturating u32), DVLE rest bytes.
  unsigned long long rest = 0;
  for (unsigned long long c0 = 0; c0 < U; c0 += CAP) {
    const unsigned cn = (unsigned)((U - c0) < (unsigned long long)CAP ? (U - c0) : CAP);
    unsigned long long cnt[ITEMS];
    T kv[ITEMS], kp[ITEMS];
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
      const unsigned i = threadIdx.x + r * NT;
      cnt[r] = 0;
      if (i < cn) {
        const unsigned long long v = c0 + i;
        const unsigned long long h0 = oc[v];
        const unsigned long long h1 = (v + 1 < U) ? (unsigned long long)oc[v + 1] : n;
        cnt[r] = h1 - h0;
        kv[r] = ok[v];
        kp[r] = v > 0 ? ok[v - 1] : T(0);
      }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
      const unsigned i = threadIdx.x + r * NT;
      if (i < cn) {
        const unsigned long long v = c0 + i;
        const uint32_t c = cnt[r] > 0xffffffffull ? 0xffffffffu : (uint32_t)cnt[r];
        oc[v] = c;
        if (v > 0) rest += (unsigned long long)(varint_len(kv[r] - kp[r]) + varint_len((uint64_t)c));
      }
    }
    __syncthreads();
  }
  unsigned long long rest_total;
  block_exclusive_scan<NT, unsigned long long>(rest, scan64, &rest_total);
  if (threadIdx.x == 0) {
    if (sstats) atomicAdd(&sstats[1], U);
    TileOut<T> o;
    o.first_key = ok[0];
    o.first_count = oc[0];
    o.last_key = ok[U - 1];
    o.rows = (uint32_t)U;
    o.rest_bytes = rest_total;
    tout[tid] = o;
  }
}

// CTAs walk the tiles big_ids[0 .. *nids) in turn.
template <class T>
__global__ void __launch_bounds__(kTileThreads, 1)
    k_big_tile_sort(T* __restrict__ keys, uint32_t* __restrict__ counts, T* __restrict__ scratch,
                    const TileDesc* __restrict__ tiles, const uint32_t* __restrict__ big_ids,
                    const unsigned* __restrict__ nids, TileOut<T>* __restrict__ tout, unsigned long long* sstats) {
  const unsigned cnt = *nids;
  for (unsigned i = blockIdx.x; i < cnt; i += gridDim.x) {
    big_sort_tile<T>(big_ids[i], keys, counts, scratch, tiles, tout, sstats);
    __syncthreads();  // shared memory is reused by the next tile
  }
}

template <class T>
void launch_big_tile_sort(T* keys, uint32_t* counts, T* scratch, const TileDesc* tiles, const uint32_t* big_ids,
                          uint32_t grid, const unsigned* nbig, TileOut<T>* out, unsigned long long* sort_stats,
                          cudaStream_t s) {
  const size_t smem = TileSmem<T>::total;
  cudaFuncSetAttribute(k_big_tile_sort<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  k_big_tile_sort<T><<<grid, kTileThreads, smem, s>>>(keys, counts, scratch, tiles, big_ids, nbig, out, sort_stats);
}
template void launch_big_tile_sort<uint64_t>(uint64_t*, uint32_t*, uint64_t*, const TileDesc*, const uint32_t*,
                                             uint32_t, const unsigned*, TileOut<uint64_t>*, unsigned long long*,
                                             cudaStream_t);
template void launch_big_tile_sort<u128>(u128*, uint32_t*, u128*, const TileDesc*, const uint32_t*, uint32_t,
                                         const unsigned*, TileOut<u128>*, unsigned long long*, cudaStream_t);

// Statistics of the tiles: stats[0] largest tile, [1] keys, [2] non-empty
// tiles, [3] keys in the tiles above `cap`, [4] those tiles, range[t] keys in
// tile index t of every bucket.  One atomic per statistic and CTA.
__global__ void __launch_bounds__(256) k_tile_stats(const uint32_t* __restrict__ lens, uint32_t ntiles, uint32_t S,
                                                    uint32_t cap, unsigned long long* __restrict__ stats,
                                                    unsigned long long* __restrict__ range) {
  __shared__ unsigned long long red[8][5];
  const uint32_t t = blockIdx.x * 256 + threadIdx.x;
  const uint32_t len = t < ntiles ? lens[t] : 0u;
  if (len && S > 1) atomicAdd(&range[t % S], (unsigned long long)len);
  unsigned long long v[5] = {len, len, len ? 1ull : 0ull, len > cap ? (unsigned long long)len : 0ull,
                             len > cap ? 1ull : 0ull};
#pragma unroll
  for (int j = 0; j < 5; ++j)
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      const unsigned long long y = __shfl_xor_sync(0xffffffffu, v[j], o);
      v[j] = j == 0 ? (y > v[j] ? y : v[j]) : v[j] + y;
    }
  if ((threadIdx.x & 31) == 0)
    for (int j = 0; j < 5; ++j) red[threadIdx.x >> 5][j] = v[j];
  __syncthreads();
  if (threadIdx.x < 5) {
    unsigned long long x = red[0][threadIdx.x];
    for (int w = 1; w < 8; ++w) {
      const unsigned long long y = red[w][threadIdx.x];
      x = threadIdx.x == 0 ? (y > x ? y : x) : x + y;
    }
    if (threadIdx.x == 0) atomicMax(&stats[0], x);
    else if (x) atomicAdd(&stats[threadIdx.x], x);
  }
}

void launch_tile_stats(const uint32_t* lens, uint32_t ntiles, uint32_t S, uint32_t cap, unsigned long long* stats,
                       unsigned long long* range, cudaStream_t s) {
  if (ntiles) k_tile_stats<<<(ntiles + 255) / 256, 256, 0, s>>>(lens, ntiles, S, cap, stats, range);
}

}  // namespace kite
