// GPU `kite merge`: decode every input chunk, k-way merge per partition with
// exact count summation, DVLE re-encode.
//
// Reference semantics restated (src/merge/mod.rs:198-214 and
// src/kiteops/mod.rs:433-859):
//   load_partition_counts   every chunk of one input's partition decoded
//                           (DVLE or RAW), equal keys summed in u64 (saturating)
//   apply_reader_filter     that input's header min/max, on the per-input sum
//   merge_vectors_total     union over inputs, u64 saturating sums
//   serialize_partition_chunk  a total above u32::MAX is an error naming the key;
//                           otherwise one DVLE chunk per non-empty partition.
//
// GPU structure:
//   decode    payload bytes cut into 8 KiB segments, one warp each, as their
//             piece of the input lands: varints per segment, per-stream scans,
//             then rows with a lane each, keys relative to the segment until
//             the start keys are added.  A "stream" is one chunk.
//   tiles     key-range tiles per partition from global splitters (or slices of
//             a partition's only stream), planned on the device; ranges above
//             the on-chip capacity are cut by bisection on the host.
//   merge     one CTA per tile: u64 rows summed in a shared-memory table, or
//             (u128, and tiles that a table does not suit) rows merged by merge
//             paths, with per-input sums, filter, cross-input sums, overflow
//             check.
//   encode    the count path's DVLE link + encode kernels.
//
// The same decode / tile / merge stages serve `kite dump` (one input):
//   LoserTreeMerger src/dump/loser_tree.rs:141-175  the chunks of a partition
//                           merged by key, equal keys summed with saturating
//                           u32 adds (= the u64 sum clamped to u32::MAX)
//   stream_partition_slabs src/dump/merge.rs:282-428  header min/max applied
//                           to that summed count, then one TSV line per row
//   decode_kmer_any src/dump/decoder.rs:27-50  the key's 2-bit codes MSB
//                           first as ACGT, "<kmer>\t<count>\n"
// with a formatting pass in place of the DVLE encode.
#include <algorithm>
#include <chrono>
#include <cstring>
#include <memory>
#include <new>
#include <string>
#include <thread>
#include <vector>

#include "merge.h"
#include "key_table.cuh"
#include "kite_internal.h"
#include "splitters.h"

namespace kite {

namespace {

constexpr uint32_t kSeg = 8192;          // decode segment bytes (one warp each)
constexpr int kMergeThreads = 512;
constexpr uint32_t kMergeCap = 4096;      // rows per merge tile
constexpr uint32_t kMaxTileStreams = 256; // streams per tile (inputs x chunks)
constexpr int kTsvThreads = 256;          // rows per formatting round
constexpr uint32_t kHistBins = 1024;      // histo: counts below this binned on chip, larger ones listed

// What the merge kernel makes of each merged key group.
enum MergeMode : int {
  kModeMerge = 0,  // kite merge: per-input filter, u64 sums, u32 overflow recorded
  kModeDump = 1,   // kite dump: sum clamped to u32, then the header filter; TSV byte counts
  kModeHisto = 2,  // kite histo: per-input filter on the u64 sum, then count -> frequency
  kModeQuery = 3,  // kite query: keys looked up in the decoded streams, no merge kernel
};

// Outputs of the histo and query modes.
struct MergeAux {
  unsigned long long* hist;      // kHistBins frequencies (histo)
  unsigned long long* spill;     // counts >= kHistBins, one entry per key (histo)
  unsigned long long* spill_n;   // entries written to spill
  unsigned long long spill_cap;
  uint32_t line_k;               // k, for TSV line lengths (dump)
};

// Decimal digits of a count.
__host__ __device__ __forceinline__ unsigned dec_digits(uint32_t v) {
  unsigned d = 1;
  for (uint32_t p = 10; d < 10 && v >= p; p *= 10) ++d;
  return d;
}

struct StreamDesc {
  uint64_t byte_off;   // payload offset in the device byte buffer
  uint64_t byte_len;
  uint64_t row_off;    // first row in the decoded arrays
  uint64_t rows;
  uint32_t codec;
  uint32_t input;
  uint32_t partition;
  uint32_t head;       // raw head bytes (12 or 20) for DVLE, 0 for RAW
};

struct SegDesc {
  uint64_t start, end;  // byte range (device buffer offsets) inside the stream's varint area
  uint32_t stream;
  uint32_t first;       // 1 if first segment of the stream
};

struct InputFilter {
  uint32_t has_min, has_max, min_count, max_count;
};

// One entry of a tile's stream list.
struct TileStream {
  uint64_t lo, hi;      // row range [lo, hi) (absolute row indices)
  uint32_t input;
  uint32_t pad;
};

struct MergeTile {
  uint64_t out_off;     // output row base (reserved = rows in)
  uint32_t first_ts;    // index into TileStream list
  uint32_t nts;
  uint32_t rows_in;
  uint32_t partition;
};

// Warp shuffle-up of a 64- or 128-bit value, a wrapping inclusive warp sum,
// and a broadcast from one lane.
template <class T>
__device__ __forceinline__ T shfl_up_t(T v, int d) {
  if constexpr (sizeof(T) == 8) {
    return (T)__shfl_up_sync(0xffffffffu, (unsigned long long)v, d);
  } else {
    const unsigned long long lo = __shfl_up_sync(0xffffffffu, (unsigned long long)v, d);
    const unsigned long long hi = __shfl_up_sync(0xffffffffu, (unsigned long long)(v >> 64), d);
    return ((T)hi << 64) | (T)lo;
  }
}
template <class T>
__device__ __forceinline__ T warp_incl_sum(T v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const T y = shfl_up_t(v, o);
    if (lane >= o) v += y;
  }
  return v;
}
template <class T>
__device__ __forceinline__ T warp_bcast_t(T v, int src) {
  if constexpr (sizeof(T) == 8) {
    return (T)__shfl_sync(0xffffffffu, (unsigned long long)v, src);
  } else {
    const unsigned long long lo = __shfl_sync(0xffffffffu, (unsigned long long)v, src);
    const unsigned long long hi = __shfl_sync(0xffffffffu, (unsigned long long)(v >> 64), src);
    return ((T)hi << 64) | (T)lo;
  }
}
// ---- warp-cooperative DVLE decode ----------------------------------------------
// A segment (kSeg bytes of one stream's varint area) is decoded by one warp in
// rounds of 512 bytes: every lane loads 16 bytes (one coalesced 512-byte load
// per warp) into a per-warp shared-memory window that also holds the 32 bytes
// before the round, and lists where the varints that end in its bytes end (top
// bit clear).  A varint is at most 19 bytes, so the one that a round's first
// byte lies in begins in the window.  Then each lane takes a whole row: the
// 32 rows' key deltas (8-byte loads from the window, their 7-bit groups packed
// by shifts of whole words) go through one warp scan, and keys and counts out
// as coalesced runs.  Key deltas and counts alternate, so which terminators end
// a row follows from the number of varints before the segment.  A row belongs
// to the segment holding its count's terminator; a final varint without one at
// the stream's end counts as ending there.
//
// Passes: varints per segment (k_seg_count), their scan per stream, rows with
// keys relative to the segment's start (k_seg_rows), the scan of the segments'
// delta sums, and the start keys added (k_seg_base).  Decoding every varint
// byte by byte in the lane that held its last byte, twice (sums first, then
// rows), took 37 warp instructions per row; this takes 15, and the 64.6M rows of 2M
// reads decode in 1.36 ms instead of 3.63.
constexpr int kDecWarps = 8;                    // warps per decode CTA
constexpr uint32_t kRound = 512;                // bytes per warp round
constexpr uint32_t kWinBytes = kRound + 32;     // window: 32 bytes before the round + the round

struct alignas(16) DecWindow {
  uint8_t b[kWinBytes + 32];   // and room for whole-word reads past the last varint
  uint16_t end[kRound + 4];    // [0], [1]: ends before the round; then its own varints' (window offset past the last byte)
};
static_assert(sizeof(DecWindow) % 16 == 0, "every window is read by 16-byte loads");

// Terminator bits of 16 bytes (bit i: byte i has its top bit clear).
__device__ __forceinline__ uint32_t term_bits16(uint4 w) {
  auto m4 = [](uint32_t x) { return (((~x & 0x80808080u) >> 7) * 0x10204080u) >> 28; };
  return m4(w.x) | (m4(w.y) << 4) | (m4(w.z) << 8) | (m4(w.w) << 12);
}

// The terminators of the 16 bytes at stream offset o that lie in [lo, hi),
// with one at the byte `forced` (the last of a stream that ends inside a varint).
__device__ __forceinline__ uint32_t own_terms(uint4 w, uint64_t o, uint64_t lo, uint64_t hi, uint64_t forced) {
  uint32_t m = term_bits16(w);
  if (forced - o < 16) m |= 1u << (uint32_t)(forced - o);
  if (o < lo) m &= lo - o >= 16 ? 0u : ~((1u << (uint32_t)(lo - o)) - 1u);
  if (o + 16 > hi) m &= hi <= o ? 0u : ((1u << (uint32_t)(hi - o)) - 1u);
  return m;
}

// Pass A, one warp per segment: the varints the segment owns.
__global__ void __launch_bounds__(32 * kDecWarps)
    k_seg_count(const uint8_t* __restrict__ bytes, uint64_t lim_pad, const SegDesc* __restrict__ segs, uint32_t nseg,
                const StreamDesc* __restrict__ streams, uint32_t* __restrict__ terms) {
  const uint32_t lane = threadIdx.x & 31, si = blockIdx.x * kDecWarps + (threadIdx.x >> 5);
  if (si >= nseg) return;
  const SegDesc d = segs[si];
  const StreamDesc sd = streams[d.stream];
  const uint64_t lim = sd.byte_off + sd.byte_len;
  uint32_t n = 0;
  constexpr int kAhead = 4;
  for (uint64_t o0 = (d.start & ~15ull) + 16 * lane; o0 - 16 * lane < d.end; o0 += kAhead * kRound) {
    uint4 w[kAhead];
#pragma unroll
    for (int j = 0; j < kAhead; ++j) {
      const uint64_t o = o0 + (uint64_t)j * kRound;
      w[j] = o < lim_pad && o < d.end ? *reinterpret_cast<const uint4*>(bytes + o) : make_uint4(~0u, ~0u, ~0u, ~0u);
    }
#pragma unroll
    for (int j = 0; j < kAhead; ++j) n += __popc(own_terms(w[j], o0 + (uint64_t)j * kRound, d.start, d.end, lim - 1));
  }
  n = __reduce_add_sync(0xffffffffu, n);
  if (lane == 0) terms[si] = n;
}

// Per stream of the list sids (one warp each): the first varint index of every
// segment [first[w], first[w + 1]) of stream sids[w] (exclusive scan of the terminator
// counts), and the check that the stream holds the 2 * (rows - 1) varints its
// rows need.
__global__ void k_stream_seg_scan(const uint32_t* __restrict__ terms, const uint32_t* __restrict__ first,
                                  const StreamDesc* __restrict__ streams, const uint32_t* __restrict__ sids,
                                  uint32_t nsid,
                                  unsigned long long* __restrict__ vstart, DevStatus* st) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t w = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
  if (w >= nsid) return;
  const uint32_t si = sids[w];
  const StreamDesc sd = streams[si];
  const uint32_t f = first[w], e = first[w + 1];
  unsigned long long cv = 0;
  for (uint32_t b = f; b < e; b += 32) {
    const uint32_t s = b + lane;
    const unsigned long long t = s < e ? terms[s] : 0ull;
    const unsigned long long ti = warp_incl_sum<unsigned long long>(t);
    if (s < e) vstart[s] = cv + ti - t;
    cv += __shfl_sync(0xffffffffu, ti, 31);
  }
  if (lane == 0 && sd.head && sd.rows && cv < 2 * (sd.rows - 1)) dev_fail(st, KITE_DEV_SHORT_VARINTS, si);
}

// Per stream of the list sids (one warp each): the key before every segment's
// first row, from the stream's head key and the segments' delta sums.
template <class T>
__global__ void k_stream_base_scan(const T* __restrict__ sums, const uint32_t* __restrict__ first,
                                   const T* __restrict__ first_keys, const uint32_t* __restrict__ sids,
                                   uint32_t nsid, T* __restrict__ kstart) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t w = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
  if (w >= nsid) return;
  const uint32_t si = sids[w], f = first[w], e = first[w + 1];
  T ck = f < e ? first_keys[si] : T(0);
  for (uint32_t b = f; b < e; b += 32) {
    const uint32_t s = b + lane;
    const T dv = s < e ? sums[s] : T(0);
    const T di = warp_incl_sum(dv);
    if (s < e) kstart[s] = ck + (di - dv);
    ck += warp_bcast_t(di, 31);
  }
}

// The 7-bit groups of eight varint bytes (continuation bits cleared), packed.
__device__ __forceinline__ uint64_t pack7(uint32_t lo, uint32_t hi) {
  auto p4 = [](uint32_t v) {
    v &= 0x7f7f7f7fu;
    v = (v & 0x007f007fu) | ((v & 0x7f007f00u) >> 1);
    return (v & 0x3fffu) | ((v & 0x3fff0000u) >> 2);
  };
  return (uint64_t)p4(lo) | ((uint64_t)p4(hi) << 28);
}

// The varint of window bytes [a, e): its low kBits bits.
template <class T>
__device__ __forceinline__ T varint_in(const DecWindow* win, uint32_t a, uint32_t e) {
  const uint32_t* w = reinterpret_cast<const uint32_t*>(win->b) + (a >> 2);
  const uint32_t sh = (a & 3u) * 8;
  const uint32_t n = e - a;
  T v = 0;
  uint32_t x0 = w[0], x1 = w[1];
#pragma unroll
  for (uint32_t g = 0; g < (sizeof(T) == 8 ? 2u : 3u); ++g) {
    if (8 * g >= n) break;
    const uint32_t x2 = w[2 * g + 2];
    uint32_t lo = __funnelshift_r(x0, x1, sh), hi = __funnelshift_r(x1, x2, sh);
    const uint32_t left = n - 8 * g;
    if (left < 4) {
      lo &= (1u << (8 * left)) - 1u;
      hi = 0;
    } else if (left < 8) {
      hi &= (1u << (8 * (left - 4))) - 1u;
    }
    const uint64_t p = pack7(lo, hi);
    if constexpr (sizeof(T) == 8) v |= g == 0 ? p : p << 56;
    else v |= (T)p << (56 * g);
    if (left <= 8) break;
    x0 = x2;
    x1 = w[2 * g + 3];
  }
  return v;
}

// Pass B, one warp per segment: (key, u64 count) rows of the segment, keys
// relative to the segment's start (wrapping sums of the deltas, as the
// reference's wrapping_add), and the segment's delta sum.
template <class T>
__global__ void __launch_bounds__(32 * kDecWarps)
    k_seg_rows(const uint8_t* __restrict__ bytes, uint64_t lim_pad, const SegDesc* __restrict__ segs, uint32_t nseg,
               const StreamDesc* __restrict__ streams, const unsigned long long* __restrict__ vstart,
               T* __restrict__ keys, unsigned long long* __restrict__ counts, T* __restrict__ sums) {
  __shared__ __align__(16) DecWindow wins[kDecWarps];
  const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const uint32_t si = blockIdx.x * kDecWarps + wid;
  if (si >= nseg) return;
  DecWindow* win = &wins[wid];
  const SegDesc d = segs[si];
  const StreamDesc sd = streams[d.stream];
  const uint64_t area = sd.byte_off + sd.head, forced = sd.byte_off + sd.byte_len - 1;
  unsigned long long v0 = vstart[si];  // stream varint index of the segment's next owned varint
  uint64_t base = d.start & ~15ull;
  // the 32 bytes before the round, and the ends of the two varints before the
  // segment's first own byte (the area's start is the first varint's)
  uint4 w = make_uint4(0, 0, 0, 0);
  if (lane < 2 && base >= 32) w = *reinterpret_cast<const uint4*>(bytes + base - 32 + 16 * lane);
  if (lane < 2) reinterpret_cast<uint4*>(win->b)[lane] = w;
  {
    uint64_t m = 0;  // window offset i: a varint ends at i (past its last byte)
    if (base >= 32) {
      const uint32_t t0 = __shfl_sync(0xffffffffu, own_terms(w, base - 32 + 16 * lane, area, d.start, forced), 0);
      const uint32_t t1 = __shfl_sync(0xffffffffu, own_terms(w, base - 32 + 16 * lane, area, d.start, forced), 1);
      m = (uint64_t)(t0 | (t1 << 16)) << 1;
    }
    // the bytes of the first round before the segment (its start rounded down)
    const uint32_t pre = (uint32_t)(d.start - base);
    uint32_t t2 = 0;
    if (pre) t2 = own_terms(*reinterpret_cast<const uint4*>(bytes + base), base, area, d.start, forced);
    m |= (uint64_t)t2 << 33;
    const int64_t at = (int64_t)(area + 32) - (int64_t)base;  // the area's window offset
    if (at >= 0 && at <= 48) m |= 1ull << at;
    const int e1 = m ? 63 - __clzll((long long)m) : 0;
    m &= ~(1ull << e1);
    const int e0 = m ? 63 - __clzll((long long)m) : 0;
    if (lane == 0) {
      win->end[0] = (uint16_t)e0;
      win->end[1] = (uint16_t)e1;
    }
  }
  T run = 0;  // the deltas of the segment's rows so far
  for (; base < d.end; base += kRound) {
    const uint64_t o = base + 16ull * lane;
    w = make_uint4(0, 0, 0, 0);
    if (o < lim_pad) w = *reinterpret_cast<const uint4*>(bytes + o);
    reinterpret_cast<uint4*>(win->b)[2 + lane] = w;
    uint32_t own = own_terms(w, o, d.start, d.end, forced);
    const uint32_t c = __popc(own);
    uint32_t incl = c;
#pragma unroll
    for (int q = 1; q < 32; q <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, incl, q);
      if (lane >= (uint32_t)q) incl += y;
    }
    for (uint32_t at = 2 + incl - c; own; own &= own - 1, ++at) win->end[at] = (uint16_t)(32 + 16 * lane + __ffs(own));
    const uint32_t n = __shfl_sync(0xffffffffu, incl, 31);
    __syncwarp();
    // row j of the round: its count is own varint i = i0 + 2 j, its key the one before
    const uint32_t i0 = (v0 & 1ull) ? 0u : 1u;
    const uint32_t nr = n > i0 ? (n - i0 + 1) / 2 : 0u;
    const unsigned long long row0 = (v0 + i0 + 1) / 2;
    for (uint32_t j0 = 0; j0 < nr; j0 += 32) {
      const uint32_t j = j0 + lane, i = i0 + 2 * j;
      const bool in = j < nr && row0 + j < sd.rows;  // bytes after the last row are ignored, as the reference decodes row_count rows
      T delta = 0;
      unsigned long long cnt = 0;
      if (in) {
        const uint32_t a = win->end[i], b = win->end[i + 1], e = win->end[i + 2];
        delta = varint_in<T>(win, a, b);
        cnt = e - b == 1 ? (unsigned long long)(win->b[b] & 0x7fu) : (unsigned long long)(uint64_t)varint_in<T>(win, b, e);
      }
      const T sum = warp_incl_sum(delta);
      if (in) {
        keys[sd.row_off + row0 + j] = run + sum;
        counts[sd.row_off + row0 + j] = cnt;
      }
      run += warp_bcast_t(sum, 31);
    }
    v0 += n;
    // for the next round: the last 32 bytes and the last two ends
    __syncwarp();
    const uint16_t e0 = win->end[n], e1 = win->end[n + 1];
    const uint4 tail = reinterpret_cast<const uint4*>(win->b)[lane < 2 ? 32 + lane : 32];
    __syncwarp();
    if (lane < 2) {
      reinterpret_cast<uint4*>(win->b)[lane] = tail;
      const uint16_t x = lane ? e1 : e0;
      win->end[lane] = x > kRound ? (uint16_t)(x - kRound) : (uint16_t)0;
    }
    __syncwarp();
  }
  if (lane == 0) sums[si] = run;
}

// The segments' start keys added to their rows, one warp per segment.
template <class T>
__global__ void __launch_bounds__(32 * kDecWarps)
    k_seg_base(const SegDesc* __restrict__ segs, uint32_t nseg, const StreamDesc* __restrict__ streams,
               const uint32_t* __restrict__ terms, const unsigned long long* __restrict__ vstart,
               const T* __restrict__ kstart, T* __restrict__ keys) {
  const uint32_t lane = threadIdx.x & 31, si = blockIdx.x * kDecWarps + (threadIdx.x >> 5);
  if (si >= nseg) return;
  const StreamDesc sd = streams[segs[si].stream];
  const unsigned long long v = vstart[si], a = (v >> 1) + 1;
  const unsigned long long e = min((v + terms[si]) / 2 + 1, (unsigned long long)sd.rows);
  const T k = kstart[si];
  T* r = keys + sd.row_off;
  constexpr int kAhead = 4;
  for (unsigned long long i0 = a + lane; i0 < e; i0 += 32 * kAhead) {
    T x[kAhead];
#pragma unroll
    for (int j = 0; j < kAhead; ++j) x[j] = i0 + 32 * j < e ? r[i0 + 32 * j] : T(0);
#pragma unroll
    for (int j = 0; j < kAhead; ++j)
      if (i0 + 32 * j < e) r[i0 + 32 * j] = x[j] + k;
  }
}

// Head row of every DVLE stream of the list sids.
template <class T>
__global__ void k_stream_heads(const uint8_t* __restrict__ bytes, const StreamDesc* __restrict__ streams,
                               const uint32_t* __restrict__ sids, uint32_t nsid, T* __restrict__ keys,
                               unsigned long long* __restrict__ counts, T* __restrict__ first_keys) {
  const uint32_t w = blockIdx.x * blockDim.x + threadIdx.x;
  if (w >= nsid) return;
  const uint32_t i = sids[w];
  const StreamDesc sd = streams[i];
  if (sd.rows == 0 || sd.head == 0) return;
  const uint8_t* p = bytes + sd.byte_off;
  T k = 0;
  for (int b = 0; b < (int)sizeof(T); ++b) k |= (T)p[b] << (8 * b);
  uint32_t c = 0;
  for (int b = 0; b < 4; ++b) c |= (uint32_t)p[sizeof(T) + b] << (8 * b);
  keys[sd.row_off] = k;
  counts[sd.row_off] = c;
  first_keys[i] = k;
}

template <class T>
__global__ void k_raw_rows(const uint8_t* __restrict__ bytes, const StreamDesc* __restrict__ streams,
                           const uint32_t* __restrict__ raw_ids, uint32_t nraw, T* __restrict__ keys,
                           unsigned long long* __restrict__ counts) {
  // one CTA per RAW stream
  if (blockIdx.x >= nraw) return;
  const StreamDesc sd = streams[raw_ids[blockIdx.x]];
  const uint32_t es = sizeof(T) + 4;
  for (uint64_t r = threadIdx.x; r < sd.rows; r += blockDim.x) {
    const uint8_t* p = bytes + sd.byte_off + r * es;
    T k = 0;
    for (int b = 0; b < (int)sizeof(T); ++b) k |= (T)p[b] << (8 * b);
    uint32_t c = 0;
    for (int b = 0; b < 4; ++b) c |= (uint32_t)p[sizeof(T) + b] << (8 * b);
    keys[sd.row_off + r] = k;
    counts[sd.row_off + r] = c;
  }
}

// lower_bound of `key` in the sorted rows [lo, hi) of the decoded key array.
template <class T>
__global__ void k_lower_bound(const T* __restrict__ keys, const uint64_t* __restrict__ qlo,
                              const uint64_t* __restrict__ qhi, const T* __restrict__ qkey, uint32_t nq,
                              uint64_t* __restrict__ out) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nq) return;
  uint64_t lo = qlo[i], hi = qhi[i];
  const T key = qkey[i];
  while (lo < hi) {
    const uint64_t mid = lo + (hi - lo) / 2;
    if (keys[mid] < key) lo = mid + 1;
    else hi = mid;
  }
  out[i] = lo;
}

// Segment descriptors: segment i belongs to the stream sids[q] with
// first[q] <= i < first[q + 1].
__global__ void k_make_segs(const StreamDesc* __restrict__ streams, const uint32_t* __restrict__ sids,
                            const uint32_t* __restrict__ first, uint32_t nsid, uint32_t nseg,
                            SegDesc* __restrict__ segs) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nseg) return;
  uint32_t lo = 0, hi = nsid;
  while (hi - lo > 1) {
    const uint32_t m = (lo + hi) >> 1;
    if (first[m] <= i) lo = m;
    else hi = m;
  }
  const StreamDesc sd = streams[sids[lo]];
  SegDesc d;
  d.start = sd.byte_off + sd.head + (uint64_t)(i - first[lo]) * kSeg;
  d.end = min(d.start + kSeg, sd.byte_off + sd.byte_len);
  d.stream = sids[lo];
  d.first = i == first[lo];
  segs[i] = d;
}

// The sum over the partition's streams of a key's counts (u64, saturating:
// load_partition_counts src/kiteops/mod.rs:433-473), 0 when absent, for
// `kite query`: one lower bound per stream, no merge.
template <class T>
__global__ void k_query_streams(const T* __restrict__ keys, const unsigned long long* __restrict__ counts,
                                const StreamDesc* __restrict__ streams, const uint32_t* __restrict__ part_first,
                                const T* __restrict__ qk, const uint32_t* __restrict__ qp, uint32_t nq,
                                unsigned long long* __restrict__ out) {
  const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= nq) return;
  const T key = qk[q];
  const uint32_t p = qp[q];
  unsigned long long c = 0;
  for (uint32_t si = part_first[p]; si < part_first[p + 1]; ++si) {
    uint64_t lo = streams[si].row_off, hi = lo + streams[si].rows;
    const uint64_t end = hi;
    while (lo < hi) {
      const uint64_t mid = lo + (hi - lo) / 2;
      if (keys[mid] < key) lo = mid + 1;
      else hi = mid;
    }
    for (; lo < end && keys[lo] == key; ++lo) c = c > ~0ull - counts[lo] ? ~0ull : c + counts[lo];
  }
  out[q] = c;
}

// Row positions that cut a stream, the only one of its partition, every
// kMergeCap rows (between two different keys), S ranges: laid out as those of
// k_range_positions.
template <class T>
__global__ void k_slice_positions(const T* __restrict__ keys, const StreamDesc* __restrict__ streams, uint32_t nst,
                                  uint32_t S, uint64_t* __restrict__ pos) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (uint64_t)nst * (S + 1)) return;
  const StreamDesc sd = streams[i / (S + 1)];
  const uint64_t end = sd.row_off + sd.rows;
  uint64_t r = sd.row_off + min((uint64_t)(i % (S + 1)) * kMergeCap, sd.rows);
  if (i % (S + 1) == S) r = end;
  while (r > sd.row_off && r < end && keys[r] == keys[r - 1]) ++r;
  pos[i] = r;
}

// The tiles of a cut into S ranges per partition, tile p * S + j for range j
// of partition p, with every stream of the partition in order (some of them
// empty in the range).  info[0]: tiles above the on-chip capacity, [1] the
// largest tile, [2] tiles with rows.
__global__ void k_plan_tiles(const uint64_t* __restrict__ pos, const StreamDesc* __restrict__ streams,
                             const uint32_t* __restrict__ part_first, uint32_t P, uint32_t S,
                             MergeTile* __restrict__ tiles, TileStream* __restrict__ ts, TileDesc* __restrict__ tds,
                             unsigned* __restrict__ info) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= P * S) return;
  const uint32_t p = t / S, j = t % S, f = part_first[p], n = part_first[p + 1] - f;
  MergeTile mt;
  mt.first_ts = f * S + j * n;
  mt.nts = n;
  mt.partition = p;
  uint64_t rows = 0, before = 0;
  for (uint32_t k = 0; k < n; ++k) {
    const uint64_t* q = pos + (size_t)(f + k) * (S + 1) + j;
    const uint64_t lo = q[0], hi = q[1];
    TileStream x;
    x.lo = lo;
    x.hi = hi;
    x.input = streams[f + k].input;
    x.pad = 0;
    ts[mt.first_ts + k] = x;
    rows += hi - lo;
    before += lo - streams[f + k].row_off;
  }
  // a partition's rows follow those of the partitions before it
  mt.out_off = (n ? streams[f].row_off : 0) + before;
  mt.rows_in = rows > kMergeCap ? 0u : (uint32_t)rows;
  tiles[t] = mt;
  TileDesc td;
  td.start = mt.out_off;
  td.len = 0;
  td.bucket = p;
  tds[t] = td;
  if (rows > kMergeCap) atomicAdd(&info[0], 1u);
  if (rows) {
    atomicMax(&info[1], (unsigned)min(rows, (uint64_t)0xffffffffu));
    atomicAdd(&info[2], 1u);
  }
}

// Row position of every splitter in every stream: pos[s * (S + 1) + j] is
// lower_bound(spl[j - 1]) in stream s's rows for 1 <= j < S, the stream's
// first row for j = 0 and its end for j = S.
template <class T>
__global__ void k_range_positions(const T* __restrict__ keys, const StreamDesc* __restrict__ streams, uint32_t nst,
                                  const T* __restrict__ spl, uint32_t S, uint64_t* __restrict__ pos) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (uint64_t)nst * (S + 1)) return;
  const uint32_t si = (uint32_t)(i / (S + 1)), j = (uint32_t)(i % (S + 1));
  const StreamDesc sd = streams[si];
  uint64_t lo = sd.row_off, hi = sd.row_off + sd.rows;
  if (j == 0 || j == S) {
    pos[i] = j == 0 ? lo : hi;
    return;
  }
  const T key = spl[j - 1];
  while (lo < hi) {
    const uint64_t mid = lo + (hi - lo) / 2;
    if (keys[mid] < key) lo = mid + 1;
    else hi = mid;
  }
  pos[i] = lo;
}

template <class T>
__global__ void k_sample_rows(const T* __restrict__ keys, uint64_t nrows, uint32_t nsample, T* __restrict__ out) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nsample) return;
  out[i] = keys[(uint64_t)((unsigned __int128)i * nrows / nsample)];
}

template <class T>
struct MergeSmem {
  static constexpr size_t keys = (size_t)kMergeCap * sizeof(T);
  static constexpr size_t cnts = (size_t)kMergeCap * 8;
  static constexpr size_t tag = (size_t)kMergeCap * 2;
  static constexpr size_t perm = (size_t)kMergeCap * 2 * 2;  // two index arrays (merge rounds ping-pong)
  static constexpr size_t head = (size_t)(kMergeCap + 1) * 2;
  // every region starts 16-byte aligned (misc holds 8-byte scan values)
  static constexpr size_t seg = ((size_t)(kMaxTileStreams + 1) * 4 + kMaxTileStreams * 4 + 15) & ~(size_t)15;
  static constexpr size_t misc = 64 * 8;
  static constexpr size_t hist = (size_t)kHistBins * 4;  // histo mode: per-CTA bins of the small counts
  static constexpr size_t total = keys + cnts + tag + perm + ((head + 15) & ~(size_t)15) + seg + misc + hist;
};

// MODE kModeMerge: `kite merge` (per-input filter on the per-input sum, u64
// totals, overflow above u32 recorded).  kModeDump: `kite dump` of one input
// (the sum clamped to u32 first, the header filter on the clamped count;
// rest_bytes of a tile = its TSV bytes, lines of k + 2 + digits).
// kModeHisto: `kite histo` of one input (load_partition_counts' u64 sum,
// apply_reader_filter_to_rows on it, then the count's frequency; no rows
// written).
template <class T, int MODE>
__device__ __forceinline__ void merge_tile(
    const uint32_t tile, const T* __restrict__ keys, const unsigned long long* __restrict__ counts,
    const MergeTile* __restrict__ tiles, const TileStream* __restrict__ ts, const InputFilter* __restrict__ filt,
    T* __restrict__ out_keys, uint32_t* __restrict__ out_counts, TileOut<T>* __restrict__ tout,
    unsigned long long* __restrict__ overflow, DevStatus* st, const MergeAux& aux) {
  constexpr bool DUMP = MODE == kModeDump;
  using L = MergeSmem<T>;
  constexpr int NT = kMergeThreads;
  extern __shared__ __align__(16) uint8_t sm[];
  T* sk = reinterpret_cast<T*>(sm);
  unsigned long long* sc = reinterpret_cast<unsigned long long*>(sm + L::keys);
  uint16_t* stag = reinterpret_cast<uint16_t*>(sm + L::keys + L::cnts);
  uint16_t* perm_a = reinterpret_cast<uint16_t*>(sm + L::keys + L::cnts + L::tag);
  uint16_t* perm_b = perm_a + kMergeCap;
  uint16_t* head = reinterpret_cast<uint16_t*>(sm + L::keys + L::cnts + L::tag + L::perm);
  uint32_t* sstart = reinterpret_cast<uint32_t*>(sm + L::keys + L::cnts + L::tag + L::perm +
                                                 ((L::head + 15) & ~(size_t)15));
  uint32_t* sinput = sstart + kMaxTileStreams + 1;
  unsigned long long* misc = reinterpret_cast<unsigned long long*>(reinterpret_cast<uint8_t*>(sstart) + L::seg);
  unsigned* hbin = reinterpret_cast<unsigned*>(reinterpret_cast<uint8_t*>(misc) + L::misc);

  const MergeTile mt = tiles[tile];
  const uint32_t nts = mt.nts, n = mt.rows_in;
  if (n == 0 || nts == 0) {
    if (threadIdx.x == 0) {
      TileOut<T> o{};
      tout[tile] = o;
    }
    return;
  }
  if (n > kMergeCap || nts > kMaxTileStreams) {
    dev_fail(st, KITE_DEV_TILE_OVERFLOW, tile, n, nts);
    return;
  }
  if (threadIdx.x < 32) {
    // stream starts inside the tile: warp 0 scans the stream lengths
    uint32_t carry = 0;
    const uint32_t lane = threadIdx.x;
    for (uint32_t i0 = 0; i0 < nts; i0 += 32) {
      const uint32_t i = i0 + lane;
      uint32_t len = 0;
      if (i < nts) {
        const TileStream t = ts[mt.first_ts + i];
        len = (uint32_t)(t.hi - t.lo);
        sinput[i] = t.input;
      }
      uint32_t incl = len;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (uint32_t)o) incl += y;
      }
      if (i < nts) sstart[i] = carry + incl - len;
      carry += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) sstart[nts] = carry;
  }
  if (MODE == kModeHisto)
    for (uint32_t b = threadIdx.x; b < kHistBins; b += NT) hbin[b] = 0;
  __syncthreads();
  // load the rows of every stream: row r of the tile belongs to the last
  // stream starting at or before it
  for (uint32_t r = threadIdx.x; r < n; r += NT) {
    uint32_t lo = 0, hi = nts - 1;
    while (lo < hi) {
      const uint32_t mid = (lo + hi + 1) >> 1;
      if (sstart[mid] <= r) lo = mid;
      else hi = mid - 1;
    }
    const uint64_t src = ts[mt.first_ts + lo].lo + (r - sstart[lo]);
    sk[r] = keys[src];
    sc[r] = counts[src];
    stag[r] = (uint16_t)lo;
  }
  __syncthreads();
  // Merged order of the rows (ties in stream order): the sorted streams are
  // merged pairwise in rounds, run 2p with run 2p + 1, each round a merge
  // path (Green, McColl and Bader, 2012): thread t takes output positions
  // [t * PER, t * PER + PER) of the tile, finds where that range starts in
  // both runs of its pair by a diagonal binary search, then merges
  // sequentially.  Stable (equal keys: the earlier run first), so a group of
  // equal keys keeps stream order, i.e. input order, then chunk order.
  constexpr uint32_t PER = kMergeCap / NT;
  uint16_t* perm = perm_a;
  {
    uint16_t* src = perm_a;
    uint16_t* dst = perm_b;
    for (uint32_t r = threadIdx.x; r < n; r += NT) src[r] = (uint16_t)r;
    __syncthreads();
    for (uint32_t w = 1; w < nts; w <<= 1) {
      const uint32_t q0 = threadIdx.x * PER;
      if (q0 < n) {
        // the pair holding output q0: pairs start at stream multiples of 2w;
        // the last pair whose first row is <= q0 (empty pairs are passed over)
        uint32_t p = 0;
        {
          uint32_t lo = 0, hi = (nts + 2 * w - 1) / (2 * w) - 1;
          while (lo < hi) {
            const uint32_t mid = (lo + hi + 1) >> 1;
            if (sstart[min(mid * 2 * w, nts)] <= q0) lo = mid;
            else hi = mid - 1;
          }
          p = lo;
        }
        uint32_t q = q0;
        const uint32_t qend = min(q0 + PER, n);
        while (q < qend) {
          const uint32_t a0 = sstart[min(p * 2 * w, nts)], a1 = sstart[min(p * 2 * w + w, nts)],
                         b1 = sstart[min(p * 2 * w + 2 * w, nts)];
          const uint32_t la = a1 - a0, lb = b1 - a1, d = q - a0;
          // i = rows of run A among the pair's first d outputs
          uint32_t lo = d > lb ? d - lb : 0, hi = d < la ? d : la;
          while (lo < hi) {
            const uint32_t mid = (lo + hi) >> 1;
            if (sk[src[a0 + mid]] <= sk[src[a1 + d - 1 - mid]]) lo = mid + 1;
            else hi = mid;
          }
          uint32_t i = lo, j = d - lo;
          const uint32_t stop = min(qend, b1);
          for (; q < stop; ++q) {
            const bool take_a = i < la && (j >= lb || sk[src[a0 + i]] <= sk[src[a1 + j]]);
            dst[q] = take_a ? src[a0 + i++] : src[a1 + j++];
          }
          ++p;  // the range continues in the next pair
        }
      }
      __syncthreads();
      uint16_t* t = src;
      src = dst;
      dst = t;
    }
    perm = src;
  }
  // key-group heads in merged order
  const uint32_t q0 = threadIdx.x * PER;
  uint32_t nh = 0;
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const uint32_t q = q0 + i;
    if (q < n && (q == 0 || sk[perm[q]] != sk[perm[q - 1]])) nh++;
  }
  unsigned G;
  unsigned* scan32 = reinterpret_cast<unsigned*>(misc);
  unsigned g = block_exclusive_scan<NT, unsigned>(nh, scan32, &G);
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const uint32_t q = q0 + i;
    if (q < n && (q == 0 || sk[perm[q]] != sk[perm[q - 1]])) head[g++] = (uint16_t)q;
  }
  if (threadIdx.x == 0) head[G] = (uint16_t)n;
  __syncthreads();
  // per group: per-input sums (u64 saturating), input filter, total.  Each
  // thread takes a run of consecutive groups (at most PER: G <= n <= the
  // capacity), keeping their totals in registers; one block scan compacts
  // the present ones in group order, and their keys go to shared memory for
  // the DVLE sizes: over the row counts (read by then) for u64 keys, over the
  // row keys for u128 (whose group keys are then kept in registers).
  constexpr bool KEEP_KEYS = sizeof(T) > 8;
  unsigned long long rest = 0;
  T first_key = T(0), last_key = T(0);
  uint32_t first_count = 0;
  unsigned* scan_b = scan32 + 40;
  const uint32_t gpt = (G + NT - 1) / NT;
  const uint32_t g_lo = min(G, threadIdx.x * gpt), g_hi = min(G, g_lo + gpt);
  T gkey[PER];
  unsigned long long gtot[PER];
  uint32_t pmask = 0, npres = 0;
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    gkey[i] = T(0);
    gtot[i] = 0;
    const uint32_t gi = g_lo + i;
    if (gi < g_hi) {
      const uint32_t a = head[gi], b = head[gi + 1];
      if (KEEP_KEYS) gkey[i] = sk[perm[a]];
      bool present = false;
      unsigned long long total = 0;
      uint32_t cur_in = 0xffffffffu;
      unsigned long long part = 0;
      for (uint32_t q = a; q <= b; ++q) {
        const uint32_t in = q < b ? sinput[stag[perm[q]]] : 0xfffffffeu;
        if (in != cur_in) {
          if (cur_in != 0xffffffffu) {
            const InputFilter f = filt[cur_in];
            const unsigned long long eff = DUMP && part > 0xffffffffull ? 0xffffffffull : part;
            const bool ok = !(f.has_min && eff < f.min_count) && !(f.has_max && eff > f.max_count);
            if (ok) {
              total = (total > ~0ull - part) ? ~0ull : total + part;
              present = true;
            }
          }
          cur_in = in;
          part = 0;
        }
        if (q < b) {
          const unsigned long long c = sc[perm[q]];
          part = (part > ~0ull - c) ? ~0ull : part + c;
        }
      }
      gtot[i] = total;
      if (present) {
        pmask |= 1u << i;
        ++npres;
      }
    }
  }
  __syncthreads();  // every row count (and for u128 every row key) has been read
  unsigned tot;
  const unsigned base = block_exclusive_scan<NT, unsigned>(npres, scan_b, &tot);
  T* outk = KEEP_KEYS ? sk : reinterpret_cast<T*>(sc);  // the present groups' keys in output order
  if (!KEEP_KEYS) {
#pragma unroll
    for (int i = 0; i < PER; ++i)
      if ((pmask >> i) & 1u) gkey[i] = sk[perm[head[g_lo + i]]];
  }
  {
    unsigned o = base;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      if (!((pmask >> i) & 1u)) continue;
      const unsigned long long total = gtot[i];
      if (MODE == kModeHisto) {
        if (total < kHistBins) {
          atomicAdd(&hbin[total], 1u);
        } else {
          const unsigned long long j = atomicAdd(aux.spill_n, 1ull);
          if (j < aux.spill_cap) aux.spill[j] = total;
        }
      } else {
        if (MODE == kModeMerge && total > 0xffffffffull)
          atomicMin(overflow, ((unsigned long long)tile << 32) | (unsigned long long)o);
        const uint32_t c32 = total > 0xffffffffull ? 0xffffffffu : (uint32_t)total;
        out_keys[mt.out_off + o] = gkey[i];
        out_counts[mt.out_off + o] = c32;
        if (o == 0) misc[60] = c32;
      }
      outk[o] = gkey[i];
      ++o;
    }
  }
  __syncthreads();
  if (MODE == kModeMerge || MODE == kModeDump) {
    // DVLE sizes of the rows after the tile's first (TSV line sizes for dump)
    unsigned o = base;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      if (!((pmask >> i) & 1u)) continue;
      const uint32_t cc = gtot[i] > 0xffffffffull ? 0xffffffffu : (uint32_t)gtot[i];
      if (DUMP) rest += aux.line_k + 2 + dec_digits(cc);
      else if (o > 0) rest += (unsigned long long)(varint_len((T)(gkey[i] - outk[o - 1])) + varint_len((uint64_t)cc));
      ++o;
    }
  }
  if (MODE != kModeHisto && threadIdx.x == 0 && tot) {
    first_key = outk[0];
    first_count = (uint32_t)misc[60];
    last_key = outk[tot - 1];
  }
  const unsigned long long out_base = tot;
  if (MODE == kModeHisto) {
    // the CTA's small-count bins into the global histogram
    for (uint32_t b = threadIdx.x; b < kHistBins; b += NT)
      if (hbin[b]) atomicAdd(&aux.hist[b], (unsigned long long)hbin[b]);
  }
  unsigned long long rest_total;
  block_exclusive_scan<NT, unsigned long long>(rest, misc + 8, &rest_total);
  if (threadIdx.x == 0) {
    TileOut<T> o;
    o.first_key = first_key;
    o.last_key = last_key;
    o.rows = (uint32_t)out_base;
    o.first_count = first_count;
    o.rest_bytes = rest_total;
    tout[tile] = o;
  }
}

// One tile per CTA, or (list) the listed ones in turn.
template <class T, int MODE>
__global__ void __launch_bounds__(kMergeThreads) k_merge_tiles(
    const T* __restrict__ keys, const unsigned long long* __restrict__ counts, const MergeTile* __restrict__ tiles,
    const TileStream* __restrict__ ts, const InputFilter* __restrict__ filt, T* __restrict__ out_keys,
    uint32_t* __restrict__ out_counts, TileOut<T>* __restrict__ tout, unsigned long long* __restrict__ overflow,
    DevStatus* st, MergeAux aux, const uint32_t* __restrict__ list, const unsigned* __restrict__ nlist) {
  const uint32_t n = list ? *nlist : gridDim.x;
  for (uint32_t i = blockIdx.x; i < n; i += gridDim.x) {
    merge_tile<T, MODE>(list ? list[i] : i, keys, counts, tiles, ts, filt, out_keys, out_counts, tout, overflow, st, aux);
    __syncthreads();
  }
}

// ---- u64 tiles by a table -------------------------------------------------------
// What bounds a tile's merge is the work per row in shared memory: the merge
// rounds above read 13 keys per row and move row indices through three rounds
// for eight streams.  Here a row goes once into a table of keys and u32 sums
// whose homes are in key order, as in the tile sort, and the slots, their
// clusters put in order, are the merged rows.  A tile of one stream needs no
// table: its rows lie in the slots in order.  A tile goes to the kernel above,
// through a list, when a row's count is 0 or 2^19 and more (4,096 of them could
// pass 32 bits), when a key lands kProbeLimit slots from home, and when a chunk
// repeats a key that a filter or the one-stream path would meet.
// k = 31: 8 databases, 96M rows 3.85 -> 1.85 ms; histo of 64.6M rows in four chunks per
// partition 2.6 -> 1.1 ms; dump of 36.2M rows in one 1.4 -> 0.6 ms.  An AT-rich
// genome, where a third of the tiles fail, is the case against: 31M rows of four
// databases 1.5 -> 1.9 ms (with 16 probes instead of 32 1.8, and the first merge
// 2.1).
struct MergeTable {
  static constexpr int NT = 512, NW = NT / 32, SLOTS = 7168, UNROLL = 4;
  static constexpr size_t o_tab = 0;
  static constexpr size_t o_cnt = o_tab + (size_t)SLOTS * 8;
  static constexpr size_t o_ord = o_cnt + (size_t)SLOTS * 4;       // occupied slots in order (u16); histo: the bins
  static constexpr size_t o_queue = o_ord + (size_t)kMergeCap * 2;  // per warp: 64 keys and counts that probe on
  static constexpr size_t o_base = o_queue + (size_t)NW * 64 * 12;  // per stream: its first row less its place
  static constexpr size_t o_start = o_base + (size_t)kMaxTileStreams * 8;
  static constexpr size_t o_misc = o_start + (size_t)(kMaxTileStreams + 4) * 4;  // u64 range (2), then u32
  static constexpr size_t o_edge = o_misc + 64;
  static constexpr size_t total = o_edge + NW * 4;
  static_assert(kHistBins * 4 <= kMergeCap * 2, "the bins fit the order list");
  static_assert(total <= 115712, "two CTAs per SM");
};

template <int MODE>
__global__ void __launch_bounds__(MergeTable::NT, 2)
    k_merge_table(const uint64_t* __restrict__ keys, const unsigned long long* __restrict__ counts,
                  const MergeTile* __restrict__ tiles, uint32_t ntiles, const TileStream* __restrict__ ts,
                  const InputFilter* __restrict__ filt, uint32_t filtered, uint64_t* __restrict__ out_keys,
                  uint32_t* __restrict__ out_counts, TileOut<uint64_t>* __restrict__ tout, uint32_t* __restrict__ list,
                  unsigned* __restrict__ nlist, unsigned* __restrict__ met, MergeAux aux) {
  using L = MergeTable;
  constexpr int NT = L::NT, NW = L::NW, UN = L::UNROLL;
  constexpr unsigned long long kFree = ~0ull;
  extern __shared__ __align__(16) uint8_t sm[];
  unsigned long long* tab = reinterpret_cast<unsigned long long*>(sm + L::o_tab);
  unsigned* cnt = reinterpret_cast<unsigned*>(sm + L::o_cnt);
  uint16_t* ord = reinterpret_cast<uint16_t*>(sm + L::o_ord);
  unsigned* hbin = reinterpret_cast<unsigned*>(sm + L::o_ord);
  unsigned long long* sbase = reinterpret_cast<unsigned long long*>(sm + L::o_base);
  uint32_t* sstart = reinterpret_cast<uint32_t*>(sm + L::o_start);
  unsigned long long* range = reinterpret_cast<unsigned long long*>(sm + L::o_misc);
  unsigned* misc = reinterpret_cast<unsigned*>(sm + L::o_misc) + 4;  // [0] failed, [1] bytes, [2 + parity] listed
  unsigned* edge = reinterpret_cast<unsigned*>(sm + L::o_edge);
  const unsigned lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1u;
  unsigned long long* qkey = reinterpret_cast<unsigned long long*>(sm + L::o_queue) + wid * 64;
  unsigned* qcnt = reinterpret_cast<unsigned*>(sm + L::o_queue + (size_t)NW * 64 * 8) + wid * 64;
  const InputFilter f0 = filt[0];
  // dump and histo filter a key's sum, merge a row (a chunk has a key once)
  auto passes = [](const InputFilter& f, uint32_t c) {
    return !(f.has_min && c < f.min_count) && !(f.has_max && c > f.max_count);
  };
  unsigned ones = 0;  // histo: sums of 1, most of them
  if (MODE == kModeHisto)
    for (uint32_t b = threadIdx.x; b < kHistBins; b += NT) hbin[b] = 0;
  if (threadIdx.x < 2) misc[threadIdx.x] = 0;
  for (uint32_t tile = blockIdx.x, par = 0; tile < ntiles; tile += gridDim.x) {
    const MergeTile mt = tiles[tile];
    const uint32_t n = mt.rows_in, nts = mt.nts;
    if (n == 0 || nts == 0) {
      if (MODE != kModeHisto && threadIdx.x == 0) tout[tile] = TileOut<uint64_t>{};
      continue;
    }
    // data whose tiles often fail (met[1] of met[0] so far) is listed without
    // the try; one tile in 16 still tries
    if (threadIdx.x == 0) {
      const unsigned tried = *(volatile unsigned*)&met[0], failed = *(volatile unsigned*)&met[1];
      misc[2 + par] = n > kMergeCap || nts > kMaxTileStreams || (tried >= 32 && 3 * failed > tried && (tile & 15u));
    }
    __syncthreads();
    // The two places of the decision take turns over the tiles that have one
    // (an empty tile has none, and no barrier): it is written again only after
    // the next such tile's barrier, when every thread has read it.
    const bool listed = misc[2 + par];
    par ^= 1;
    if (listed) {
      if (threadIdx.x == 0) list[atomicAdd(nlist, 1u)] = tile;
      continue;
    }
    const bool single = nts == 1;
    // slots: twice the rows, in whole threads' shares
    const uint32_t slots = single ? (n + 15) & ~15u
                           : n < (uint32_t)L::SLOTS / 2 - 288 ? (2 * n + 64 + 511) & ~511u : (uint32_t)L::SLOTS;
    // ---- the streams (warp 0); the others clear the slots ----
    if (wid == 0) {
      uint32_t carry = 0;
      unsigned long long mn = ~0ull, mx = 0;
      for (uint32_t i0 = 0; i0 < nts; i0 += 32) {
        const uint32_t i = i0 + lane;
        TileStream t{};
        if (i < nts) t = ts[mt.first_ts + i];
        const uint32_t len = (uint32_t)(t.hi - t.lo);
        if (len) {
          mn = min(mn, (unsigned long long)keys[t.lo]);
          mx = max(mx, (unsigned long long)keys[t.hi - 1]);
        }
        const uint32_t incl = warp_inclusive(len, lane);
        if (i < nts) {
          sstart[i] = carry + incl - len;
          // the stream's input rides in the top bits: rows are far below 2^40
          sbase[i] = (t.lo - (carry + incl - len)) & ((1ull << 40) - 1) | (unsigned long long)t.input << 40;
        }
        carry += __shfl_sync(0xffffffffu, incl, 31);
      }
#pragma unroll
      for (int o = 16; o; o >>= 1) {
        mn = min(mn, __shfl_xor_sync(0xffffffffu, mn, o));
        mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      }
      if (lane == 0) {
        range[0] = mn;
        range[1] = mx;
      }
    } else {
      const uint32_t j0 = threadIdx.x - 32;
      if (!single)
        for (uint32_t j = j0; j < slots / 2; j += NT - 32) reinterpret_cast<uint4*>(tab)[j] = make_uint4(~0u, ~0u, ~0u, ~0u);
      for (uint32_t j = j0; j < slots / 4; j += NT - 32) reinterpret_cast<uint4*>(cnt)[j] = make_uint4(0, 0, 0, 0);
    }
    __syncthreads();
    // ---- the rows, UN at a time per thread so that their loads overlap ----
    {
      const RangeMap<uint64_t> map(range[0], range[1]);
      const HomeLinear<uint64_t> home(map, range[1], single ? 1u : slots - 2 * kProbeLimit);
      bool bad = false;
      uint32_t nq = 0;
      auto probe = [&](uint32_t m) {  // the last m queued rows
        __syncwarp();
        nq -= m;
        if (lane < m) {
          const unsigned long long v = qkey[nq + lane];
          uint32_t s = home(v);
          const uint32_t end = s + kProbeLimit;
          for (;;) {
            if (++s == end) {
              bad = true;
              break;
            }
            const unsigned long long x = atomicCAS(&tab[s], kFree, v);
            if (x == kFree || x == v) {
              atomicAdd(&cnt[s], qcnt[nq + lane]);
              break;
            }
          }
        }
        __syncwarp();
      };
      uint32_t si = 0;  // the stream of the thread's row
      for (uint32_t r0 = threadIdx.x; r0 - threadIdx.x < n; r0 += NT * UN) {
        unsigned long long v[UN], old[UN];
        uint32_t c[UN], h[UN];
        bool in[UN];
#pragma unroll
        for (int q = 0; q < UN; ++q) {
          const uint32_t r = r0 + q * NT;
          in[q] = r < n;
          v[q] = kFree;
          c[q] = 0;
          if (in[q]) {
            if (!single) {  // the last stream that starts at or before the row
              uint32_t hi = nts - 1;
              while (si < hi) {
                const uint32_t mid = (si + hi + 1) >> 1;
                if (sstart[mid] <= r) si = mid;
                else hi = mid - 1;
              }
            }
            const unsigned long long sb = sbase[si];
            const uint64_t src = (sb + r) & ((1ull << 40) - 1);
            v[q] = keys[src];
            const unsigned long long w = counts[src];
            bad |= w - 1 >= (1u << 19) - 1 || v[q] == kFree;
            c[q] = (uint32_t)w;
            // the row before it in its stream must have another key
            if ((single || (MODE == kModeMerge && filtered)) && r > sstart[si]) bad |= keys[src - 1] >= v[q];
            if (MODE == kModeMerge && filtered) in[q] = passes(filt[sb >> 40], c[q]);
          }
        }
        if (single) {
#pragma unroll
          for (int q = 0; q < UN; ++q)
            if (r0 + q * NT < n) {
              tab[r0 + q * NT] = v[q];
              cnt[r0 + q * NT] = in[q] ? c[q] : 0u;
            }
          continue;
        }
#pragma unroll
        for (int q = 0; q < UN; ++q) {
          h[q] = home(v[q]);
          old[q] = in[q] ? atomicCAS(&tab[h[q]], kFree, v[q]) : kFree;
        }
#pragma unroll
        for (int q = 0; q < UN; ++q) {
          const bool hit = old[q] == kFree || old[q] == v[q];
          if (hit && in[q]) atomicAdd(&cnt[h[q]], c[q]);
          const unsigned miss = __ballot_sync(0xffffffffu, !hit);
          if (miss) {
            if (!hit) {
              const uint32_t j = nq + __popc(miss & lt);
              qkey[j] = v[q];
              qcnt[j] = c[q];
            }
            nq += __popc(miss);
            if (nq >= 32) probe(32);
          }
        }
        if (__any_sync(0xffffffffu, bad)) break;
      }
      if (nq) probe(nq);
      if (bad) misc[0] = 1;
    }
    __syncthreads();
    if (misc[0]) {
      __syncthreads();
      if (threadIdx.x == 0) {
        list[atomicAdd(nlist, 1u)] = tile;
        misc[0] = 0;
        atomicAdd(&met[1], 1u);
        atomicAdd(&met[0], 1u);
      }
      continue;
    }
    if (threadIdx.x == 0) atomicAdd(&met[0], 1u);
    if (MODE == kModeHisto) {
      for (uint32_t j = threadIdx.x; j < slots; j += NT) {
        const uint32_t c = cnt[j];
        if (c == 0 || !passes(f0, c)) continue;
        if (c == 1) {
          ++ones;
        } else if (c < kHistBins) {
          atomicAdd(&hbin[c], 1u);
        } else {
          const unsigned long long at = atomicAdd(aux.spill_n, 1ull);
          if (at < aux.spill_cap) aux.spill[at] = c;
        }
      }
      __syncthreads();
      continue;
    }
    // ---- clusters in order (one lane each), then the thread's 16 slots listed ----
    const uint32_t a = threadIdx.x * 16;
    auto used = [&](auto&& ok) {
      uint32_t m = 0;
      if (a < slots) {
        const uint4* c4 = reinterpret_cast<const uint4*>(cnt + a);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint4 x = c4[j];
          m |= (ok(x.x) ? 1u << (4 * j) : 0u) | (ok(x.y) ? 2u << (4 * j) : 0u) | (ok(x.z) ? 4u << (4 * j) : 0u) |
               (ok(x.w) ? 8u << (4 * j) : 0u);
        }
      }
      return m;
    };
    uint32_t mine = used([](uint32_t c) { return c != 0; });
    if (!single) {
      const uint32_t before = a && a < slots && cnt[a - 1], after = a + 16 < slots && cnt[a + 16];
      const uint32_t multi = mine & ~((mine << 1) | before) & ((mine >> 1) | (after << 15));
      const unsigned inc = warp_inclusive(__popc(multi), lane);
      uint16_t* first = reinterpret_cast<uint16_t*>(qkey);
      unsigned p = inc - __popc(multi);
      for (uint32_t m = multi; m; m &= m - 1) first[p++] = (uint16_t)(a + __ffs(m) - 1);
      const unsigned nc = __shfl_sync(0xffffffffu, inc, 31);
      __syncthreads();  // every warp has read the counts
      for (unsigned j = lane; j < nc; j += 32) order_cluster(tab, cnt, first[j], slots);
      __syncthreads();
    }
    if (MODE == kModeDump && filtered) mine = used([&](uint32_t c) { return c != 0 && passes(f0, c); });
    unsigned U;
    {
      const unsigned inc = warp_inclusive(__popc(mine), lane);
      if (lane == 31) edge[wid] = inc;
      __syncthreads();
      const unsigned wt = lane < (unsigned)NW ? edge[lane] : 0u;
      const unsigned wi = warp_inclusive(wt, lane);
      U = __shfl_sync(0xffffffffu, wi, NW - 1);
      unsigned u = __shfl_sync(0xffffffffu, wi - wt, wid) + inc - __popc(mine);
      for (uint32_t m = mine; m; m &= m - 1) ord[u++] = (uint16_t)(a + __ffs(m) - 1);
    }
    __syncthreads();
    if (U == 0) {
      if (threadIdx.x == 0) tout[tile] = TileOut<uint64_t>{};
      continue;
    }
    const uint32_t line = aux.line_k + 2;
    write_rows<NT>(
        U, out_keys + mt.out_off, out_counts + mt.out_off, &misc[1], &tout[tile],
        [&](unsigned u, uint64_t* key, uint32_t* c) {
          const uint32_t s = ord[u];
          *key = tab[s];
          *c = cnt[s];
        },
        [&](unsigned u, uint64_t delta, uint32_t c) {
          return MODE == kModeDump ? line + dec_digits(c) : dvle_size<uint64_t>(u, delta, c);
        });
  }
  if (MODE == kModeHisto) {
    __syncthreads();
    ones = __reduce_add_sync(0xffffffffu, ones);
    if (lane == 0 && ones) atomicAdd(&hbin[1], ones);
    __syncthreads();
    for (uint32_t b = threadIdx.x; b < kHistBins; b += NT)
      if (hbin[b]) atomicAdd(&aux.hist[b], (unsigned long long)hbin[b]);
  }
}

// TSV lines of one merged tile: rows in rounds of kTsvThreads, each round's
// lines assembled in shared memory (block scan of the line lengths), then
// stored as one contiguous run of bytes at the tile's output offset.
template <class T>
__global__ void __launch_bounds__(kTsvThreads) k_tsv_tiles(const T* __restrict__ keys,
                                                           const uint32_t* __restrict__ counts,
                                                           const MergeTile* __restrict__ tiles,
                                                           const TileOut<T>* __restrict__ tout,
                                                           const unsigned long long* __restrict__ tboff, uint32_t k,
                                                           uint8_t* __restrict__ out) {
  constexpr int NT = kTsvThreads;
  extern __shared__ __align__(16) uint8_t sm[];
  unsigned* scan = reinterpret_cast<unsigned*>(sm);
  char* buf = reinterpret_cast<char*>(sm + 256);
  const uint64_t base = tiles[blockIdx.x].out_off;
  const uint32_t rows = tout[blockIdx.x].rows;
  unsigned long long dst = tboff[blockIdx.x];
  for (uint32_t r0 = 0; r0 < rows; r0 += NT) {
    const uint32_t r = r0 + threadIdx.x;
    T key = T(0);
    uint32_t c = 0;
    unsigned len = 0;
    if (r < rows) {
      key = keys[base + r];
      c = counts[base + r];
      len = k + 2 + dec_digits(c);
    }
    unsigned tot;
    const unsigned o = block_exclusive_scan<NT, unsigned>(len, scan, &tot);
    if (len) {
      char* p = buf + o;
      for (uint32_t i = 0; i < k; ++i) p[i] = "ACGT"[(unsigned)(key >> (2 * (k - 1 - i))) & 3u];
      p[k] = '\t';
      uint32_t v = c;
      for (unsigned i = len - 2; i > k; --i) {
        p[i] = (char)('0' + v % 10);
        v /= 10;
      }
      p[len - 1] = '\n';
    }
    __syncthreads();
    // 4-byte stores on 4-byte aligned addresses; the unaligned head and tail
    // bytes one by one
    uint8_t* d8 = out + dst;
    const unsigned head = (unsigned)((4u - ((uintptr_t)d8 & 3u)) & 3u);
    if (tot < head + 8u) {
      for (unsigned i = threadIdx.x; i < tot; i += NT) d8[i] = (uint8_t)buf[i];
    } else {
      const unsigned body = (tot - head) & ~3u, tail = tot - head - body;
      if (threadIdx.x < head) d8[threadIdx.x] = (uint8_t)buf[threadIdx.x];
      if (threadIdx.x < tail) d8[head + body + threadIdx.x] = (uint8_t)buf[head + body + threadIdx.x];
      uint32_t* dw = reinterpret_cast<uint32_t*>(d8 + head);
      for (unsigned i = threadIdx.x; i < body / 4; i += NT) {
        const uint8_t* b = reinterpret_cast<const uint8_t*>(buf) + head + 4 * i;
        dw[i] = (uint32_t)b[0] | ((uint32_t)b[1] << 8) | ((uint32_t)b[2] << 16) | ((uint32_t)b[3] << 24);
      }
    }
    dst += tot;
    __syncthreads();
  }
}

// Dump: a partition's lines, bytes and key range from its tiles' records, one
// warp per partition; tile byte counts for the scan of their offsets.
struct PartLines {
  unsigned long long rows, bytes, kmin_lo, kmin_hi, kmax_lo, kmax_hi;
};
template <class T>
__global__ void k_part_lines(const TileOut<T>* __restrict__ tout, const uint32_t* __restrict__ tile_first, uint32_t P,
                             unsigned long long* __restrict__ tile_bytes, PartLines* __restrict__ out) {
  const uint32_t lane = threadIdx.x & 31, p = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (p >= P) return;
  PartLines x{};
  bool have = false;
  T kmin = T(0), kmax = T(0);
  for (uint32_t t0 = tile_first[p]; t0 < tile_first[p + 1]; t0 += 32) {
    const uint32_t t = t0 + lane;
    TileOut<T> o{};
    if (t < tile_first[p + 1]) {
      o = tout[t];
      tile_bytes[t] = o.rest_bytes;
    }
    const unsigned any = __ballot_sync(0xffffffffu, o.rows > 0);
    if (!any) continue;
    x.rows += __reduce_add_sync(0xffffffffu, o.rows);
    x.bytes += warp_bcast_t(warp_incl_sum((unsigned long long)o.rest_bytes), 31);
    const T lo = warp_bcast_t(o.first_key, __ffs(any) - 1);
    kmax = warp_bcast_t(o.last_key, 31 - __clz(any));
    if (!have) kmin = lo;
    have = true;
  }
  if (lane == 0) {
    x.kmin_lo = (unsigned long long)kmin;
    x.kmin_hi = hi64(kmin);
    x.kmax_lo = (unsigned long long)kmax;
    x.kmax_hi = hi64(kmax);
    out[p] = x;
  }
}

// ---- host side -----------------------------------------------------------------
// A device buffer of the call: its own allocation, or a slot of the
// context's pool (kept after the call).
struct Dev {
  MergePoolSlot own;
  MergePoolSlot* sl = &own;
  void* p = nullptr;
  size_t cap = 0;
  Dev() = default;
  Dev(MergePool* pool, int slot) : sl(pool ? &pool->slot[slot] : &own) {}
  Dev(const Dev&) = delete;
  Dev& operator=(const Dev&) = delete;
  bool ensure(size_t b) {
    if (b > sl->cap) {
      cudaFree(sl->p);
      sl->p = nullptr;
      sl->cap = 0;
      if (cudaMalloc(&sl->p, b + 256) != cudaSuccess) return false;
      sl->cap = b + 256;
    }
    p = sl->p;
    cap = sl->cap;
    return true;
  }
  ~Dev() {
    if (sl == &own) cudaFree(own.p);
  }
  template <class U> U* as() { return static_cast<U*>(p); }
};

// Pinned host memory of the call, its own or a slot of the pool's.
struct Pinned {
  MergePoolSlot own;
  MergePoolSlot* sl = &own;
  explicit Pinned(MergePoolSlot* slot) : sl(slot ? slot : &own) {}
  Pinned(const Pinned&) = delete;
  Pinned& operator=(const Pinned&) = delete;
  bool ensure(size_t b) {
    if (b <= sl->cap) return true;
    if (sl->p) cudaFreeHost(sl->p);
    sl->p = nullptr;
    sl->cap = 0;
    if (cudaMallocHost(&sl->p, b) != cudaSuccess) return false;
    sl->cap = b;
    return true;
  }
  ~Pinned() {
    if (own.p) cudaFreeHost(own.p);
  }
  template <class U> U* as() { return static_cast<U*>(sl->p); }
};

// What the host reads back in fixed sizes.
struct HostResults {
  DevStatus decode, run, encode;
  unsigned plan[3];                         // see k_plan_tiles
  unsigned long long over[8];               // per group: its first overflowing row
  unsigned long long hist[kHistBins + 1];   // histo: the bins, and the counts listed
};

template <class T>
int merge_typed(uint32_t P, uint32_t key_bits, const kite_gpu_merge_input* in, int n, cudaStream_t s,
                uint32_t timeout_ms, int mode, kite_gpu_emit_fn emit, void* user, std::string* msg,
                kite_gpu_stats* stat, const StagingFn& staging, const MergeExtra* ex) {
  const bool dump = mode == kModeDump;
  auto fail = [&](int code, const std::string& m) {
    *msg = m;
    return code;
  };
#define MCU(call)                                                                      \
  do {                                                                                 \
    cudaError_t _e = (call);                                                           \
    if (_e != cudaSuccess) return fail(KITE_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(_e)); \
  } while (0)
  auto bad_delta = [&]() {
    return fail(KITE_ERR_BAD_INPUT, sizeof(T) == 8 ? "invalid u64 DVLE delta" : "invalid u128 DVLE delta");
  };
  auto sync = [&]() { return bounded_sync(s, timeout_ms); };
  const uint32_t head_bytes = sizeof(T) + 4;
  // stage timing: [0] decode, [1] tile planning, [2] merge, [3] encode or
  // TSV formatting, [4] copy of the output to the host (events 0-3 back to
  // back, then 4-6 around the last two stages)
  cudaEvent_t sev[7];
  for (auto& e : sev)
    if (cudaEventCreate(&e) != cudaSuccess) return fail(KITE_ERR_CUDA, "event create");
  struct EvGuard {
    cudaEvent_t* e;
    ~EvGuard() {
      for (int i = 0; i < 7; ++i) cudaEventDestroy(e[i]);
    }
  } ev_guard{sev};
  for (int i = 0; i < 12; ++i) stat->stage_ms[i] = 0;
  // ---- streams (one per input chunk), bytes to the device ----
  std::vector<StreamDesc> streams;
  std::vector<uint64_t> in_base(n);
  uint64_t total_bytes = 0, total_rows = 0;
  std::vector<std::pair<uint64_t, uint64_t>> in_span(n);  // file [lo, hi) of payload bytes
  for (int i = 0; i < n; ++i) {
    uint64_t lo = UINT64_MAX, hi = 0;
    uint64_t nch = 0;
    for (uint32_t p = 0; p < P; ++p) nch = std::max<uint64_t>(nch, in[i].part_first[p] + in[i].part_count[p]);
    for (uint64_t c = 0; c < nch; ++c) {
      const uint64_t off = in[i].chunk_offset[c], len = in[i].chunk_len[c];
      if (off > in[i].base_len || len > in[i].base_len - off)
        return fail(KITE_ERR_BAD_INPUT, "chunk out of bounds in input #" + std::to_string(i + 1));
      lo = std::min(lo, off);
      hi = std::max(hi, off + len);
    }
    if (nch == 0) lo = hi = 0;
    in_span[i] = {lo, hi};
    in_base[i] = total_bytes;
    total_bytes += (hi - lo + 15) & ~15ull;
  }
  for (uint32_t p = 0; p < P; ++p)
    for (int i = 0; i < n; ++i)
      for (uint64_t c = in[i].part_first[p]; c < in[i].part_first[p] + in[i].part_count[p]; ++c) {
        const uint32_t codec = in[i].chunk_codec[c];
        if (codec & KITE_CODEC_ZSTD) return fail(KITE_ERR_UNSUPPORTED, "zstd chunks are not supported by the GPU merge");
        StreamDesc sd{};
        sd.byte_off = in_base[i] + in[i].chunk_offset[c] - in_span[i].first;
        sd.byte_len = in[i].chunk_len[c];
        sd.rows = in[i].chunk_rows[c];
        sd.row_off = total_rows;
        sd.codec = codec;
        sd.input = (uint32_t)i;
        sd.partition = p;
        sd.head = (codec & KITE_CODEC_DVLE) ? head_bytes : 0;
        if (sd.rows && (codec & KITE_CODEC_DVLE) && sd.byte_len < head_bytes)
          return fail(KITE_ERR_BAD_INPUT, sizeof(T) == 8 ? "u64 DVLE payload too small" : "u128 DVLE payload too small");
        // two varints a row, of a byte at least (the decode counts them)
        if (sd.rows && sd.head && sd.rows - 1 > (sd.byte_len - head_bytes) / 2) return bad_delta();
        if (sd.rows && !(codec & KITE_CODEC_DVLE) && sd.rows > sd.byte_len / head_bytes)
          return fail(KITE_ERR_BAD_INPUT, "raw row payload truncated");
        total_rows += sd.rows;
        streams.push_back(sd);
      }
  stat->h2d_bytes += total_bytes;
  MergePool* pool = ex ? ex->pool : nullptr;
  // The host reads device memory back into pinned memory, or into its own
  // after a wait: a copy to pageable memory that is queued behind kernels waits
  // for them inside the copy call, without the deadline.
  Pinned h_results(pool ? &pool->results : nullptr), h_rows(pool ? &pool->rows : nullptr);
  if (!h_results.ensure(sizeof(HostResults))) return fail(KITE_ERR_OOM, "merge results (pinned)");
  HostResults* hr = h_results.as<HostResults>();
  Dev d_bytes(pool, 0), d_streams(pool, 1), d_segs(pool, 2), d_terms(pool, 3), d_vstart(pool, 4), d_dsum(pool, 5),
      d_qseg(pool, 6), d_pfirst(pool, 7), d_status(pool, 8), d_sids(pool, 9), d_kstart(pool, 10), d_keys(pool, 11),
      d_counts(pool, 12), d_first(pool, 13), d_raw(pool, 14);
  if (!d_bytes.ensure(total_bytes + 64)) return fail(KITE_ERR_OOM, "device bytes");
  // ---- pieces: runs of an input's streams in file order, of about a
  // sixteenth of all bytes (8 MiB at least).  Each piece's bytes come in on a
  // side stream and its streams are decoded as soon as they have landed, so
  // the copies of later pieces overlap the decode of earlier ones ----
  struct Piece {
    uint64_t lo, hi;        // device byte range copied for it
    int input;
    uint32_t q0, q1;        // its streams in sids
  };
  std::vector<Piece> pieces;
  std::vector<uint32_t> raw_ids, sids, qseg;  // RAW streams; DVLE streams with rows; each one's first segment
  uint64_t nseg64 = 0;
  {
    std::vector<std::vector<uint32_t>> by_input(n);
    for (uint32_t si = 0; si < streams.size(); ++si) by_input[streams[si].input].push_back(si);
    const uint64_t target = std::max<uint64_t>(8ull << 20, total_bytes / 16);
    for (int i = 0; i < n; ++i) {
      auto& v = by_input[i];
      std::sort(v.begin(), v.end(),
                [&](uint32_t x, uint32_t y) { return streams[x].byte_off < streams[y].byte_off; });
      const uint64_t in_end = in_base[i] + (in_span[i].second - in_span[i].first);
      uint64_t at = in_base[i], reach = at;
      uint32_t q0 = (uint32_t)sids.size();
      for (size_t j = 0; j < v.size(); ++j) {
        const StreamDesc& sd = streams[v[j]];
        if (sd.byte_off > reach + (1u << 20)) {
          // a query's partitions lie apart: what lies between is not copied
          if (reach > at) pieces.push_back(Piece{at, reach, i, q0, (uint32_t)sids.size()});
          at = reach = sd.byte_off;
          q0 = (uint32_t)sids.size();
        }
        if (sd.rows && sd.head) {
          sids.push_back(v[j]);
          qseg.push_back((uint32_t)nseg64);
          nseg64 += (sd.byte_len - sd.head + kSeg - 1) / kSeg;
        } else if (sd.rows) {
          raw_ids.push_back(v[j]);
        }
        reach = std::max(reach, sd.byte_off + sd.byte_len);
        if (reach - at >= target && j + 1 < v.size()) {
          pieces.push_back(Piece{at, reach, i, q0, (uint32_t)sids.size()});
          at = reach;
          q0 = (uint32_t)sids.size();
        }
      }
      pieces.push_back(Piece{at, mode == kModeQuery ? reach : in_end, i, q0, (uint32_t)sids.size()});
    }
    qseg.push_back((uint32_t)nseg64);
  }
  const uint32_t nseg = (uint32_t)nseg64, nst = (uint32_t)streams.size(), nsid = (uint32_t)sids.size();
  std::vector<uint32_t> part_first_stream(P + 1, 0);
  uint32_t most_streams = 0;   // of a partition
  uint64_t most_rows = 0;
  {
    uint32_t si = 0;
    for (uint32_t p = 0; p < P; ++p) {
      part_first_stream[p] = si;
      uint64_t rows = 0;
      while (si < nst && streams[si].partition == p) rows += streams[si++].rows;
      most_streams = std::max(most_streams, si - part_first_stream[p]);
      most_rows = std::max(most_rows, rows);
    }
    part_first_stream[P] = nst;
  }
  if (!d_streams.ensure(nst * sizeof(StreamDesc) + 8) || !d_segs.ensure(nseg * sizeof(SegDesc) + 8) ||
      !d_terms.ensure(nseg * 4 + 8) || !d_vstart.ensure(nseg * 8 + 8) || !d_dsum.ensure(nseg * sizeof(T) + 16) ||
      !d_kstart.ensure(nseg * sizeof(T) + 16) || !d_keys.ensure(total_rows * sizeof(T) + 16) ||
      !d_counts.ensure(total_rows * 8 + 16) || !d_first.ensure(nst * sizeof(T) + 16) ||
      !d_raw.ensure(raw_ids.size() * 4 + 8) || !d_qseg.ensure(qseg.size() * 4 + 8) ||
      !d_pfirst.ensure((P + 1) * 4) || !d_sids.ensure(nsid * 4 + 8) || !d_status.ensure(2 * sizeof(DevStatus) + 64))
    return fail(KITE_ERR_OOM, "merge decode buffers");
  DevStatus* dst = d_status.as<DevStatus>();
  DevStatus* est = dst + 1;                                           // of the encode
  unsigned* plan_info = reinterpret_cast<unsigned*>(est + 1);         // of the tile plan
  MCU(cudaMemsetAsync(d_status.p, 0, 2 * sizeof(DevStatus) + 64, s));
  // copy lane: the side stream, one landing event per piece, timing events
  // around the copies ([0], [1]) and around each piece's decode ([2 + 2i],
  // [3 + 2i]: recorded after the wait, so they time the kernels only)
  struct CopyLane {
    cudaStream_t cs = nullptr;
    std::vector<cudaEvent_t> ev, tev;
    ~CopyLane() {
      for (auto e : ev) cudaEventDestroy(e);
      for (auto e : tev) cudaEventDestroy(e);
      if (cs) cudaStreamDestroy(cs);
    }
  } cl;
  const size_t np = pieces.size();
  MCU(cudaStreamCreateWithFlags(&cl.cs, cudaStreamNonBlocking));
  cl.ev.resize(np, nullptr);
  for (auto& e : cl.ev) MCU(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  cl.tev.resize(2 + 2 * np, nullptr);
  for (auto& e : cl.tev) MCU(cudaEventCreate(&e));
  MCU(cudaEventRecord(sev[0], s));
  MCU(cudaEventRecord(cl.tev[0], cl.cs));
  for (size_t i = 0; i < np; ++i) {
    const Piece& pc = pieces[i];
    if (pc.hi > pc.lo)
      MCU(cudaMemcpyAsync(d_bytes.as<uint8_t>() + pc.lo,
                          in[pc.input].base + in_span[pc.input].first + (pc.lo - in_base[pc.input]), pc.hi - pc.lo,
                          cudaMemcpyHostToDevice, cl.cs));
    MCU(cudaEventRecord(cl.ev[i], cl.cs));
  }
  MCU(cudaEventRecord(cl.tev[1], cl.cs));
  MCU(cudaMemcpyAsync(d_pfirst.p, part_first_stream.data(), (P + 1) * 4, cudaMemcpyHostToDevice, s));
  if (nst) MCU(cudaMemcpyAsync(d_streams.p, streams.data(), nst * sizeof(StreamDesc), cudaMemcpyHostToDevice, s));
  if (nsid) {
    MCU(cudaMemcpyAsync(d_sids.p, sids.data(), nsid * 4, cudaMemcpyHostToDevice, s));
    MCU(cudaMemcpyAsync(d_qseg.p, qseg.data(), qseg.size() * 4, cudaMemcpyHostToDevice, s));
  }
  if (!raw_ids.empty())
    MCU(cudaMemcpyAsync(d_raw.p, raw_ids.data(), raw_ids.size() * 4, cudaMemcpyHostToDevice, s));
  int launches = 0;
  if (nseg) {
    k_make_segs<<<(nseg + 255) / 256, 256, 0, s>>>(d_streams.as<StreamDesc>(), d_sids.as<uint32_t>(),
                                                   d_qseg.as<uint32_t>(), nsid, nseg, d_segs.as<SegDesc>());
    launches++;
  }
  const uint64_t lim_pad = total_bytes + 64;  // every aligned 16-byte block below this is readable
  for (size_t i = 0; i < np; ++i) {
    const Piece& pc = pieces[i];
    MCU(cudaStreamWaitEvent(s, cl.ev[i], 0));
    MCU(cudaEventRecord(cl.tev[2 + 2 * i], s));
    const uint32_t q0 = pc.q0, nq = pc.q1 - pc.q0, s0 = qseg[pc.q0], ns = qseg[pc.q1] - s0;
    if (nq) {
      k_stream_heads<T><<<(nq + 255) / 256, 256, 0, s>>>(d_bytes.as<uint8_t>(), d_streams.as<StreamDesc>(),
                                                         d_sids.as<uint32_t>() + q0, nq, d_keys.as<T>(),
                                                         d_counts.as<unsigned long long>(), d_first.as<T>());
      launches++;
    }
    const unsigned gsegs = (ns + kDecWarps - 1) / kDecWarps;
    if (ns)
      k_seg_count<<<gsegs, 32 * kDecWarps, 0, s>>>(d_bytes.as<uint8_t>(), lim_pad, d_segs.as<SegDesc>() + s0, ns,
                                                   d_streams.as<StreamDesc>(), d_terms.as<uint32_t>() + s0);
    if (nq)
      k_stream_seg_scan<<<(nq + 7) / 8, 256, 0, s>>>(d_terms.as<uint32_t>(), d_qseg.as<uint32_t>() + q0,
                                                     d_streams.as<StreamDesc>(), d_sids.as<uint32_t>() + q0, nq,
                                                     d_vstart.as<unsigned long long>(), dst);
    if (ns) {
      k_seg_rows<T><<<gsegs, 32 * kDecWarps, 0, s>>>(d_bytes.as<uint8_t>(), lim_pad, d_segs.as<SegDesc>() + s0, ns,
                                                     d_streams.as<StreamDesc>(), d_vstart.as<unsigned long long>() + s0,
                                                     d_keys.as<T>(), d_counts.as<unsigned long long>(),
                                                     d_dsum.as<T>() + s0);
      k_stream_base_scan<T><<<(nq + 7) / 8, 256, 0, s>>>(d_dsum.as<T>(), d_qseg.as<uint32_t>() + q0, d_first.as<T>(),
                                                         d_sids.as<uint32_t>() + q0, nq, d_kstart.as<T>());
      k_seg_base<T><<<gsegs, 32 * kDecWarps, 0, s>>>(d_segs.as<SegDesc>() + s0, ns, d_streams.as<StreamDesc>(),
                                                     d_terms.as<uint32_t>() + s0,
                                                     d_vstart.as<unsigned long long>() + s0, d_kstart.as<T>() + s0,
                                                     d_keys.as<T>());
      launches += 5;
    }
    MCU(cudaEventRecord(cl.tev[3 + 2 * i], s));
  }
  if (!raw_ids.empty()) {
    k_raw_rows<T><<<(unsigned)raw_ids.size(), 256, 0, s>>>(d_bytes.as<uint8_t>(), d_streams.as<StreamDesc>(),
                                                           d_raw.as<uint32_t>(), (uint32_t)raw_ids.size(),
                                                           d_keys.as<T>(), d_counts.as<unsigned long long>());
    launches++;
  }
  // stage times of the decode ([0], its kernels alone) and the copies in ([5])
  auto copy_times = [&]() {
    float ms = 0, dec = 0;
    for (size_t i = 0; i < np; ++i)
      if (cudaEventElapsedTime(&ms, cl.tev[2 + 2 * i], cl.tev[3 + 2 * i]) == cudaSuccess) dec += ms;
    stat->stage_ms[0] = dec;
    if (cudaEventElapsedTime(&ms, cl.tev[0], cl.tev[1]) == cudaSuccess) stat->stage_ms[5] = ms;
  };
  MCU(cudaMemcpyAsync(&hr->decode, dst, sizeof(DevStatus), cudaMemcpyDeviceToHost, s));
  MCU(cudaEventRecord(sev[1], s));
  auto stage_times = [&]() {
    static const int pairs[5][2] = {{0, 1}, {1, 2}, {2, 3}, {4, 5}, {5, 6}};
    float ms = 0;
    for (int i = 0; i < 5; ++i)
      if (cudaEventElapsedTime(&ms, sev[pairs[i][0]], sev[pairs[i][1]]) == cudaSuccess) stat->stage_ms[i] = ms;
    // [0] the decode kernels alone (the wait for each piece's bytes left
    // out), [5] the copies of the inputs in, which the decode overlaps
    copy_times();
  };
  if (mode == kModeQuery) {
    // ---- query: every key looked up in the streams of its partition ----
    const uint32_t nq = (uint32_t)ex->nq;
    Dev d_qk(pool, 28), d_qp(pool, 29), d_qout(pool, 30);
    if (!d_qk.ensure(nq * sizeof(T) + 16) || !d_qp.ensure(nq * 4 + 8) || !d_qout.ensure(nq * 8 + 8) ||
        !h_rows.ensure((size_t)nq * (sizeof(T) + 12) + 16))
      return fail(KITE_ERR_OOM, "query buffers");
    T* qk = h_rows.as<T>();
    uint64_t* found = reinterpret_cast<uint64_t*>(qk + nq);
    uint32_t* qp = reinterpret_cast<uint32_t*>(found + nq);
    for (uint32_t q = 0; q < nq; ++q) {
      qk[q] = (T)(((unsigned __int128)ex->keys[2 * q + 1] << 64) | ex->keys[2 * q]);
      qp[q] = ex->parts[q];
    }
    for (int i = 2; i < 5; ++i) MCU(cudaEventRecord(sev[i], s));
    if (nq) {
      MCU(cudaMemcpyAsync(d_qk.p, qk, nq * sizeof(T), cudaMemcpyHostToDevice, s));
      MCU(cudaMemcpyAsync(d_qp.p, qp, nq * 4, cudaMemcpyHostToDevice, s));
      k_query_streams<T><<<(nq + 255) / 256, 256, 0, s>>>(d_keys.as<T>(), d_counts.as<unsigned long long>(),
                                                          d_streams.as<StreamDesc>(), d_pfirst.as<uint32_t>(),
                                                          d_qk.as<T>(), d_qp.as<uint32_t>(), nq,
                                                          d_qout.as<unsigned long long>());
      launches++;
    }
    MCU(cudaEventRecord(sev[5], s));
    if (nq) MCU(cudaMemcpyAsync(found, d_qout.p, nq * 8, cudaMemcpyDeviceToHost, s));
    MCU(cudaEventRecord(sev[6], s));
    if (sync()) return fail(KITE_ERR_TIMEOUT, "query wait");
    MCU(cudaGetLastError());
    if (hr->decode.code == KITE_DEV_SHORT_VARINTS) return bad_delta();
    if (nq) std::memcpy(ex->counts_out, found, nq * 8);
    stage_times();
    stat->kernel_launches = launches;
    return KITE_OK;
  }
  // planning phases, host wall clock (the decode's kernels run meanwhile until
  // the first wait): [6] splitters, [7] first cut, [8] bisection, [9] tile lists
  auto wall = []() { return std::chrono::steady_clock::now(); };
  auto ms_since = [](std::chrono::steady_clock::time_point a) {
    return std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - a).count();
  };
  auto tp0 = wall();
  // ---- tiles.  Partitions of one stream each are cut every kMergeCap rows;
  // others by global splitters from a row sample into tiles of three quarters
  // of the on-chip capacity on average (the merge kernel's cost per tile is
  // mostly fixed, so fuller tiles cost less per row).  The cut, the tiles and
  // their stream ranges are made on the device; only when one of its ranges is
  // above the capacity (skewed keys) does the host cut again, with bisection.
  // (The host's lists and the copies of the position matrix and the tiles took
  // 3.0 - 4.7 ms of each call at 50 - 100M rows, 0.1 - 0.2 ms now.)
  uint32_t S = 1;
  auto want_ranges = [&]() {
    const double want = (double)total_rows / ((double)P * 0.75 * kMergeCap);
    return want > 1.0 ? (uint32_t)std::min(4096.0, std::ceil(want)) : 1u;
  };
  Dev d_spl(pool, 28), d_pos(pool, 31);
  auto make_splitters = [&]() -> int {  // S - 1 of them
    const uint32_t ns = (uint32_t)std::min<uint64_t>(total_rows, 1u << 20);
    Dev d_sample(pool, 29), d_hist(pool, 30);
    if (!d_sample.ensure(ns * sizeof(T)) || !d_spl.ensure(S * sizeof(T)) || !d_hist.ensure(65536 * 4))
      return fail(KITE_ERR_OOM, "merge splitters");
    k_sample_rows<T><<<(ns + 255) / 256, 256, 0, s>>>(d_keys.as<T>(), total_rows, ns, d_sample.as<T>());
    // sampling every m-th row of the concatenated streams is a uniform sample
    // of the key multiset; key bits from the input k
    launches += 1 + compute_hist_splitters<T>(d_sample.as<T>(), ns, key_bits, S, d_spl.as<T>(),
                                              d_hist.as<unsigned>(), s);
    stat->splitter_used = KITE_SPLIT_SAMPLED;
    if (ex && ex->mlp && ex->splitter_mode == KITE_SPLIT_LEARNED) {
      // the learned CDF of the row sample, on request: its training (650 ms)
      // is longer than most merges, and ranges that the histogram cuts badly
      // are bisected
      double hist_imb = 0.0;
      if (predict_imbalance<T>(ex->mlp, d_sample.as<T>(), ns, d_spl.as<T>(), S, s, timeout_ms, &hist_imb))
        return fail(KITE_ERR_TIMEOUT, "merge splitter evaluation did not finish");
      Dev d_spl2;
      if (!d_spl2.ensure(S * sizeof(T))) return fail(KITE_ERR_OOM, "merge splitters");
      MlpReport rep;
      if (mlp_splitters<T>(ex->mlp, d_sample.as<T>(), ns, key_bits, S, d_spl2.as<T>(), s, timeout_ms, &rep))
        return fail(KITE_ERR_CUDA, "learned splitter training failed");
      launches += 1 + rep.launches;
      stat->hist_pred_imbalance = hist_imb;
      stat->mlp_pred_imbalance = rep.pred_imbalance;
      stat->mlp_loss = rep.loss;
      stat->mlp_reused = rep.reused ? 1u : 0u;
      if (rep.pred_imbalance < 1e29) {
        MCU(cudaMemcpyAsync(d_spl.p, d_spl2.p, (S - 1) * sizeof(T), cudaMemcpyDeviceToDevice, s));
        stat->splitter_used = KITE_SPLIT_LEARNED;
      }
      if (sync()) return fail(KITE_ERR_TIMEOUT, "merge splitter wait");
    }
    return KITE_OK;
  };
  auto range_positions = [&]() -> int {
    const uint64_t nq = (uint64_t)nst * (S + 1);
    if (!d_pos.ensure(nq * 8)) return fail(KITE_ERR_OOM, "merge range positions");
    k_range_positions<T><<<(unsigned)((nq + 255) / 256), 256, 0, s>>>(d_keys.as<T>(), d_streams.as<StreamDesc>(), nst,
                                                                     d_spl.as<T>(), S, d_pos.as<uint64_t>());
    launches++;
    return KITE_OK;
  };
  std::vector<MergeTile> mts;  // the host's cut; empty when the device made the tiles
  std::vector<TileDesc> tds;
  std::vector<uint32_t> tile_first(P + 1, 0);
  const uint64_t out_off = total_rows;  // rows reserved for the output
  uint32_t ntiles = 0;
  Pinned h_lists(pool ? &pool->host : nullptr);  // the host's cut: the tiles' stream ranges on their way to the device
  size_t nts_all = 0;
  Dev d_mt(pool, 15), d_ts(pool, 16), d_tds(pool, 22);
  bool planned = false;  // the tiles are on the device
  uint32_t cut = 1;      // ranges whose splitters and positions are on the device
  unsigned* const info = hr->plan;
  if (total_rows && most_streams <= kMaxTileStreams) {
    const bool slices = most_streams <= 1;
    S = slices ? (uint32_t)((most_rows + kMergeCap - 1) / kMergeCap) : want_ranges();
    if ((uint64_t)P * S <= 4 * (total_rows / kMergeCap + P)) {
      const uint64_t nt = (uint64_t)P * S, npos = (uint64_t)nst * (S + 1);
      if (!slices && S > 1) {
        if (const int rc = make_splitters()) return rc;
        if (const int rc = range_positions()) return rc;
        cut = S;
      } else {
        if (!d_pos.ensure(npos * 8)) return fail(KITE_ERR_OOM, "merge range positions");
        k_slice_positions<T><<<(unsigned)((npos + 255) / 256), 256, 0, s>>>(
            d_keys.as<T>(), d_streams.as<StreamDesc>(), nst, S, d_pos.as<uint64_t>());
        launches++;
        stat->splitter_used = KITE_SPLIT_SAMPLED;
      }
      if (!d_mt.ensure(nt * sizeof(MergeTile) + 8) || !d_ts.ensure((size_t)nst * S * sizeof(TileStream) + 8) ||
          !d_tds.ensure(nt * sizeof(TileDesc) + 8))
        return fail(KITE_ERR_OOM, "merge tile buffers");
      k_plan_tiles<<<(unsigned)((nt + 255) / 256), 256, 0, s>>>(
          d_pos.as<uint64_t>(), d_streams.as<StreamDesc>(), d_pfirst.as<uint32_t>(), P, S, d_mt.as<MergeTile>(),
          d_ts.as<TileStream>(), d_tds.as<TileDesc>(), plan_info);
      launches++;
      MCU(cudaMemcpyAsync(info, plan_info, sizeof hr->plan, cudaMemcpyDeviceToHost, s));
      if (sync()) return fail(KITE_ERR_TIMEOUT, "merge tile wait");
      if (hr->decode.code == KITE_DEV_SHORT_VARINTS) return bad_delta();
      planned = info[0] == 0;
      if (planned) {
        ntiles = (uint32_t)nt;
        nts_all = (size_t)nst * S;
        for (uint32_t p = 0; p <= P; ++p) tile_first[p] = p * S;
      }
    }
  }
  stat->stage_ms[6] = ms_since(tp0);
  if (!planned) {
  // ---- the host's cut ----
  S = total_rows ? want_ranges() : 1;
  std::vector<T> spl(S - 1);
  if (S > 1 && S != cut) {  // else the plan's are the same
    if (const int rc = make_splitters()) return rc;
  }
  auto tp1 = wall();
  // ---- first cut on the device: the row position of every splitter in every
  // stream (one binary search each), read back as one matrix
  const size_t SP = (size_t)S + 1;
  std::vector<uint64_t> pos((size_t)nst * SP);
  if (nst && S > 1) {
    if (S != cut) {
      if (const int rc = range_positions()) return rc;
    }
    if (sync()) return fail(KITE_ERR_TIMEOUT, "merge range wait");
    MCU(cudaMemcpyAsync(spl.data(), d_spl.p, (S - 1) * sizeof(T), cudaMemcpyDeviceToHost, s));
    MCU(cudaMemcpyAsync(pos.data(), d_pos.p, pos.size() * 8, cudaMemcpyDeviceToHost, s));
    if (sync()) return fail(KITE_ERR_TIMEOUT, "merge range wait");
  } else {
    if (sync()) return fail(KITE_ERR_TIMEOUT, "merge splitter wait");
    for (uint32_t si = 0; si < nst; ++si) {
      pos[si * SP] = streams[si].row_off;
      pos[si * SP + 1] = streams[si].row_off + streams[si].rows;
    }
  }
  // A finished range: partition, low key, and the offset of its per-stream
  // [lo, hi) row positions in dlo / dhi (one entry per stream of the
  // partition).  Ranges above the on-chip capacity are bisected by key.
  struct Done {
    uint32_t p;
    T lo;
    uint64_t off;
  };
  struct Range {
    uint32_t p;
    T lo, hi;
    bool open_hi;
  };
  // First cut, partitions in parallel on the host threads: each range that
  // fits on chip becomes a finished range of its partition, the rest go to
  // the bisection below.
  const unsigned hthreads = std::max(1u, std::min(32u, std::thread::hardware_concurrency()));
  auto parallel_parts = [&](auto&& fn) {
    std::vector<std::thread> th;
    for (unsigned t = 0; t < hthreads; ++t)
      th.emplace_back([&, t]() {
        for (uint32_t p = t; p < P; p += hthreads) fn(p);
      });
    for (auto& x : th) x.join();
  };
  struct PartCut {
    std::vector<Done> done;
    std::vector<uint64_t> dlo, dhi;
    std::vector<Range> work;
  };
  std::vector<PartCut> cut(P);
  parallel_parts([&](uint32_t p) {
    PartCut& c = cut[p];
    const uint32_t f = part_first_stream[p], nstr = part_first_stream[p + 1] - f;
    if (!nstr) return;
    for (uint32_t j = 0; j < S; ++j) {
      const T lo = j ? spl[j - 1] : T(0);
      const bool open_hi = j + 1 == S;
      const T hi = open_hi ? T(0) : spl[j];
      if (!open_hi && hi <= lo) continue;  // empty (repeated splitter)
      uint64_t rows = 0;
      for (uint32_t k2 = 0; k2 < nstr; ++k2) rows += pos[(f + k2) * SP + j + 1] - pos[(f + k2) * SP + j];
      if (rows == 0) continue;
      if (rows <= kMergeCap && nstr <= kMaxTileStreams) {
        c.done.push_back(Done{p, lo, (uint64_t)c.dlo.size()});
        for (uint32_t k2 = 0; k2 < nstr; ++k2) {
          c.dlo.push_back(pos[(f + k2) * SP + j]);
          c.dhi.push_back(pos[(f + k2) * SP + j + 1]);
        }
      } else {
        c.work.push_back(Range{p, lo, hi, open_hi});
      }
    }
  });
  stat->stage_ms[7] = ms_since(tp1);
  auto tp2 = wall();
  std::vector<Done> done;  // ranges finished by the bisection (offsets into dlo / dhi)
  std::vector<uint64_t> dlo, dhi;
  std::vector<Range> work;
  for (uint32_t p = 0; p < P; ++p) work.insert(work.end(), cut[p].work.begin(), cut[p].work.end());
  std::vector<uint64_t>().swap(pos);
  // the decode's status arrived with the sync above
  if (hr->decode.code == KITE_DEV_SHORT_VARINTS) return bad_delta();
  Dev d_qlo, d_qhi, d_qkey, d_qout;
  std::vector<uint64_t> lp, hp;
  for (int round = 0; !work.empty() && round < 200; ++round) {
    // queries: for every range and stream, lower_bound(lo) and lower_bound(hi)
    std::vector<uint64_t> qlo, qhi;
    std::vector<T> qkey;
    for (auto& r : work)
      for (uint32_t si = part_first_stream[r.p]; si < part_first_stream[r.p + 1]; ++si) {
        const uint64_t a = streams[si].row_off, b = a + streams[si].rows;
        qlo.push_back(a);
        qhi.push_back(b);
        qkey.push_back(r.lo);
        qlo.push_back(a);
        qhi.push_back(b);
        qkey.push_back(r.open_hi ? T(0) : r.hi);
      }
    const uint32_t nq = (uint32_t)qlo.size();
    if (!d_qlo.ensure(nq * 8) || !d_qhi.ensure(nq * 8) || !d_qkey.ensure(nq * sizeof(T)) || !d_qout.ensure(nq * 8))
      return fail(KITE_ERR_OOM, "merge tile queries");
    MCU(cudaMemcpyAsync(d_qlo.p, qlo.data(), nq * 8, cudaMemcpyHostToDevice, s));
    MCU(cudaMemcpyAsync(d_qhi.p, qhi.data(), nq * 8, cudaMemcpyHostToDevice, s));
    MCU(cudaMemcpyAsync(d_qkey.p, qkey.data(), nq * sizeof(T), cudaMemcpyHostToDevice, s));
    k_lower_bound<T><<<(nq + 255) / 256, 256, 0, s>>>(d_keys.as<T>(), d_qlo.as<uint64_t>(), d_qhi.as<uint64_t>(),
                                                      d_qkey.as<T>(), nq, d_qout.as<uint64_t>());
    launches++;
    std::vector<uint64_t> qout(nq);
    if (sync()) return fail(KITE_ERR_TIMEOUT, "merge tile wait");
    MCU(cudaMemcpyAsync(qout.data(), d_qout.p, nq * 8, cudaMemcpyDeviceToHost, s));
    if (sync()) return fail(KITE_ERR_TIMEOUT, "merge tile wait");
    std::vector<Range> next;
    size_t q = 0;
    for (auto& r : work) {
      uint64_t rows = 0;
      lp.clear();
      hp.clear();
      for (uint32_t si = part_first_stream[r.p]; si < part_first_stream[r.p + 1]; ++si) {
        const uint64_t a = qout[q++], b0 = qout[q++];
        const uint64_t b = r.open_hi ? streams[si].row_off + streams[si].rows : b0;
        lp.push_back(a);
        hp.push_back(b);
        rows += b - a;
      }
      const uint32_t nstr = part_first_stream[r.p + 1] - part_first_stream[r.p];
      const T hi_eff = r.open_hi ? (sizeof(T) == 8 ? (T)~0ull : ~T(0)) : r.hi;
      if (rows > kMergeCap && hi_eff - r.lo > T(1)) {
        const T mid = r.lo + (hi_eff - r.lo) / 2;
        Range a = r, b = r;
        a.hi = mid;
        a.open_hi = false;
        b.lo = mid;
        next.push_back(a);
        next.push_back(b);
      } else {
        if (rows > kMergeCap || nstr > kMaxTileStreams)
          return fail(KITE_ERR_UNSUPPORTED, "merge tile cannot be split below the on-chip capacity");
        if (rows) {
          done.push_back(Done{r.p, r.lo, (uint64_t)dlo.size()});
          dlo.insert(dlo.end(), lp.begin(), lp.end());
          dhi.insert(dhi.end(), hp.begin(), hp.end());
        }
      }
    }
    work.swap(next);
  }
  if (!work.empty()) return fail(KITE_ERR_UNSUPPORTED, "merge tile refinement did not converge");
  stat->stage_ms[8] = ms_since(tp2);
  auto tp3 = wall();
  // ---- tile lists: per partition (in parallel) its finished ranges in key
  // order, then the partitions concatenated with their offsets ----
  std::vector<std::vector<Done>> refined(P);
  for (const Done& d : done) refined[d.p].push_back(d);
  struct PartTiles {
    std::vector<MergeTile> mts;
    std::vector<TileStream> tss;
    uint64_t rows = 0;
  };
  std::vector<PartTiles> pt(P);
  parallel_parts([&](uint32_t p) {
    PartTiles& o = pt[p];
    PartCut& c = cut[p];
    std::vector<Done>& rf = refined[p];
    std::sort(rf.begin(), rf.end(), [](const Done& a, const Done& b) { return a.lo < b.lo; });
    const uint32_t f = part_first_stream[p], nstr = part_first_stream[p + 1] - f;
    size_t i = 0, r = 0;
    while (i < c.done.size() || r < rf.size()) {
      const bool from_cut = r >= rf.size() || (i < c.done.size() && c.done[i].lo < rf[r].lo);
      const Done& d = from_cut ? c.done[i++] : rf[r++];
      const uint64_t* lo_v = from_cut ? c.dlo.data() : dlo.data();
      const uint64_t* hi_v = from_cut ? c.dhi.data() : dhi.data();
      MergeTile mt{};
      mt.out_off = o.rows;  // relative to the partition until concatenated
      mt.first_ts = (uint32_t)o.tss.size();
      mt.partition = p;
      uint64_t rows = 0;
      for (uint32_t k2 = 0; k2 < nstr; ++k2) {
        const uint64_t lo = lo_v[d.off + k2], hi = hi_v[d.off + k2];
        if (hi == lo) continue;
        o.tss.push_back(TileStream{lo, hi, streams[f + k2].input, 0});
        rows += hi - lo;
      }
      mt.nts = (uint32_t)(o.tss.size() - mt.first_ts);
      mt.rows_in = (uint32_t)rows;
      o.rows += rows;
      o.mts.push_back(mt);
    }
    std::vector<Done>().swap(c.done);
    std::vector<uint64_t>().swap(c.dlo);
    std::vector<uint64_t>().swap(c.dhi);
  });
  // the partitions' offsets, then every partition's tiles and stream ranges
  // written in place in parallel, the stream ranges straight into pinned
  // memory for their copy to the device
  std::vector<uint64_t> ts_first(P + 1, 0), row_first(P + 1, 0);
  for (uint32_t p = 0; p < P; ++p) {
    tile_first[p + 1] = tile_first[p] + (uint32_t)pt[p].mts.size();
    ts_first[p + 1] = ts_first[p] + pt[p].tss.size();
    row_first[p + 1] = row_first[p] + pt[p].rows;
  }
  nts_all = (size_t)ts_first[P];
  mts.resize(tile_first[P]);
  tds.resize(tile_first[P]);
  if (!h_lists.ensure(nts_all * sizeof(TileStream) + 64)) return fail(KITE_ERR_OOM, "merge tile lists (pinned)");
  TileStream* tss = h_lists.as<TileStream>();
  parallel_parts([&](uint32_t p) {
    PartTiles& o = pt[p];
    const uint32_t t0 = tile_first[p], s0 = (uint32_t)ts_first[p];
    for (size_t i = 0; i < o.mts.size(); ++i) {
      MergeTile mt = o.mts[i];
      mt.out_off += row_first[p];
      mt.first_ts += s0;
      tds[t0 + i] = TileDesc{mt.out_off, 0, p};
      mts[t0 + i] = mt;
    }
    if (!o.tss.empty()) std::memcpy(tss + s0, o.tss.data(), o.tss.size() * sizeof(TileStream));
    PartTiles().mts.swap(o.mts);
    PartTiles().tss.swap(o.tss);
  });
  stat->stage_ms[9] = ms_since(tp3);
  ntiles = (uint32_t)mts.size();
  }  // the host's cut
  std::vector<InputFilter> filt(n);
  for (int i = 0; i < n; ++i)
    filt[i] = InputFilter{(uint32_t)in[i].has_min, (uint32_t)in[i].has_max, in[i].min_count, in[i].max_count};
  Dev d_filt(pool, 17), d_okeys(pool, 18), d_ocounts(pool, 19), d_tout(pool, 20), d_over(pool, 21), d_tf(pool, 23),
      d_boff(pool, 24), d_prev(pool, 25), d_meta(pool, 26), d_out(pool, 27);
  if (!d_mt.ensure(ntiles * sizeof(MergeTile) + 8) || !d_ts.ensure(nts_all * sizeof(TileStream) + 8) ||
      !d_filt.ensure(n * sizeof(InputFilter)) || !d_okeys.ensure(out_off * sizeof(T) + 16) ||
      !d_ocounts.ensure(out_off * 4 + 16) || !d_tout.ensure(ntiles * sizeof(TileOut<T>) + 16) ||
      !d_over.ensure(8) || !d_tds.ensure(ntiles * sizeof(TileDesc) + 8) || !d_tf.ensure((P + 1) * 4) ||
      !d_boff.ensure(ntiles * 8 + 8) || !d_prev.ensure(ntiles * sizeof(T) + 16) || !d_meta.ensure(P * sizeof(BucketMeta)))
    return fail(KITE_ERR_OOM, "merge tile buffers");
  if (!mts.empty()) {
    MCU(cudaMemcpyAsync(d_mt.p, mts.data(), ntiles * sizeof(MergeTile), cudaMemcpyHostToDevice, s));
    MCU(cudaMemcpyAsync(d_ts.p, h_lists.as<TileStream>(), nts_all * sizeof(TileStream), cudaMemcpyHostToDevice, s));
    MCU(cudaMemcpyAsync(d_tds.p, tds.data(), ntiles * sizeof(TileDesc), cudaMemcpyHostToDevice, s));
  }
  MCU(cudaMemcpyAsync(d_tf.p, tile_first.data(), (P + 1) * 4, cudaMemcpyHostToDevice, s));
  MCU(cudaMemcpyAsync(d_filt.p, filt.data(), n * sizeof(InputFilter), cudaMemcpyHostToDevice, s));
  MCU(cudaMemsetAsync(d_over.p, 0xff, 8, s));
  auto tile_imbalance = [&]() {
    uint64_t tmax = info[1], tne = info[2];
    if (!planned) {
      tmax = tne = 0;
      for (auto& m : mts) {
        tmax = std::max<uint64_t>(tmax, m.rows_in);
        tne += m.rows_in != 0;
      }
    }
    return tne ? (double)tmax / ((double)out_off / (double)tne) : 0.0;
  };
  const size_t smem = MergeSmem<T>::total;
  auto kmerge = mode == kModeDump    ? k_merge_tiles<T, kModeDump>
                : mode == kModeHisto ? k_merge_tiles<T, kModeHisto>
                                     : k_merge_tiles<T, kModeMerge>;
  cudaFuncSetAttribute(kmerge, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  // u64 tiles go through the table, those that it lists through kmerge: always
  // for dump and histo, for merge unless an input with a filter has several
  // chunks in a partition (their sum is what is filtered)
  bool by_table = sizeof(T) == 8, filtered = false;
  for (int i = 0; i < n; ++i) {
    if (!in[i].has_min && !in[i].has_max) continue;
    filtered = true;
    for (uint32_t p = 0; mode == kModeMerge && p < P; ++p) by_table &= in[i].part_count[p] <= 1;
  }
  Dev d_list(pool, 34);  // listed tiles, behind the groups' counters and the tiles met
  if (!d_list.ensure(((size_t)ntiles + 16) * 4)) return fail(KITE_ERR_OOM, "merge tile buffers");
  if (by_table) MCU(cudaMemsetAsync(d_list.p, 0, 16 * 4, s));
  int dev = 0, sms = 0;
  MCU(cudaGetDevice(&dev));
  MCU(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  MergeAux aux{};
  // The merge of tiles [ta, tb), group g of at most 8.
  auto merge_tiles = [&](uint32_t ta, uint32_t tb, uint32_t g) {
    if (tb <= ta) return;
    const uint32_t nt = tb - ta;
    uint32_t* list = nullptr;
    unsigned* nlist = nullptr;
    if constexpr (sizeof(T) == 8) {
      if (by_table) {
        nlist = d_list.as<unsigned>() + g;
        list = d_list.as<uint32_t>() + 16 + ta;
        auto ktable = mode == kModeDump    ? k_merge_table<kModeDump>
                      : mode == kModeHisto ? k_merge_table<kModeHisto>
                                           : k_merge_table<kModeMerge>;
        cudaFuncSetAttribute(ktable, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MergeTable::total);
        // histo's CTAs keep their bins over all their tiles
        const uint32_t grid = mode == kModeHisto ? std::min<uint32_t>(nt, 2 * sms) : nt;
        ktable<<<grid, MergeTable::NT, MergeTable::total, s>>>(
            d_keys.as<T>(), d_counts.as<unsigned long long>(), d_mt.as<MergeTile>() + ta, nt, d_ts.as<TileStream>(),
            d_filt.as<InputFilter>(), filtered ? 1u : 0u, d_okeys.as<T>(), d_ocounts.as<uint32_t>(),
            d_tout.as<TileOut<T>>() + ta, list, nlist, d_list.as<unsigned>() + 8, aux);
        launches++;
      }
    }
    kmerge<<<list ? std::min<uint32_t>(nt, 2 * sms) : nt, kMergeThreads, smem, s>>>(
        d_keys.as<T>(), d_counts.as<unsigned long long>(), d_mt.as<MergeTile>() + ta, d_ts.as<TileStream>(),
        d_filt.as<InputFilter>(), d_okeys.as<T>(), d_ocounts.as<uint32_t>(), d_tout.as<TileOut<T>>() + ta,
        d_over.as<unsigned long long>() + g, dst, aux, list, nlist);
  };
  aux.line_k = key_bits / 2;
  Dev d_hist(pool, 30);
  if (mode == kModeHisto) {
    if (!d_hist.ensure((kHistBins + 1) * 8)) return fail(KITE_ERR_OOM, "histo buffers");
    MCU(cudaMemsetAsync(d_hist.p, 0, (kHistBins + 1) * 8, s));
    aux.hist = d_hist.as<unsigned long long>();
    aux.spill_n = aux.hist + kHistBins;
    aux.spill = d_okeys.as<unsigned long long>();  // no rows are written in this mode
    aux.spill_cap = out_off;
  }
  if (mode == kModeMerge && ntiles) {
    // ---- merge, encode and copy-out pipelined over partition groups: group
    // g's payload copies to the host (on the input copy lane, idle by now)
    // while group g + 1 merges.  The offsets kernel writes each group's
    // partition records into mapped pinned memory, so the host sizes the
    // group's encode without a copy that would queue on a copy engine. ----
    const uint32_t NG = std::min<uint32_t>(8, P);
    std::vector<uint32_t> pb(NG + 1);
    for (uint32_t g = 0; g <= NG; ++g) pb[g] = (uint32_t)((uint64_t)P * g / NG);
    if (NG == 8 && P >= 64) {
      // tapering groups (weights 6,6,6,6,6,5,3,2 of 40): the last copy-out,
      // which nothing overlaps, carries about a twentieth of the output
      static const uint32_t cw[9] = {0, 6, 12, 18, 24, 30, 35, 38, 40};
      for (uint32_t g = 0; g <= NG; ++g) pb[g] = (uint32_t)((uint64_t)P * cw[g] / 40);
    }
    if (!d_over.ensure((size_t)NG * 8)) return fail(KITE_ERR_OOM, "merge tile buffers");
    MCU(cudaMemsetAsync(d_over.p, 0xff, (size_t)NG * 8, s));  // per group: its first overflowing row
    // pinned partition records
    Pinned h_records(pool ? &pool->records : nullptr);
    if (!h_records.ensure((size_t)P * sizeof(BucketMeta))) return fail(KITE_ERR_OOM, "merge records (pinned)");
    BucketMeta* hm = h_records.as<BucketMeta>();
    BucketMeta* hm_dev = nullptr;
    MCU(cudaHostGetDevicePointer(reinterpret_cast<void**>(&hm_dev), hm, 0));
    // output buffers: the inputs' payload size to start with (a merged
    // partition's rows are at most its inputs' rows); a group that needs more
    // grows them once every queued encode and copy has finished
    uint64_t cap = std::max<uint64_t>(total_bytes, 1ull << 20) + 16;
    if (!d_out.ensure(cap)) return fail(KITE_ERR_OOM, "merge output");
    uint8_t* hout = staging ? staging(cap) : nullptr;
    std::unique_ptr<uint8_t[]> hown;
    if (!hout) {
      hown.reset(new (std::nothrow) uint8_t[cap]);
      if (!hown) return fail(KITE_ERR_OOM, "merge output host buffer");
      hout = hown.get();
    }
    struct Evs {
      std::vector<cudaEvent_t> e;
      ~Evs() {
        for (auto x : e) cudaEventDestroy(x);
      }
    } gv;
    gv.e.resize(7 * (size_t)NG, nullptr);
    for (auto& e : gv.e) MCU(cudaEventCreate(&e));
    cudaEvent_t* ge = gv.e.data();  // per group: merge, merged, linked | encode start, end | copy start, end
    MCU(cudaEventRecord(sev[2], s));
    auto queue_merge = [&](uint32_t g) -> cudaError_t {
      const uint32_t pa = pb[g], pe = pb[g + 1], ta = tile_first[pa], tb = tile_first[pe];
      cudaEventRecord(ge[7 * g], s);
      merge_tiles(ta, tb, g);
      cudaEventRecord(ge[7 * g + 1], s);
      if (pe > pa) {
        launch_tile_link_ranges<T>(d_tout.as<TileOut<T>>(), pe - pa, d_tf.as<uint32_t>() + pa,
                                   d_boff.as<unsigned long long>(), d_prev.as<T>(), d_meta.as<BucketMeta>() + pa, s);
        launch_bucket_offsets(d_meta.as<BucketMeta>() + pa, pe - pa, hm_dev + pa, s);
      }
      cudaEventRecord(ge[7 * g + 2], s);
      return cudaGetLastError();
    };
    std::vector<uint64_t> gbase(NG, 0);
    uint64_t total_out = 0, out_rows = 0;
    MCU(queue_merge(0));
    for (uint32_t g = 0; g < NG; ++g) {
      if (g + 1 < NG) MCU(queue_merge(g + 1));
      launches += 3;
      if (bounded_event_wait(ge[7 * g + 2], timeout_ms)) return fail(KITE_ERR_TIMEOUT, "merge group wait");
      const uint32_t pa = pb[g], pe = pb[g + 1], ta = tile_first[pa], tb = tile_first[pe];
      uint64_t gbytes = 0;
      for (uint32_t p = pa; p < pe; ++p) {
        gbytes += hm[p].bytes;
        out_rows += hm[p].rows;
      }
      if (total_out + gbytes + 16 > cap) {
        // every earlier group's bytes are on the host once the copy lane is
        // idle: the device buffer is replaced, the host one grown with them
        if (bounded_sync(s, timeout_ms) || bounded_sync(cl.cs, timeout_ms))
          return fail(KITE_ERR_TIMEOUT, "merge output wait");
        const uint64_t ncap = total_out + gbytes + 16 + (total_out + gbytes) / 4;
        if (!d_out.ensure(ncap)) return fail(KITE_ERR_OOM, "merge output");
        std::unique_ptr<uint8_t[]> nh(new (std::nothrow) uint8_t[ncap]);
        if (!nh) return fail(KITE_ERR_OOM, "merge output host buffer");
        std::memcpy(nh.get(), hout, total_out);
        hown = std::move(nh);
        hout = hown.get();
        cap = ncap;
      }
      gbase[g] = total_out;
      MCU(cudaEventRecord(ge[7 * g + 3], s));
      // k_encode places a partition's bytes at its record's offset (relative
      // to the group) plus the tile's: the group's slice of the output
      if (tb > ta)
        launch_encode<T>(d_okeys.as<T>(), d_ocounts.as<uint32_t>(), d_tds.as<TileDesc>() + ta,
                         d_tout.as<TileOut<T>>() + ta, d_boff.as<unsigned long long>() + ta, d_prev.as<T>() + ta,
                         d_meta.as<BucketMeta>(), tb - ta, d_out.as<uint8_t>() + total_out, gbytes, est, s);
      MCU(cudaEventRecord(ge[7 * g + 4], s));
      MCU(cudaStreamWaitEvent(cl.cs, ge[7 * g + 4], 0));
      MCU(cudaEventRecord(ge[7 * g + 5], cl.cs));
      if (gbytes)
        MCU(cudaMemcpyAsync(hout + total_out, d_out.as<uint8_t>() + total_out, gbytes, cudaMemcpyDeviceToHost, cl.cs));
      MCU(cudaEventRecord(ge[7 * g + 6], cl.cs));
      total_out += gbytes;
    }
    MCU(cudaEventRecord(sev[3], s));
    unsigned long long* const overs = hr->over;
    const DevStatus &hst = hr->run, &hest = hr->encode;
    MCU(cudaMemcpyAsync(&hr->run, dst, sizeof(DevStatus), cudaMemcpyDeviceToHost, s));
    MCU(cudaMemcpyAsync(&hr->encode, est, sizeof(DevStatus), cudaMemcpyDeviceToHost, s));
    MCU(cudaMemcpyAsync(overs, d_over.p, (size_t)NG * 8, cudaMemcpyDeviceToHost, s));
    if (bounded_sync(s, timeout_ms) || bounded_sync(cl.cs, timeout_ms)) return fail(KITE_ERR_TIMEOUT, "merge wait");
    if (hst.code) {
      char b[160];
      snprintf(b, sizeof b, "merge: device status %u (%u, %u, %u)", hst.code, hst.a, hst.b, hst.c);
      return fail(hst.code == KITE_DEV_BAD_INPUT ? KITE_ERR_BAD_INPUT : KITE_ERR_DEVICE, b);
    }
    for (uint32_t g = 0; g < NG; ++g) {
      if (overs[g] == ~0ull) continue;
      // first overflowing row in (partition, key) order: name its key like the reference
      const uint32_t t = tile_first[pb[g]] + (uint32_t)(overs[g] >> 32), r = (uint32_t)(overs[g] & 0xffffffffu);
      T key{};
      MergeTile mt{};
      MCU(cudaMemcpy(&mt, d_mt.as<MergeTile>() + t, sizeof mt, cudaMemcpyDeviceToHost));
      MCU(cudaMemcpy(&key, d_okeys.as<T>() + mt.out_off + r, sizeof(T), cudaMemcpyDeviceToHost));
      unsigned __int128 v = (unsigned __int128)key;
      std::string ks;
      if (v == 0) ks = "0";
      while (v) {
        ks.insert(ks.begin(), (char)('0' + (int)(v % 10)));
        v /= 10;
      }
      return fail(KITE_ERR_COUNT_OVERFLOW, "merged count exceeds u32 for key " + ks);
    }
    if (hest.code) return fail(KITE_ERR_DEVICE, "merge encode failed");
    // stage times: decode, planning and the input copy as the other modes;
    // merge, link + offsets + encode, and the copy-out summed over the groups
    {
      static const int pairs[2][2] = {{0, 1}, {1, 2}};
      float ms = 0;
      for (int i = 0; i < 2; ++i)
        if (cudaEventElapsedTime(&ms, sev[pairs[i][0]], sev[pairs[i][1]]) == cudaSuccess) stat->stage_ms[i] = ms;
      copy_times();
      double mg = 0, en = 0, cp = 0;
      for (uint32_t g = 0; g < NG; ++g) {
        if (cudaEventElapsedTime(&ms, ge[7 * g], ge[7 * g + 1]) == cudaSuccess) mg += ms;
        if (cudaEventElapsedTime(&ms, ge[7 * g + 1], ge[7 * g + 2]) == cudaSuccess) en += ms;
        if (cudaEventElapsedTime(&ms, ge[7 * g + 3], ge[7 * g + 4]) == cudaSuccess) en += ms;
        if (cudaEventElapsedTime(&ms, ge[7 * g + 5], ge[7 * g + 6]) == cudaSuccess) cp += ms;
      }
      stat->stage_ms[2] = mg;
      stat->stage_ms[3] = en;
      stat->stage_ms[4] = cp;
    }
    stat->d2h_bytes += total_out;
    stat->rows = out_rows;
    stat->payload_bytes = total_out;
    stat->tiles = ntiles;
    stat->kernel_launches = launches;
    stat->tile_imbalance = tile_imbalance();
    if (!emit) return KITE_OK;
    for (uint32_t g = 0; g < NG; ++g)
      for (uint32_t p = pb[g]; p < pb[g + 1]; ++p) {
        const BucketMeta& m = hm[p];
        if (!m.rows) continue;
        kite_chunk_meta cm{};
        cm.partition_id = p;
        cm.codec = KITE_CODEC_DVLE;
        cm.row_count = m.rows;
        cm.raw_bytes = m.bytes;
        cm.key_min_lo[0] = m.kmin_lo;
        cm.key_min_lo[1] = m.kmin_hi;
        cm.key_max_lo[0] = m.kmax_lo;
        cm.key_max_lo[1] = m.kmax_hi;
        if (emit(user, &cm, hout + gbase[g] + m.byte_off, (size_t)m.bytes))
          return fail(KITE_ERR_CALLBACK, "emit callback aborted");
      }
    return KITE_OK;
  }
  MCU(cudaEventRecord(sev[2], s));
  if (ntiles) {
    merge_tiles(0, ntiles, 0);
    launches++;
  }
  MCU(cudaEventRecord(sev[3], s));
  stat->tiles = ntiles;
  const DevStatus& hst = hr->run;
  MCU(cudaMemcpyAsync(&hr->run, dst, sizeof(DevStatus), cudaMemcpyDeviceToHost, s));
  auto bad_status = [&]() {
    char b[160];
    snprintf(b, sizeof b, "%s: device status %u (%u, %u, %u)", dump ? "dump" : "merge", hst.code, hst.a, hst.b,
             hst.c);
    return fail(hst.code == KITE_DEV_BAD_INPUT ? KITE_ERR_BAD_INPUT : KITE_ERR_DEVICE, b);
  };
  if (mode == kModeHisto) {
    // ---- count -> frequency: the small bins, then the listed large counts ----
    unsigned long long* const hb = hr->hist;
    MCU(cudaMemcpyAsync(hb, d_hist.p, sizeof hr->hist, cudaMemcpyDeviceToHost, s));
    if (sync()) return fail(KITE_ERR_TIMEOUT, "histo wait");
    if (hst.code) return bad_status();
    const unsigned long long ns = std::min<unsigned long long>(hb[kHistBins], out_off);
    if (!h_rows.ensure(ns * 8 + 8)) return fail(KITE_ERR_OOM, "histo counts (pinned)");
    unsigned long long* const big = h_rows.as<unsigned long long>();
    MCU(cudaEventRecord(sev[4], s));
    if (ns) MCU(cudaMemcpyAsync(big, d_okeys.p, ns * 8, cudaMemcpyDeviceToHost, s));
    MCU(cudaEventRecord(sev[5], s));
    MCU(cudaEventRecord(sev[6], s));
    if (sync()) return fail(KITE_ERR_TIMEOUT, "histo wait");
    stage_times();
    std::sort(big, big + ns);
    uint64_t keys_out = 0;
    for (uint32_t b = 0; b < kHistBins; ++b) keys_out += hb[b];
    stat->rows = keys_out + ns;
    stat->kernel_launches = launches;
    if (!ex || !ex->histo) return KITE_OK;
    for (uint32_t b = 0; b < kHistBins; ++b)
      if (hb[b] && ex->histo(ex->user, b, hb[b])) return fail(KITE_ERR_CALLBACK, "histo callback aborted");
    for (size_t i = 0; i < ns;) {
      size_t j = i;
      while (j < ns && big[j] == big[i]) ++j;
      if (ex->histo(ex->user, big[i], j - i)) return fail(KITE_ERR_CALLBACK, "histo callback aborted");
      i = j;
    }
    return KITE_OK;
  }
  if (dump) {
    // ---- TSV: tile byte offsets in (partition, key) order on the device, the
    // partitions' records back to the host, then formatting ----
    Dev d_lines(pool, 32), d_scan(pool, 33);
    if (!d_boff.ensure((ntiles + 1) * 8) || !d_lines.ensure(P * sizeof(PartLines)) ||
        !d_scan.ensure(scan_tmp_elems(ntiles + 1) * 8 + 64))
      return fail(KITE_ERR_OOM, "dump output");
    if (!h_rows.ensure(P * sizeof(PartLines))) return fail(KITE_ERR_OOM, "dump records (pinned)");
    PartLines* const lines = h_rows.as<PartLines>();
    std::memset(lines, 0, P * sizeof(PartLines));
    if (ntiles) {
      k_part_lines<T><<<(P + 7) / 8, 256, 0, s>>>(d_tout.as<TileOut<T>>(), d_tf.as<uint32_t>(), P,
                                                  d_boff.as<unsigned long long>(), d_lines.as<PartLines>());
      launches += 1 + exclusive_scan_u64(d_boff.as<unsigned long long>(), d_boff.as<unsigned long long>(), ntiles,
                                         d_scan.as<unsigned long long>(), s);
      MCU(cudaMemcpyAsync(lines, d_lines.p, P * sizeof(PartLines), cudaMemcpyDeviceToHost, s));
    }
    if (sync()) return fail(KITE_ERR_TIMEOUT, "merge wait");
    if (hst.code) return bad_status();
    unsigned long long acc = 0;
    uint64_t out_rows = 0;
    for (uint32_t p = 0; p < P; ++p) {
      acc += lines[p].bytes;
      out_rows += lines[p].rows;
    }
    if (!d_out.ensure(acc + 16)) return fail(KITE_ERR_OOM, "dump output");
    MCU(cudaEventRecord(sev[4], s));
    if (ntiles && acc) {
      const size_t tsm = 256 + (size_t)kTsvThreads * (key_bits / 2 + 12);
      k_tsv_tiles<T><<<ntiles, kTsvThreads, tsm, s>>>(d_okeys.as<T>(), d_ocounts.as<uint32_t>(), d_mt.as<MergeTile>(),
                                                      d_tout.as<TileOut<T>>(), d_boff.as<unsigned long long>(),
                                                      key_bits / 2, d_out.as<uint8_t>());
      launches++;
    }
    MCU(cudaEventRecord(sev[5], s));
    stat->d2h_bytes += emit ? acc : 0;
    stat->rows = out_rows;
    stat->payload_bytes = acc;
    stat->kernel_launches = launches;
    if (!emit || acc == 0) {
      MCU(cudaEventRecord(sev[6], s));
      if (sync()) return fail(KITE_ERR_TIMEOUT, "dump wait");
      MCU(cudaGetLastError());
      stage_times();
      return KITE_OK;
    }
    // ---- copy-out in groups of whole partitions through two pinned halves:
    // group i+2 is queued once group i has been emitted, so the copy of the
    // next group overlaps the callback's work on this one
    uint64_t maxpart = 0;
    for (uint32_t p = 0; p < P; ++p) maxpart = std::max<uint64_t>(maxpart, lines[p].bytes);
    const uint64_t half = std::max<uint64_t>(std::min<uint64_t>(acc, 256ull << 20), maxpart);
    std::vector<uint32_t> gfirst{0};  // first partition of every group
    std::vector<uint64_t> goff{0};
    {
      uint64_t g = 0, off = 0;
      for (uint32_t p = 0; p < P; ++p) {
        if (g + lines[p].bytes > half) {
          gfirst.push_back(p);
          goff.push_back(off);
          g = 0;
        }
        g += lines[p].bytes;
        off += lines[p].bytes;
      }
      gfirst.push_back(P);
      goff.push_back(off);
    }
    const uint32_t ngroups = (uint32_t)gfirst.size() - 1;
    uint8_t* stage = staging ? staging(ngroups > 1 ? 2 * half : half) : nullptr;
    std::unique_ptr<uint8_t[]> fallback;
    if (!stage) {
      // no pinned staging offered: one pageable buffer for everything
      fallback.reset(new (std::nothrow) uint8_t[acc]);
      if (!fallback) return fail(KITE_ERR_OOM, "dump host buffer");
    }
    auto group_dst = [&](uint32_t g) { return stage ? stage + (g & 1) * half : fallback.get() + goff[g]; };
    cudaEvent_t cev[2];
    for (auto& e : cev)
      if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) return fail(KITE_ERR_CUDA, "event");
    struct CevGuard {
      cudaEvent_t* e;
      ~CevGuard() {
        cudaEventDestroy(e[0]);
        cudaEventDestroy(e[1]);
      }
    } cev_guard{cev};
    auto queue_copy = [&](uint32_t g) -> cudaError_t {
      const uint64_t n = goff[g + 1] - goff[g];
      cudaError_t e = n ? cudaMemcpyAsync(group_dst(g), d_out.as<uint8_t>() + goff[g], n, cudaMemcpyDeviceToHost, s)
                        : cudaSuccess;
      if (e == cudaSuccess) e = cudaEventRecord(cev[g & 1], s);
      return e;
    };
    MCU(queue_copy(0));
    if (ngroups > 1) MCU(queue_copy(1));
    for (uint32_t g = 0; g < ngroups; ++g) {
      const int w = bounded_event_wait(cev[g & 1], timeout_ms);
      if (w) return fail(w == -3 ? KITE_ERR_TIMEOUT : KITE_ERR_CUDA, "dump copy wait");
      const uint8_t* src = group_dst(g);
      uint64_t off = 0;
      for (uint32_t p = gfirst[g]; p < gfirst[g + 1]; ++p) {
        const PartLines& l = lines[p];
        if (!l.rows) continue;
        kite_chunk_meta cm{};
        cm.partition_id = p;
        cm.codec = 0;
        cm.row_count = l.rows;
        cm.raw_bytes = l.bytes;
        cm.key_min_lo[0] = l.kmin_lo;
        cm.key_min_lo[1] = l.kmin_hi;
        cm.key_max_lo[0] = l.kmax_lo;
        cm.key_max_lo[1] = l.kmax_hi;
        if (emit(user, &cm, src + off, (size_t)l.bytes)) return fail(KITE_ERR_CALLBACK, "emit callback aborted");
        off += l.bytes;
      }
      if (g + 2 < ngroups) MCU(queue_copy(g + 2));
    }
    MCU(cudaEventRecord(sev[6], s));
    if (sync()) return fail(KITE_ERR_TIMEOUT, "dump wait");
    MCU(cudaGetLastError());
    stage_times();
    return KITE_OK;
  }
  // a merge of inputs without rows
  if (sync()) return fail(KITE_ERR_TIMEOUT, "merge wait");
  if (hst.code) return bad_status();
  stage_times();
  stat->rows = 0;
  stat->payload_bytes = 0;
  stat->kernel_launches = launches;
  stat->tile_imbalance = 0.0;
  return KITE_OK;
#undef MCU
}

}  // namespace

int merge_run(int k, uint32_t partitions, const kite_gpu_merge_input* inputs, int n, cudaStream_t s,
              uint32_t timeout_ms, int mode, kite_gpu_emit_fn emit, void* user, std::string* msg,
              kite_gpu_stats* st, const StagingFn& staging, const MergeExtra* ex) {
  if (k <= 31)
    return merge_typed<uint64_t>(partitions, 2 * k, inputs, n, s, timeout_ms, mode, emit, user, msg, st, staging,
                                 ex);
  return merge_typed<u128>(partitions, 2 * k, inputs, n, s, timeout_ms, mode, emit, user, msg, st, staging, ex);
}

}  // namespace kite
