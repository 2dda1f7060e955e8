// kite_gpu_count_rows_noalloc: exact k-mer counting of one small FASTQ chunk
// that allocates nothing.
//
// Some callers cannot allocate device memory when they want a count: a
// process whose framework has already reserved the device's memory for its
// own caching pool, or a loop that counts small read batches between other
// GPU work and cannot accept the device-wide synchronisation that cudaMalloc
// and cudaFree imply, nor an out-of-memory failure half way through a run.
// The context API (kite_gpu_open) grows its buffers on demand with cudaMalloc;
// this entry point works only in g_noalloc_scratch below, a fixed array in
// this file's device data, and writes its results into buffers the caller
// already owns.
//
// Limits and sharing:
//  * at most KITE_NOALLOC_MAX_BYTES (512 KiB) of FASTQ per call; a larger
//    chunk is rejected with KITE_ERR_UNSUPPORTED before any launch.
//  * the array (kScratchBytes, about 19 MiB) exists once per device in the
//    process.  Every call on a device uses the same array, so calls that
//    overlap on the GPU (two host threads, or two streams without ordering
//    between them) race and corrupt each other's results: serialise them.
//  * the first call on a device looks the array's address up with
//    cudaGetSymbolAddress (which also loads this module on that device); make
//    that first call before any stream capture begins.  The address is kept
//    with the id of the device's context and looked up again when a new
//    context replaces it (after cudaDeviceReset, for example).
//  * the call returns once the work has finished, waiting at most timeout_ms.
//
// The chunk is small, so what counts is the number of dependent steps and how
// many SMs share each.  Six launches: newlines per 2 KiB segment; k-mers, one
// CTA per segment (KmerIter::next, src/count/kmer.rs:241-267 and :311-337);
// keys to their tile, a key range of a Fibonacci-hash partition
// (src/count/kmer.rs:67-71, :111-116) of about 256 keys; one CTA per tile
// sorts on chip and reduces to (key, count) rows, as the reference's
// flush_bucket does per bucket (src/count/worker.rs:296-449); tiles above the
// on-chip capacity through global memory; rows to the caller.  The two scans
// that need every CTA's result are done by the last CTA to finish.  254 KB of
// reads (93,134 k-mers, k = 31, 256 partitions) take 43 us on the device; one
// CTA finding the lines, one thread per 256 bases and one CTA per partition
// sorting through global memory took about 250.
#include <algorithm>
#include <cstring>
#include <mutex>
#include <tuple>
#include <utility>

#include "kite_gpu.h"
#include "kite_internal.h"
#include "kmer_words.cuh"

namespace kite {
namespace na {

constexpr uint32_t kMaxBytes = KITE_NOALLOC_MAX_BYTES;
constexpr uint32_t kMaxParts = 65536;
constexpr uint32_t kMaxTiles = 65536;
constexpr uint32_t kSegment = 2048;    // bytes of text per extraction CTA
constexpr uint32_t kTileKeys = 256;    // keys a tile is meant to have
constexpr uint32_t kTileCap = 2048;    // keys of a tile sorted on chip
constexpr int kMaxDevices = 64;
constexpr int kExtractThreads = 256;
constexpr int kTileSortThreads = 128;
constexpr int kSortThreads = 512;
constexpr uint32_t kMaxSegments = kMaxBytes / kSegment + 1;  // the text may start inside its first 16 bytes

struct Counters {
  unsigned long long reads, bases, kmers;
  unsigned int nkeys, nrows, nbig, extracted, sorted, pad;
};

constexpr size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }
constexpr size_t kOffKeysA = 0;
constexpr size_t kOffKeysB = align256(kOffKeysA + (size_t)kMaxBytes * 16);
constexpr size_t kOffCounts = align256(kOffKeysB + (size_t)kMaxBytes * 16);
constexpr size_t kOffSegLines = align256(kOffCounts + (size_t)kMaxBytes * 4);
constexpr size_t kOffTileCount = align256(kOffSegLines + (size_t)kMaxSegments * 4);
constexpr size_t kOffTileOff = align256(kOffTileCount + (size_t)kMaxTiles * 4);
constexpr size_t kOffTileRows = align256(kOffTileOff + (size_t)(kMaxTiles + 1) * 4);
constexpr size_t kOffRowOff = align256(kOffTileRows + (size_t)kMaxTiles * 4);
constexpr size_t kOffBig = align256(kOffRowOff + (size_t)(kMaxTiles + 1) * 4);
constexpr size_t kOffCounters = align256(kOffBig + (size_t)kMaxTiles * 4);
constexpr size_t kScratchBytes = align256(kOffCounters + sizeof(Counters));

// Typed views of the scratch array.
struct View {
  uint8_t* s;
  template <class T> __device__ T* keys_a() const { return reinterpret_cast<T*>(s + kOffKeysA); }
  template <class T> __device__ T* keys_b() const { return reinterpret_cast<T*>(s + kOffKeysB); }
  __device__ uint32_t* counts() const { return reinterpret_cast<uint32_t*>(s + kOffCounts); }
  __device__ uint32_t* seg_lines() const { return reinterpret_cast<uint32_t*>(s + kOffSegLines); }
  __device__ uint32_t* tile_count() const { return reinterpret_cast<uint32_t*>(s + kOffTileCount); }
  __device__ uint32_t* tile_off() const { return reinterpret_cast<uint32_t*>(s + kOffTileOff); }
  __device__ uint32_t* tile_rows() const { return reinterpret_cast<uint32_t*>(s + kOffTileRows); }
  __device__ uint32_t* row_off() const { return reinterpret_cast<uint32_t*>(s + kOffRowOff); }
  __device__ uint32_t* big() const { return reinterpret_cast<uint32_t*>(s + kOffBig); }
  __device__ Counters* counters() const { return reinterpret_cast<Counters*>(s + kOffCounters); }
};

}  // namespace na
}  // namespace kite

// The only working memory of kite_gpu_count_rows_noalloc (one per device).
static __device__ __align__(256) unsigned char g_noalloc_scratch[kite::na::kScratchBytes];

namespace kite {
namespace na {
namespace {

// The chunk in 16-byte granules of its address: a caller's pointer may have any
// alignment, so the text starts `skew` bytes into the first granule.
struct Text {
  const uint8_t* base;  // 16-byte aligned
  uint32_t skew, end;   // the text is bytes [skew, end) from base
};

__device__ __forceinline__ uint4 text_granule(const Text& t, uint32_t at) {
  if (at >= t.skew && at + 16 <= t.end) return *reinterpret_cast<const uint4*>(t.base + at);
  uint32_t w[4] = {0, 0, 0, 0};
  if (at < t.end)  // its first or last granule: only its own bytes are read
    for (uint32_t i = 0; i < 16; ++i)
      if (at + i >= t.skew && at + i < t.end) w[i >> 2] |= (uint32_t)t.base[at + i] << (8 * (i & 3u));
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// The tile of a key: ranges of equal width (a power of two per partition)
// over the keys' 2k bits, so that tile order is partition, then key order.
struct TileOf {
  uint32_t shift, bits, key_bits;
  template <class T>
  __device__ __forceinline__ uint32_t operator()(T key) const {
    return bits ? (bucket_of(key, shift) << bits) | (uint32_t)(uint64_t)(key >> (key_bits - bits))
                : bucket_of(key, shift);
  }
};

// Newlines per segment; what later kernels add to starts at zero.
__global__ void __launch_bounds__(128) k_prepare(Text t, uint32_t tiles, uint8_t* scr) {
  __shared__ unsigned sm[40];
  const View v{scr};
  const uint32_t at = blockIdx.x * kSegment + threadIdx.x * 16;
  for (uint32_t i = blockIdx.x * 128 + threadIdx.x; i < tiles; i += gridDim.x * 128) v.tile_count()[i] = 0;
  if (blockIdx.x == 0 && threadIdx.x == 0) *v.counters() = Counters{};
  const uint4 w = text_granule(t, at);
  const unsigned n = (__popc(__vcmpeq4(w.x, 0x0a0a0a0au)) + __popc(__vcmpeq4(w.y, 0x0a0a0a0au)) +
                      __popc(__vcmpeq4(w.z, 0x0a0a0a0au)) + __popc(__vcmpeq4(w.w, 0x0a0a0a0au))) >> 3;
  unsigned tot;
  block_exclusive_scan<128, unsigned>(n, sm, &tot);
  if (threadIdx.x == 0) v.seg_lines()[blockIdx.x] = tot;
}
static_assert(kSegment == 128 * 16, "a thread of k_prepare counts one granule");

// True in every thread of the last CTA to get here; what the others wrote
// before is then visible to it.
__device__ __forceinline__ bool last_cta(unsigned* done) {
  __shared__ bool last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(done, 1u) == gridDim.x - 1;
  __syncthreads();
  if (last) __threadfence();
  return last;
}

// Exclusive scan of n counters into out[0..n] by one CTA, four per thread and step.
template <int NT>
__device__ __forceinline__ void cta_scan(const uint32_t* in, uint32_t n, uint32_t* out, unsigned* sm) {
  unsigned carry = 0;
  for (uint32_t i0 = 0; i0 < n; i0 += NT * 4) {
    const uint32_t i = i0 + threadIdx.x * 4;
    unsigned x[4], sum = 0;
#pragma unroll
    for (uint32_t j = 0; j < 4; ++j) {
      x[j] = i + j < n ? __ldcg(in + i + j) : 0u;
      sum += x[j];
    }
    unsigned tot;
    unsigned at = carry + block_exclusive_scan<NT, unsigned>(sum, sm, &tot);
#pragma unroll
    for (uint32_t j = 0; j < 4; ++j) {
      if (i + j < n) out[i + j] = at;
      at += x[j];
    }
    carry += tot;
  }
  if (threadIdx.x == 0) out[n] = carry;
}

// K-mers of one segment: its 64 words and the two before it are encoded by one
// thread each (lines 1 mod 4 of a chunk that starts with '@' are sequences,
// parse_sequences, src/count/parser.rs:19-65; a k-mer cannot cross a newline,
// so only its last byte's line matters), then each warp takes words in turn
// with one lane per end byte.  A key's place in its tile is the tile counter's
// value, kept beside the key; the last CTA scans the counters.
template <class T>
__global__ void __launch_bounds__(kExtractThreads) k_extract(Text t, uint32_t k, uint32_t canonical, TileOf tile_of,
                                                             uint32_t tiles, uint8_t* scr) {
  constexpr int NT = kExtractThreads, W = kSegment / 32, WARPS = NT / 32;
  __shared__ uint64_t code[W + 2], rcode[W + 2];
  __shared__ uint32_t vb[W + 2], nl[W + 2], ends[W], place[W];
  __shared__ unsigned long long scan_sm[40];
  __shared__ unsigned scan32[40];
  __shared__ uint32_t base;
  const View v{scr};
  Counters* c = v.counters();
  const int tid = threadIdx.x;
  // this thread's word: tid - 2 of the segment
  const uint32_t at = blockIdx.x * kSegment + tid * 32 - 64;  // wraps below zero for the first two of the text
  const bool mine = tid < W + 2 && (blockIdx.x > 0 || tid >= 2) && at < t.end;
  Word32 w{0, 0, 0, 0};
  if (mine) w = encode_word(text_granule(t, at), text_granule(t, at + 16));
  if (tid < W + 2) {
    code[tid] = w.code;
    rcode[tid] = w.rcode;
    vb[tid] = w.vb;
    nl[tid] = w.nl;
  }
  const bool own = mine && tid >= 2;
  unsigned long long sum = own ? __popc(w.nl) : 0u;
  for (uint32_t i = tid; i < blockIdx.x; i += NT) sum += (unsigned long long)v.seg_lines()[i] << 32;
  unsigned long long tot;
  const unsigned long long before = block_exclusive_scan<NT, unsigned long long>(sum, scan_sm, &tot);
  unsigned ph = ((unsigned)(tot >> 32) + (unsigned)before) & 3u;  // the line's phase at the word
  const bool chunk_ok = t.end > t.skew && t.base[t.skew] == '@';
  uint32_t V = 0;
  unsigned long long reads = 0, bases = 0;
  if (own && chunk_ok) {
    // bytes outside the text are no newlines and no bases
    uint32_t in = 0xffffffffu;
    if (at < t.skew) in &= 0xffffffffu << (t.skew - at);
    if (t.end - at < 32) in &= (1u << (t.end - at)) - 1u;
    const uint32_t seq = seq_mask(w.nl, ph) & in;
    if constexpr (sizeof(T) == 8) {
      V = (uint32_t)(runs_of((uint64_t)vb[tid - 1] | (uint64_t)w.vb << 32, k) >> (33 - k)) & seq;
    } else {
      const u128 ok = (u128)((uint64_t)vb[tid - 2] | (uint64_t)vb[tid - 1] << 32) | (u128)w.vb << 64;
      V = (uint32_t)(runs_of128(ok, k) >> (65 - k)) & seq;
    }
    bases = __popc(seq);
    reads = __popc(seq & (w.nl << 1 | nl[tid - 1] >> 31));  // a line's first byte follows a newline
  }
  unsigned n;
  const unsigned first = block_exclusive_scan<NT, unsigned>(__popc(V), scan32, &n);
  if (tid >= 2 && tid < W + 2) {
    ends[tid - 2] = V;
    place[tid - 2] = first;
  }
  if (tid == 0) base = n ? atomicAdd(&c->nkeys, n) : 0u;
  for (int m = 16; m; m >>= 1) {
    reads += __shfl_xor_sync(0xffffffffu, reads, m);
    bases += __shfl_xor_sync(0xffffffffu, bases, m);
  }
  if ((tid & 31) == 0 && bases) {
    atomicAdd(&c->reads, reads);
    atomicAdd(&c->bases, bases);
  }
  __syncthreads();
  const unsigned lane = tid & 31;
  const T mask = (2 * k == (uint32_t)KeyTraits<T>::kBits) ? ~T(0) : ((T(1) << (2 * k)) - T(1));
  const uint32_t fs = 2 * (31 - lane);
  T* keys = v.keys_a<T>() + base;
  uint32_t* ranks = v.counts() + base;
  uint32_t* counts = v.tile_count();
  uint32_t rank[W / WARPS];
#pragma unroll
  for (int j = 0; j < W / WARPS; ++j) {
    const int i = (tid >> 5) + j * WARPS;  // word i of the segment is entry i + 2
    const uint32_t Vi = ends[i];
    rank[j] = 0;
    if (!((Vi >> lane) & 1u)) continue;
    T fwd, rc;
    const u128 x = (u128)code[i + 1] << 64 | code[i + 2];
    if constexpr (sizeof(T) == 8) {
      fwd = (uint64_t)(x >> fs) & mask;
      rc = (uint64_t)(((u128)rcode[i + 2] << 64 | rcode[i + 1]) >> (2 * (33 + lane - k))) & mask;
    } else {
      fwd = (fs ? x >> fs | (u128)code[i] << (128 - fs) : x) & mask;
      const uint32_t rs = 2 * (65 + lane - k);  // 2 .. 128
      const u128 lo = (u128)rcode[i + 1] << 64 | rcode[i];
      rc = rs < 64 ? lo >> rs | (u128)rcode[i + 2] << (128 - rs)
                   : ((u128)rcode[i + 2] << 64 | rcode[i + 1]) >> (rs - 64);
      rc &= mask;
    }
    const T key = canonical && rc < fwd ? rc : fwd;
    keys[place[i] + __popc(Vi & ((1u << lane) - 1u))] = key;
    rank[j] = atomicAdd(&counts[tile_of(key)], 1u);
  }
#pragma unroll
  for (int j = 0; j < W / WARPS; ++j) {
    const int i = (tid >> 5) + j * WARPS;
    const uint32_t Vi = ends[i];
    if ((Vi >> lane) & 1u) ranks[place[i] + __popc(Vi & ((1u << lane) - 1u))] = rank[j];
  }
  if (last_cta(&c->extracted)) {
    cta_scan<NT>(v.tile_count(), tiles, v.tile_off(), scan32);
    if (tid == 0) c->kmers = __ldcg(&c->nkeys);
  }
}

// Keys to their tiles: keys_a -> keys_b.
template <class T>
__global__ void __launch_bounds__(256) k_scatter(TileOf tile_of, uint8_t* scr) {
  const View v{scr};
  const uint32_t n = v.counters()->nkeys;
  const T* a = v.keys_a<T>();
  T* b = v.keys_b<T>();
  const uint32_t* off = v.tile_off();
  const uint32_t* rank = v.counts();
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const T key = a[i];
    b[off[tile_of(key)] + rank[i]] = key;
  }
}

// One CTA per tile of at most kTileCap keys: a bitonic sort in shared memory,
// then the run-length reduction to rows, written to keys_a / counts at the
// tile's offset.  A warp's 32 pairs of a step with stride <= 32 are 64
// consecutive keys, the same in every such step, so only longer strides need
// the whole CTA.  Larger tiles are listed.
template <class T>
__global__ void __launch_bounds__(kTileSortThreads) k_sort_tiles(uint8_t* scr) {
  constexpr uint32_t NT = kTileSortThreads;
  __shared__ T buf[kTileCap];
  __shared__ uint16_t head[kTileCap];
  __shared__ unsigned sm[40];
  const View v{scr};
  const uint32_t tile = blockIdx.x, tid = threadIdx.x;
  const uint32_t n = v.tile_count()[tile];
  if (n == 0 || n > kTileCap) {
    if (tid == 0) {
      if (n == 0) v.tile_rows()[tile] = 0;
      else v.big()[atomicAdd(&v.counters()->nbig, 1u)] = tile;
    }
    return;
  }
  const uint32_t off = v.tile_off()[tile];
  const T* src = v.keys_b<T>() + off;
  uint32_t m = 64;
  while (m < n) m *= 2;
  for (uint32_t i = tid; i < m; i += NT) buf[i] = i < n ? src[i] : ~T(0);
  __syncthreads();
  for (uint32_t size = 2; size <= m; size *= 2) {
    for (uint32_t stride = size / 2; stride; stride /= 2) {
      for (uint32_t i = tid; i < m / 2; i += NT) {
        const uint32_t a = 2 * i - (i & (stride - 1)), b = a + stride;
        const T x = buf[a], y = buf[b];
        if ((y < x) == ((a & size) == 0) && x != y) {
          buf[a] = y;
          buf[b] = x;
        }
      }
      // the next step's keys may be another warp's when its stride, or this one's, is long
      if (stride > 32 || (stride == 1 && size > 32)) __syncthreads();
      else __syncwarp();
    }
  }
  __syncthreads();
  const uint32_t per = (n + NT - 1) / NT, b0 = min(tid * per, n), e0 = min(b0 + per, n);
  unsigned heads = 0;
  for (uint32_t i = b0; i < e0; ++i) heads += i == 0 || buf[i] != buf[i - 1];
  unsigned U;
  unsigned u = block_exclusive_scan<NT, unsigned>(heads, sm, &U);
  for (uint32_t i = b0; i < e0; ++i)
    if (i == 0 || buf[i] != buf[i - 1]) head[u++] = (uint16_t)i;
  __syncthreads();
  T* ok = v.keys_a<T>() + off;
  uint32_t* oc = v.counts() + off;
  for (uint32_t r = tid; r < U; r += NT) {
    const uint32_t h = head[r];
    ok[r] = buf[h];
    oc[r] = (r + 1 < U ? head[r + 1] : n) - h;
  }
  if (tid == 0) v.tile_rows()[tile] = U;
}

// One CTA per tile above the on-chip capacity: LSD radix sort of its keys through
// global memory (8-bit digits over the bits that vary, each chunk of CAP keys
// ranked stably on chip), then the run-length reduction to (key, count) rows
// written to keys_a / counts at the tile's offset, and the tile's row count.
template <class T>
__device__ void sort_big(const View& v, uint32_t bk) {
  constexpr int NT = kSortThreads, ITEMS = tile_items<T>(), CAP = NT * ITEMS, NW = NT / 32;
  __shared__ unsigned warp_hist[256 * NW];
  __shared__ unsigned scan_sm[40];
  __shared__ unsigned dtot[256], dstart[256];
  __shared__ unsigned long long run_off[256];
  __shared__ T red_mn[NW], red_mx[NW];
  const uint32_t n = v.tile_count()[bk];
  const uint32_t off = v.tile_off()[bk];
  T* src = v.keys_b<T>() + off;
  T* dst = v.keys_a<T>() + off;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;

  T mn = ~T(0), mx = T(0);
  for (uint32_t i = threadIdx.x; i < n; i += NT) {
    const T x = src[i];
    mn = x < mn ? x : mn;
    mx = x > mx ? x : mx;
  }
  for (int m = 16; m; m >>= 1) {
    const T a = shfl_xor_key(mn, m), b = shfl_xor_key(mx, m);
    mn = a < mn ? a : mn;
    mx = b > mx ? b : mx;
  }
  if (lane == 0) {
    red_mn[wid] = mn;
    red_mx[wid] = mx;
  }
  __syncthreads();
  mn = red_mn[0];
  mx = red_mx[0];
  for (int w = 1; w < NW; ++w) {
    mn = red_mn[w] < mn ? red_mn[w] : mn;
    mx = red_mx[w] > mx ? red_mx[w] : mx;
  }
  const int nbits = mn == mx ? 0 : KeyTraits<T>::kBits - clz_key(T(mn ^ mx));
  const unsigned pos0 = (unsigned)wid * 32u * ITEMS + lane;
  for (int sh = 0; sh < nbits; sh += 8) {
    for (int d = threadIdx.x; d < 256; d += NT) dtot[d] = 0;
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < n; i += NT) atomicAdd(&dtot[digit_of(src[i], sh)], 1u);
    __syncthreads();
    if (threadIdx.x == 0) {
      unsigned long long acc = 0;
      for (int d = 0; d < 256; ++d) {
        run_off[d] = acc;
        acc += dtot[d];
      }
    }
    __syncthreads();
    for (uint32_t c0 = 0; c0 < n; c0 += CAP) {
      const uint32_t cn = min(n - c0, (uint32_t)CAP);
      T key[ITEMS];
      unsigned dig[ITEMS], dest[ITEMS];
      bool valid[ITEMS];
#pragma unroll
      for (int r = 0; r < ITEMS; ++r) {
        const unsigned pos = pos0 + r * 32u;
        valid[r] = pos < cn;
        key[r] = valid[r] ? src[c0 + pos] : T(0);
        dig[r] = digit_of(key[r], sh);
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
  // Run-length reduction of the sorted keys in src.  Unique keys go to
  // keys_a at the partition offset (in place when src is keys_a: the u-th
  // head is written only after the whole chunk holding position u was read,
  // and u never passes the position being read).  Pass A stores the head
  // positions in counts, pass B turns them into run lengths.
  T* ok = v.keys_a<T>() + off;
  uint32_t* oc = v.counts() + off;
  uint32_t U = 0;
  for (uint32_t c0 = 0; c0 < n; c0 += CAP) {
    const uint32_t cn = min(n - c0, (uint32_t)CAP);
    const uint32_t b0 = threadIdx.x * ITEMS;
    T kv[ITEMS];
    bool hd[ITEMS];
    unsigned nh = 0;
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
      const uint32_t i = b0 + r;
      hd[r] = false;
      if (i < cn) {
        const uint32_t gi = c0 + i;
        kv[r] = src[gi];
        hd[r] = gi == 0 || kv[r] != src[gi - 1];
        nh += hd[r];
      }
    }
    unsigned tot;
    uint32_t u = U + block_exclusive_scan<NT, unsigned>(nh, scan_sm, &tot);
#pragma unroll
    for (int r = 0; r < ITEMS; ++r)
      if (hd[r]) {
        ok[u] = kv[r];
        oc[u] = c0 + b0 + r;
        u++;
      }
    U += tot;
    __syncthreads();
  }
  for (uint32_t c0 = 0; c0 < U; c0 += CAP) {
    const uint32_t cn = min(U - c0, (uint32_t)CAP);
    uint32_t cnt[ITEMS];
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
      const uint32_t i = threadIdx.x + r * NT;
      cnt[r] = 0;
      if (i < cn) {
        const uint32_t q = c0 + i;
        cnt[r] = ((q + 1 < U) ? oc[q + 1] : n) - oc[q];
      }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
      const uint32_t i = threadIdx.x + r * NT;
      if (i < cn) oc[c0 + i] = cnt[r];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) v.tile_rows()[bk] = U;
  __syncthreads();
}

// The listed tiles, then (by the last CTA) the row offsets of all tiles.
template <class T>
__global__ void __launch_bounds__(kSortThreads) k_sort_listed(uint32_t tiles, uint8_t* scr) {
  __shared__ unsigned sm[40];
  const View v{scr};
  Counters* c = v.counters();
  const uint32_t n = c->nbig;
  for (uint32_t i = blockIdx.x; i < n; i += gridDim.x) sort_big<T>(v, v.big()[i]);
  if (last_cta(&c->sorted)) cta_scan<kSortThreads>(v.tile_rows(), tiles, v.row_off(), sm);
}

// One CTA per tile: copies its rows to the caller's arrays at the tile's row
// offset (rows past max_rows are dropped; the host reports the shortfall); a
// partition's first tile stores the partition's row count.
template <class T>
__global__ void __launch_bounds__(128) k_emit(uint8_t* scr, uint32_t tiles, uint32_t per_part, T* __restrict__ out_keys,
                                              uint32_t* __restrict__ out_counts, unsigned long long max_rows,
                                              uint32_t* __restrict__ part_rows) {
  const View v{scr};
  const uint32_t bk = blockIdx.x;
  const uint32_t rows = v.tile_rows()[bk];
  const unsigned long long ro = v.row_off()[bk];
  const uint32_t off = v.tile_off()[bk];
  const T* ok = v.keys_a<T>() + off;
  const uint32_t* oc = v.counts() + off;
  for (uint32_t i = threadIdx.x; i < rows; i += blockDim.x) {
    if (ro + i >= max_rows) break;
    out_keys[ro + i] = ok[i];
    out_counts[ro + i] = oc[i];
  }
  if (threadIdx.x == 0) {
    if (bk % per_part == 0) part_rows[bk / per_part] = v.row_off()[bk + per_part] - (uint32_t)ro;
    if (bk == 0) v.counters()->nrows = v.row_off()[tiles];
  }
}

// Per device: the scratch array's address and the SM count, and the CUDA
// context they belong to.  A context that is destroyed and made again (for
// example after cudaDeviceReset) loads this module afresh, so its array can
// sit elsewhere: the entry is looked up again whenever the device's current
// context has another id.
struct DeviceEntry {
  unsigned long long ctx_id = 0;
  uint8_t* scratch = nullptr;
  uint32_t sms = 0;
};
std::mutex g_mu;
DeviceEntry g_dev[kMaxDevices];

typedef int (*CtxGetCurrentFn)(void**);
typedef int (*CtxGetIdFn)(void*, unsigned long long*);

// Id of the calling thread's current context (0 when it cannot be had).
unsigned long long current_ctx_id() {
  static CtxGetCurrentFn get_current = nullptr;
  static CtxGetIdFn get_id = nullptr;
  static bool looked = false;
  if (!looked) {
    looked = true;
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      get_current = reinterpret_cast<CtxGetCurrentFn>(f);
    f = nullptr;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      get_id = reinterpret_cast<CtxGetIdFn>(f);
  }
  if (!get_current || !get_id) return 0;
  void* ctx = nullptr;
  unsigned long long id = 0;
  if (get_current(&ctx) != 0 || !ctx || get_id(ctx, &id) != 0) return 0;
  return id;
}

// Address of this device's scratch array and its SM count, with that device
// current: looked up on the first call in each context of the device (on
// every call when the context id is unavailable).
int device_entry(int device, uint8_t** scratch, uint32_t* sms) {
  std::lock_guard<std::mutex> lock(g_mu);
  DeviceEntry& d = g_dev[device];
  const unsigned long long id = current_ctx_id();
  if (!d.scratch || id == 0 || id != d.ctx_id) {
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess || p == nullptr) return KITE_ERR_CUDA;
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || n < 1)
      return KITE_ERR_CUDA;
    d.scratch = static_cast<uint8_t*>(p);
    d.sms = (uint32_t)n;
    d.ctx_id = id;
  }
  *scratch = d.scratch;
  *sms = d.sms;
  return KITE_OK;
}

// Launches kernel f and returns the error of this launch alone (a launch
// error the caller had left pending is neither reported nor cleared).
template <class... KArgs, class... Args, size_t... I>
cudaError_t launch_impl(void (*f)(KArgs...), dim3 g, dim3 b, cudaStream_t s, std::index_sequence<I...>,
                        Args... args) {
  std::tuple<KArgs...> t(static_cast<KArgs>(args)...);
  void* p[sizeof...(KArgs) + 1] = {static_cast<void*>(&std::get<I>(t))...};
  return cudaLaunchKernel(reinterpret_cast<const void*>(f), g, b, p, 0, s);
}
template <class... KArgs, class... Args>
cudaError_t launch(void (*f)(KArgs...), dim3 g, dim3 b, cudaStream_t s, Args... args) {
  static_assert(sizeof...(KArgs) == sizeof...(Args), "kernel argument count");
  return launch_impl(f, g, b, s, std::index_sequence_for<KArgs...>{}, args...);
}

// Polls the stream until its work is done; no event or other object is made.
int wait_idle(cudaStream_t s, uint32_t timeout_ms) {
  PollPause pause(timeout_ms);
  for (;;) {
    const cudaError_t q = cudaStreamQuery(s);
    if (q == cudaSuccess) return KITE_OK;
    if (q != cudaErrorNotReady) return KITE_ERR_CUDA;
    if (!pause()) return KITE_ERR_TIMEOUT;
  }
}

template <class T>
int run(uint8_t* scr, uint32_t sms, uint32_t k, bool canonical, uint32_t P, const uint8_t* d_fastq, uint32_t len,
        void* d_keys, uint32_t* d_counts, uint64_t max_rows, uint32_t* d_part_rows, uint64_t* totals,
        cudaStream_t s, uint32_t timeout_ms) {
  uint32_t log2p = 0;
  while ((1u << log2p) < P) ++log2p;
  // Tiles: a partition's keys by their top bits, kTileKeys each when every
  // second byte ends a k-mer (reads with qualities) and the keys are even.
  uint32_t bits = 0;
  while (bits < 2 * k && (P << (bits + 1)) <= kMaxTiles && (P << bits) * kTileKeys < len / 2) ++bits;
  const uint32_t tiles = P << bits;
  const TileOf tile_of{64 - log2p, bits, 2 * k};
  Text t;
  t.skew = (uint32_t)(reinterpret_cast<uintptr_t>(d_fastq) & 15u);
  t.base = d_fastq - t.skew;
  t.end = t.skew + len;
  const uint32_t segments = std::max<uint32_t>((t.end + kSegment - 1) / kSegment, 1);
  if (len == 0) t.end = t.skew = 0;  // nothing is read
  const uint32_t g_keys = std::min<uint32_t>(len / 512 + 1, 4 * sms);
  const cudaError_t le[6] = {
      launch(k_prepare, segments, 128, s, t, tiles, scr),
      launch(k_extract<T>, segments, kExtractThreads, s, t, k, canonical ? 1u : 0u, tile_of, tiles, scr),
      launch(k_scatter<T>, g_keys, 256, s, tile_of, scr),
      launch(k_sort_tiles<T>, tiles, kTileSortThreads, s, scr),
      launch(k_sort_listed<T>, std::min(tiles, sms), kSortThreads, s, tiles, scr),
      launch(k_emit<T>, tiles, 128, s, scr, tiles, 1u << bits, static_cast<T*>(d_keys), d_counts,
             (unsigned long long)max_rows, d_part_rows)};
  for (const cudaError_t e : le)
    if (e != cudaSuccess) return KITE_ERR_CUDA;
  int rc = wait_idle(s, timeout_ms);
  if (rc) return rc;
  Counters hc;
  if (cudaMemcpyAsync(&hc, scr + kOffCounters, sizeof hc, cudaMemcpyDeviceToHost, s) != cudaSuccess)
    return KITE_ERR_CUDA;
  rc = wait_idle(s, timeout_ms);
  if (rc) return rc;
  totals[0] = hc.reads;
  totals[1] = hc.bases;
  totals[2] = hc.kmers;
  totals[3] = hc.nrows;
  if (hc.nrows > max_rows) return KITE_ERR_BAD_INPUT;
  return KITE_OK;
}

}  // namespace
}  // namespace na
}  // namespace kite

extern "C" int kite_gpu_count_rows_noalloc(int device, int k, int canonical, uint32_t partitions,
                                           const uint8_t* d_fastq, size_t len, void* d_keys, uint32_t* d_counts,
                                           uint64_t max_rows, uint32_t* d_partition_rows, uint64_t* totals,
                                           void* stream, uint32_t timeout_ms) {
  using namespace kite::na;
  if (!totals) return KITE_ERR_BAD_INPUT;
  for (int i = 0; i < 4; ++i) totals[i] = 0;
  if (k < 1 || k > 64 || partitions < 2 || partitions > kMaxParts || (partitions & (partitions - 1)) ||
      !d_partition_rows || (max_rows && (!d_keys || !d_counts)) || (len && !d_fastq) || device < 0 ||
      device >= kMaxDevices)
    return KITE_ERR_BAD_INPUT;
  if (len > kMaxBytes) return KITE_ERR_UNSUPPORTED;
  int prev = 0;
  if (cudaGetDevice(&prev) != cudaSuccess) return KITE_ERR_CUDA;
  // with the device current its primary context is initialised, so the
  // context id below is that of the context the kernels will run in
  if (cudaSetDevice(device) != cudaSuccess) return KITE_ERR_CUDA;
  uint8_t* scr = nullptr;
  uint32_t sms = 0;
  int rc = device_entry(device, &scr, &sms);
  if (rc == KITE_OK) {
    const cudaStream_t s = static_cast<cudaStream_t>(stream);
    const uint32_t t = timeout_ms ? timeout_ms : 600000u;
    rc = k <= 31 ? run<uint64_t>(scr, sms, (uint32_t)k, canonical != 0, partitions, d_fastq, (uint32_t)len,
                                 d_keys, d_counts, max_rows, d_partition_rows, totals, s, t)
                 : run<u128>(scr, sms, (uint32_t)k, canonical != 0, partitions, d_fastq, (uint32_t)len, d_keys,
                             d_counts, max_rows, d_partition_rows, totals, s, t);
  }
  if (prev != device) cudaSetDevice(prev);
  return rc;
}
