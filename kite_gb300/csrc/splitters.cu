// Tile splitters over the key space.  Splitters never change which .kite
// partition a key lands in (that is the Fibonacci hash); they only cut each
// hash bucket into key ranges small enough for the on-chip sort.
//
// Sampled-histogram splitters: a 2^16-bin histogram of the top key bits of
// sampled keys, cut at equal cumulative mass.  Sample quantiles: of up to 2^17
// sampled keys, sorted, for keys whose top bits are too skewed for the
// histogram.  The learned alternative lives in mlp_kernels.cu and produces
// splitters in the same format.
#include "kite_internal.h"
#include "splitters.h"

namespace kite {

template <class T>
__global__ void k_sample_hist(const T* __restrict__ sample, uint32_t n, uint32_t key_bits, uint32_t hbits,
                              unsigned* __restrict__ hist) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    atomicAdd(&hist[sample_bin(sample[i], key_bits, hbits)], 1u);
}

// One CTA: turns the histogram into its inclusive cumulative counts (in
// place), then splitter j = upper edge of the first bin whose cumulative
// count reaches ceil(j*total/S).  Each thread takes consecutive bins (64 of
// 65536, by 16-byte loads), so one block scan serves them all: what bounds it
// is the latency of that chain, 135 us with a scan per 1024 bins
// beside the bucket scatter, 47 us now.
template <class T>
__global__ void __launch_bounds__(1024) k_hist_splitters(unsigned* __restrict__ cum, uint32_t hbits,
                                                         uint32_t key_bits, uint32_t S, T* __restrict__ spl) {
  __shared__ unsigned sm[34];
  const uint32_t nb = 1u << hbits;
  unsigned carry = 0;
  if (nb >= 4096) {
    const uint32_t per = nb / 1024;  // a multiple of 4, at most 64
    uint4* c4 = reinterpret_cast<uint4*>(cum) + threadIdx.x * (per / 4);
    unsigned sum = 0;
    for (uint32_t j0 = 0; j0 < per / 4; j0 += 4) {
      uint4 v[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] = j0 + j < per / 4 ? c4[j0 + j] : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int j = 0; j < 4; ++j) sum += v[j].x + v[j].y + v[j].z + v[j].w;
    }
    unsigned at = block_exclusive_scan<1024, unsigned>(sum, sm, &carry);
    for (uint32_t j0 = 0; j0 < per / 4; j0 += 4) {
      uint4 v[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] = j0 + j < per / 4 ? c4[j0 + j] : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        v[j].x += at;
        v[j].y += v[j].x;
        v[j].z += v[j].y;
        v[j].w += v[j].z;
        at = v[j].w;
        if (j0 + j < per / 4) c4[j0 + j] = v[j];
      }
    }
  } else {
    for (uint32_t b0 = 0; b0 < nb; b0 += 1024) {
      const uint32_t b = b0 + threadIdx.x;
      const unsigned v = b < nb ? cum[b] : 0;
      unsigned tot;
      const unsigned ex = block_exclusive_scan<1024, unsigned>(v, sm, &tot);
      if (b < nb) cum[b] = carry + ex + v;
      carry += tot;
    }
  }
  __syncthreads();
  const unsigned long long total = carry;
  const uint32_t sh = key_bits - hbits;
  for (uint32_t j = threadIdx.x + 1; j < S; j += blockDim.x) {
    T s;
    if (total == 0) {
      // no sample: uniform cut of [0, 2^key_bits): j/S as a 32-bit fraction, scaled
      const unsigned long long f = ((unsigned long long)j << 32) / S;
      s = key_bits >= 32 ? ((T)f << (key_bits - 32)) : (T)(f >> (32 - key_bits));
    } else {
      const unsigned long long target = (total * (unsigned long long)j + S - 1) / S;
      uint32_t lo = 0, hi = nb - 1;
      while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if ((unsigned long long)cum[mid] >= target) hi = mid;
        else lo = mid + 1;
      }
      // keys of bins <= lo fall below the splitter
      s = (lo + 1 == nb && key_bits == (uint32_t)KeyTraits<T>::kBits) ? ~T(0) : ((T)(lo + 1) << sh);
    }
    spl[j - 1] = s;
  }
}

template <class T>
int compute_hist_splitters(const T* d_sample, uint32_t nsample, uint32_t key_bits, uint32_t S, T* d_spl,
                           unsigned* d_hist /* 65536 */, cudaStream_t s) {
  const uint32_t hbits = key_bits < 16 ? key_bits : 16;
  cudaMemsetAsync(d_hist, 0, sizeof(unsigned) << hbits, s);
  if (nsample) k_sample_hist<T><<<256, 256, 0, s>>>(d_sample, nsample, key_bits, hbits, d_hist);
  k_hist_splitters<T><<<1, 1024, 0, s>>>(d_hist, hbits, key_bits, S, d_spl);
  return nsample ? 2 : 1;
}
// ---- sample quantiles ---------------------------------------------------------
// n keys, evenly taken from the sample, in blocks of kSortBlock sorted by one
// CTA each (bitonic, in shared memory); a key's rank is its place in its block
// plus the keys before it in every other block (binary searches, all in L1 and
// L2).  Up to 64 blocks: one launch of searches costs less than six of merging.
// 188M keys of an AT-rich genome at k = 63, 214 ranges per bucket: the largest
// holds 1.10 times the mean (3.8 times with the histogram), in 0.08 + 0.36 ms
// beside the bucket scatter; training the learned CDF took 650 ms in a context's
// first call.
constexpr uint32_t kSortBlock = 2048;
constexpr uint32_t kMaxQuantileKeys = 1u << 17;

template <class T>
__global__ void __launch_bounds__(512) k_sort_sample(const T* __restrict__ sample, uint32_t nsample, uint32_t n,
                                                     T* __restrict__ out) {
  __shared__ T buf[kSortBlock];
  const uint32_t b0 = blockIdx.x * kSortBlock;
  for (uint32_t i = threadIdx.x; i < kSortBlock; i += 512)
    buf[i] = b0 + i < n ? sample[(uint64_t)(b0 + i) * nsample / n] : ~T(0);
  __syncthreads();
  for (uint32_t size = 2; size <= kSortBlock; size *= 2) {
    for (uint32_t stride = size / 2; stride; stride /= 2) {
      for (uint32_t i = threadIdx.x; i < kSortBlock / 2; i += 512) {
        const uint32_t a = 2 * i - (i & (stride - 1)), b = a + stride;
        const T x = buf[a], y = buf[b];
        if (x != y && (y < x) == ((a & size) == 0)) {
          buf[a] = y;
          buf[b] = x;
        }
      }
      // a warp's pairs of a step with stride <= 32 are 64 consecutive keys
      if (stride > 32 || (stride == 1 && size > 32)) __syncthreads();
      else __syncwarp();
    }
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < kSortBlock; i += 512)
    if (b0 + i < n) out[b0 + i] = buf[i];
}

// Splitter j (1 <= j < S) = the key of rank j * n / S.
template <class T>
__global__ void __launch_bounds__(256) k_quantiles(const T* __restrict__ keys, uint32_t n, uint32_t S,
                                                   T* __restrict__ spl) {
  const uint32_t at = blockIdx.x * 256 + threadIdx.x;
  if (at >= n) return;
  const T key = keys[at];
  const uint32_t mine = at / kSortBlock;
  uint32_t rank = at % kSortBlock;
  constexpr int U = 8;  // searches side by side: each step waits for L2
  for (uint32_t c0 = 0; c0 * kSortBlock < n; c0 += U) {
    uint32_t pos[U];
#pragma unroll
    for (int u = 0; u < U; ++u) pos[u] = 0;
    for (uint32_t w = kSortBlock; w; w /= 2) {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const uint64_t b = (uint64_t)(c0 + u) * kSortBlock;
        if (pos[u] + w > kSortBlock || b + pos[u] + w > n) continue;
        const T x = keys[b + pos[u] + w - 1];
        if (x < key || (x == key && c0 + u < mine)) pos[u] += w;  // equal keys of earlier blocks come first
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) rank += c0 + u == mine ? 0u : pos[u];
  }
  for (uint64_t j = ((uint64_t)rank * S + n - 1) / n; j < S && j * n / S == rank; ++j)
    if (j) spl[j - 1] = key;
}

template <class T>
int compute_quantile_splitters(const T* d_sample, uint32_t nsample, uint32_t S, T* d_spl, T* d_keys, cudaStream_t s) {
  const uint32_t n = nsample < kMaxQuantileKeys ? nsample : kMaxQuantileKeys;
  k_sort_sample<T><<<(n + kSortBlock - 1) / kSortBlock, 512, 0, s>>>(d_sample, nsample, n, d_keys);
  k_quantiles<T><<<(n + 255) / 256, 256, 0, s>>>(d_keys, n, S, d_spl);
  return 2;
}
uint32_t quantile_keys() { return kMaxQuantileKeys; }
template int compute_quantile_splitters<uint64_t>(const uint64_t*, uint32_t, uint32_t, uint64_t*, uint64_t*, cudaStream_t);
template int compute_quantile_splitters<u128>(const u128*, uint32_t, uint32_t, u128*, u128*, cudaStream_t);
template int compute_hist_splitters<uint64_t>(const uint64_t*, uint32_t, uint32_t, uint32_t, uint64_t*, unsigned*,
                                              cudaStream_t);
template int compute_hist_splitters<u128>(const u128*, uint32_t, uint32_t, uint32_t, u128*, unsigned*,
                                          cudaStream_t);

}  // namespace kite
