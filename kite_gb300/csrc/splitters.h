// Splitter producers (sampled histogram, sample quantiles, learned CDF).  Internal.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "kite_common.cuh"

namespace kite {

// The key, or the largest one of key_bits bits when it is above that.  Sampled
// rows of a database are as its bytes say: a wrong head key, or rows that its
// chunk does not hold (the decode's status tells later), may be any value.
template <class T>
__host__ __device__ __forceinline__ T within_bits(T key, uint32_t key_bits) {
  const T last = key_bits < 8 * sizeof(T) ? (T(1) << key_bits) - T(1) : ~T(0);
  return key < last ? key : last;
}
// Bin of a sampled key in a histogram of its top hbits bits.
template <class T>
__host__ __device__ __forceinline__ uint32_t sample_bin(T key, uint32_t key_bits, uint32_t hbits) {
  return (uint32_t)(uint64_t)(within_bits(key, key_bits) >> (key_bits - hbits));
}
// The key's 48 top bits, the learned CDF's view of it (a shorter key's bits on top).
template <class T>
__host__ __device__ __forceinline__ uint64_t view48(T key, uint32_t key_bits) {
  const T x = within_bits(key, key_bits);
  return key_bits >= 48 ? (uint64_t)(x >> (key_bits - 48)) : ((uint64_t)x << (48 - key_bits));
}

// S-1 ascending splitters from a 2^16-bin histogram of the sampled keys'
// top bits (key_bits = 2k).  With no sample, splitters cut [0, 2^key_bits)
// uniformly.
// Returns the number of kernels launched.
template <class T>
int compute_hist_splitters(const T* d_sample, uint32_t nsample, uint32_t key_bits, uint32_t S, T* d_spl,
                           unsigned* d_hist, cudaStream_t s);

// S-1 ascending splitters (some may be equal) at the quantiles of up to
// quantile_keys() of the sampled keys, which d_keys has room for; at least S of
// them.  Returns the number of kernels launched.
template <class T>
int compute_quantile_splitters(const T* d_sample, uint32_t nsample, uint32_t S, T* d_spl, T* d_keys, cudaStream_t s);
uint32_t quantile_keys();

}  // namespace kite
