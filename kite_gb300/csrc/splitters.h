// Splitter producers (sampled histogram, sample quantiles, learned CDF).  Internal.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "kite_common.cuh"

namespace kite {

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
