// sort_launch.cuh -- host launchers of the radix sort, instantiated per key width in
// sort_k{1,2,4,8,16,32,64}.cu.
#pragma once

#include <algorithm>

#include "host_common.h"
#include "sort_cluster.cuh"
#include "sort_kernels.cuh"

namespace rfx {

struct SortPlan {
  uint8_t* keys;
  uint8_t* vals;
  const uint8_t* src_keys;   // when set, the sort reads these and leaves them (out of place)
  const uint8_t* src_vals;
  uint8_t* alt_keys;
  uint8_t* alt_vals;
  uint8_t* alt2_keys;   // a second pair of alternate buffers, with 3 or more passes
  uint8_t* alt2_vals;
  uint64_t n;
  uint32_t begin_bit;
  uint32_t end_bit;     // end_bit - begin_bit <= 128
  uint32_t passes;
  uint32_t* ghist;      // [passes][256]
  uint32_t* route;      // [passes]
  uint32_t* done;       // 1
  uint32_t* counters;   // [passes]
  uint32_t* status;     // [passes][tiles][256]
  uint64_t tiles;
  uint32_t* err;
  cudaStream_t stream;
};

struct SortTiles {
  uint64_t tiles;
  uint64_t most;
};

struct ClusterSort {
  const uint8_t* keys_in;
  const uint8_t* vals_in;
  uint8_t* keys_out;   // keys_in, or an array that does not overlap it
  uint8_t* vals_out;
  uint64_t n;
  uint32_t begin_bit, end_bit;
  cudaStream_t stream;
};

// Whether n elements take the pass's small tiles, and how many tiles they make.
template <int K, int V>
bool sort_small(uint64_t n) {
  return kSortHasSmall<K, V> && n <= kSortSmallBelow * SortTuning<K, V>::TILE;
}

template <int K, int V>
uint64_t sort_tiles(uint64_t n) {
  const uint64_t tile = sort_small<K, V>(n) ? SortTuning<K, V, kSortHasSmall<K, V>>::TILE : SortTuning<K, V>::TILE;
  return (n + tile - 1) / tile;
}

// The most tiles that any input of up to n elements makes: a workspace with look-back words
// for that many serves them all.
template <int K, int V>
uint64_t sort_tiles_most(uint64_t n) {
  constexpr uint64_t kSmallMost = kSortHasSmall<K, V> ? kSortSmallBelow * SortTuning<K, V>::TILE : 0;
  const uint64_t tiles = sort_tiles<K, V>(n);
  return n > kSmallMost ? std::max(tiles, sort_tiles<K, V>(kSmallMost)) : tiles;
}

// Histogram of every digit; clears the look-back words.
template <int K, int P>
rfx_status launch_histogram(SortPlan& s) {
  auto k = sort_histogram_kernel<K, P>;
  constexpr size_t smem = P * (size_t)kHistPlaceBytes;
  RFX_CUDA_TRY(allow_smem((const void*)k, smem));
  const uint64_t per_block = (uint64_t)kHistThreads * kHistLoads * 16;   // bytes of one round of loads
  const int grid = persistent_grid((const void*)k, kHistThreads, smem, (s.n * K + per_block - 1) / per_block);
  k<<<grid, kHistThreads, smem, s.stream>>>(s.src_keys ? s.src_keys : s.keys, s.n, s.begin_bit, s.end_bit, s.passes,
                                            s.ghist, s.route, !s.src_keys, s.done, reinterpret_cast<uint4*>(s.status),
                                            s.passes * s.tiles * (kRadix / 4));
  RFX_CUDA_TRY(cudaGetLastError());
  return RFX_OK;
}

template <int K, int V, bool SMALL>
rfx_status run_passes(SortPlan& s) {
  using T = SortTuning<K, V, SMALL>;
  auto pass = sort_pass_kernel<K, V, SMALL>;
  constexpr size_t smem = T::SMEM;
  RFX_CUDA_TRY(allow_smem((const void*)pass, smem));
  const int grid = persistent_grid((const void*)pass, T::THREADS, smem, s.tiles);
  for (uint32_t p = 0; p < s.passes; ++p) {
    SortPassArgs a;
    a.keys[0] = s.src_keys ? const_cast<uint8_t*>(s.src_keys) : s.keys;   // out of place: never written
    a.vals[0] = s.src_keys ? const_cast<uint8_t*>(s.src_vals) : s.vals;
    a.keys[1] = s.keys;
    a.vals[1] = s.vals;
    a.keys[2] = s.alt_keys;
    a.vals[2] = s.alt_vals;
    a.keys[3] = s.alt2_keys;
    a.vals[3] = s.alt2_vals;
    a.route = s.route + p;
    a.n = s.n;
    a.shift = s.begin_bit + 8 * p;
    const uint32_t w = s.end_bit - a.shift < 8 ? s.end_bit - a.shift : 8;
    a.mask = (1u << w) - 1;
    a.gexcl = s.ghist + p * kRadix;
    a.status = s.status + (uint64_t)p * s.tiles * kRadix;
    a.tile_counter = s.counters + p;
    a.err = s.err;
    RFX_CUDA_TRY(launch_chained(pass, grid, T::THREADS, smem, s.stream, a));
  }
  return RFX_OK;
}

template <int K, int V>
rfx_status run_sort_kv(SortPlan& s) {
  rfx_status hst = s.passes == 1   ? launch_histogram<K, 1>(s)
                   : s.passes == 2 ? launch_histogram<K, 2>(s)
                   : s.passes == 3 ? launch_histogram<K, 3>(s)
                                   : launch_histogram<K, kHistPlaces>(s);
  if (hst != RFX_OK) return hst;
  if constexpr (kSortHasSmall<K, V>) {
    if (sort_small<K, V>(s.n)) return run_passes<K, V, true>(s);
  }
  return run_passes<K, V, false>(s);
}

// The one-launch sort of small inputs; RFX_ERR_UNSUPPORTED when it does not take this one
// (nothing is launched then).  Any bit range, in place or out of place.
template <int K, int V>
rfx_status run_cluster_kv(const ClusterSort& c) {
  using T = ClusterTuning<K, V>;
  if (c.n > T::MAX) return RFX_ERR_UNSUPPORTED;
  // as many blocks as give each about kClusterThreads elements: fewer leave SMs idle, more
  // only add to the exchange
  uint32_t blocks = 1;
  while (blocks < (uint32_t)kClusterMax && blocks * kClusterThreads < c.n) blocks *= 2;
  const uint32_t slice = ((c.n + blocks - 1) / blocks + 31) / 32 * 32;
  auto k = sort_cluster_kernel<K, V>;
  // the largest slice's shared memory, so that the lookups are one per cluster size
  const size_t smem = cluster_smem<K, V>(T::SLICE);
  if (!cluster_fits((const void*)k, kClusterThreads, smem, (int)blocks)) return RFX_ERR_UNSUPPORTED;
  ClusterArgs a;
  a.keys_in = c.keys_in;
  a.vals_in = c.vals_in;
  a.keys_out = c.keys_out;
  a.vals_out = c.vals_out;
  a.n = (uint32_t)c.n;
  a.slice = slice;
  a.inverse = (uint32_t)(((1ull << 32) + slice - 1) / slice);
  a.begin_bit = c.begin_bit;
  a.end_bit = c.end_bit;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(kClusterThreads);
  cfg.dynamicSmemBytes = cluster_smem<K, V>(slice);
  cfg.stream = c.stream;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = blocks;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  RFX_CUDA_TRY(cudaLaunchKernelEx(&cfg, k, a));
  return RFX_OK;
}

template <int K>
rfx_status run_cluster(const ClusterSort& c, uint32_t vbytes) {
  switch (vbytes) {
    case 0: return run_cluster_kv<K, 0>(c);
    case 1: return run_cluster_kv<K, 1>(c);
    case 2: return run_cluster_kv<K, 2>(c);
    case 4: return run_cluster_kv<K, 4>(c);
    case 8: return run_cluster_kv<K, 8>(c);
    case 16: return run_cluster_kv<K, 16>(c);
    default: return RFX_ERR_UNSUPPORTED;
  }
}

template <int K>
rfx_status run_sort(SortPlan& s, uint32_t vbytes) {
  switch (vbytes) {
    case 0: return run_sort_kv<K, 0>(s);
    case 1: return run_sort_kv<K, 1>(s);
    case 2: return run_sort_kv<K, 2>(s);
    case 4: return run_sort_kv<K, 4>(s);
    case 8: return run_sort_kv<K, 8>(s);
    case 16: return run_sort_kv<K, 16>(s);
    default: return RFX_ERR_UNSUPPORTED;
  }
}

// The tiles of n elements, and the most of up to n.
template <int K>
SortTiles sort_tiles_for(uint64_t n, uint32_t vbytes) {
  switch (vbytes) {
    case 0: return {sort_tiles<K, 0>(n), sort_tiles_most<K, 0>(n)};
    case 1: return {sort_tiles<K, 1>(n), sort_tiles_most<K, 1>(n)};
    case 2: return {sort_tiles<K, 2>(n), sort_tiles_most<K, 2>(n)};
    case 4: return {sort_tiles<K, 4>(n), sort_tiles_most<K, 4>(n)};
    case 8: return {sort_tiles<K, 8>(n), sort_tiles_most<K, 8>(n)};
    default: return {sort_tiles<K, 16>(n), sort_tiles_most<K, 16>(n)};
  }
}

#define RFX_INSTANTIATE_SORT(K)                                  \
  template rfx_status run_sort<K>(SortPlan&, uint32_t);          \
  template rfx_status run_cluster<K>(const ClusterSort&, uint32_t); \
  template SortTiles sort_tiles_for<K>(uint64_t, uint32_t);

}  // namespace rfx
