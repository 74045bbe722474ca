// sort_cluster.cuh -- the radix sort of small inputs in one launch: the whole input in the
// shared memory of one thread-block cluster, every digit pass within the cluster.
#pragma once

#include <cooperative_groups.h>
#include <utility>

#include "sort_kernels.cuh"

namespace rfx {

// The general path costs a launch per digit plus the histogram's and a clear, each a few
// microseconds however small the input (10K rows of 8 bytes: 52 us for four passes), on one
// to a few SMs.  Here block c of the cluster holds elements [c * slice, (c + 1) * slice) in
// shared memory.  Per pass: rank as the general pass does (sort_kernels.cuh), exchange the
// blocks' digit counts through distributed shared memory, and write every element to its
// place in the other buffer of the block that owns it; two cluster barriers.  The last pass
// writes to global memory.  Four passes, us a call back to back, general -> here (the general
// path on either side of the largest input that fits):
//   4 B rows   10K 45 -> 18.6, 65536 51 -> 25.8      8 B   10K 45 -> 18.6, 65536 51 -> 28.9
//   16 B       10K 45 -> 18.6, 65536 43 -> 33.4
// so everything that fits the cluster's shared memory comes here.
constexpr int kClusterThreads = 512;
constexpr int kClusterWarps = kClusterThreads / 32;
constexpr int kClusterSteps = 8;     // elements per lane at the most
constexpr int kClusterMax = 16;      // blocks (above 8 not portable, but resident on this part)

template <int K, int V>
struct ClusterTuning {
  // elements per block: two buffers of 64 KB at the most, and kClusterSteps per lane
  static constexpr uint32_t FIT = 65536 / (K + V) / 32 * 32;
  static constexpr uint32_t SLICE = FIT < kClusterThreads * kClusterSteps ? FIT : kClusterThreads * kClusterSteps;
  static constexpr uint32_t MAX = SLICE * kClusterMax;
};

// Dynamic shared memory for a slice of `slice` elements (a multiple of 32): two key and two
// value buffers, the entries, the warps' counters, two rounds of all blocks' digit counts.
template <int K, int V>
__host__ __device__ constexpr size_t cluster_smem(uint32_t slice) {
  return (size_t)slice * (2 * (K + V) + 4) + (kClusterWarps + 2 * kClusterMax) * kRadix * 4;
}

struct ClusterArgs {
  const uint8_t* keys_in;
  const uint8_t* vals_in;
  uint8_t* keys_out;     // may be keys_in: every block has loaded its slice before any writes
  uint8_t* vals_out;
  uint32_t n;
  uint32_t slice;        // elements per block, a multiple of 32
  uint32_t inverse;      // ceil(2^32 / slice): position / slice = mulhi(position, inverse)
  uint32_t begin_bit, end_bit;
};

template <int K, int V>
__global__ void __launch_bounds__(kClusterThreads, 1) sort_cluster_kernel(const ClusterArgs a) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  const uint32_t blocks = cluster.num_blocks(), me = cluster.block_rank();
  extern __shared__ __align__(16) uint8_t sbuf[];
  uint8_t* keys = sbuf;                                       // this pass's elements, then the next's
  uint8_t* keys_next = keys + (size_t)a.slice * K;
  uint8_t* vals = keys_next + (size_t)a.slice * K;
  uint8_t* vals_next = vals + (size_t)a.slice * V;
  uint32_t* const entries = reinterpret_cast<uint32_t*>(sbuf + (size_t)a.slice * 2 * (K + V));
  uint32_t* const counters = entries + a.slice;               // [warps][256]
  uint32_t* counts = counters + kClusterWarps * kRadix;       // [blocks][256] of this pass, then the next's
  uint32_t* counts_next = counts + kClusterMax * kRadix;
  __shared__ uint32_t s_base[kRadix];
  __shared__ uint32_t s_scan[2][kRadix / 32];
  const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const uint32_t lo = min(me * a.slice, a.n), count_me = min(a.slice, a.n - lo);
  for (uint32_t i = t; i < count_me; i += kClusterThreads) {
    store_elem<K>(keys, i, load_elem<K>(a.keys_in, lo + i));
    if constexpr (V > 0) store_elem<V>(vals, i, load_elem<V>(a.vals_in, lo + i));
  }
  cluster.sync();   // every block runs: its shared memory can be written from the others
  // warp w owns elements [w * span, (w + 1) * span) of the slice
  const uint32_t steps = (a.slice / 32 + kClusterWarps - 1) / kClusterWarps, span = steps * 32;
  uint32_t* const wcount = counters + warp * kRadix;
  bool written = false;
  for (uint32_t bit = a.begin_bit; bit < a.end_bit; bit += 8) {
    const uint32_t width = min(8u, a.end_bit - bit), mask = (1u << width) - 1;
    const uint32_t q = bit >> 5, sh = bit & 31;
    const bool straddle = sh + width > 32;
    for (uint32_t k = t; k < kClusterWarps * kRadix / 4; k += kClusterThreads)
      reinterpret_cast<uint4*>(counters)[k] = make_uint4(0, 0, 0, 0);
    __syncthreads();
    uint32_t key[kClusterSteps];   // digit << 16 | rank among the warp's elements of that digit
#pragma unroll
    for (int j = 0; j < kClusterSteps; ++j) {
      const uint32_t i = warp * span + j * 32 + lane;
      key[j] = 0xffffffffu;
      if ((uint32_t)j < steps && i < count_me) {
        const uint32_t d = raw_digit<K>(keys, i, q, sh, straddle) & mask;
        key[j] = d << 16 | atomicAdd(&wcount[d], 1u);
      }
    }
    __syncthreads();
    uint32_t before[kClusterWarps], count = 0, start = 0;
    if (t < kRadix) {
#pragma unroll
      for (int w = 0; w < kClusterWarps; ++w) before[w] = counters[w * kRadix + t];
#pragma unroll
      for (int w = 0; w < kClusterWarps; ++w) {
        const uint32_t c = before[w];
        before[w] = count;
        count += c;
      }
      for (uint32_t b = 0; b < blocks; ++b) *cluster.map_shared_rank(counts + me * kRadix + t, b) = count;
      uint32_t incl = count;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (uint32_t)o) incl += v;
      }
      if (lane == 31) s_scan[0][warp] = incl;
      start = incl - count;
    }
    auto counted = cluster.barrier_arrive();
    __syncthreads();
    if (t < kRadix) {
#pragma unroll
      for (uint32_t w = 0; w < kRadix / 32; ++w) start += w < warp ? s_scan[0][w] : 0u;
#pragma unroll
      for (int w = 0; w < kClusterWarps; ++w) counters[w * kRadix + t] = before[w] + start;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kClusterSteps; ++j)
      if (key[j] != 0xffffffffu)
        entries[wcount[key[j] >> 16] + (key[j] & 0xffffu)] = (key[j] & 0xffff0000u) | (warp * span + j * 32 + lane);
    cluster.barrier_wait(std::move(counted));
    // all blocks' counts: the digit's global start and what lower blocks hold of it
    uint32_t total = 0, lower = 0, incl = 0;
    if (t < kRadix) {
      for (uint32_t b = 0; b < blocks; ++b) {
        const uint32_t c = counts[b * kRadix + t];
        total += c;
        lower += b < me ? c : 0u;
      }
      incl = total;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (uint32_t)o) incl += v;
      }
      if (lane == 31) s_scan[1][warp] = incl;
    }
    // a digit that every element has: the pass is the identity (every block sees the same)
    const bool trivial = __syncthreads_or(t < kRadix && total == a.n);
    uint32_t* const swap_counts = counts;
    counts = counts_next;
    counts_next = swap_counts;
    if (trivial) continue;
    if (t < kRadix) {
      uint32_t first = incl - total;
#pragma unroll
      for (uint32_t w = 0; w < kRadix / 32; ++w) first += w < warp ? s_scan[1][w] : 0u;
      s_base[t] = first + lower - start;
    }
    bool disorder = false;   // see sort_pass_kernel
    for (uint32_t i = t + 1; i < count_me; i += kClusterThreads) disorder = disorder || entries[i - 1] > entries[i];
    if (__syncthreads_or(disorder)) order_entries(entries, count_me, kClusterThreads);
    const bool last = bit + 8 >= a.end_bit;
    for (uint32_t i = t; i < count_me; i += kClusterThreads) {
      const uint32_t e = entries[i], li = e & 0xffffu, pos = s_base[e >> 16] + i;
      const Elem<K> k = load_elem<K>(keys, li);
      if (last) {
        store_elem<K>(a.keys_out, pos, k);
        if constexpr (V > 0) store_elem<V>(a.vals_out, pos, load_elem<V>(vals, li));
      } else {
        const uint32_t owner = __umulhi(pos, a.inverse), at = pos - owner * a.slice;
        store_elem<K>(cluster.map_shared_rank(keys_next, owner), at, k);
        if constexpr (V > 0) store_elem<V>(cluster.map_shared_rank(vals_next, owner), at, load_elem<V>(vals, li));
      }
    }
    written = last;
    cluster.sync();   // every element is in place, and no block leaves while another writes to it
    uint8_t* const swap_keys = keys;
    keys = keys_next;
    keys_next = swap_keys;
    uint8_t* const swap_vals = vals;
    vals = vals_next;
    vals_next = swap_vals;
  }
  if (!written) {
    // the last pass moved nothing (its barrier was every block's last access to another)
    for (uint32_t i = t; i < count_me; i += kClusterThreads) {
      store_elem<K>(a.keys_out, lo + i, load_elem<K>(keys, i));
      if constexpr (V > 0) store_elem<V>(a.vals_out, lo + i, load_elem<V>(vals, i));
    }
  }
}

}  // namespace rfx
