// sort_kernels.cuh -- stable LSD radix sort of packed keys (with optional values):
// one histogram pass over the keys for every digit, then one kernel per 8-bit digit that
// ranks a tile with shared-memory counters, publishes per-digit tile counts through
// decoupled look-back, and writes the tile out in digit runs.
//
// Keys are containers of K bytes (1..64), sorted on bits [begin_bit, end_bit) as
// unsigned integers, values V bytes (0 = keys only).  The sort is stable, so it orders
// exactly like b40c's LSD sort on bits [0, key_bits) (b40cSort.cu:58-1022) and like
// moderngpu's stable merge sort when the range covers the whole key (ModernGPUSort.cu).
#pragma once

#include "rfx_device.cuh"
#include "tile_ring.cuh"

namespace rfx {

constexpr int kRadix = 256;
constexpr int kMaxSortPasses = 16;  // up to 128 key bits per call
constexpr int kSortLookWindow = 8;  // predecessors examined per look-back round trip (16: 2 % slower, 32: 8 %)

// The tile of a digit pass by the bytes of a key and its value.  Two blocks per SM: as large
// a tile as their shared memory allows (the per-tile costs -- barriers, the look-back -- and
// the number of digit runs a tile is written in fall with its size), over as many threads as
// that leaves registers for.  Whole sorts of four passes, us, at 1M / 4M / 60M elements:
//   4 B   512 x 20: 63 / 117 / 942 (64 registers, 28 bytes of spills); 512 x 22: 68 / 122 / 930;
//         384 x 28: 74 / 133 / 1060
//   8 B   512 x 14: 62 / 120 / 1170; 512 x 12: 62 / 125 / 1211; 384 x 16: 62 / 138 / 1281
//   4 B keys with 8 B values   512 x 10: 65 / 141 / 1447; 384 x 12: 63 / 148 / 1510; 384 x 16: 71 / 153 / 1389
//   16 B  512 x 9: 67 / 162 / 1688; 512 x 8: 65 / 166 / 1746; 384 x 12: 71 / 167 / 1710
// Inputs of fewer large tiles than SMs take small tiles instead (elements of 4 to 16 bytes):
// a tile's chain is shorter and more SMs work.  Large -> small, us:
//   4 B   100K 51 -> 38, 1M (98 large tiles) 61 -> 52, 2M (196) 70 -> 75
//   8 B   300K 48 -> 42, 1M (140) 59 -> 58, 2M (280) 67 -> 84
//   16 B  100K 42 -> 36, 300K (66) 46 -> 44, 1M (218) 62 -> 71
constexpr uint64_t kSortSmallBelow = 148;   // large tiles

template <int K, int V>
constexpr bool kSortHasSmall = (K == 4 || K == 8 || K == 16) && K + V <= 16;

template <int K, int V, bool SMALL = false>
struct SortTuning {
  static constexpr int B = K + V;
  static constexpr int THREADS = B <= 16 ? 512 : B <= 48 ? 384 : 256;
  static constexpr int LARGE = B <= 4 ? 20 : B <= 8 ? 14 : B <= 12 ? 10 : B <= 16 ? 9 : B <= 32 ? 6 : 4;
  static constexpr int IPT = !SMALL ? LARGE : B <= 4 ? 8 : B <= 8 ? 6 : B <= 12 ? 5 : 4;
  static constexpr int WARPS = THREADS / 32;
  static constexpr int TILE = THREADS * IPT;
  // dynamic shared memory: the tile's keys and values as they lie in global memory, every
  // warp's digit counters, one 32-bit entry per element
  static constexpr size_t KEYS = (size_t)TILE * K;
  static constexpr size_t VALS = (size_t)TILE * V;
  static constexpr size_t COUNTERS = (size_t)WARPS * 256 * 4;
  static constexpr size_t SMEM = KEYS + VALS + COUNTERS + (size_t)TILE * 4;
  static_assert(THREADS >= 256, "one thread per digit");
  static_assert(TILE <= 0x10000, "an element's place in its tile fits 16 bits");
  static_assert(KEYS % 16 == 0 && VALS % 16 == 0 && COUNTERS % 16 == 0, "16-byte aligned parts");
  static_assert(2 * (SMEM + 4096) <= 228 * 1024, "two blocks per SM");
};

// A K-byte element as 32-bit words (1- and 2-byte elements zero-extended into w[0]).
template <int B>
struct Elem {
  static constexpr int NW = B <= 4 ? 1 : B / 4;
  uint32_t w[NW];
};

template <int B>
__device__ __forceinline__ Elem<B> load_elem(const uint8_t* base, uint64_t i) {
  Elem<B> e;
  if constexpr (B == 1) {
    e.w[0] = base[i];
  } else if constexpr (B == 2) {
    e.w[0] = reinterpret_cast<const uint16_t*>(base)[i];
  } else if constexpr (B == 4) {
    e.w[0] = reinterpret_cast<const uint32_t*>(base)[i];
  } else if constexpr (B == 8) {
    uint2 v = reinterpret_cast<const uint2*>(base)[i];
    e.w[0] = v.x;
    e.w[1] = v.y;
  } else {
    const uint4* p = reinterpret_cast<const uint4*>(base + i * B);
#pragma unroll
    for (int k = 0; k < B / 16; ++k) {
      uint4 v = p[k];
      e.w[4 * k] = v.x;
      e.w[4 * k + 1] = v.y;
      e.w[4 * k + 2] = v.z;
      e.w[4 * k + 3] = v.w;
    }
  }
  return e;
}

template <int B>
__device__ __forceinline__ void store_elem(uint8_t* base, uint64_t i, const Elem<B>& e) {
  if constexpr (B == 1) {
    base[i] = (uint8_t)e.w[0];
  } else if constexpr (B == 2) {
    reinterpret_cast<uint16_t*>(base)[i] = (uint16_t)e.w[0];
  } else if constexpr (B == 4) {
    reinterpret_cast<uint32_t*>(base)[i] = e.w[0];
  } else if constexpr (B == 8) {
    reinterpret_cast<uint2*>(base)[i] = make_uint2(e.w[0], e.w[1]);
  } else {
    uint4* p = reinterpret_cast<uint4*>(base + i * B);
#pragma unroll
    for (int k = 0; k < B / 16; ++k) p[k] = make_uint4(e.w[4 * k], e.w[4 * k + 1], e.w[4 * k + 2], e.w[4 * k + 3]);
  }
}

// Where the passes read and write.  A pass whose digit is the same in every key moves
// nothing; which passes those are is known on the device only (from the histogram), so the
// histogram's last block plans the sequence and every pass kernel looks its part up:
//   bits 0..1 source, 2..3 destination buffer (0 the source, 1 the output, 2 / 3 the
//   alternates; in place 0 and 1 are the same), and what to do.
constexpr uint32_t kRouteSort = 16;
constexpr uint32_t kRouteCopy = 32;

__host__ __device__ constexpr uint32_t sort_route(uint32_t what, uint32_t from, uint32_t to) {
  return what | from | to << 2;
}

__host__ __device__ __forceinline__ uint32_t bit_count(uint32_t x) {
#ifdef __CUDA_ARCH__
  return __popc(x);
#else
  return (uint32_t)__builtin_popcount(x);
#endif
}

// The part of pass p of `passes`; bit p of `moving`: pass p's digits are not all the same.
// The result ends in buffer 1, but for a single pass in place, which ends in 2 (the caller
// copies it back; it always runs).  An even number of passes that move keys goes back and
// forth between 1 and 2; in place an odd number from 3 on takes 2, 3, 1 first; a single one
// is copied, before or after, by a pass that moves nothing itself.
__host__ __device__ __forceinline__ uint32_t sort_plan(uint32_t moving, uint32_t passes, bool in_place, uint32_t p) {
  if (passes == 1) moving = 1;
  const uint32_t m = bit_count(moving);
  if (m == 0) return !in_place && p == passes - 1 ? sort_route(kRouteCopy, 0, 1) : 0u;
  const bool moves = moving >> p & 1;
  if (in_place && m == 1 && passes > 1) {
    if (!(moving >> (passes - 1) & 1))
      return moves ? sort_route(kRouteSort, 0, 2) : p == passes - 1 ? sort_route(kRouteCopy, 2, 1) : 0u;
    return moves ? sort_route(kRouteSort, 2, 1) : p == 0 ? sort_route(kRouteCopy, 0, 2) : 0u;
  }
  if (!moves) return 0;
  auto to = [&](uint32_t j) -> uint32_t {   // of the j-th pass that moves
    if (!in_place || m % 2 == 0) return (m - 1 - j) % 2 ? 2 : 1;
    return j == 1 ? 3 : j == 0 || j % 2 ? 2 : 1;
  };
  const uint32_t j = bit_count(moving & ((1u << p) - 1));
  return sort_route(kRouteSort, j ? to(j - 1) : 0u, to(j));
}

struct SortPassArgs {
  uint8_t* keys[4];     // the buffers of the routes (keys[0] is only read when it is not keys[1])
  uint8_t* vals[4];
  const uint32_t* route;  // this pass's part
  uint64_t n;
  uint32_t shift;       // first bit of this digit
  uint32_t mask;        // digit mask (0xff, or fewer bits for the last digit)
  const uint32_t* gexcl;  // exclusive global digit offsets of this pass [256]
  uint32_t* status;     // [tiles][256] look-back words of this pass
  uint32_t* tile_counter;
  uint32_t* err;
};

// 32-bit look-back words: bits 31..30 flag (1 aggregate, 2 inclusive), 29..0 value.
constexpr uint32_t kSFlagAgg = 1u << 30;
constexpr uint32_t kSFlagInc = 2u << 30;
constexpr uint32_t kSValMask = (1u << 30) - 1;

__device__ __forceinline__ uint32_t ld_relaxed_u32(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed_u32(uint32_t* p, uint32_t v) {
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// ------------------------------------------------------------------ histogram
// Counts the digits of up to kHistPlaces passes in one read of the keys (more passes: one
// read per kHistPlaces), then the last block turns the counts into exclusive offsets and
// plans the passes (sort_plan).  Also clears the look-back words of every pass.
//
// Every lane counts in bins of its own (bin d of lane l at word d * 32 + l, so that the 32
// lanes always hit 32 banks): a digit is two or three instructions and one wavefront,
// whatever its distribution; one funnel shift brings a group's digits into one word.  Bins
// shared by the block, with a warp vote that took digits equal in all lanes together, were
// bound by instruction issue and bank conflicts: 60M 4-byte keys with four digits 337 us (now
// 60), 60M 16-byte rows 483 us (178).  16 bytes per load and
// thread, kHistLoads loads in flight.
constexpr int kHistThreads = 1024;
constexpr int kHistPlaces = 4;
constexpr int kHistLoads = 4;
constexpr uint32_t kHistPlaceBytes = kRadix * 32 * 4;

template <int PLACE>
__device__ __forceinline__ void hist_count(uint32_t at) {
  asm volatile("red.shared.add.u32 [%0 + %1], 1;" ::"r"(at), "n"(PLACE * kHistPlaceBytes) : "memory");
}

// The 32 bits of an element from bit `begin` on hold every digit of a group of up to four
// places; digit p is bits [8 p, 8 p + 8) of them.
template <int K, int P>
struct HistDigits {
  uint32_t q, sh;      // the word and the bit in it where the group's digits begin
  uint32_t mask[P];    // each place's digit mask, at bit 7
  uint32_t at;         // this lane's bin 0 of place 0
  __device__ __forceinline__ HistDigits(uint32_t bins, uint32_t begin, uint32_t end) : at(bins + (threadIdx.x & 31) * 4) {
    q = begin >> 5;
    sh = begin & 31;
#pragma unroll
    for (int p = 0; p < P; ++p) {
      const uint32_t s = begin + 8 * p;
      const uint32_t w = s >= end ? 0u : end - s < 8 ? end - s : 8u;   // places past the last pass: digit 0
      mask[p] = ((1u << w) - 1) << 7;
    }
  }
  template <int PLACE = 0>
  __device__ __forceinline__ void count_places(uint32_t w) const {
    if constexpr (PLACE < P) {
      hist_count<PLACE>(at + (__funnelshift_r(w, w, (8 * PLACE - 7) & 31) & mask[PLACE]));
      count_places<PLACE + 1>(w);
    }
  }
  __device__ __forceinline__ void count(const Elem<K>& e) const {
    if constexpr (Elem<K>::NW == 1) {
      count_places(e.w[0] >> sh);
    } else {
      uint32_t lo = e.w[0], hi = e.w[1];
#pragma unroll
      for (int k = 1; k < Elem<K>::NW; ++k) {
        if ((int)q == k) {
          lo = e.w[k];
          hi = k + 1 < Elem<K>::NW ? e.w[k + 1] : 0u;
        }
      }
      count_places(__funnelshift_r(lo, hi, sh));
    }
  }
};

// The digits of the elements in one 16-byte chunk.
template <int K, int P>
__device__ __forceinline__ void hist_chunk(const HistDigits<K, P>& h, const uint4& v) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
  if constexpr (K <= 4) {
#pragma unroll
    for (int k = 0; k < 16 / K; ++k) {
      Elem<K> e;
      e.w[0] = w[k * K / 4] >> (8 * (k * K % 4));
      h.count(e);
    }
  } else if constexpr (K == 8) {
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      Elem<8> e;
      e.w[0] = w[2 * k];
      e.w[1] = w[2 * k + 1];
      h.count(e);
    }
  } else {
    Elem<16> e;
#pragma unroll
    for (int k = 0; k < 4; ++k) e.w[k] = w[k];
    h.count(e);
  }
}

template <int K, int P>
__global__ void __launch_bounds__(kHistThreads)
sort_histogram_kernel(const uint8_t* __restrict__ keys, uint64_t n, uint32_t begin_bit, uint32_t end_bit,
                      uint32_t passes, uint32_t* __restrict__ ghist, uint32_t* __restrict__ route, bool in_place,
                      uint32_t* __restrict__ done_counter, uint4* __restrict__ status, uint64_t status_chunks) {
  extern __shared__ __align__(16) uint32_t bins[];   // [P][256][32]
  __shared__ bool s_last;
  __shared__ uint32_t s_moving;   // bit p: pass p has more than one digit
  const uint32_t t = threadIdx.x, lane = t & 31;
  const uint64_t tid = (uint64_t)blockIdx.x * kHistThreads + t, stride = (uint64_t)gridDim.x * kHistThreads;
  grid_release();
  for (uint64_t k = tid; k < status_chunks; k += stride) status[k] = make_uint4(0, 0, 0, 0);
  // whole 16-byte chunks where the elements tile them; the rest element by element
  const bool vec = K <= 16 && (reinterpret_cast<uintptr_t>(keys) & 15u) == 0;
  const uint64_t chunks = vec ? n * K / 16 : 0;
  for (uint32_t p0 = 0; p0 < passes; p0 += P) {
    for (uint32_t k = t; k < P * kHistPlaceBytes / 16; k += kHistThreads)
      reinterpret_cast<uint4*>(bins)[k] = make_uint4(0, 0, 0, 0);
    __syncthreads();
    const HistDigits<K, P> h(smem_u32(bins), begin_bit + 8 * p0, end_bit);
    if constexpr (K <= 16) {
      const uint4* src = reinterpret_cast<const uint4*>(keys);
      for (uint64_t c = tid; c < chunks; c += kHistLoads * stride) {
        uint4 v[kHistLoads];
#pragma unroll
        for (int u = 0; u < kHistLoads; ++u)
          if (c + u * stride < chunks) v[u] = __ldg(src + c + u * stride);
#pragma unroll
        for (int u = 0; u < kHistLoads; ++u)
          if (c + u * stride < chunks) hist_chunk<K, P>(h, v[u]);
      }
    }
    for (uint64_t i = chunks * 16 / K + tid; i < n; i += stride) h.count(load_elem<K>(keys, i));
    __syncthreads();
    // bin b of the group, its 32 lanes' counts read in a rotated order (one bank per thread)
    for (uint32_t b = t; b < min((uint32_t)P, passes - p0) * kRadix; b += kHistThreads) {
      uint32_t sum = 0;
#pragma unroll 8
      for (uint32_t l = 0; l < 32; ++l) sum += bins[b * 32 + ((l + t) & 31)];
      if (sum) atomicAdd(&ghist[p0 * kRadix + b], sum);
    }
    __syncthreads();
  }
  __threadfence();
  __syncthreads();
  if (t == 0) s_last = atomicAdd(done_counter, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  if (t == 0) s_moving = 0;
  __syncthreads();
  // exclusive scan per pass (one warp per pass)
  for (uint32_t p = t >> 5; p < passes; p += kHistThreads / 32) {
    uint32_t run = 0, maxc = 0, cnt[kRadix / 32];
#pragma unroll
    for (int r = 0; r < kRadix / 32; ++r) cnt[r] = ld_relaxed_u32(&ghist[p * kRadix + r * 32 + lane]);
#pragma unroll
    for (int r = 0; r < kRadix / 32; ++r) {
      const uint32_t c = cnt[r], d0 = r * 32;
      maxc = max(maxc, c);
      uint32_t incl = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (uint32_t)o) incl += v;
      }
      ghist[p * kRadix + d0 + lane] = run + incl - c;
      run += __shfl_sync(0xffffffffu, incl, 31);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) maxc = max(maxc, __shfl_xor_sync(0xffffffffu, maxc, o));
    if (lane == 0 && maxc != (uint32_t)n) atomicOr(&s_moving, 1u << p);
  }
  __syncthreads();
  if (t < passes) route[t] = sort_plan(s_moving, passes, in_place, t);
}

// ------------------------------------------------------------------ digit pass
// Per tile:
//   load     one thread copies the tile into shared memory by bulk copies (elements of
//            arrays that are not 16-byte aligned, and the last elements of the last tile,
//            by plain loads), after the previous tile has been written out;
//   rank     every key takes the next count of its digit from its warp's counters by one
//            shared-memory atomic add; the keys themselves stay where they are;
//   count    per digit: the warps' counts become starts within the tile, the tile's count
//            is published for the successors' look-back;
//   order    every key's entry (digit << 16 | place in the tile) goes to its slot;
//   prefix   the digits' global offsets, by decoupled look-back;
//   write    the slots are written out in order, the keys read through their entries: one
//            run of consecutive addresses per digit.
//
// What bounds it: shared-memory wavefronts (accesses by digit hit random banks) for narrow
// keys, HBM for 16-byte ones.  The ranks were found by an atomic OR of the lane into a
// per-digit mask, two reads, a count update and a clear before (29 wavefronts per 32 keys
// in all, now about 20), and a tile was claimed one ahead of its turn: a claimed tile waits
// for its block's current one, and every later tile's look-back waits for it, so all
// blocks ran at the pace of the slowest.  A tile is now claimed while the one before it is
// written out, and what a block will claim about a round later is brought into L2 by a
// prefetch.  60M keys, us per pass, before -> now: 4 B 325 -> 220, 8 B 430 -> 270, 16 B 605 -> 385.
//
// Stability.  The order in which one atomic instruction serves the lanes that share a digit
// is not specified, so the keys of one warp step may come out exchanged.  Entries must
// ascend over the tile; the block looks at every neighbouring pair (read anyway for the
// write-out) and, should any be out of order, sorts the entries by odd-even transposition.
// Every exchange is between neighbouring slots, so that ends after a few rounds.

// The bits of element i of a raw shared-memory array from bit 32 * q + sh on, at least the
// digit's; `straddle`: the digit reaches into the next word.
template <int K>
__device__ __forceinline__ uint32_t raw_digit(const uint8_t* raw, uint32_t i, uint32_t q, uint32_t sh, bool straddle) {
  if constexpr (K == 1) {
    return raw[i] >> sh;
  } else if constexpr (K == 2) {
    return reinterpret_cast<const uint16_t*>(raw)[i] >> sh;
  } else {
    const uint32_t* p = reinterpret_cast<const uint32_t*>(raw) + i * (K / 4) + q;
    if (!straddle) return p[0] >> sh;
    return __funnelshift_r(p[0], q + 1 < K / 4 ? p[1] : 0u, sh);
  }
}

// The exclusive prefix of digit threadIdx.x over the tiles before `tile` (tile > 0): the
// words of kSortLookWindow predecessors per round trip, taken up to the first inclusive or
// missing one.
__device__ __forceinline__ uint32_t sort_lookback(const uint32_t* status, uint32_t tile, uint32_t* err) {
  uint32_t prefix = 0, spins = 0;
  int32_t base = (int32_t)tile - 1;
  while (base >= 0) {
    uint32_t w[kSortLookWindow];
    // predecessor base - r sits r * kRadix words below base's word: constant offsets from
    // one pointer (a window reaching past tile 0 reads "inclusive 0" there)
    const uint32_t* p = status + (uint64_t)base * kRadix + threadIdx.x;
    if (base >= kSortLookWindow - 1) {
#pragma unroll
      for (int r = 0; r < kSortLookWindow; ++r) w[r] = ld_relaxed_u32(p - r * kRadix);
    } else {
#pragma unroll
      for (int r = 0; r < kSortLookWindow; ++r) w[r] = r <= base ? ld_relaxed_u32(p - r * kRadix) : kSFlagInc;
    }
    // the whole window ready and none inclusive, as in most rounds but a tile's last: the
    // flags of eight words (2^30 each) add up to a multiple of 2^32
    static_assert(kSortLookWindow == 8, "see above");
    const uint32_t all = w[0] & w[1] & w[2] & w[3] & w[4] & w[5] & w[6] & w[7];
    if (all & kSFlagAgg) {
      prefix += ((w[0] + w[1]) + (w[2] + w[3])) + ((w[4] + w[5]) + (w[6] + w[7]));
      base -= kSortLookWindow;
      continue;
    }
    bool open = true, done = false;
    uint32_t used = 0;
#pragma unroll
    for (int r = 0; r < kSortLookWindow; ++r) {
      if (open && w[r] != 0) {
        prefix += w[r] & kSValMask;
        ++used;
        done = (w[r] & kSFlagInc) != 0;
      }
      open = open && w[r] != 0 && !done;
    }
    if (done) break;
    base -= (int32_t)used;
    if (used == 0) {
      if (++spins > kSpinLimit) {
        raise_error(err, kErrTimeout);
        break;
      }
      if (spins > 4) __nanosleep(spins < 16 ? 20 : 128);
    }
  }
  return prefix;
}

// Sorts the block's `count` entries in shared memory (ends with a barrier).
static __device__ __noinline__ void order_entries(uint32_t* entries, uint32_t count, uint32_t threads) {
  bool more = true;
  while (more) {
    bool moved = false;
    for (uint32_t odd = 0; odd < 2; ++odd) {
      for (uint32_t i = 2 * threadIdx.x + odd; i + 1 < count; i += 2 * threads) {
        const uint32_t x = entries[i], y = entries[i + 1];
        if (x > y) {
          entries[i] = y;
          entries[i + 1] = x;
          moved = true;
        }
      }
      __syncthreads();
    }
    more = __syncthreads_or(moved);
  }
}

__device__ __forceinline__ void prefetch_l2(const void* p, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

// All n elements of B bytes from `src` to `dst`, by the whole grid.
template <int B>
__device__ void grid_copy(uint8_t* dst, const uint8_t* src, uint64_t n) {
  const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (uint64_t)gridDim.x * blockDim.x;
  const bool vec = ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15u) == 0;
  const uint64_t chunks = vec ? n * B / 16 : 0;
  for (uint64_t c = tid; c < chunks; c += stride)
    reinterpret_cast<uint4*>(dst)[c] = reinterpret_cast<const uint4*>(src)[c];
  for (uint64_t i = chunks * 16 / B + tid; i < n; i += stride) store_elem<B>(dst, i, load_elem<B>(src, i));
}

template <int K, int V, bool SMALL>
__global__ void __launch_bounds__((SortTuning<K, V, SMALL>::THREADS), 2)
sort_pass_kernel(const __grid_constant__ SortPassArgs a) {
  using T = SortTuning<K, V, SMALL>;
  constexpr int IPT = T::IPT, WARPS = T::WARPS;
  constexpr uint32_t TILE = T::TILE, THREADS = T::THREADS;
  extern __shared__ __align__(16) uint8_t sbuf[];
  uint8_t* const raw = sbuf;
  uint8_t* const rawv = sbuf + T::KEYS;
  uint32_t* const counters = reinterpret_cast<uint32_t*>(sbuf + T::KEYS + T::VALS);
  uint32_t* const entries = counters + T::COUNTERS / 4;
  __shared__ uint32_t s_base[kRadix];   // output index of slot i = s_base[digit] + i (modulo 2^32)
  __shared__ uint32_t s_scan[kRadix / 32];
  __shared__ uint32_t s_tile;
  __shared__ __align__(8) uint64_t s_bar;
  const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
  // chained launch: what needs no other kernel's results comes before the wait
  if (t == 0) {
    mbar_init(&s_bar, 1);
    mbar_fence_init();
  }
  for (uint32_t k = t; k < T::COUNTERS / 16; k += THREADS) reinterpret_cast<uint4*>(counters)[k] = make_uint4(0, 0, 0, 0);
  grid_wait();
  grid_release();
  const uint32_t route = *a.route;
  const uint32_t n = (uint32_t)a.n;   // below 2^30
  const uint32_t num_tiles = (n + TILE - 1) / TILE;
  const uint32_t q = a.shift >> 5, sh = a.shift & 31, mask = a.mask;
  const bool straddle = sh + (32 - __clz(mask)) > 32;
  uint32_t* const wcount = counters + warp * kRadix;
  const uint32_t gexcl = t < kRadix ? a.gexcl[t] : 0u;
  // a tile is claimed while the route is on its way; a pass that turns out not to sort has no
  // use for its tile numbers
  if (t == 0) s_tile = atomicAdd(a.tile_counter, 1u);
  __syncthreads();
  // the buffers are looked up in the parameters where they are used, which leaves no register
  // to their addresses
  const uint32_t from = route & 3, to = route >> 2 & 3;
  if (!(route & kRouteSort)) {
    if (route & kRouteCopy) {
      grid_copy<K>(a.keys[to], a.keys[from], a.n);
      if constexpr (V > 0) grid_copy<V>(a.vals[to], a.vals[from], a.n);
    }
    return;
  }
  const bool bulk =
      ((reinterpret_cast<uintptr_t>(a.keys[from]) | (V ? reinterpret_cast<uintptr_t>(a.vals[from]) : 0u)) & 15u) == 0;

  auto load = [&](uint32_t tile) {
    const uint32_t base = tile * TILE, cnt = min(TILE, n - base);
    uint32_t k0 = 0, v0 = 0;   // elements the bulk copies bring
    if (bulk) {
      const uint32_t kb = cnt * K & ~15u, vb = cnt * V & ~15u;
      if (t == 0) {
        fence_proxy_async_smem();   // the buffers were read and written by plain accesses
        mbar_arrive_tx(&s_bar, kb + vb);
        if (kb) bulk_copy_g2s(raw, a.keys[from] + (uint64_t)base * K, kb, &s_bar);
        if (vb) bulk_copy_g2s(rawv, a.vals[from] + (uint64_t)base * V, vb, &s_bar);
      }
      k0 = kb / K;
      if constexpr (V > 0) v0 = vb / V;
    }
    for (uint32_t i = k0 + t; i < cnt; i += THREADS) store_elem<K>(raw, i, load_elem<K>(a.keys[from], (uint64_t)base + i));
    if constexpr (V > 0)
      for (uint32_t i = v0 + t; i < cnt; i += THREADS)
        store_elem<V>(rawv, i, load_elem<V>(a.vals[from], (uint64_t)base + i));
  };

  uint32_t tile = s_tile;
  if (tile < num_tiles) load(tile);
  for (uint32_t parity = 0; tile < num_tiles; parity ^= 1u) {
    const uint32_t tcount = min(TILE, n - tile * TILE);
    const bool full = tcount == TILE;
    if (!full || !bulk) __syncthreads();   // elements brought by plain loads
    if (bulk && !mbar_wait(&s_bar, parity)) {
      raise_error(a.err, kErrTimeout);
      mbar_wait(&s_bar, parity);   // the copy is this block's own: no exit before it lands
    }
    // warp w owns elements [w * 32 * IPT, (w + 1) * 32 * IPT) of the tile, element j of lane l
    // at j * 32 + l; the first nv of a lane's elements exist
    const uint32_t first = warp * 32 * IPT + lane;
    const uint32_t nv = first >= tcount ? 0u : (tcount - first + 31) / 32;
    uint32_t key[IPT];   // digit << 16 | rank among the warp's keys of that digit
#pragma unroll
    for (int j = 0; j < IPT; ++j) key[j] = raw_digit<K>(raw, first + j * 32, q, sh, straddle) & mask;
    if (full) {
#pragma unroll
      for (int j = 0; j < IPT; ++j) key[j] = key[j] << 16 | atomicAdd(&wcount[key[j]], 1u);
    } else {
#pragma unroll
      for (int j = 0; j < IPT; ++j)
        if ((uint32_t)j < nv) key[j] = key[j] << 16 | atomicAdd(&wcount[key[j]], 1u);
    }
    __syncthreads();
    const uint32_t ahead = tile + gridDim.x;   // claimed by some block about a round from now
    if (bulk && t == THREADS - 1 && ahead < num_tiles) {
      const uint32_t ab = ahead * TILE, ac = min(TILE, n - ab), kb = ac * K & ~15u, vb = ac * V & ~15u;
      if (kb) prefetch_l2(a.keys[from] + (uint64_t)ab * K, kb);
      if (vb) prefetch_l2(a.vals[from] + (uint64_t)ab * V, vb);
    }
    // thread t < 256, digit t: the warps' counts as exclusive sums, the tile's count
    // (published at once), the tile-local start
    uint32_t before[WARPS], count = 0, start = 0;
    uint32_t* const status = a.status + (uint64_t)tile * kRadix + t;
    if (t < kRadix) {
#pragma unroll
      for (int w = 0; w < WARPS; ++w) before[w] = counters[w * kRadix + t];
#pragma unroll
      for (int w = 0; w < WARPS; ++w) {
        const uint32_t c = before[w];
        before[w] = count;
        count += c;
      }
      st_relaxed_u32(status, tile == 0 ? kSFlagInc | (gexcl + count) : kSFlagAgg | count);
      uint32_t incl = count;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (uint32_t)o) incl += v;
      }
      if (lane == 31) s_scan[warp] = incl;
      start = incl - count;
    }
    __syncthreads();
    if (t < kRadix) {
#pragma unroll
      for (uint32_t w = 0; w < kRadix / 32; ++w) start += w < warp ? s_scan[w] : 0u;
#pragma unroll
      for (int w = 0; w < WARPS; ++w) counters[w * kRadix + t] = before[w] + start;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < IPT; ++j)
      if (full || (uint32_t)j < nv)
        entries[wcount[key[j] >> 16] + (key[j] & 0xffffu)] = (key[j] & 0xffff0000u) | (first + j * 32);
    __syncthreads();
    // the look-back comes last before the write-out, which gives the predecessors that long
    for (uint32_t k = t; k < T::COUNTERS / 16; k += THREADS)
      reinterpret_cast<uint4*>(counters)[k] = make_uint4(0, 0, 0, 0);
    uint32_t entry[IPT];
    bool disorder = false;
#pragma unroll
    for (int j = 0; j < IPT; ++j) {
      const uint32_t i = j * THREADS + t;
      entry[j] = entries[i];
      disorder = disorder || (i > 0 && i < tcount && entries[i - 1] > entry[j]);
    }
    if (t < kRadix) {
      uint32_t prefix = gexcl;
      if (tile > 0) {
        prefix = sort_lookback(a.status, tile, a.err);
        st_relaxed_u32(status, kSFlagInc | ((prefix + count) & kSValMask));
      }
      s_base[t] = prefix - start;
    }
    if (__syncthreads_or(disorder)) {
      order_entries(entries, tcount, THREADS);
#pragma unroll
      for (int j = 0; j < IPT; ++j) entry[j] = entries[j * THREADS + t];
    }
    if (t == 0) s_tile = atomicAdd(a.tile_counter, 1u);   // the round trip hides behind the write-out
#pragma unroll
    for (int j = 0; j < IPT; ++j) {
      const uint32_t i = j * THREADS + t, li = entry[j] & 0xffffu;
      if (full || i < tcount) {
        const uint32_t pos = s_base[entry[j] >> 16] + i;
        if (pos < n) {
          store_elem<K>(a.keys[to], pos, load_elem<K>(raw, li));
          if constexpr (V > 0) store_elem<V>(a.vals[to], pos, load_elem<V>(rawv, li));
        }
      }
    }
    __syncthreads();
    tile = s_tile;
    if (tile < num_tiles) load(tile);
  }
}

}  // namespace rfx
