// reduce_f64_abi.cu -- reduce-by-key over double values: the reference's total_*_double
// (thrust::reduce_by_key with plus<double>), min_32_double (minimum<double>) and the
// scalar total_double / max_double / count of Reduce.cu:742-1536.
//
// Sums are exact, then rounded once (round to nearest, ties to even), in up to three passes.
//   * The first keeps a run's sum as an unevaluated pair of doubles hi + lo.  Every addition
//     is an error-free transformation (Knuth's TwoSum, both parts): the error of the high
//     addition goes to the low part, and an error of the low addition raises a flag.  While
//     the flag stays down hi + lo is the exact sum whatever the order of the additions, and
//     one rounding of hi + lo finishes it.  This holds for values whose bits span about 100
//     binary places, such as amounts of money, with or without infinities and NaNs.
//   * Where the flag went up (a wider span, a finite value from 2^1000 on), a second pass sums
//     the runs that lost bits again, in integers: every double is a 53-bit integer times a
//     power of two, so a run's sum is accumulated as a two's-complement integer in units of 2^L
//     over W 64-bit limbs (add with carry).  W = 3 limbs with L set from the largest exponent in
//     the units that are summed again: exact for every value within 2^107 of the largest, with
//     room for 2^30 terms.
//   * A value below that window with bits that would be lost raises a flag too, and a third
//     pass with W = 34 limbs and L = -1074, which covers every finite double, does the same.
// The kernels of the later passes are always enqueued and return at once unless their flag is
// set, so no host round trip is needed.  Specials follow IEEE addition: NaN if any NaN or both
// infinities, else the infinity, and an exact zero is -0 only when every term is -0.
//
// The minimum follows the reference's fold acc = (acc < v ? acc : v) exactly: a later
// element replaces an equal one (so -0 / +0 ties go to the later), a NaN sets the
// accumulator and the next element replaces it.  That fold is associative as a
// combination of run summaries, so the parallel result equals the sequential one bit for
// bit.
//
// Structure: units of up to 4096 elements, one warp per unit.  A pre-pass counts each unit's
// run heads, and its last block scans the counts into each unit's first run index; the main
// pass folds a unit in registers and warp shuffles, writes every run that starts and ends
// inside it at its final index, and leaves the partial before its first head and the partial
// from its last head for the fix-up, which closes the runs crossing units.
#include <algorithm>
#include <cstring>

#include "host_common.h"
#include "rfx_device.cuh"

namespace rfx {
namespace {

constexpr int kNarrowLimbs = 3;   // 192 bits: every value within 2^107 of the largest
constexpr int kWideLimbs = 34;    // 2176 bits: every finite double
constexpr int kWideL = -1074;

enum : uint32_t { kSumNaN = 1, kSumPosInf = 2, kSumNegInf = 4, kSumNotNegZero = 8 };

// ------------------------------------------------------------------ exact sum
// W 64-bit limbs holding a two's-complement integer (limb 0 lowest) in units of 2^L.
// Additions are exact modulo 2^(64W); the true sum stays inside the signed range by the
// choice of L, so the result is exact and independent of the order of the additions.
// TENTATIVE: the pass finds out where it loses bits; AGAIN: the pass does those units over.
template <int W>
struct SumOp {
  static constexpr bool TENTATIVE = false, AGAIN = true;
  static constexpr bool COMMUTES = W == 3;   // (the 34 limbs are not worth another copy)
  static constexpr int BLOCKS = W == 3 ? 2 : 1;   // of 256 threads per SM: the limbs live in registers
  struct P {
    unsigned long long l[W];
    uint32_t flags;
    uint32_t pad;
  };
  __device__ __forceinline__ static P identity() {
    P p;
#pragma unroll
    for (int k = 0; k < W; ++k) p.l[k] = 0;
    p.flags = 0;
    p.pad = 0;
    return p;
  }
  // acc += a (neg: acc -= a) where a has limbs lo at q, hi at q + 1.
  __device__ __forceinline__ static void accumulate(unsigned long long* acc, int q, unsigned long long lo,
                                                    unsigned long long hi, bool neg) {
    if constexpr (W == 3) {
      const unsigned long long a0 = q == 0 ? lo : 0ull, a1 = q == 0 ? hi : lo, a2 = q == 0 ? 0ull : hi;
      if (!neg)
        asm("add.cc.u64 %0, %0, %3;\n\taddc.cc.u64 %1, %1, %4;\n\taddc.u64 %2, %2, %5;"
            : "+l"(acc[0]), "+l"(acc[1]), "+l"(acc[2])
            : "l"(a0), "l"(a1), "l"(a2));
      else
        asm("sub.cc.u64 %0, %0, %3;\n\tsubc.cc.u64 %1, %1, %4;\n\tsubc.u64 %2, %2, %5;"
            : "+l"(acc[0]), "+l"(acc[1]), "+l"(acc[2])
            : "l"(a0), "l"(a1), "l"(a2));
    } else {
      unsigned long long c = 0;
      for (int k = q; k < W; ++k) {
        const unsigned long long a = k == q ? lo : k == q + 1 ? hi : 0ull;
        if (!neg) {
          const unsigned __int128 t = (unsigned __int128)acc[k] + a + c;
          acc[k] = (unsigned long long)t;
          c = (unsigned long long)(t >> 64);
        } else {
          const unsigned __int128 t = (unsigned __int128)acc[k] - a - c;
          acc[k] = (unsigned long long)t;
          c = (unsigned long long)(t >> 64) ? 1ull : 0ull;
        }
        if (k > q && c == 0) break;
      }
    }
  }
  __device__ __forceinline__ static void add(P& p, double x, int L, uint32_t* inexact, bool&) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    const uint32_t eb = (uint32_t)(b >> 52) & 0x7ffu;
    const unsigned long long frac = b & ((1ull << 52) - 1);
    const bool neg = (b >> 63) != 0;
    if (b != 0x8000000000000000ull) p.flags |= kSumNotNegZero;
    if (eb == 0x7ffu) {
      p.flags |= frac ? kSumNaN : (neg ? kSumNegInf : kSumPosInf);
      return;
    }
    if (eb == 0 && frac == 0) return;
    unsigned long long m = eb ? (frac | (1ull << 52)) : frac;
    int s = (int)(eb ? eb : 1u) - 1075 - L;  // the mantissa's LSB in units of 2^L
    if (s < 0) {
      const int r = -s;
      if (r >= 64 ? m != 0 : (m & ((1ull << r) - 1)) != 0) atomicOr(inexact, 1u);
      m = r >= 64 ? 0 : m >> r;
      s = 0;
    }
    const int q = s >> 6, o = s & 63;
    if (q + 1 >= W) {  // above the window: only when L was not set from this input's maximum
      atomicOr(inexact, 1u);
      return;
    }
    const unsigned long long lo = m << o;
    const unsigned long long hi = o ? m >> (64 - o) : 0ull;
    accumulate(p.l, q, lo, hi, neg);
  }
  __device__ __forceinline__ static P combine(const P& a, const P& b, bool&) {
    P r;
    if constexpr (W == 3) {
      r.l[0] = a.l[0];
      r.l[1] = a.l[1];
      r.l[2] = a.l[2];
      asm("add.cc.u64 %0, %0, %3;\n\taddc.cc.u64 %1, %1, %4;\n\taddc.u64 %2, %2, %5;"
          : "+l"(r.l[0]), "+l"(r.l[1]), "+l"(r.l[2])
          : "l"(b.l[0]), "l"(b.l[1]), "l"(b.l[2]));
    } else {
      unsigned long long c = 0;
      for (int k = 0; k < W; ++k) {
        const unsigned __int128 t = (unsigned __int128)a.l[k] + b.l[k] + c;
        r.l[k] = (unsigned long long)t;
        c = (unsigned long long)(t >> 64);
      }
    }
    r.flags = a.flags | b.flags;
    r.pad = 0;
    return r;
  }
  // Bits [pos, pos + len) of the limbs (len <= 64, pos >= 0).
  __device__ static unsigned long long bits_at(const unsigned long long* l, int pos, int len) {
    if (len <= 0) return 0;
    const int k = pos >> 6, o = pos & 63;
    const unsigned long long d0 = k < W ? l[k] : 0ull, d1 = k + 1 < W ? l[k + 1] : 0ull;
    unsigned long long v = (d0 >> o) | (o ? d1 << (64 - o) : 0ull);
    if (len < 64) v &= (1ull << len) - 1;
    return v;
  }
  __device__ static bool any_below(const unsigned long long* l, int pos) {
    const int k = pos >> 6;
    for (int i = 0; i < k && i < W; ++i)
      if (l[i]) return true;
    if (k < W && (pos & 63) && (l[k] & ((1ull << (pos & 63)) - 1))) return true;
    return false;
  }
  // The correctly rounded double of the accumulated value, as bits.
  __device__ static unsigned long long finalize(const P& p, int L) {
    if ((p.flags & kSumNaN) || ((p.flags & kSumPosInf) && (p.flags & kSumNegInf))) return 0x7ff8000000000000ull;
    if (p.flags & kSumPosInf) return 0x7ff0000000000000ull;
    if (p.flags & kSumNegInf) return 0xfff0000000000000ull;
    unsigned long long r[W];
#pragma unroll
    for (int k = 0; k < W; ++k) r[k] = p.l[k];
    const bool neg = (r[W - 1] >> 63) != 0;
    if (neg) {  // magnitude = two's complement negation
      unsigned long long c = 1;
#pragma unroll
      for (int k = 0; k < W; ++k) {
        const unsigned long long t = ~r[k] + c;
        c = (c && t == 0) ? 1ull : 0ull;
        r[k] = t;
      }
    }
    int top = -1;
    for (int k = W - 1; k >= 0; --k)
      if (r[k]) {
        top = 64 * k + 63 - __clzll(r[k]);
        break;
      }
    if (top < 0) return (p.flags & kSumNotNegZero) ? 0ull : 0x8000000000000000ull;
    const unsigned long long sgn = neg ? 0x8000000000000000ull : 0ull;
    int e = top + L;  // the value lies in [2^e, 2^(e+1))
    if (e > 1023) return sgn | 0x7ff0000000000000ull;
    const bool normal = e >= -1022;
    const int lsb = normal ? top - 52 : -1074 - L;  // bit that becomes the result's LSB
    unsigned long long mant;
    if (lsb <= 0) {
      mant = bits_at(r, 0, top + 1) << (-lsb);
    } else {
      mant = bits_at(r, lsb, top - lsb + 1);
      const bool round = (bits_at(r, lsb - 1, 1) & 1ull) != 0;
      const bool sticky = any_below(r, lsb - 1);
      if (round && (sticky || (mant & 1ull))) ++mant;
    }
    if (normal) {
      if (mant == (1ull << 53)) {
        mant >>= 1;
        if (++e > 1023) return sgn | 0x7ff0000000000000ull;
      }
      return sgn | ((unsigned long long)(e + 1023) << 52) | (mant & ((1ull << 52) - 1));
    }
    return sgn | mant;  // subnormal; 2^52 after rounding is the smallest normal
  }
};

// ------------------------------------------------------------------ exact sum in two doubles
// The sum is hi + lo exactly as long as no flag (`bad`) went up.  Finite values from 2^1000 on
// raise it by themselves: no sum of 2^30 smaller ones overflows, so a high part that is not
// finite comes from an infinity or a NaN among the terms, and is what IEEE addition makes of
// them.  The errors are NaN from there on and say nothing.
struct PairOp {
  static constexpr int BLOCKS = 4;
  static constexpr bool TENTATIVE = true, AGAIN = false;
  static constexpr bool COMMUTES = true;
  struct P {
    double hi, lo;
  };
  __device__ __forceinline__ static P identity() { return P{-0.0, 0.0}; }   // -0 + x is x for every x
  // a + b = s + e exactly (Knuth's TwoSum) when s is finite.
  __device__ __forceinline__ static double two_sum(double a, double b, double& e) {
    const double s = __dadd_rn(a, b);
    const double bb = __dadd_rn(s, -a);
    e = __dadd_rn(__dadd_rn(a, -__dadd_rn(s, -bb)), __dadd_rn(b, -bb));
    return s;
  }
  __device__ __forceinline__ static bool lost(double e) { return fabs(e) > 0.0; }   // not for a NaN
  // Twice the high word without the sign, infinities and NaNs wrapped round to the low end.
  __device__ __forceinline__ static bool large(double x) {
    constexpr uint32_t kFrom = ((1000u + 1023u) << 21) + (1u << 21);
    return ((uint32_t)__double2hiint(x) << 1) + (1u << 21) >= kFrom;
  }
  __device__ __forceinline__ static void add(P& p, double x, int, uint32_t*, bool& bad) {
    double e, e2;
    p.hi = two_sum(p.hi, x, e);
    p.lo = two_sum(p.lo, e, e2);
    bad = bad || lost(e2);
  }
  __device__ __forceinline__ static P combine(const P& a, const P& b, bool& bad) {
    double e, e2, e3, r;
    const double s = two_sum(a.hi, b.hi, e);
    const double l = two_sum(a.lo, b.lo, e2);
    const double t = two_sum(l, e, e3);
    bad = bad || lost(e2) || lost(e3);
    const double h = two_sum(s, t, r);   // keeps the low part below the high one's last place
    return fabs(t) > 0.0 ? P{h, r} : P{s, 0.0};   // (s + 0 would lose the sign of a zero)
  }
  __device__ __forceinline__ static unsigned long long finalize(const P& p, int) {
    if (!isfinite(p.hi)) return p.hi != p.hi ? 0x7ff8000000000000ull : (unsigned long long)__double_as_longlong(p.hi);
    return (unsigned long long)__double_as_longlong(p.lo == 0.0 ? p.hi : __dadd_rn(p.hi, p.lo));
  }
};

// ------------------------------------------------------------------ minimum (the fold)
struct MinOp {
  static constexpr int BLOCKS = 4;
  static constexpr bool TENTATIVE = false, AGAIN = false;
  static constexpr bool COMMUTES = false;
  struct P {
    unsigned long long v;  // bits of the fold value (a NaN while pending)
    uint32_t any;          // an element after the last NaN was folded
    uint32_t nan;          // a NaN occurs in the summarised range
  };
  __device__ __forceinline__ static P identity() { return P{0ull, 0u, 0u}; }
  __device__ __forceinline__ static void add(P& p, double x, int, uint32_t*, bool&) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    if (x != x) {
      p = P{b, 0u, 1u};
    } else if (!p.any) {
      p.v = b;
      p.any = 1u;
    } else {
      const double a = __longlong_as_double((long long)p.v);
      p.v = a < x ? p.v : b;
    }
  }
  // a is the earlier range, b the later one.
  __device__ __forceinline__ static P combine(const P& a, const P& b, bool&) {
    if (b.nan) return b;
    if (!b.any) return a;
    if (!a.any) return P{b.v, 1u, a.nan};
    const double x = __longlong_as_double((long long)a.v), y = __longlong_as_double((long long)b.v);
    return P{x < y ? a.v : b.v, 1u, a.nan};
  }
  __device__ static unsigned long long finalize(const P& p, int) { return p.v; }
};

__device__ __forceinline__ uint32_t ld_relaxed_u32(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// ------------------------------------------------------------------ keys
struct Key {
  unsigned long long lo, hi;
};

template <int KB>
__device__ __forceinline__ Key load_key(const uint8_t* keys, uint32_t i) {
  if constexpr (KB == 0) return Key{0ull, 0ull};
  if constexpr (KB == 1) return Key{keys[i], 0ull};
  if constexpr (KB == 2) return Key{reinterpret_cast<const uint16_t*>(keys)[i], 0ull};
  if constexpr (KB == 4) return Key{reinterpret_cast<const uint32_t*>(keys)[i], 0ull};
  if constexpr (KB == 8) return Key{reinterpret_cast<const unsigned long long*>(keys)[i], 0ull};
  if constexpr (KB == 16) {
    const ulonglong2 v = reinterpret_cast<const ulonglong2*>(keys)[i];
    return Key{v.x, v.y};
  }
  return Key{0ull, 0ull};
}

template <int KB>
__device__ __forceinline__ void store_key(uint8_t* out, uint32_t r, const Key& k) {
  if constexpr (KB == 1) out[r] = (uint8_t)k.lo;
  if constexpr (KB == 2) reinterpret_cast<uint16_t*>(out)[r] = (uint16_t)k.lo;
  if constexpr (KB == 4) reinterpret_cast<uint32_t*>(out)[r] = (uint32_t)k.lo;
  if constexpr (KB == 8) reinterpret_cast<unsigned long long*>(out)[r] = k.lo;
  if constexpr (KB == 16) reinterpret_cast<ulonglong2*>(out)[r] = make_ulonglong2(k.lo, k.hi);
}

// ------------------------------------------------------------------ shuffles
template <typename T>
__device__ __forceinline__ T shfl_up_any(const T& x, int delta) {
  constexpr int W = (int)((sizeof(T) + 3) / 4);
  uint32_t w[W];
  memcpy(w, &x, sizeof(T));
#pragma unroll
  for (int i = 0; i < W; ++i) w[i] = __shfl_up_sync(0xffffffffu, w[i], delta);
  T r;
  memcpy(&r, w, sizeof(T));
  return r;
}

template <typename T>
__device__ __forceinline__ T shfl_down_any(const T& x, int delta) {
  constexpr int W = (int)((sizeof(T) + 3) / 4);
  uint32_t w[W];
  memcpy(w, &x, sizeof(T));
#pragma unroll
  for (int i = 0; i < W; ++i) w[i] = __shfl_down_sync(0xffffffffu, w[i], delta);
  T r;
  memcpy(&r, w, sizeof(T));
  return r;
}

template <typename T>
__device__ __forceinline__ T shfl_any(const T& x, int src) {
  constexpr int W = (int)((sizeof(T) + 3) / 4);
  uint32_t w[W];
  memcpy(w, &x, sizeof(T));
#pragma unroll
  for (int i = 0; i < W; ++i) w[i] = __shfl_sync(0xffffffffu, w[i], src);
  T r;
  memcpy(&r, w, sizeof(T));
  return r;
}

// ------------------------------------------------------------------ kernels
struct F64Args {
  const uint8_t* keys;
  const double* vals;
  uint64_t n;
  uint32_t unit;        // elements per unit, a multiple of kF64Step
  const unsigned long long* emit;  // if set, out key of a run = emit[head] (8 bytes)
  uint8_t* out_keys;
  double* out_vals;
  uint64_t* d_groups;
  uint32_t* done;       // blocks of the count that have finished
  uint32_t* heads;      // run heads per unit
  uint32_t* base;       // index of the unit's first run (heads before it)
  void* first;          // Op::P per unit: before its first head (the whole unit if it has none)
  void* last;           // Op::P per unit: from its last head
  uint32_t* need;       // per unit: what the integer passes do over (kLossy, kInvolved, kReclose)
  int* emax;            // max biased exponent of the finite values (the 3-limb pass's window)
  int fixed_L;          // used when emax is null
  uint32_t* inexact;    // raised when the pass was not exact everywhere
  const uint32_t* gate; // if set, the kernels do nothing unless *gate != 0
  uint32_t* err;
};

// Why a unit is summed again in integers: bits were lost in it; a run that lost bits goes through
// it; that run ends at its first head (or with it).
enum : uint32_t { kLossy = 1, kInvolved = 2, kReclose = 4 };

__device__ __forceinline__ bool gated_off(const F64Args& a) { return a.gate && *a.gate == 0u; }

__device__ __forceinline__ int window_L(const F64Args& a) {
  if (!a.emax) return a.fixed_L;
  const int e = *a.emax;
  return (e > 1 ? e : 1) - 1182;
}

constexpr int kF64WarpIPT = 8;
constexpr int kF64Step = 32 * kF64WarpIPT;   // elements a warp folds at a time
constexpr int kF64UnitMost = 4096;

// Eight consecutive keys from element `first` (a multiple of 8) of a 16-byte aligned array.
template <int KB>
__device__ __forceinline__ void load_keys8(const uint8_t* keys, uint32_t first, Key (&k)[8]) {
  const uint8_t* p = keys + (size_t)first * KB;
  if constexpr (KB == 1) {
    const uint2 v = *reinterpret_cast<const uint2*>(p);
#pragma unroll
    for (int j = 0; j < 8; ++j) k[j] = Key{((j < 4 ? v.x : v.y) >> (8 * (j & 3))) & 0xffu, 0ull};
  } else if constexpr (KB == 2) {
    const uint4 v = *reinterpret_cast<const uint4*>(p);
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 8; ++j) k[j] = Key{(w[j >> 1] >> (16 * (j & 1))) & 0xffffu, 0ull};
  } else if constexpr (KB == 4) {
    const uint4 a = reinterpret_cast<const uint4*>(p)[0], b = reinterpret_cast<const uint4*>(p)[1];
    const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
    for (int j = 0; j < 8; ++j) k[j] = Key{w[j], 0ull};
  } else if constexpr (KB == 8) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const ulonglong2 v = reinterpret_cast<const ulonglong2*>(p)[j];
      k[2 * j] = Key{v.x, 0ull};
      k[2 * j + 1] = Key{v.y, 0ull};
    }
  } else if constexpr (KB == 16) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const ulonglong2 v = reinterpret_cast<const ulonglong2*>(p)[j];
      k[j] = Key{v.x, v.y};
    }
  }
}

// Keys first .. first + 7 of the elements before `end`; vec: the array is 16-byte aligned.
template <int KB>
__device__ __forceinline__ void load_keys(const uint8_t* keys, uint32_t first, uint32_t end, bool vec, Key (&k)[8]) {
  if constexpr (KB == 0) {
#pragma unroll
    for (int j = 0; j < 8; ++j) k[j] = Key{0ull, 0ull};
  } else if (vec && first + 8 <= end) {
    load_keys8<KB>(keys, first, k);
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j) k[j] = first + j < end ? load_key<KB>(keys, first + j) : Key{0ull, 0ull};
  }
}

// The heads among a lane's keys (bit j: element first + j starts a run).
template <int KB>
__device__ __forceinline__ uint32_t head_bits(const F64Args& a, const Key (&k)[8], uint32_t first, uint32_t end) {
  uint32_t hm = first == 0 && end > 0 ? 1u : 0u;
  if constexpr (KB > 0) {
    const uint32_t lane = threadIdx.x & 31;
    Key pk;
    pk.lo = __shfl_up_sync(0xffffffffu, k[7].lo, 1);
    pk.hi = KB == 16 ? __shfl_up_sync(0xffffffffu, k[7].hi, 1) : 0ull;
    if (lane == 0 && first > 0 && first < end) pk = load_key<KB>(a.keys, first - 1);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const Key q = j ? k[j - 1] : pk;
      const bool h = first + j > 0 && first + j < end && (k[j].lo != q.lo || k[j].hi != q.hi);
      hm |= (uint32_t)h << j;
    }
  }
  return hm;
}

// Run heads per unit, one warp per unit; the last block to finish turns the counts into each
// unit's first run index and writes the number of runs.
template <int KB>
__global__ void __launch_bounds__(256) f64_unit_count(F64Args a, uint64_t units) {
  __shared__ uint64_t s_warp[8];
  __shared__ bool s_last;
  const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const bool vec = (reinterpret_cast<uintptr_t>(a.keys) & 15u) == 0;
  grid_wait();   // chained launch
  grid_release();
  const uint64_t nw = (uint64_t)gridDim.x * 8;
  for (uint64_t u = (uint64_t)blockIdx.x * 8 + warp; u < units; u += nw) {
    const uint32_t e0 = (uint32_t)u * a.unit, e1 = min(e0 + a.unit, (uint32_t)a.n);
    uint32_t c = 0;
#pragma unroll 4
    for (uint32_t tb = e0; tb < e1; tb += kF64Step) {
      const uint32_t first = tb + 8 * lane;
      Key k[8];
      load_keys<KB>(a.keys, first, e1, vec, k);
      c += (uint32_t)__popc(head_bits<KB>(a, k, first, e1));
    }
    c = __reduce_add_sync(0xffffffffu, c);
    if (lane == 0) {
      a.heads[u] = c;
      a.need[u] = 0;
    }
  }
  __threadfence();
  __syncthreads();
  if (t == 0) s_last = atomicAdd(a.done, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  // consecutive counts per thread, 8 at a time
  uint64_t carry = 0;
  for (uint64_t b = 0; b < units; b += 8 * 256) {
    uint32_t c[8], sum = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const uint64_t u = b + 8ull * t + j;
      c[j] = u < units ? ld_relaxed_u32(a.heads + u) : 0u;
      sum += c[j];
    }
    uint64_t inc = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint64_t y = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= (uint32_t)o) inc += y;
    }
    if (lane == 31) s_warp[warp] = inc;
    __syncthreads();
    uint64_t run = carry + inc - sum;
#pragma unroll
    for (uint32_t w = 0; w < 8; ++w) {
      run += w < warp ? s_warp[w] : 0ull;
      carry += s_warp[w];
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const uint64_t u = b + 8ull * t + j;
      if (u < units) a.base[u] = (uint32_t)run;
      run += c[j];
    }
    __syncthreads();
  }
  if (t == 0) *a.d_groups = carry;
}

// The largest biased exponent of the finite values of the units that are summed again (the 3-limb
// pass's window), one warp per unit, 16 bytes per load and four loads in flight.
__global__ void __launch_bounds__(256) f64_emax(F64Args a, uint64_t units) {
  grid_wait();   // chained launch
  grid_release();
  if (gated_off(a)) return;
  const uint32_t lane = threadIdx.x & 31;
  const bool vec = (reinterpret_cast<uintptr_t>(a.vals) & 15u) == 0;
  int m = 1;
  auto take = [&](double x) {
    const int eb = (__double2hiint(x) >> 20) & 0x7ff;
    if (eb != 0x7ff && eb > m) m = eb;
  };
  for (uint32_t u = blockIdx.x * 8 + (threadIdx.x >> 5); u < units; u += gridDim.x * 8) {
    if (!a.need[u]) continue;
    const uint32_t e0 = u * a.unit, e1 = min(e0 + a.unit, (uint32_t)a.n);
    uint32_t i = e0;
    if (vec) {
      for (; i + kF64Step <= e1; i += kF64Step) {
        double2 v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = reinterpret_cast<const double2*>(a.vals + i)[32 * k + lane];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          take(v[k].x);
          take(v[k].y);
        }
      }
    }
    for (i += lane; i < e1; i += 32) take(a.vals[i]);
  }
  m = __reduce_max_sync(0xffffffffu, m);
  if (lane == 0) atomicMax(a.emax, m);
}

// The main pass: a warp folds its unit 256 elements at a time, 8 consecutive ones per lane
// (16-byte loads).  A lane folds its elements, writing the runs that start and end among
// them; a segmented warp scan gives every lane what is open before it.  Bound by the latency
// of a step's chain (loads, fold, scan), so by the warps resident: 19.3M elements, 256K runs,
// SUM with 32 warps per SM (64 registers, 20 bytes of spills) 91 us, MIN 67, the 3-limb integers
// with 16 warps 152.  An earlier form of the pair took 87 with 32 warps, 105 with 24, 106 with 16
// and the next step's loads in flight.
//
// A unit in which an addition of the pair lost bits is left at the next step and marked; the
// integer passes do the marked units over.  us a call with the integer pass alone / now: all units
// done over (values over 80 binary places) 319 / 262, a few (one value that does not fit) 322 / 247,
// of 60M elements and 1M runs 690 / 462, one run over 19.3M with one such value 278 / 248 to 284.
template <int KB, class Op>
__global__ void __launch_bounds__(256, Op::BLOCKS) f64_unit_kernel(F64Args a, uint64_t units) {
  grid_wait();   // chained launch
  grid_release();
  if (gated_off(a)) return;
  using P = typename Op::P;
  constexpr int V = kF64WarpIPT;
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t gw = blockIdx.x * 8 + (threadIdx.x >> 5);
  const uint32_t nw = gridDim.x * 8;
  const int L = window_L(a);
  const bool vk = (reinterpret_cast<uintptr_t>(a.keys) & 15u) == 0;
  const bool vv = (reinterpret_cast<uintptr_t>(a.vals) & 15u) == 0;
  // one run over everything: bits lost in any unit have all done over, so each warp looks whether
  // another has lost some (the flag is asked for a step before it is used)
  const bool one_run = Op::TENTATIVE && (KB == 0 || *a.d_groups == 1);
  bool bad = false, raised = false;
  for (uint32_t u = gw; u < units; u += nw) {
    if (Op::AGAIN && !a.need[u]) continue;
    const uint32_t e0 = u * a.unit, e1 = min(e0 + a.unit, (uint32_t)a.n);   // below 2^30
    uint32_t run_base = a.base[u];   // index of the next head's run
    P carry = Op::identity();
    bool carry_head = false;
    // sums of steps without a head stay in their lanes until a head or the unit's end comes
    P held = Op::identity();
    bool holding = false;
    auto release = [&] {
      if (Op::COMMUTES && holding) {
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const P y = shfl_down_any(held, o);
          if (lane + o < 32) held = Op::combine(held, y, bad);
        }
        carry = Op::combine(carry, shfl_any(held, 0), bad);
        held = Op::identity();
        holding = false;
      }
    };
    for (uint32_t tb = e0; tb < e1; tb += kF64Step) {
      if constexpr (Op::TENTATIVE) {
        if (one_run && (tb / kF64Step & 3) == 3) bad = bad || raised;
        if (__any_sync(0xffffffffu, bad)) break;   // the unit is done over
        if (one_run && (tb / kF64Step & 3) == 2) raised = ld_relaxed_u32(a.inexact) != 0;
      }
      const uint32_t first = tb + lane * V;
      Key keys[V];
      double vals[V];
      load_keys<KB>(a.keys, first, e1, vk, keys);
      if (vv && first + V <= e1) {
#pragma unroll
        for (int j = 0; j < V / 2; ++j) {
          const double2 v = reinterpret_cast<const double2*>(a.vals + first)[j];
          vals[2 * j] = v.x;
          vals[2 * j + 1] = v.y;
        }
      } else {
#pragma unroll
        for (int j = 0; j < V; ++j) vals[j] = first + j < e1 ? a.vals[first + j] : 0.0;
      }
      if constexpr (Op::TENTATIVE) {
#pragma unroll
        for (int j = 0; j < V; ++j) bad = bad || Op::large(vals[j]);
      }
      const uint32_t hm = head_bits<KB>(a, keys, first, e1);
      if (Op::COMMUTES && !__any_sync(0xffffffffu, hm != 0)) {
#pragma unroll
        for (int j = 0; j < V; ++j)
          if (first + j < e1) Op::add(held, vals[j], L, a.inexact, bad);
        holding = true;
        continue;
      }
      release();
      // run index of this lane's first head
      const uint32_t cnt = (uint32_t)__popc(hm);
      uint32_t inc = cnt;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= (uint32_t)o) inc += y;
      }
      const uint32_t lane_run = run_base + inc - cnt;
      // keys at heads; runs that end inside this lane
      P cur = Op::identity(), pfirst = Op::identity();
      uint32_t r = lane_run;
#pragma unroll
      for (int j = 0; j < V; ++j) {
        if (first + j < e1) {
          if ((hm >> j) & 1u) {
            if (a.emit)
              reinterpret_cast<unsigned long long*>(a.out_keys)[r] = a.emit[first + j];
            else
              store_key<KB>(a.out_keys, r, keys[j]);
            if (r != lane_run)
              a.out_vals[r - 1] = __longlong_as_double((long long)Op::finalize(cur, L));
            else
              pfirst = cur;
            cur = Op::identity();
            ++r;
          }
          Op::add(cur, vals[j], L, a.inexact, bad);
        }
      }
      const bool seen = cnt != 0;
      if (!seen) pfirst = cur;
      // what is open before each lane: inclusive scan of the lanes' last partials, from the
      // nearest lane with a head on
      const uint32_t seen_mask = __ballot_sync(0xffffffffu, seen);
      const uint32_t upto = seen_mask & (0xffffffffu >> (31 - lane));
      const uint32_t start = upto ? 31u - __clz(upto) : 0u;
      P incl = cur;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const P y = shfl_up_any(incl, o);
        if (lane >= start + o) incl = Op::combine(y, incl, bad);
      }
      P X = shfl_up_any(incl, 1);
      if (lane == 0) X = Op::identity();
      const bool before = (seen_mask & ((1u << lane) - 1)) != 0;
      const P all = shfl_any(incl, 31);
      if (seen) {
        // the run that ends before this lane's first head
        const P y = Op::combine(before ? X : Op::combine(carry, X, bad), pfirst, bad);
        if (before || carry_head)
          a.out_vals[lane_run - 1] = __longlong_as_double((long long)Op::finalize(y, L));
        else
          reinterpret_cast<P*>(a.first)[u] = y;   // the run began before this unit
      }
      carry = seen_mask ? all : Op::combine(carry, all, bad);
      carry_head = carry_head || seen_mask != 0;
      run_base += __shfl_sync(0xffffffffu, inc, 31);
    }
    release();
    if (Op::TENTATIVE && __any_sync(0xffffffffu, bad)) {
      if (lane == 0) {
        a.need[u] = kLossy;
        if (!raised) *static_cast<volatile uint32_t*>(a.inexact) = 1u;   // the only value ever written
      }
      bad = false;
      continue;
    }
    if (lane == 0) reinterpret_cast<P*>(carry_head ? a.last : a.first)[u] = carry;
  }
}

// The runs that cross units, one warp per unit: a unit with a head closes the run of the last
// head before it, the last unit also the last run.  The warp looks back over 32 units; where
// none of them has a head, which is one warp of a block at the most (the later ones find its
// unit's), the block walks on over 256 units, then 4096 at a time.  Every unit is walked over
// by one block only.  The longest walk is one run over everything, us a call with the one warp
// walking on by 512 / with its block: SUM of 19.3M values (4712 units) 191 / 146, of 60M 467 / 331,
// of 200M 1398 / 855; MIN 201 / 153, 473 / 322, 1470 / 894.
//
// A run that loses bits here, or that goes through a unit which did, is not written: its units
// are marked for the integer passes, which close the marked runs alone.
template <class Op>
__global__ void __launch_bounds__(256) f64_fix(F64Args a, uint64_t units) {
  grid_wait();   // chained launch
  grid_release();
  if (gated_off(a)) return;
  using P = typename Op::P;
  __shared__ P s_part[8];
  __shared__ bool s_head[8], s_lost[8], s_again;
  __shared__ int32_t s_stop[8], s_pos;
  const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const uint32_t u = blockIdx.x * 8 + warp;   // below 2^22
  const int L = window_L(a);
  const uint32_t mine = u < units ? a.need[u] : 0u;
  const bool head = u < units && a.heads[u] > 0, last = u + 1 == units;
  const bool closes = u > 0 && (head || last) && (!Op::AGAIN || (mine & kReclose));   // the run open before the unit
  const P* first_of = reinterpret_cast<const P*>(a.first);
  const P* last_of = reinterpret_cast<const P*>(a.last);
  auto lossy = [&](int32_t v) { return Op::TENTATIVE && (a.need[v] & kLossy); };
  // The sum of the lanes' parts up to the nearest lane with a head, in order (a higher lane holds
  // earlier units), in lane 0.  `lost`: bits were lost in the lane's part; then in the sum (lanes
  // beyond the nearest head hold units of earlier runs).  Returns that lane, 32 if there is none.
  auto join = [&](P& x, bool h, bool& lost) -> uint32_t {
    const uint32_t m = __ballot_sync(0xffffffffu, h);
    const uint32_t stop = m ? __ffs(m) - 1 : 32u;
    if (lane > stop) {
      x = Op::identity();
      lost = false;
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const P y = shfl_down_any(x, o);
      if ((lane & (2 * o - 1)) == 0) x = Op::combine(y, x, lost);   // the lanes that lead to lane 0
    }
    lost = __any_sync(0xffffffffu, lost);
    return stop;
  };
  bool bad = false, open = false;
  uint32_t stop = 0;
  P acc = Op::identity();
  if (closes) {
    const int32_t v = (int32_t)u - 1 - (int32_t)lane;
    const bool h = v >= 0 && a.heads[v] > 0;
    bad = v >= 0 && lossy(v);
    if (v >= 0) acc = h ? last_of[v] : first_of[v];
    stop = join(acc, h, bad);
    open = stop == 32;   // (unit 0 has a head)
  }
  const bool walk = __syncthreads_or(open);
  if (walk) {
    constexpr int R = 16;
    if (open && lane == 0) s_pos = (int32_t)u - 33;
    __syncthreads();
    int32_t pos = s_pos;
    for (int r = 1;; r = R) {
      // this thread's units, the newest first, up to one with a head
      P x = Op::identity();
      bool h = false, lost = false;
      int32_t at = pos - (int32_t)t * r;
      if (r == 1) {
        if (at >= 0) {
          h = a.heads[at] > 0;
          lost = lossy(at);
          x = h ? last_of[at] : first_of[at];
        }
      } else {
        const int32_t p0 = at;
#pragma unroll(sizeof(P) <= 32 ? 8 : 1)
        for (int k = 0; k < R; ++k) {
          const int32_t v = p0 - k;
          const int32_t c = v >= 0 ? v : 0;   // loaded whether it counts or not: the loads overlap
          const bool hk = a.heads[c] > 0, lk = lossy(c);
          const P y = hk ? last_of[c] : first_of[c];
          if (v >= 0 && !h) {
            x = Op::combine(y, x, lost);
            lost = lost || lk;
            h = hk;
            at = v;
          }
        }
      }
      const uint32_t near = join(x, h, lost);
      if (lane == 0) {
        s_part[warp] = x;
        s_lost[warp] = lost;
        s_head[warp] = near < 32;
      }
      if (lane == near) s_stop[warp] = at;
      __syncthreads();
      bool found = false;
      uint32_t used = 0;   // warps up to the nearest one with a head
      for (; used < 8 && !found; ++used) {
        if (open && lane == 0) acc = Op::combine(s_part[used], acc, bad);
        bad = bad || (open && s_lost[used]);
        found = s_head[used];
      }
      if (found) pos = s_stop[used - 1];
      else pos -= 256 * r;
      if (found || pos < 0) break;
      __syncthreads();   // the parts are written again
    }
    if (open && lane == 0) s_pos = pos;   // the run's first unit
  }
  if (lane == 0 && u < units) {
    const uint32_t base = a.base[u];
    if (closes) {
      const P y = Op::combine(acc, first_of[u], bad);
      bad = bad || lossy((int32_t)u);
      if (!Op::TENTATIVE || !bad) a.out_vals[base - 1] = __longlong_as_double((long long)Op::finalize(y, L));
    }
    if (last && head && (Op::AGAIN ? mine != 0 : !(Op::TENTATIVE && (mine & kLossy))))
      a.out_vals[base + a.heads[u] - 1] = __longlong_as_double((long long)Op::finalize(last_of[u], L));
  }
  if constexpr (Op::TENTATIVE) {
    const bool again = __any_sync(0xffffffffu, bad);
    if (again) {
      if (lane == 0) {
        atomicOr(a.need + u, kInvolved | kReclose);
        *static_cast<volatile uint32_t*>(a.inexact) = 1u;
      }
      if (lane <= stop && (int32_t)(u - 1 - lane) >= 0) atomicOr(a.need + (u - 1 - lane), kInvolved);
    }
    if (walk) {
      if (open && lane == 0) s_again = again;
      __syncthreads();
      const int32_t from = s_pos;
      if (s_again)
        for (int32_t v = from + (int32_t)t; v < (int32_t)(blockIdx.x * 8); v += 256) atomicOr(a.need + v, kInvolved);
    }
  }
}

// ------------------------------------------------------------------ scalar reductions
__global__ void max_u64_kernel(const unsigned long long* v, uint64_t n, unsigned long long* out) {
  unsigned long long m = 0;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
    m = v[i] > m ? v[i] : m;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long y = __shfl_down_sync(0xffffffffu, m, o);
    m = y > m ? y : m;
  }
  if ((threadIdx.x & 31) == 0) atomicMax(out, m);
}

__global__ void sum_u32_kernel(const uint32_t* v, uint64_t n, uint32_t* out) {
  uint32_t s = 0;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
    s += v[i];
  s = __reduce_add_sync(0xffffffffu, s);
  if ((threadIdx.x & 31) == 0) atomicAdd(out, s);
}

// ------------------------------------------------------------------ host side
// Elements per unit: one unit per resident warp of the main pass where that gives full units
// (32 warps on each of 148 SMs), fewer elements for short inputs.
constexpr uint64_t kF64Warps = 32 * 148;

uint32_t f64_unit_items(uint64_t n) {
  const uint64_t per = (n + kF64Warps - 1) / kF64Warps;
  const uint64_t steps = (per + kF64Step - 1) / kF64Step;
  return (uint32_t)(steps * kF64Step < kF64UnitMost ? steps * kF64Step : kF64UnitMost);
}

// done, the exponent maximum and the two passes' flags (cleared), then the counts and first run
// indices, which every pass shares, then the partials of the pass that runs.
struct F64Layout {
  uint32_t* done;
  int* emax;
  uint32_t* inexact_pair;
  uint32_t* inexact_narrow;
  size_t clear;
  uint32_t* heads;
  uint32_t* base;
  uint32_t* need;
  uint8_t* first;
  uint8_t* last;
  size_t total;
};

F64Layout f64_layout(void* ws, uint64_t n) {
  const uint64_t unit = f64_unit_items(n);
  // room for as many units as any smaller input makes (up to one per resident warp while units
  // of 256 elements give no more), so that a workspace serves every smaller input too
  const uint64_t fewest = (n + kF64Step - 1) / kF64Step;
  const uint64_t units = std::max(unit ? (n + unit - 1) / unit : 0, std::min(fewest, kF64Warps));
  constexpr size_t partial = sizeof(SumOp<kWideLimbs>::P);   // the largest
  static_assert(partial % 16 == 0 || partial % 8 == 0, "aligned partials");
  F64Layout l;
  Carver c(ws);
  uint32_t* words = c.take<uint32_t>(4);
  l.done = words;
  l.emax = reinterpret_cast<int*>(words) + 1;
  l.inexact_pair = words + 2;
  l.inexact_narrow = words + 3;
  l.clear = 4 * sizeof(uint32_t);
  l.heads = c.take<uint32_t>(units + 1);
  l.base = c.take<uint32_t>(units + 1);
  l.need = c.take<uint32_t>(units + 1);
  l.first = c.take<uint8_t>((units + 1) * partial);
  l.last = c.take<uint8_t>((units + 1) * partial);
  l.total = align_up(c.used + 256, 256);
  return l;
}

size_t f64_workspace(uint64_t n) { return f64_layout(nullptr, n).total; }

// One pass over the units and its fix-up.
template <int KB, class Op>
rfx_status f64_run_units(const F64Args& a, uint64_t units, cudaStream_t s) {
  const uint64_t want = (units + 7) / 8;
  const int gm = persistent_grid((const void*)f64_unit_kernel<KB, Op>, 256, 0, want);
  RFX_CUDA_TRY(launch_chained(f64_unit_kernel<KB, Op>, gm, 256, 0, s, a, units));
  RFX_CUDA_TRY(launch_chained(f64_fix<Op>, (int)want, 256, 0, s, a, units));
  return RFX_OK;
}

template <int KB>
rfx_status f64_dispatch_op(F64Args a, uint32_t op, void* ws, cudaStream_t s) {
  const F64Layout l = f64_layout(ws, a.n);
  a.unit = f64_unit_items(a.n);
  const uint64_t units = (a.n + a.unit - 1) / a.unit;
  a.done = l.done;
  a.heads = l.heads;
  a.base = l.base;
  a.need = l.need;
  a.first = l.first;
  a.last = l.last;
  a.inexact = l.inexact_pair;
  RFX_CUDA_TRY(cudaMemsetAsync(ws, 0, l.clear, s));
  const int gc = persistent_grid((const void*)f64_unit_count<KB>, 256, 0, (units + 7) / 8);
  f64_unit_count<KB><<<gc, 256, 0, s>>>(a, units);
  RFX_CUDA_TRY(cudaGetLastError());
  if (op == RFX_F64_MIN) return f64_run_units<KB, MinOp>(a, units, s);
  rfx_status st = f64_run_units<KB, PairOp>(a, units, s);
  if (st != RFX_OK) return st;
  // each further pass runs on the device only if the one before lost bits, over the marked units
  a.gate = l.inexact_pair;
  a.inexact = l.inexact_narrow;
  a.emax = l.emax;
  const int ge = persistent_grid((const void*)f64_emax, 256, 0, (units + 7) / 8);
  RFX_CUDA_TRY(launch_chained(f64_emax, ge, 256, 0, s, a, units));
  st = f64_run_units<KB, SumOp<kNarrowLimbs>>(a, units, s);
  if (st != RFX_OK) return st;
  a.gate = l.inexact_narrow;
  a.emax = nullptr;
  a.fixed_L = kWideL;
  return f64_run_units<KB, SumOp<kWideLimbs>>(a, units, s);
}

rfx_status f64_dispatch(F64Args a, uint32_t key_bytes, uint32_t op, void* ws, cudaStream_t s) {
  switch (key_bytes) {
    case 0: return f64_dispatch_op<0>(a, op, ws, s);
    case 1: return f64_dispatch_op<1>(a, op, ws, s);
    case 2: return f64_dispatch_op<2>(a, op, ws, s);
    case 4: return f64_dispatch_op<4>(a, op, ws, s);
    case 8: return f64_dispatch_op<8>(a, op, ws, s);
    case 16: return f64_dispatch_op<16>(a, op, ws, s);
    default: return RFX_ERR_UNSUPPORTED;
  }
}

struct DevScratch {
  void* p = nullptr;
  ~DevScratch() {
    if (p) cudaFreeAsync(p, 0);
  }
};

}  // namespace

rfx_status string_codes(const unsigned long long* ptrs, uint64_t n, uint32_t* codes, uint32_t* perm,
                        uint64_t* ndistinct, cudaStream_t s);

rfx_status reduce_f64_impl(const void* keys, uint64_t n, uint32_t key_bytes, const double* values,
                           const unsigned long long* emit, uint32_t op, void* out_keys, double* out_values,
                           uint64_t* d_groups, void* ws, size_t wsb, cudaStream_t s) {
  if (op != RFX_F64_SUM && op != RFX_F64_MIN) return RFX_ERR_INVALID;
  if (key_bytes != 0 && key_bytes != 1 && key_bytes != 2 && key_bytes != 4 && key_bytes != 8 && key_bytes != 16)
    return RFX_ERR_UNSUPPORTED;
  if (!d_groups) return RFX_ERR_INVALID;
  if (n >= (1ull << 30)) return RFX_ERR_UNSUPPORTED;
  if (n == 0) {
    RFX_CUDA_TRY(cudaMemsetAsync(d_groups, 0, sizeof(uint64_t), s));
    return RFX_OK;
  }
  if (!values || !out_values || (key_bytes && !keys) || ((key_bytes || emit) && !out_keys)) return RFX_ERR_INVALID;
  if (!ws || wsb < f64_workspace(n)) return RFX_ERR_WORKSPACE;
  uint32_t* err = device_error_word();
  if (!err) return RFX_ERR_CUDA;
  F64Args a;
  std::memset(&a, 0, sizeof(a));
  a.keys = static_cast<const uint8_t*>(keys);
  a.vals = values;
  a.n = n;
  a.emit = emit;
  a.out_keys = static_cast<uint8_t*>(out_keys);
  a.out_vals = out_values;
  a.d_groups = d_groups;
  a.err = err;
  return f64_dispatch(a, key_bytes, op, ws, s);
}

}  // namespace rfx

using namespace rfx;

extern "C" size_t rfx_reduce_f64_workspace(uint64_t n) { return f64_workspace(n); }

extern "C" rfx_status rfx_reduce_f64(const void* keys, uint64_t n, uint32_t key_bytes, const double* values,
                                     uint32_t op, void* out_keys, double* out_values, uint64_t* d_groups,
                                     void* workspace, size_t workspace_bytes, void* stream) {
  return reduce_f64_impl(keys, n, key_bytes, values, nullptr, op, out_keys, out_values, d_groups, workspace,
                         workspace_bytes, as_stream(stream));
}

namespace {

// The byte-size convention of Reduce.cu: *key_size / *value_size are device byte counts,
// read on entry, replaced by the output byte counts.
rfx_status f64_compat(const void* key_begin, const void* value_begin, void* result_key_begin,
                      void* result_value_begin, uint64_t* key_size, uint64_t* value_size, uint32_t key_bytes,
                      uint32_t op, bool string_keys) {
  if (!key_size || !value_size) return RFX_ERR_INVALID;
  cudaStream_t s = 0;
  uint64_t kbytes = 0;
  RFX_CUDA_TRY(cudaMemcpy(&kbytes, key_size, sizeof(kbytes), cudaMemcpyDeviceToHost));
  const uint64_t n = kbytes / (string_keys ? 8 : key_bytes);
  uint64_t g = 0;
  if (n) {
    DevScratch ws, codes, groups;
    const size_t wsb = f64_workspace(n);
    RFX_CUDA_TRY(cudaMallocAsync(&ws.p, wsb, s));
    RFX_CUDA_TRY(cudaMallocAsync(&groups.p, 16, s));
    const void* keys = key_begin;
    const unsigned long long* emit = nullptr;
    if (string_keys) {
      RFX_CUDA_TRY(cudaMallocAsync(&codes.p, n * 4, s));
      rfx_status st = string_codes(static_cast<const unsigned long long*>(key_begin), n,
                                   static_cast<uint32_t*>(codes.p), nullptr, nullptr, s);
      if (st != RFX_OK) return st;
      keys = codes.p;
      emit = static_cast<const unsigned long long*>(key_begin);
    }
    rfx_status st = reduce_f64_impl(keys, n, key_bytes, static_cast<const double*>(value_begin), emit, op,
                                    result_key_begin, static_cast<double*>(result_value_begin),
                                    static_cast<uint64_t*>(groups.p), ws.p, wsb, s);
    if (st != RFX_OK) return st;
    RFX_CUDA_TRY(cudaMemcpyAsync(&g, groups.p, sizeof(g), cudaMemcpyDeviceToHost, s));
    RFX_CUDA_TRY(cudaStreamSynchronize(s));
  }
  const uint64_t sizes[2] = {g * (string_keys ? 8 : key_bytes), g * 8};
  RFX_CUDA_TRY(cudaMemcpy(key_size, &sizes[0], sizeof(uint64_t), cudaMemcpyHostToDevice));
  RFX_CUDA_TRY(cudaMemcpy(value_size, &sizes[1], sizeof(uint64_t), cudaMemcpyHostToDevice));
  return RFX_OK;
}

}  // namespace

extern "C" rfx_status rfx_total_double_compat(const void* key_begin, const void* value_begin, void* result_key_begin,
                                              void* result_value_begin, uint64_t* key_size, uint64_t* value_size,
                                              uint32_t key_bytes) {
  if (key_bytes != 1 && key_bytes != 2 && key_bytes != 4 && key_bytes != 8 && key_bytes != 16)
    return RFX_ERR_UNSUPPORTED;
  return f64_compat(key_begin, value_begin, result_key_begin, result_value_begin, key_size, value_size, key_bytes,
                    RFX_F64_SUM, false);
}

extern "C" rfx_status rfx_total_string_double_compat(const void* key_begin, const void* value_begin,
                                                     void* result_key_begin, void* result_value_begin,
                                                     uint64_t* key_size, uint64_t* value_size) {
  return f64_compat(key_begin, value_begin, result_key_begin, result_value_begin, key_size, value_size, 4,
                    RFX_F64_SUM, true);
}

extern "C" rfx_status rfx_min_32_double_compat(const void* key_begin, const void* value_begin,
                                               void* result_key_begin, void* result_value_begin, uint64_t* key_size,
                                               uint64_t* value_size) {
  return f64_compat(key_begin, value_begin, result_key_begin, result_value_begin, key_size, value_size, 4,
                    RFX_F64_MIN, false);
}

extern "C" rfx_status rfx_sum_double_compat(void* result, const void* begin, const void* end) {
  if (!result || (!begin && begin != end)) return RFX_ERR_INVALID;
  const uint64_t n = (static_cast<const char*>(end) - static_cast<const char*>(begin)) / 8;
  cudaStream_t s = 0;
  if (n == 0) {  // thrust::reduce of an empty range returns its initial value, 0.0
    RFX_CUDA_TRY(cudaMemset(result, 0, sizeof(double)));
    return RFX_OK;
  }
  DevScratch ws, groups;
  const size_t wsb = f64_workspace(n);
  RFX_CUDA_TRY(cudaMallocAsync(&ws.p, wsb, s));
  RFX_CUDA_TRY(cudaMallocAsync(&groups.p, 16, s));
  rfx_status st = reduce_f64_impl(nullptr, n, 0, static_cast<const double*>(begin), nullptr, RFX_F64_SUM, nullptr,
                                  static_cast<double*>(result), static_cast<uint64_t*>(groups.p), ws.p, wsb, s);
  if (st != RFX_OK) return st;
  RFX_CUDA_TRY(cudaStreamSynchronize(s));
  return RFX_OK;
}

extern "C" rfx_status rfx_max_double_compat(void* result, const void* begin, const void* end) {
  if (!result || (!begin && begin != end)) return RFX_ERR_INVALID;
  const uint64_t n = (static_cast<const char*>(end) - static_cast<const char*>(begin)) / 8;
  cudaStream_t s = 0;
  RFX_CUDA_TRY(cudaMemsetAsync(result, 0, sizeof(unsigned long long), s));
  if (n) {
    const uint64_t blocks = (n + 255) / 256, cap = (uint64_t)device_sms() * 8;
    max_u64_kernel<<<(int)(blocks < cap ? blocks : cap), 256, 0, s>>>(
        static_cast<const unsigned long long*>(begin), n, static_cast<unsigned long long*>(result));
    RFX_CUDA_TRY(cudaGetLastError());
  }
  RFX_CUDA_TRY(cudaStreamSynchronize(s));
  return RFX_OK;
}

extern "C" rfx_status rfx_count_u32_compat(void* result, const void* begin, const void* end) {
  if (!result || (!begin && begin != end)) return RFX_ERR_INVALID;
  const uint64_t n = (static_cast<const char*>(end) - static_cast<const char*>(begin)) / 4;
  cudaStream_t s = 0;
  RFX_CUDA_TRY(cudaMemsetAsync(result, 0, sizeof(uint32_t), s));
  if (n) {
    const uint64_t blocks = (n + 255) / 256, cap = (uint64_t)device_sms() * 8;
    sum_u32_kernel<<<(int)(blocks < cap ? blocks : cap), 256, 0, s>>>(static_cast<const uint32_t*>(begin), n,
                                                                     static_cast<uint32_t*>(result));
    RFX_CUDA_TRY(cudaGetLastError());
  }
  RFX_CUDA_TRY(cudaStreamSynchronize(s));
  return RFX_OK;
}
