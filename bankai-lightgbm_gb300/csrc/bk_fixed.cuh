// The float path's fixed-point numbers: 96-bit multiples of a unit that a tree chooses for its gradients
// and one for its hessians (JobState::red_maxg / red_maxh hold the largest biased exponents, Params::
// fix_bits the bits of the largest value), such that every value is a multiple and no sum of the tree's
// rows overflows. Sums are exact, in any order. All of it runs on the integer pipes: an f64 instruction
// takes 64 cycles of a scheduler.
#pragma once
#include "bk_common.cuh"

namespace bk {

namespace {

// A 96-bit two's complement multiple of the tree's unit.
struct Fixed {
  uint32_t lo, mid, hi;
};

// v's 24-bit mantissa shifted up by its exponent's distance from the smallest one that fits: `shift0`
// = the shift of biased exponent 0. The tree's rule (JobState::fix_ok) makes 0 <= shift.
__device__ __forceinline__ Fixed to_fixed(float v, int shift0) {
  const uint32_t u = __float_as_uint(v), e = (u >> 23) & 0xffu, m = (u & 0x7fffffu) | (e ? 0x800000u : 0u);
  const uint32_t s = m ? (uint32_t)((int)max(e, 1u) + shift0) : 0u;
  const uint64_t x = (uint64_t)m << (s & 31u);
  const uint32_t x0 = (uint32_t)x, x1 = (uint32_t)(x >> 32), w = s >> 5;
  Fixed f;
  f.lo = w == 0u ? x0 : 0u;
  uint64_t top = w == 0u ? (uint64_t)x1 : (w == 1u ? x : x << 32);
  if (u >> 31) {
    f.lo = 0u - f.lo;
    top = ~top + (f.lo == 0u ? 1u : 0u);
  }
  f.mid = (uint32_t)top;
  f.hi = (uint32_t)(top >> 32);
  return f;
}

// (hi:mid:lo) * 2^exp as a double, rounded to nearest even. In integer instructions: the f64 unit takes
// 64 cycles of a scheduler for each conversion or addition of a warp.
__device__ __forceinline__ double fixed_to_double(uint32_t lo, uint32_t mid, uint32_t hi, int exp) {
  const bool neg = (hi >> 31) != 0u;
  if (neg) {
    lo = 0u - lo;
    const uint64_t t = ~(((uint64_t)hi << 32) | mid) + (lo == 0u ? 1u : 0u);
    mid = (uint32_t)t;
    hi = (uint32_t)(t >> 32);
  }
  if (!(lo | mid | hi)) return 0.0;
  if (hi == 0u) {  // two words at the top
    hi = mid, mid = lo, lo = 0u, exp -= 32;
    if (hi == 0u) hi = mid, mid = 0u, exp -= 32;
  }
  const int z = __clz((int)hi);
  uint64_t top = ((uint64_t)__funnelshift_l(mid, hi, z) << 32) | __funnelshift_l(lo, mid, z);  // bit 63 set
  const bool sticky = (lo << z) != 0u;
  const uint32_t rest = (uint32_t)top & 0x7ffu;
  top >>= 11;
  if (rest > 0x400u || (rest == 0x400u && (sticky || (top & 1u)))) ++top;
  // top in [2^52, 2^53], so its bit 52 adds one to the exponent field
  const int64_t field = exp + 95 - z + 1022;
  return __longlong_as_double((long long)(top + ((uint64_t)field << 52)) | (neg ? (long long)(1ull << 63) : 0));
}

__device__ __forceinline__ Fixed operator+(const Fixed& a, const Fixed& b) {
  Fixed r;
  r.lo = a.lo + b.lo;
  const uint64_t top = (((uint64_t)a.hi << 32) | a.mid) + (((uint64_t)b.hi << 32) | b.mid) + (r.lo < a.lo ? 1u : 0u);
  r.mid = (uint32_t)top;
  r.hi = (uint32_t)(top >> 32);
  return r;
}
__device__ __forceinline__ Fixed operator-(const Fixed& a, const Fixed& b) {
  Fixed r;
  r.lo = a.lo - b.lo;
  const uint64_t top = (((uint64_t)a.hi << 32) | a.mid) - (((uint64_t)b.hi << 32) | b.mid) - (a.lo < b.lo ? 1u : 0u);
  r.mid = (uint32_t)top;
  r.hi = (uint32_t)(top >> 32);
  return r;
}
__device__ __forceinline__ bool operator<(const Fixed& a, const Fixed& b) {
  if (a.hi != b.hi) return (int32_t)a.hi < (int32_t)b.hi;
  return a.mid != b.mid ? a.mid < b.mid : a.lo < b.lo;
}

// The exponent of a tree's unit: the value of biased exponent e and mantissa m is m 2^(e - 150), and the
// largest exponent's values end at bit fix_bits.
__device__ __forceinline__ int fixed_unit(const Params& p, uint32_t emax) { return (int)emax - p.fix_bits - 126; }

// x in units of 2^exp: bits below the unit are dropped (sums of a tree's values have none), values past
// 95 bits saturate.
__device__ __forceinline__ Fixed double_to_fixed(double x, int exp) {
  const uint64_t b = (uint64_t)__double_as_longlong(x);
  const int e = (int)((b >> 52) & 0x7ffu);
  uint64_t m = b & 0xfffffffffffffULL;
  if (e) m |= 0x10000000000000ULL;
  const int s = max(e, 1) - 1075 - exp;
  Fixed r;
  if (s <= 0) {
    m >>= min(-s, 63);
    r.lo = (uint32_t)m;
    r.mid = (uint32_t)(m >> 32);
    r.hi = 0u;
  } else {
    const uint32_t t = (uint32_t)s & 31u;
    const uint64_t x0 = m << t;
    const uint32_t over = (uint32_t)((m >> 32) >> (32u - t));  // t = 0: nothing (53 bits)
    r.lo = s < 32 ? (uint32_t)x0 : 0u;
    r.mid = s < 32 ? (uint32_t)(x0 >> 32) : (uint32_t)x0;
    r.hi = s < 32 ? over : (uint32_t)(x0 >> 32);
    if (s > 42 && m) r = Fixed{0xffffffffu, 0xffffffffu, 0x7fffffffu};
  }
  if (b >> 63) r = Fixed{0u, 0u, 0u} - r;
  return r;
}

// x 2^exp as a float, truncated: within 2^-23 of it (zero below the normal range).
__device__ __forceinline__ float fixed_to_float(Fixed x, int exp) {
  const bool neg = (x.hi >> 31) != 0u;
  if (neg) x = Fixed{0u, 0u, 0u} - x;
  if (x.hi == 0u) {
    x.hi = x.mid, x.mid = x.lo, exp -= 32;
    if (x.hi == 0u) x.hi = x.mid, x.mid = 0u, exp -= 32;
  }
  if (x.hi == 0u) return 0.f;
  const int z = __clz((int)x.hi), field = exp + 95 - z + 127;
  const uint32_t top = __funnelshift_l(x.mid, x.hi, z) >> 8;
  uint32_t r = ((uint32_t)field << 23) | (top & 0x7fffffu);
  if (field <= 0) r = 0u;
  if (field >= 255) r = 0x7f800000u;
  return __uint_as_float(neg ? r | 0x80000000u : r);
}
// A double truncated to a float, the same way.
__device__ __forceinline__ float double_to_float(double x) {
  const uint64_t b = (uint64_t)__double_as_longlong(x);
  const uint32_t hi = (uint32_t)(b >> 32), abs_hi = hi & 0x7fffffffu;
  uint32_t f = __funnelshift_l((uint32_t)b, abs_hi - (896u << 20), 3);
  if (abs_hi < (897u << 20)) f = 0u;
  if (abs_hi >= (1151u << 20)) f = 0x7f800000u;
  return __uint_as_float(f | (hi & 0x80000000u));
}

__device__ __forceinline__ Fixed shfl_fixed(const Fixed& x, int from) {
  return Fixed{__shfl_sync(0xffffffffu, x.lo, from), __shfl_sync(0xffffffffu, x.mid, from),
               __shfl_sync(0xffffffffu, x.hi, from)};
}
__device__ __forceinline__ Fixed shfl_up_fixed(const Fixed& x, int o, int width) {
  return Fixed{__shfl_up_sync(0xffffffffu, x.lo, o, width), __shfl_up_sync(0xffffffffu, x.mid, o, width),
               __shfl_up_sync(0xffffffffu, x.hi, o, width)};
}

}  // namespace

}  // namespace bk
