// Pairs of fp32 numbers (hi + lo, about 46 bits; Dekker 1971, Knuth's two-sum) for the row-wise
// kernels whose reference arithmetic is f64. An f64 instruction holds a scheduler's pipe for 64 cycles
// per warp on this part, an fp32 one for one, so a value that ends as fp32 is computed as a pair and
// rounded from it wherever the pair's error cannot move the rounding; the rest (a few rows in a
// hundred thousand) are computed in f64. Both give the fp32 number that the f64 arithmetic gives.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace bk {

struct Pair {
  float hi, lo;
};

__device__ __forceinline__ Pair quick_two_sum(float a, float b) {  // |a| >= |b| or a = 0
  const float s = __fadd_rn(a, b);
  return Pair{s, __fsub_rn(b, __fsub_rn(s, a))};
}
__device__ __forceinline__ Pair two_sum(float a, float b) {
  const float s = __fadd_rn(a, b), bb = __fsub_rn(s, a);
  return Pair{s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb))};
}
__device__ __forceinline__ Pair two_prod(float a, float b) {
  const float x = __fmul_rn(a, b);
  return Pair{x, __fmaf_rn(a, b, -x)};
}
__device__ __forceinline__ Pair pair_add(Pair a, Pair b) {  // error at most 2^-45 of |a| + |b|
  Pair s = two_sum(a.hi, b.hi);
  return quick_two_sum(s.hi, __fadd_rn(s.lo, __fadd_rn(a.lo, b.lo)));
}
__device__ __forceinline__ Pair pair_mul(Pair a, Pair b) {  // relative error at most 2^-45
  const Pair x = two_prod(a.hi, b.hi);
  return quick_two_sum(x.hi, __fmaf_rn(a.hi, b.lo, __fmaf_rn(a.lo, b.hi, x.lo)));
}
__device__ __forceinline__ Pair pair_div(Pair a, Pair b) {  // relative error at most 2^-44
  const float q = __fdiv_rn(a.hi, b.hi);
  float r = __fmaf_rn(-q, b.hi, a.hi);  // exact
  r = __fadd_rn(r, __fmaf_rn(-q, b.lo, a.lo));
  return quick_two_sum(q, __fdividef(r, b.hi));
}
__device__ __forceinline__ Pair pair_neg(Pair a) { return Pair{-a.hi, -a.lo}; }

// An f64 value as a pair, by integer operations: the high 24 bits of its significand, then the other
// 29 rounded to 24 (error 2^-53 of the value). ok = false above 2^60 and for NaN, and for magnitudes
// below 2^-60 but zero, whose parts an fp32 pair cannot hold. ABSOLUTE: the caller needs an error below
// 2^-60 only, not one relative to the value, so those become 0 with ok true.
template <bool ABSOLUTE = false>
__device__ __forceinline__ Pair pair_of(double x, bool* ok) {
  const uint32_t h = (uint32_t)__double2hiint(x), l = (uint32_t)__double2loint(x);
  const int e = (int)((h >> 20) & 0x7ffu) - 1023;
  *ok = e < 60 && (ABSOLUTE || e >= -60 || ((h << 1) | l) == 0u);
  if (e < -60 || e >= 60) return Pair{0.f, 0.f};
  const uint32_t sign = h & 0x80000000u;
  const float hi = __uint_as_float(sign | ((uint32_t)(e + 127) << 23) | ((h & 0xfffffu) << 3) | (l >> 29));
  const float lo = __fmul_rn((float)(l & 0x1fffffffu), __uint_as_float(sign | ((uint32_t)(e - 52 + 127) << 23)));
  return quick_two_sum(hi, lo);
}

// 2^(j / 32) as pairs.
struct ExpTable {
  float hi[32], lo[32];
};

// exp(z), |z| <= 60, relative error at most 2^-43: z = (32 m + j) ln2 / 32 + r, |r| <= 0.0109,
// exp(z) = 2^m 2^(j/32) (1 + p(r)) with p the series to r^6 (Tang, "Table-driven implementation of the
// exponential function in IEEE floating-point arithmetic", 1989); r, r^2 / 2 and the product are
// pairs. ln2 / 32 is split in parts of 13 (exact products with n < 2^11) and 24 + 24 bits.
__device__ __forceinline__ Pair pair_exp(Pair z, const ExpTable& T) {
  const float n = rintf(__fmul_rn(z.hi, 46.16624130844683f));
  const int ni = (int)n, j = ni & 31, m = ni >> 5;
  constexpr double kStep = 0.021660849392498290;  // ln2 / 32
  constexpr float c1 = 0.0216598510742187500f;     // 13 significant bits
  constexpr float c2 = (float)(kStep - (double)c1);
  constexpr float c3 = (float)(kStep - (double)c1 - (double)c2);
  const float r0 = __fmaf_rn(-n, c1, z.hi);  // exact: both are multiples of the result's last bit
  const Pair q = two_prod(n, c2);
  Pair r = two_sum(r0, -q.hi);
  r = quick_two_sum(r.hi, __fadd_rn(r.lo, __fadd_rn(z.lo, __fmaf_rn(-n, c3, -q.lo))));
  const float x = r.hi;
  // r^3 (1/6 + r/24 + r^2/120 + r^3/720), then r^2 / 2 and r in pairs
  const float t = __fmaf_rn(x, __fmaf_rn(x, __fmaf_rn(x, 1.f / 720.f, 1.f / 120.f), 1.f / 24.f), 1.f / 6.f);
  const Pair sq = two_prod(x, x);
  const float sql = __fmaf_rn(2.f * x, r.lo, sq.lo);
  Pair p = two_sum(x, 0.5f * sq.hi);
  p = quick_two_sum(p.hi, __fadd_rn(p.lo, __fadd_rn(r.lo, __fmaf_rn(0.5f, sql, __fmul_rn(__fmul_rn(sq.hi, x), t)))));
  const Pair tj{T.hi[j], T.lo[j]};
  const Pair tp = pair_mul(tj, p);
  const Pair e = pair_add(tj, tp);
  const float s = __uint_as_float((uint32_t)(m + 127) << 23);
  return Pair{__fmul_rn(e.hi, s), __fmul_rn(e.lo, s)};
}

// Rounds a (normalized) pair to fp32: false when a relative error `rel` of it could change the result,
// or when the pair is so small that its low part, or the result itself, is not held in full (zero too).
__device__ __forceinline__ bool pair_round(Pair a, float rel, float* out) {
  *out = a.hi;
  const uint32_t u = __float_as_uint(a.hi), b = u & 0x7fffffffu;
  uint32_t half = (b & 0x7f800000u) - (24u << 23);  // half a unit in the last place
  // below a power of two the units are half as large
  if ((b & 0x7fffffu) == 0u && (a.lo == 0.f || ((u ^ __float_as_uint(a.lo)) >> 31) != 0u)) half -= 1u << 23;
  return b - (40u << 23) < (210u << 23) &&
         fabsf(__fsub_rn(__uint_as_float(half), fabsf(a.lo))) > __fmul_rn(rel, fabsf(a.hi));
}

}  // namespace bk
