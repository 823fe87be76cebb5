// What the split searches share: scans, the scan directions' geometry, one side of an exact
// evaluation, key comparisons.
#pragma once
#include "bk_decide.cuh"
#include "bk_math.cuh"

namespace bk {

namespace {

template <typename T>
__device__ __forceinline__ T warp_incl_scan(T v, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    T u = __shfl_up_sync(FULL, v, o);
    if (lane >= o) v += u;
  }
  return v;
}

// Inclusive scan towards lower lanes: lane l gets the sum over lanes l .. 31.
template <typename T>
__device__ __forceinline__ T warp_incl_scan_down(T v, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    T u = __shfl_down_sync(FULL, v, o);
    if (lane + o < 32) v += u;
  }
  return v;
}

template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
  return v;
}


__device__ __forceinline__ int64_t unpack_g(int64_t pk) { return pk >> 32; }
__device__ __forceinline__ int64_t unpack_h(int64_t pk) { return pk & 0xffffffffLL; }

// Order-preserving integer keys of non-NaN floats and doubles (negative zero counts as zero),
// computed with integer operations only.
__device__ __forceinline__ int32_t float_key(float x) {
  int32_t b = __float_as_int(x);
  if (b == (int32_t)0x80000000) b = 0;
  return b ^ ((b >> 31) & 0x7fffffff);
}
__device__ void cand_reset(Cand* c, int32_t real, int32_t inner) {
  c->gain = -CUDART_INF;
  c->left_output = c->right_output = 0.0;
  c->lsg = c->lsh = c->rsg = c->rsh = 0.0;
  c->lint = c->rint = 0;
  c->feature = real;
  c->inner = inner;
  c->threshold = 0;
  c->left_count = c->right_count = 0;
  c->default_left = 1;
  c->splittable = 0;
  c->categorical = 0;
}

// Direction geometry of FindBestThreshold[Int] (feature_histogram.rs:219-357, :673-830): direction
// 0 is the reverse scan (right side accumulates, default left, positions t = tf_r down to 1 - off),
// direction 1 the forward scan (left side accumulates, positions t = -1 or 0 up to t_end).
struct ScanGeom {
  bool two, skip, fwd_rest;
  int off, tf_r, t_end;
};

__device__ __forceinline__ ScanGeom scan_geom(const DevFeature& m) {
  ScanGeom G;
  G.two = m.num_bin > 2 && m.missing != 0;
  G.skip = G.two && m.missing == 1;
  const bool na = G.two && m.missing == 2;
  G.off = m.offset;
  G.tf_r = m.num_bin - 1 - G.off - (na ? 1 : 0);
  G.t_end = m.num_bin - 2 - G.off;
  // with NaN missing and the most-frequent bin 0, the forward scan's left side starts as
  // everything outside the slice, at position t = -1 (held by the last thread)
  G.fwd_rest = na && G.off == 1;
  return G;
}

// One quarter of a queued position's evaluation, as one lane computes it (plain gains: no L1,
// max_delta_step or path_smooth). Role 0 / 1: the left / right leaf gain (simd.rs:6-8,
// feature_histogram.rs:148-176: left + right = the split gain, in that order); role 2 / 3: the
// left / right output (feature_histogram.rs:79-104) with the side's SplitInfo sums and count
// (feature_histogram.rs:240-357, :700-830). Both are one division, num / (den + lambda_l2), so all
// four lanes run the same instructions: gain = g^2 / (h + l2), output = -g / (h + l2).
struct SidePart {
  double val;     // the leaf gain (roles 0, 1) or the output (roles 2, 3)
  double sg, sh;  // the side's sums as the SplitInfo stores them (roles 2, 3)
  int32_t n;      // the side's count (roles 2, 3)
};

// Role `role` of an integer threshold with left sums (lg, lh): the hessian gets kEpsilon added for
// the gain (feature_histogram.rs:878-925), the output and the SplitInfo use the plain sums, the
// counts are round_int(hess * cnt_factor) — exactly as int_split_gain and eval_int compute them.
__device__ __forceinline__ SidePart int_side(const Params& p, int64_t lg, int64_t lh, int64_t tg, int64_t th,
                                             double gs, double hs, double cnt_factor, int role) {
  const bool right = (role & 1) != 0, gain = role < 2;
  const int64_t sg = right ? tg - lg : lg, sh = right ? th - lh : lh;
  const double dg = (double)(int32_t)sg * gs, dh = (double)(uint32_t)sh * hs;
  SidePart r;
  r.n = round_int((double)(uint32_t)sh * cnt_factor);
  const double sq = dg * dg;
  const double he = dh + BK_EPS;
  const double num = gain ? sq : -dg;
  const double den = (gain ? he : dh) + p.l2;
  r.val = num / den;
  r.sg = dg;
  r.sh = dh;
  return r;
}

// Role `role` of a float threshold of direction d with accumulated sums (ag, ah, c): the gain
// takes the sums split_gains gets (the reverse scan's right side is the accumulated one), the
// output and the SplitInfo the right side from the left sums, as eval_float computes them.
__device__ __forceinline__ SidePart float_side(const Params& p, int d, double ag, double ah, int32_t c, double sum_g,
                                               double sum_h, int32_t num_data, int role) {
  const bool right = (role & 1) != 0, gain = role < 2;
  const double slg = d == 0 ? sum_g - ag : ag, slh = d == 0 ? sum_h - ah : ah;
  const int32_t lc = d == 0 ? num_data - c : c;
  // the gain's sums: the accumulated side as accumulated, the other as total minus it
  const double gg = !right ? slg : (d == 0 ? ag : sum_g - ag);
  const double gh = !right ? slh : (d == 0 ? ah : sum_h - ah);
  // the SplitInfo's sums: the right side from the left sums
  const double og = !right ? slg : sum_g - slg, oh = !right ? slh : sum_h - slh;
  SidePart r;
  r.n = !right ? lc : num_data - lc;
  const double sq = gg * gg;
  const double num = gain ? sq : -og;
  const double den = (gain ? gh : oh) + p.l2;
  r.val = num / den;
  r.sg = og;
  r.sh = oh - BK_EPS;
  return r;
}

constexpr int kNoneLo = -0x7fffffff, kNoneHi = 0x7fffffff;

// !(gain <= mgs) without an f64 comparison.
__device__ __forceinline__ bool gain_passes(double gain, double mgs) {
  return dnan(gain) || dnan(mgs) || dkey(gain) > dkey(mgs);
}
__device__ __forceinline__ bool is_neg_inf(double x) {
  return (unsigned long long)__double_as_longlong(x) == 0xfff0000000000000ULL;
}

}  // namespace

}  // namespace bk
