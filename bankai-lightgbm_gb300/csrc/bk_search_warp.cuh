// The quantized, plain (no L1 / max_delta_step / path_smooth) search of a grow round: one warp per
// (leaf, numerical feature), eight features per CTA.
//
// A round searches up to 32 leaves, thousands of (leaf, feature) slices of at most 255 bins. With a
// CTA per slice a round was six or seven waves of CTAs, each a chain of barriers; with a warp per
// slice (lane l holds the NB consecutive positions from NB l) every slice of a round is resident at
// once, the scans are a few shuffles, and the eight warps of a CTA read the same pool sectors.
//
// f64 is slow on this part (64 cycles of a scheduler's pipe per warp instruction), so a threshold
// gets its exact gain only if it can matter. The reference's gain of a threshold,
// gl^2/(hl+l2) + gr^2/(hr+l2), differs from the leaf-wide constant s0 = g^2/(h+2 l2) by exactly
//   d = (gl (hr+l2) - gr (hl+l2))^2 / ((hl+l2) (hr+l2) (h+2 l2)),
// so thresholds compare by d. The numerator is a difference of products of integer sums, exact in
// 64 bits, so fp32 carries d to a few ulps of d itself; comparing the gains in fp32 instead would
// lose everything below 1e-6 of the gain, which in a leaf whose mean gradient is far from zero is
// more than the whole difference between its thresholds (then nearly all of them went to f64).
// Error bound (u = 2^-24), with t = a + b the numerator's root, a the integer part times the scales
// (4u) and b the l2 part (5u): |d - exact| <= 44 u (|a| + |b|)^2 / denominator, plus the f64
// rounding of the reference's own evaluation and its +kEpsilon on the hessians, together below
// (4e-15 + 1.01e-15 / ymin) (s0 + d), where ymin is the smallest denominator of a valid position
// (bk_leaf.cuh), plus 1e-24 where products underflow; all of it with the gradients' scale brought to [1, 2). So only the thresholds whose
// upper bound reaches the best lower bound of the CTA's features (when no feature is penalized) can
// be the leaf's best split among them, and a feature is splittable if a lower bound passes
// min_gain_shift; a feature with no certain answer evaluates every threshold that may pass. The
// chosen split, its gain and the splittable flags are exactly the reference's. On the 10M x 100
// workload a feature queues no or one position, where a bound on the gains themselves queued up to
// all of its 254.
#pragma once
#include "bk_search.cuh"

namespace bk {

namespace {

constexpr int kWarpFeatures = 8;  // features per CTA, one warp each

// Shared memory of one warp: the feature's bins on the way in, then the packed sums of the
// accumulated bins below each position and their total. Position t sits at slice_at(t), so the lanes'
// runs of eight start in different banks, and the rows of a CTA's features are offset by two, so that
// storing two bins of eight features covers all banks.
constexpr int kSliceRow = 290;
__device__ __forceinline__ int slice_at(int t) { return t + (t >> 3); }
struct WarpSlice {
  int64_t e[kSliceRow];
  float2 up[kSliceRow];  // the positions' upper bounds (reverse, forward)
  uint16_t q[512];       // queued positions: direction << 15 | position + 1
};
static_assert(kSliceRow >= 256 + 32 + 1 && kSliceRow % 16 == 2, "257 positions, rows two banks apart");

struct WarpSearchSmem {
  WarpSlice w[kWarpFeatures];
  int32_t m[kWarpFeatures];          // best lower-bound key of each feature
  long long key[kWarpFeatures];      // the candidates: dkey of the gain, real feature
  int32_t real[kWarpFeatures];
};

// fp32 bounds on d (see above). Leaves outside the range where they hold (LeafConst::bk1 < 0), sides
// without hessian and results that overflow give lo / up = -inf / +inf. Sums fit in 32 signed bits there.
struct Bound {
  float lo, up;
};
__device__ __forceinline__ Bound bound_int(int64_t left, int32_t tg, int32_t th, const LeafConst& C, float cgh) {
  const int32_t lg = (int32_t)(left >> 32), lh = (int32_t)left, rh = th - lh;
  const int64_t num = (int64_t)lg * th - (int64_t)tg * lh;  // = lg rh - rg lh
  float t = __fmul_rn((float)num, cgh), tm = t;
  if (C.l2f != 0.f) {  // uniform
    const float b = __fmul_rn(__fmul_rn((float)((int64_t)lg - (int64_t)(tg - lg)), C.gsf), C.l2f);
    tm = __fadd_rn(fabsf(t), fabsf(b));
    t = __fadd_rn(t, b);
  }
  const float yl = fmaf((float)lh, C.hsf, C.l2f), yr = fmaf((float)rh, C.hsf, C.l2f);
  const float q = __fdividef(1.0f, __fmul_rn(__fmul_rn(yl, yr), C.hs2));
  const float d = __fmul_rn(__fmul_rn(t, t), q), dm = __fmul_rn(__fmul_rn(tm, tm), q);
  const float e = fmaf(dm, C.bk1, C.bk0);
  Bound r{__fsub_rn(d, e), __fadd_rn(d, e)};
  if (!(r.up < 1e30f) || C.bk1 < 0.f || lh == 0 || rh == 0) r = Bound{-CUDART_INF_F, CUDART_INF_F};
  if ((lg | tg) == 0) r = Bound{0.f, 0.f};  // no gradient on either side: gain and s0 are exactly 0
  return r;
}

// FindBestThresholdInt (feature_histogram.rs:673-830, scans :839-1142) of one (leaf, feature) on one
// warp, its bins in the warp's slice (0 at the most frequent bin and past the last one): lane l holds
// the nb positions from nb l (nb 8, or 2 for at most 63 bins). bounds() fixes the most frequent bin
// in the leaf's slot, bounds every threshold and returns the best lower-bound key; queue() collects
// the positions to evaluate exactly. The position loops stay rolled and keep their state in shared
// memory: a warp runs this code once per launch, so unrolled it would spend more time fetching
// instructions than executing them (bounds() measured 6 us unrolled, alone on its SM).
struct WarpSearch {
  int64_t T, base_f;
  float xup;     // upper bound of the forward scan's position -1
  int n;         // queued positions
  bool certain;  // the splittable flag is certain

  // own: the leaf's slot at the feature
  __device__ __forceinline__ int32_t bounds(const DevFeature& m, const ScanGeom& G, const LeafConst& C, int64_t* own,
                                            WarpSlice& sm, int nb, int lane) {
    const int64_t l_int = C.ls.int_sum;
    const int t0 = lane * nb;
    int64_t all = 0, acc = 0;
#pragma unroll 1
    for (int i = 0; i < nb; ++i) {
      const int t = t0 + i;
      const int64_t v = sm.e[slice_at(t)];
      all += v;
      if (!(G.skip && t + G.off == m.default_bin) && t <= G.tf_r) acc += v;
    }
    if (m.mfb > 0) {  // FixHistogram: the most frequent bin is the leaf total minus every other bin
      const int64_t rest = l_int - warp_sum(all);
      if (m.mfb >= t0 && m.mfb < t0 + nb) {
        sm.e[slice_at(m.mfb)] = rest;
        own[(size_t)(m.mfb + 1) * TILE] = rest;
        if (!(G.skip && m.mfb + G.off == m.default_bin) && m.mfb <= G.tf_r) acc += rest;
      }
    }
    // the forward scan starts with everything outside the slice (never with a fixed bin: offset 1)
    base_f = G.fwd_rest ? l_int - warp_sum(all) : 0;
    // the accumulated bins' prefix sums (packed arithmetic is exact componentwise)
    const int64_t incl = warp_incl_scan(acc, lane);
    T = __shfl_sync(FULL, incl, 31);
    const int32_t tg = (int32_t)unpack_g(l_int);
    const int32_t th = (int32_t)unpack_h(l_int);
    // the candidate positions and the first `break` of each direction
    int lb0 = kNoneLo, lb1 = kNoneHi;
    uint32_t cand = 0u;  // bits 2 i, 2 i + 1
    int64_t x = incl - acc;
#pragma unroll 1
    for (int i = 0; i < nb; ++i) {
      const int t = t0 + i;
      const bool skip_t = G.skip && t + G.off == m.default_bin;
      const int64_t v = (skip_t || t > G.tf_r) ? 0 : sm.e[slice_at(t)];
      sm.e[slice_at(t)] = x;
      const int64_t r_h = unpack_h(T - x);
      if (t >= 1 - G.off && !skip_t && t <= G.tf_r && r_h >= C.first_x) {
        cand |= 1u << (2 * i);
        if (r_h >= C.brk_x) lb0 = t;  // ascending: the highest
      }
      x += v;
      const int64_t l_h = unpack_h(base_f + x);
      if (G.two && t <= G.t_end && !skip_t && l_h >= C.first_x) {
        cand |= 2u << (2 * i);
        if (l_h >= C.brk_x && lb1 == kNoneHi) lb1 = t;
      }
    }
    if (lane == 31) sm.e[slice_at(32 * nb)] = x;
    lb0 = __reduce_max_sync(FULL, lb0);
    lb1 = __reduce_min_sync(FULL, lb1);
    const bool firstx = G.fwd_rest && unpack_h(base_f) >= C.first_x;
    if (firstx && unpack_h(base_f) >= C.brk_x) lb1 = -1;
    __syncwarp();
    const float cgh = __fmul_rn(C.gsf, C.hsf);
    float best = -CUDART_INF_F;
    x = sm.e[slice_at(t0)];
#pragma unroll 2
    for (int i = 0; i < nb; ++i) {
      const int t = t0 + i;
      const int64_t xn = sm.e[slice_at(t + 1)];
      const bool empty = xn == x;
      // a position whose bin adds nothing repeats its scan predecessor's gain and comes after it
      const Bound b0 = bound_int(l_int - (T - x), tg, th, C, cgh);
      const bool v0 = ((cand >> (2 * i)) & 1u) && t > lb0;
      const bool r0 = empty && t + 1 <= G.tf_r && !(G.skip && t + 1 + G.off == m.default_bin);
      if (v0) best = fmaxf(best, b0.lo);
      float2 u = make_float2(v0 && !r0 ? b0.up : -CUDART_INF_F, -CUDART_INF_F);
      if (G.two) {
        const Bound b1 = bound_int(base_f + xn, tg, th, C, cgh);
        const bool v1 = ((cand >> (2 * i)) & 2u) && t < lb1;
        const bool r1 = empty && ((t >= 1 && !(G.skip && t - 1 + G.off == m.default_bin)) || (t == 0 && G.fwd_rest));
        if (v1) best = fmaxf(best, b1.lo);
        if (v1 && !r1) u.y = b1.up;
      }
      sm.up[slice_at(t)] = u;
      x = xn;
    }
    // the forward scan's position -1 (every lane evaluates it, lane 0 queues it)
    xup = -CUDART_INF_F;
    if (firstx && lb1 != -1) {
      const Bound b = bound_int(base_f, tg, th, C, cgh);
      best = fmaxf(best, b.lo);
      xup = b.up;
    }
    certain = __any_sync(FULL, best > C.d_up);
    return __reduce_max_sync(FULL, float_key(best));
  }

  // Queues the positions that need their exact gain: those that may pass min_gain_shift and reach
  // the best lower bound M; every one that may pass when the flag is not certain.
  __device__ __forceinline__ void queue(const LeafConst& C, int32_t M, WarpSlice& sm, int nb, int lane) {
    uint32_t need = 0u;
#pragma unroll 1
    for (int i = 0; i < nb; ++i) {
      const float2 u = sm.up[slice_at(lane * nb + i)];
      if (u.x > C.d_dn && (!certain || float_key(u.x) >= M)) need |= 1u << (2 * i);
      if (u.y > C.d_dn && (!certain || float_key(u.y) >= M)) need |= 2u << (2 * i);
    }
    const bool needx = lane == 0 && xup > C.d_dn && (!certain || float_key(xup) >= M);
    const int cnt = __popc(need) + (needx ? 1 : 0);
    n = 0;
    if (!__any_sync(FULL, cnt != 0)) return;
    const int incl = warp_incl_scan(cnt, lane);
    n = __shfl_sync(FULL, incl, 31);
    int at = incl - cnt;
    if (needx) sm.q[at++] = (uint16_t)0x8000u;
    while (need) {
      const int b = __ffs(need) - 1;
      need &= need - 1u;
      sm.q[at++] = (uint16_t)((lane * nb + (b >> 1) + 1) | ((b & 1) << 15));
    }
    __syncwarp();
  }
};

// One direction's best exact position (in every lane).
struct ExactBest {
  long long key;
  double gain, lsg, lsh, rsg, rsh, lo, ro;
  int64_t left;  // packed sums of the left side
  int32_t lc, rc, t;
  int split;     // a position passed min_gain_shift
};

// The exact gains, outputs and sums of the queued positions (int_side): eight positions a batch,
// four lanes each, both directions together; each direction's arg-max (highest gain, ties to the
// earliest position in scan order).
__device__ __forceinline__ void exact_batches(const Params& p, const WarpSlice& sm, int n, int64_t T, int64_t base_f,
                                              const LeafConst& C, int lane, ExactBest (&r)[2]) {
#pragma unroll
  for (int d = 0; d < 2; ++d) {
    r[d].key = kNoKey;
    r[d].gain = -CUDART_INF;
    r[d].t = d == 0 ? kNoneLo : kNoneHi;
    r[d].split = 0;
  }
  const int64_t l_int = C.ls.int_sum, tg = unpack_g(l_int), th = unpack_h(l_int);
  const int k = lane >> 2, role = lane & 3;
#pragma unroll 1
  for (int b0 = 0; b0 < n; b0 += 8) {
    const bool have = b0 + k < n;
    const uint32_t ent = sm.q[have ? b0 + k : n - 1];
    const int t = (int)(ent & 0x7fffu) - 1, d = (int)(ent >> 15);
    const int64_t left = d == 0 ? l_int - (T - sm.e[slice_at(t)]) : base_f + sm.e[slice_at(t + 1)];
    const int64_t lg = unpack_g(left), lh = unpack_h(left);
    const SidePart sp = int_side(p, lg, lh, tg, th, C.gs, C.hs, C.cnt_factor, role);
    const int q0 = lane & ~3;
    const double gl = __shfl_sync(FULL, sp.val, q0), gr = __shfl_sync(FULL, sp.val, q0 | 1);
    const double g = gl + gr;
    const bool passed = have && gain_passes(g, C.mgs);
    const bool elig = passed && !dnan(g) && !is_neg_inf(g);  // NaN never wins
#pragma unroll
    for (int dd = 0; dd < 2; ++dd) {
      if (!__any_sync(FULL, passed && d == dd)) continue;
      r[dd].split = 1;
      const bool mine = elig && d == dd;
      const long long key = warp_max64(mine ? dkey(g) : kNoKey);
      if (key == kNoKey) continue;
      const bool at = mine && dkey(g) == key;
      const int tb = dd == 0 ? __reduce_max_sync(FULL, at ? t : kNoneLo) : __reduce_min_sync(FULL, at ? t : kNoneHi);
      const int wl = (__ffs(__ballot_sync(FULL, at && t == tb)) - 1) & ~3;
      const bool better = key > r[dd].key || (key == r[dd].key && (dd == 0 ? tb > r[dd].t : tb < r[dd].t));
      ExactBest x;
      x.key = key;
      x.gain = __shfl_sync(FULL, g, wl);
      x.lsg = __shfl_sync(FULL, sp.sg, wl + 2);
      x.lsh = __shfl_sync(FULL, sp.sh, wl + 2);
      x.lo = __shfl_sync(FULL, sp.val, wl + 2);
      x.lc = __shfl_sync(FULL, sp.n, wl + 2);
      x.rsg = __shfl_sync(FULL, sp.sg, wl + 3);
      x.rsh = __shfl_sync(FULL, sp.sh, wl + 3);
      x.ro = __shfl_sync(FULL, sp.val, wl + 3);
      x.rc = __shfl_sync(FULL, sp.n, wl + 3);
      x.left = (int64_t)__shfl_sync(FULL, (long long)left, wl);
      x.t = tb;
      x.split = 1;
      if (better) r[dd] = x;
    }
  }
}

// The combination of the directions (feature_histogram.rs:700-830): the reverse scan first, the
// forward scan replaces it only with a strictly larger gain; then the penalty.
__device__ __forceinline__ Cand warp_cand(const DevFeature& m, const ScanGeom& G, int32_t f, const LeafConst& C,
                                          const ExactBest (&r)[2], int split) {
  const int nd = G.two ? 2 : 1;
  // the forward scan replaces a reverse one only with a gain above (reverse gain - shift) + shift
  int ch = r[0].key != kNoKey ? 0 : -1;
  if (nd == 2 && r[1].key != kNoKey && (ch < 0 || r[1].gain > (r[0].gain - C.mgs) + C.mgs)) ch = 1;
  Cand c;
  cand_reset(&c, m.real, f);
  if (ch >= 0) {
    const int64_t l_int = C.ls.int_sum;
    const int64_t left = ch == 0 ? r[0].left : r[1].left;
    const int32_t t = ch == 0 ? r[0].t : r[1].t;
    c.threshold = (uint32_t)(ch == 0 ? t - 1 + G.off : t + G.off);
    c.left_output = ch == 0 ? r[0].lo : r[1].lo;
    c.right_output = ch == 0 ? r[0].ro : r[1].ro;
    c.left_count = ch == 0 ? r[0].lc : r[1].lc;
    c.right_count = ch == 0 ? r[0].rc : r[1].rc;
    c.lsg = ch == 0 ? r[0].lsg : r[1].lsg;
    c.lsh = ch == 0 ? r[0].lsh : r[1].lsh;
    c.rsg = ch == 0 ? r[0].rsg : r[1].rsg;
    c.rsh = ch == 0 ? r[0].rsh : r[1].rsh;
    c.lint = left;
    c.rint = (int64_t)(((uint64_t)(unpack_g(l_int) - unpack_g(left)) << 32) |
                       ((uint64_t)(unpack_h(l_int) - unpack_h(left)) & 0xffffffffull));
    c.gain = (ch == 0 ? r[0].gain : r[1].gain) - C.mgs;
    c.default_left = ch == 0 ? 1 : 0;
  }
  if (nd == 1 && m.missing == 2) c.default_left = 0;
  if (m.penalty != 1.0) c.gain *= m.penalty;
  c.splittable = split;
  c.missing = m.missing;
  return c;
}

}  // namespace

}  // namespace bk
