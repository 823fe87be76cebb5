// FindBestSplitsFromHistograms (serial.rs:1322-1566, int: :1212-1300) and the grow-loop
// bookkeeping kernels (serial.rs:578-628, :779-825, :1685-1876), GB300 form.
//
// k_search: one 256-thread CTA per (leaf side, feature), thread t owning local bin t (a feature
// slice holds at most 255 bins). The CTA fixes the smaller leaf's most-frequent bin (FixHistogram,
// serial.rs:2205-2238), derives the larger leaf's slice as parent minus the fixed smaller slice in
// place (serial.rs:1407-1437, :1218-1242), and evaluates both directional threshold scans of the
// reference (FindBestThresholdSequentially[Int], feature_histogram.rs:363-663 / 839-1142) at once,
// thread t holding the reverse scan's position t and the forward scan's position t. The sequential
// scan's `break` (the first threshold whose other side falls under min_data / min_hessian ends the
// scan) becomes "the first such position in scan order and everything after it is excluded";
// `current_gain > best_gain` becomes an arg-max with ties going to the earliest position in scan
// order. Every reduction is a warp reduction plus one barrier.
//
// The quantized path scans the packed (grad << 32) + hess sums with one block prefix scan; the
// reverse scan's sums are the total minus the prefix, exact in integers, so its candidates are
// bit-identical to the reference's. The float path scans exact 96-bit integers (search_float_fixed); trees
// without fixed-point histograms, and gains with L1 / max_delta_step / path_smooth, scan f64 prefix and
// suffix sums (associated differently from the sequential scan, about 1e-16 relative).
//
// f64 is slow on this part, so it stays off the common path: the leaf constants the scans share
// come precomputed from the histogram launch (bk_leaf.cuh), plain gains are filtered in fp32 with
// a rigorous error bound, and every comparison of the fold and the arg-max runs on integer keys.
// The last CTA of k_search folds the per-feature candidates of each searched leaf in feature order
// with `better_than`, takes the arg-max leaf (split_info.rs:88-96), stops the tree when its gain is
// <= 0, and builds the route table of the chosen split (data_partition.rs:299-410). The post-split
// bookkeeping (bk_grow.cuh) runs in the last CTA of the partition scatter.
#include <math_constants.h>

#include <type_traits>

#include "bk_decide.cuh"
#include "bk_grow.cuh"
#include "bk_launch.cuh"
#include "bk_leaf.cuh"
#include "bk_math.cuh"
#include "bk_fixed.cuh"
#include "bk_search.cuh"
#include "bk_search_warp.cuh"

namespace bk {

namespace {

constexpr int kSearchThreads = kDecideThreads;  // one thread per local bin
constexpr int kSearchWarps = kSearchThreads / 32;

// ---- fp32 prefilter of the plain split gain (no L1 / max_delta_step / path_smooth) ----
// The reference evaluates gl^2/(hl+l2) + gr^2/(hr+l2) in f64 for every threshold. Each candidate is
// first evaluated in fp32 together with a rigorous bound E on |fp32 - f64| (u = 2^-24): the
// numerators' conversions and scaling (3u), the denominators' (4u, plus kEpsilon, below 0.02u for
// denominators >= 1e-6), the square (u), the division (__fdividef: at most 2 ulp = 4u for divisors
// in [2^-126, 2^126]) and the sum (u) add up to at most 16.1u relative to the non-negative result;
// the fp32 bound computations round once more. E uses 24u. The largest gain G* of a direction is
// at least the best certified lower bound M over its valid thresholds, so only the thresholds
// whose upper bound reaches M (and exceeds min_gain_shift) can hold it, and the direction is
// splittable exactly when G* passes min_gain_shift. Those few thresholds (and any whose fp32
// evaluation is uncertain) are evaluated in f64, so the chosen split, its gain and the splittable
// flag are exactly the reference's. A threshold whose accumulated side gained nothing since its
// predecessor in scan order (an empty bin between them) has that predecessor's gain exactly and
// comes after it, so it is never queued.
constexpr float kPrefilterRel = 24.0f * 5.9604645e-08f;

struct Approx {
  float g, e;
  bool uncertain;
};

__device__ __forceinline__ Approx approx_from(float xl, float yl, float xr, float yr) {
  Approx a;
  float tl = __fdividef(__fmul_rn(xl, xl), yl);
  float tr = __fdividef(__fmul_rn(xr, xr), yr);
  a.g = __fadd_rn(tl, tr);
  a.e = __fadd_rn(__fmul_rn(kPrefilterRel, a.g), 1e-30f);
  // non-finite values, denominators outside [1e-6, 1e30] (where the reference's +kEpsilon matters
  // or the fast division leaves its accuracy range) and huge results go to f64
  a.uncertain = !(yl >= 1e-6f) || !(yr >= 1e-6f) || !(yl <= 1e30f) || !(yr <= 1e30f) || !(a.g < 1e30f) ||
                isnan(a.g);
  return a;
}

// GetSplitGains of one integer threshold (feature_histogram.rs:878-925: the hessians get
// kEpsilon added, counts are round_int(hess * cnt_factor)).
__device__ __forceinline__ double int_split_gain(const Params& p, int64_t lg, int64_t lh, int64_t tg, int64_t th,
                                                 double gs, double hs, double cnt_factor, double parent, bool plain) {
  // the sums fit in 32 bits (signed gradients, unsigned hessians): 32-bit conversions, exact
  const int64_t rg = tg - lg, rh = th - lh;
  const double slh = (double)(uint32_t)lh * hs, srh = (double)(uint32_t)rh * hs;
  const int32_t lc = plain ? 0 : round_int((double)(uint32_t)lh * cnt_factor);
  const int32_t rc = plain ? 0 : round_int((double)(uint32_t)rh * cnt_factor);
  return split_gains(p, (double)(int32_t)lg * gs, slh + BK_EPS, (double)(int32_t)rg * gs, srh + BK_EPS, lc, rc,
                     parent);
}

// What one search CTA needs of the job state, loaded in one round of independent loads: the
// searched leaf's constants and sums (computed by the histogram launch), the smaller leaf's sums
// (for FixHistogram), and the pool slots of the smaller and larger leaf.
struct SearchIn {
  LeafConst C;
  LeafSum S0;
  int32_t sslot, lslot;  // pool slots: the smaller leaf's, and the larger one's, which holds its parent's
  int32_t group; // a grow round's search: the feature group of the candidate, else -1
  int32_t crow;  // row of the compact candidate copies: the side, or 2 e + side in a grow round
  // the integer search's two pool entries of this thread (IntPool), loaded from the slots known
  // before the wait; valid when those slots are the state's
  int64_t sv, lv;
  bool pre;
};

// The pool entries thread t of an integer search scans: the smaller leaf's bin t + 1 of feature
// f (none at the most-frequent bin, which the fix rewrites) and, on side 1, its parent's.
struct IntPool {
  int64_t sv, lv;
};
__device__ __forceinline__ IntPool int_pool(const Job& J, const Params& p, const DevFeature& m, int side, int32_t f,
                                            int32_t sslot, int32_t lslot) {
  const int t = threadIdx.x;
  const size_t slot_stride = (size_t)p.T * p.B * TILE;
  const size_t feat_off = (size_t)(f / TILE) * p.B * TILE + (f % TILE) + (size_t)(t + 1) * TILE;
  const int64_t* pool = reinterpret_cast<const int64_t*>(J.pool);
  const bool fix = m.mfb > 0;
  const bool in = t < m.len;
  IntPool r;
  r.sv = (in && !(fix && t == m.mfb)) ? pool[(size_t)sslot * slot_stride + feat_off] : 0;
  r.lv = (side && in) ? pool[(size_t)lslot * slot_stride + feat_off] : 0;
  return r;
}

// Scan order: the reverse scan visits higher bins first, the forward scan lower bins first.
__device__ __forceinline__ bool earlier(int d, int ta, int tb) { return d == 0 ? ta > tb : ta < tb; }

// The best position of one direction within a warp (and, combined, within the CTA).
// Everything a candidate threshold contributes to its SplitInfo: the gain, the left / right sums,
// counts and outputs.
struct Eval {
  double gain, lsg, lsh, rsg, rsh, lo, ro;
  int32_t lc, rc;
  int64_t lint, rint;
};

struct DirBest {
  long long key;  // dkey of the gain; kNoKey when no position qualified
  int64_t a, b;   // int: left (grad, hess) sums; float: bit patterns of the accumulated (grad, hess)
  int32_t t, c;   // position; float: accumulated count
  Eval ev;        // ev.gain: -inf when none
};


// The chosen threshold's SplitInfo: lane 0 evaluates the left side, lane 1 the right side, in one
// instruction stream (FindBestThresholdInt's output assembly, feature_histogram.rs:700-830: 32-bit
// conversions of the packed sums, exact since they fit in 32 bits).
__device__ __forceinline__ Eval eval_int(const Params& p, int64_t lg, int64_t lh, int64_t tg, int64_t th, double gs,
                                         double hs, double cnt_factor, double parent, double gain, int lane) {
  const int64_t rg = tg - lg, rh = th - lh;
  const int64_t sg = lane == 0 ? lg : rg, sh = lane == 0 ? lh : rh;
  const double dg = (double)(int32_t)sg * gs, dh = (double)(uint32_t)sh * hs;
  const int32_t n = round_int((double)(uint32_t)sh * cnt_factor);
  const double out = lane < 2 ? split_output(p, dg, dh, n, parent) : 0.0;
  Eval v;
  v.gain = gain;
  v.lsg = dg;
  v.lsh = dh;
  v.lc = n;
  v.lo = out;
  v.rsg = __shfl_sync(FULL, dg, 1);
  v.rsh = __shfl_sync(FULL, dh, 1);
  v.rc = __shfl_sync(FULL, n, 1);
  v.ro = __shfl_sync(FULL, out, 1);
  v.lint = (int64_t)(((uint64_t)lg << 32) | ((uint64_t)lh & 0xffffffffull));
  v.rint = (int64_t)(((uint64_t)rg << 32) | ((uint64_t)rh & 0xffffffffull));
  return v;
}

// FindBestThreshold's output assembly (feature_histogram.rs:240-357): (ag, ah, c) is the
// accumulated side of direction d (0: right, 1: left); the right side of the outputs derives from
// the left sums. Lane 0 evaluates the left output, lane 1 the right one.
__device__ __forceinline__ Eval eval_float(const Params& p, int d, double ag, double ah, int32_t c, double sum_g,
                                           double sum_h, int32_t num_data, double parent, double gain, int lane) {
  const double slg = d == 0 ? sum_g - ag : ag, slh = d == 0 ? sum_h - ah : ah;
  const int32_t lc = d == 0 ? num_data - c : c;
  const double sg = lane == 0 ? slg : sum_g - slg, sh = lane == 0 ? slh : sum_h - slh;
  const int32_t n = lane == 0 ? lc : num_data - lc;
  const double out = lane < 2 ? split_output(p, sg, sh, n, parent) : 0.0;
  Eval v;
  v.gain = gain;
  v.lsg = slg;
  v.lsh = slh - BK_EPS;
  v.lc = lc;
  v.lo = out;
  v.rsg = sum_g - slg;
  v.rsh = (sum_h - slh) - BK_EPS;
  v.rc = num_data - lc;
  v.ro = __shfl_sync(FULL, out, 1);
  v.lint = v.rint = 0;
  return v;
}

// One direction's stop / prefilter summary of a warp (published before one barrier).
struct WarpFilt {
  int32_t lb;      // the warp's first `break` position in scan order (kNoneLo / kNoneHi: none)
  int32_t mb, ma;  // best certified fp32 lower-bound key of positions before lb / of all positions
};

// A position queued for its f64 gain (PLAIN gains): evaluated by warp 0.
struct QEnt {
  int64_t a, b;  // int: left (grad, hess) sums; float: bit patterns of the accumulated (grad, hess)
  int32_t c;     // float: accumulated count
  int16_t t, d;  // position, direction
};

// The shared memory of a numerical search CTA of NW warps (32 * NW threads, one per local bin).
template <int NW>
struct SearchSmemT {
  QEnt q[2][32 * NW];  // per direction: every position at most once
  int32_t qn[2];
  DirBest pres[2][4];  // per direction and batch lane (below): the arg-max of its batches
  int32_t psplit[2][4];
  int64_t wi[2][NW];
  double wd[10][NW];
  int32_t wc[3][NW];
  WarpFilt wf[2][NW];
  WarpFilt xf;  // the forward scan's position -1 (last thread)
  Fixed fx[3][NW], top[3];  // search_float_fixed: the warps' sums of gradients, hessians, counts; the top bin's
  int32_t spl[2][NW];
  DirBest wb[2][NW];
};
using SearchSmem = SearchSmemT<kSearchWarps>;

// This warp's arg-max of direction d (highest key, then the earliest position in scan order) into w.
__device__ __forceinline__ void warp_best(int d, bool elig, double gain, int t, int64_t a, int64_t b, int32_t c,
                                          int lane, DirBest* w) {
  const long long key = elig ? dkey(gain) : kNoKey;
  const long long km = warp_max64(key);
  if (km == kNoKey) {
    if (lane == 0) {
      w->key = kNoKey;
      w->ev.gain = -CUDART_INF;
      w->t = 0;
    }
    return;
  }
  const bool at = elig && key == km;
  const int tb = d == 0 ? __reduce_max_sync(FULL, at ? t : kNoneLo) : __reduce_min_sync(FULL, at ? t : kNoneHi);
  if (at && t == tb) {
    w->key = km;
    w->a = a;
    w->b = b;
    w->t = t;
    w->c = c;
    w->ev.gain = gain;
  }
}

// Warp 0 after the barrier: the CTA's best of each direction (lane 0: direction 0, lane 8:
// direction 1), broadcast to every lane of the warp.
template <int NW>
__device__ __forceinline__ void combine_best(const SearchSmemT<NW>& sm, int lane, DirBest (&r)[2], int (&split)[2]) {
  const int d = (lane >> 3) & 1;
  long long key = kNoKey;
  double gain = -CUDART_INF;
  int64_t a = 0, b = 0;
  int32_t t = 0, c = 0;
  int sp = 0;
  if (lane < 16 && (lane & 7) < NW) {
    const DirBest& e = sm.wb[d][lane & 7];
    key = e.key;
    if (key != kNoKey) {
      gain = e.ev.gain;
      a = e.a;
      b = e.b;
      t = e.t;
      c = e.c;
    }
    sp = sm.spl[d][lane & 7];
  }
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) {
    const long long xk = __shfl_xor_sync(FULL, key, o);
    const double xg = __shfl_xor_sync(FULL, gain, o);
    const int64_t xa = __shfl_xor_sync(FULL, a, o), xb = __shfl_xor_sync(FULL, b, o);
    const int32_t xt = __shfl_xor_sync(FULL, t, o), xc = __shfl_xor_sync(FULL, c, o);
    sp |= __shfl_xor_sync(FULL, sp, o);
    if (xk > key || (xk == key && xk != kNoKey && earlier(d, xt, t))) {
      key = xk;
      gain = xg;
      a = xa;
      b = xb;
      t = xt;
      c = xc;
    }
  }
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const int src = 8 * k;
    r[k].key = __shfl_sync(FULL, key, src);
    r[k].ev.gain = __shfl_sync(FULL, gain, src);
    r[k].a = __shfl_sync(FULL, a, src);
    r[k].b = __shfl_sync(FULL, b, src);
    r[k].t = __shfl_sync(FULL, t, src);
    r[k].c = __shfl_sync(FULL, c, src);
    split[k] |= __shfl_sync(FULL, sp, src);
  }
}

// The fp32 view of one position: certified lower-bound key lo, upper-bound key up, and whether it
// may pass min_gain_shift (mp).
struct Filt {
  bool mp, unc;
  int32_t lo, up;
};

__device__ __forceinline__ Filt filt_of(bool cand, const Approx& a, const LeafConst& C) {
  Filt f;
  f.unc = a.uncertain;
  f.mp = cand && (a.uncertain || __fadd_rn(a.g, a.e) > C.mgs_dn);
  f.lo = (cand && !a.uncertain) ? float_key(__fsub_rn(a.g, a.e)) : float_key(-CUDART_INF_F);
  f.up = a.uncertain ? 0 : float_key(__fadd_rn(a.g, a.e));
  return f;
}

// Before the barrier: the warp's summary of direction d for positions `pos` (thread order = t).
template <bool PLAIN, int NW>
__device__ __forceinline__ void publish_dir(SearchSmemT<NW>& sm, int d, bool brk, int pos, const Filt& f, int lane,
                                            int warp) {
  const int lb = d == 0 ? __reduce_max_sync(FULL, brk ? pos : kNoneLo) : __reduce_min_sync(FULL, brk ? pos : kNoneHi);
  WarpFilt w;
  w.lb = lb;
  w.mb = w.ma = float_key(-CUDART_INF_F);
  if (PLAIN) {
    const bool none = d == 0 ? lb == kNoneLo : lb == kNoneHi;
    const bool before = none || (d == 0 ? pos > lb : pos < lb);
    w.ma = __reduce_max_sync(FULL, f.lo);
    w.mb = __reduce_max_sync(FULL, before ? f.lo : float_key(-CUDART_INF_F));
  }
  if (lane == 0) sm.wf[d][warp] = w;
}

// After the barrier: direction d's stop S (the first `break` in scan order; positions from it on
// are invalid) and the best certified lower bound M over the valid positions. Warp w holds
// positions 32w .. 32w + 31; the forward scan's position -1 (when `has_x`) comes first in its
// scan order. The maximal gain G* of the direction is at least M, so only positions whose upper
// bound reaches M can hold it; and any position passes min_gain_shift exactly when G* does.
template <bool PLAIN, int NW>
__device__ __forceinline__ void resolve_dir(const SearchSmemT<NW>& sm, int d, bool has_x, int* S, int32_t* M) {
  int s = d == 0 ? kNoneLo : kNoneHi;
#pragma unroll
  for (int w = 0; w < NW; ++w) s = d == 0 ? max(s, sm.wf[d][w].lb) : min(s, sm.wf[d][w].lb);
  if (d == 1 && has_x && sm.xf.lb == -1) s = -1;
  *S = s;
  int32_t m = float_key(-CUDART_INF_F);
  if (PLAIN) {
    const bool none = d == 0 ? s == kNoneLo : s == kNoneHi;
    if (d == 1 && has_x && s != -1) m = sm.xf.ma;
#pragma unroll
    for (int w = 0; w < NW; ++w) {
      const WarpFilt& f = sm.wf[d][w];
      const bool contains = !none && f.lb == s;
      const bool all_before = none || (d == 0 ? 32 * w > s : 32 * w + 31 < s);
      if (contains)
        m = max(m, f.mb);
      else if (all_before)
        m = max(m, f.ma);
    }
  }
  *M = m;
}

// Appends this thread's entry (when `push`) to direction d's queue, one shared atomic per warp.
template <int NW>
__device__ __forceinline__ void queue_push(SearchSmemT<NW>& sm, int d, bool push, const QEnt& e, int lane) {
  const unsigned bal = __ballot_sync(FULL, push);
  int base = 0;
  if (lane == 0 && bal) base = atomicAdd(&sm.qn[d], __popc(bal));
  base = __shfl_sync(FULL, base, 0);
  if (push) sm.q[d][base + __popc(bal & ((1u << lane) - 1u))] = e;
}

// Queue batches of 8 positions, four lanes per position: lanes 4k, 4k + 1 evaluate the left and
// right leaf gains of position k, lanes 4k + 2, 4k + 3 its left and right outputs (SidePart). An
// f64 instruction costs a scheduler the same whether one lane or 32 run it, so spreading a
// position's two gains and two outputs over four lanes (one division each, in the same
// instructions) shortens its instruction chain to a quarter of the work, and evaluating every
// queued position's outputs with its gain leaves none to evaluate after the arg-max. Batch k of direction d runs on warp
// d + 2 (k mod 4), so the first batches of the two directions run on two schedulers and longer
// queues spread over all four. One warp: its batches k0, k0 + 4, ...; their arg-max (highest gain,
// ties to the earliest position in scan order) with its SplitInfo, and whether any passed, into
// sm.pres[d][k0] / sm.psplit[d][k0]. (With NW warps, batch k runs on warp d + 2 (k mod NW / 2).)
template <int NW, typename SideOf>
__device__ __forceinline__ void eval_batches(SearchSmemT<NW>& sm, int d, int k0, int lane, double mgs, SideOf side_of) {
  DirBest r;
  r.key = kNoKey;
  r.ev.gain = -CUDART_INF;
  r.a = r.b = 0;
  r.t = d == 0 ? kNoneLo : kNoneHi;
  r.c = 0;
  int split = 0;
  const int n = sm.qn[d];
  const int k = lane >> 2, role = lane & 3;
  auto batch = [&](int b0) {
    // quads past the queue's end evaluate its last entry and discard the result: an all-zero
    // entry would send the whole warp through the f64 division's slow path (zero dividend, tiny
    // divisor), which costs more than the gain itself on this part
    const bool have = b0 + k < n;
    const QEnt e = sm.q[d][have ? b0 + k : n - 1];
    const SidePart sp = side_of(e, role);
    const int q0 = lane & ~3;
    const double gl = __shfl_sync(FULL, sp.val, q0);
    const double gr = __shfl_sync(FULL, sp.val, q0 | 1);
    double g = gl + gr;
    if (!have) g = -CUDART_INF;
    const bool passed = have && gain_passes(g, mgs);
    if (__any_sync(FULL, passed)) split = 1;
    const bool elig = passed && !dnan(g) && !is_neg_inf(g);  // NaN never wins
    const long long key = warp_max64(elig ? dkey(g) : kNoKey);
    if (key == kNoKey) return;
    const bool at = elig && dkey(g) == key;
    const int tb = d == 0 ? __reduce_max_sync(FULL, at ? (int)e.t : kNoneLo)
                          : __reduce_min_sync(FULL, at ? (int)e.t : kNoneHi);
    const int wl = __ffs(__ballot_sync(FULL, at && (int)e.t == tb)) - 1 & ~3;  // the quad's first lane
    Eval v;
    v.gain = __shfl_sync(FULL, g, wl);
    v.lsg = __shfl_sync(FULL, sp.sg, wl + 2);
    v.lsh = __shfl_sync(FULL, sp.sh, wl + 2);
    v.lo = __shfl_sync(FULL, sp.val, wl + 2);
    v.lc = __shfl_sync(FULL, sp.n, wl + 2);
    v.rsg = __shfl_sync(FULL, sp.sg, wl + 3);
    v.rsh = __shfl_sync(FULL, sp.sh, wl + 3);
    v.ro = __shfl_sync(FULL, sp.val, wl + 3);
    v.rc = __shfl_sync(FULL, sp.n, wl + 3);
    v.lint = v.rint = 0;
    const int64_t wa = __shfl_sync(FULL, e.a, wl), wb = __shfl_sync(FULL, e.b, wl);
    const int32_t wc = __shfl_sync(FULL, e.c, wl);
    if (key > r.key || (key == r.key && earlier(d, tb, r.t))) {
      r.key = key;
      r.t = tb;
      r.ev = v;
      r.a = wa;
      r.b = wb;
      r.c = wc;
    }
  };
  // the first batch outside the loop: the f64 gain evaluated inside a loop measured about twice
  // as slow as the same code in straight-line form
  constexpr int kLanes = NW / 2;  // batch lanes per direction
  if (8 * k0 < n) batch(8 * k0);
  for (int b0 = 8 * (k0 + kLanes); b0 < n; b0 += 8 * kLanes) batch(b0);
  if (lane == 0) {
    sm.pres[d][k0] = r;
    sm.psplit[d][k0] = split;
  }
}

// After the queues are filled (barrier 3): the NW warps evaluate the queue batches (warp w takes
// direction w & 1, batches w >> 1, (w >> 1) + NW / 2, ...). Barrier 4; then warp 0 combines the
// batch results of each direction into r / rs, the winner's SplitInfo included.
template <int NW, typename SideOf>
__device__ __forceinline__ void eval_queues(SearchSmemT<NW>& sm, int warp, int lane, double mgs, SideOf side_of,
                                            DirBest (&r)[2], int (&rs)[2]) {
  static_assert(NW >= 2 && NW <= 8 && NW % 2 == 0, "one batch lane of each direction per pair of warps");
  const int d = warp & 1, k0 = warp >> 1;
  if (k0 < NW / 2) eval_batches<NW>(sm, d, k0, lane, mgs, side_of);
  __syncthreads();
  if (warp != 0) return;
#pragma unroll
  for (int dd = 0; dd < 2; ++dd) {
    r[dd] = sm.pres[dd][0];
    rs[dd] = sm.psplit[dd][0];
#pragma unroll
    for (int k = 1; k < NW / 2; ++k) {
      const DirBest& x = sm.pres[dd][k];
      rs[dd] |= sm.psplit[dd][k];
      if (x.key != kNoKey && (x.key > r[dd].key || (x.key == r[dd].key && earlier(dd, x.t, r[dd].t)))) r[dd] = x;
    }
  }
}

// A grow round's candidate of feature group `g` (its node's record is in J.cand already) and the
// node's splittable flag of feature f.
__device__ __forceinline__ void store_round_cand(const Job& J, const Params& p, int crow, int g, int32_t node, int32_t f,
                                                 const Cand& c) {
  RoundCand r;
  r.key = dnan(c.gain) ? kNoKey : dkey(c.gain);
  r.pk = ((uint32_t)f << 9) | ((uint32_t)(c.default_left != 0) << 8) | c.threshold;
  r.real = c.feature;
  round_view(J, p).cand[(size_t)crow * p.n_groups + g] = r;
  J.splittable[(size_t)node * p.F + f] = (uint8_t)c.splittable;
}

// `row`: the leaf (or, in a grow round, the node) the candidate belongs to; `crow`: its place among
// the search's compact copies. In a grow round the node's splittable flag is written here; otherwise
// the split decision writes it to the leaf's slot.
__device__ __forceinline__ void store_cand(const Job& J, const Params& p, const SearchIn& si, int32_t row, int32_t f,
                                           const Cand& c) {
  J.cand[(size_t)row * p.F + f] = c;
  if (si.group >= 0) {
    store_round_cand(J, p, si.crow, si.group, row, f, c);
    return;
  }
  J.cgain[(size_t)si.crow * p.F + f] = c.gain;
  J.cthr[(size_t)si.crow * p.F + f] = c.threshold | ((uint32_t)(c.default_left != 0) << 31);
  J.csplit[(size_t)si.crow * p.F + f] = (uint8_t)c.splittable;
}

// The combination of the directions (feature_histogram.rs:240-357, :700-830): the reverse scan
// first, the forward scan replaces it only with a strictly larger gain; then the chosen threshold's
// SplitInfo (`eval_of(best, direction)`), the penalty and the feature's candidate record. Warp 0,
// every lane with the same values.
template <typename EvalOf>
__device__ __forceinline__ void finish_cand(const Job& J, const Params& p, const DevFeature& m, const SearchIn& si,
                                            int32_t leaf, int32_t f, const ScanGeom& G, double mgs, const DirBest (&r)[2],
                                            const int (&rs)[2], int lane, EvalOf eval_of) {
  const int nd = G.two ? 2 : 1;
  int sp = 0, ch = -1;
  double cgain = -CUDART_INF;
  for (int i = 0; i < nd; ++i) {
    sp |= rs[i];
    if (rs[i] && r[i].ev.gain > cgain + mgs) {
      ch = i;
      cgain = r[i].ev.gain - mgs;
    }
  }
  Cand c;
  cand_reset(&c, m.real, f);
  if (ch >= 0) {
    // field-wise selects keep the chosen direction in registers
    DirBest b;
    b.key = ch == 0 ? r[0].key : r[1].key;
    b.a = ch == 0 ? r[0].a : r[1].a;
    b.b = ch == 0 ? r[0].b : r[1].b;
    b.c = ch == 0 ? r[0].c : r[1].c;
    b.t = ch == 0 ? r[0].t : r[1].t;
    b.ev = ch == 0 ? r[0].ev : r[1].ev;
    const Eval e = eval_of(b, ch);
    const int32_t t = b.t;
    c.threshold = (uint32_t)(ch == 0 ? t - 1 + G.off : t + G.off);
    c.left_output = e.lo;
    c.left_count = e.lc;
    c.lsg = e.lsg;
    c.lsh = e.lsh;
    c.right_output = e.ro;
    c.right_count = e.rc;
    c.rsg = e.rsg;
    c.rsh = e.rsh;
    c.lint = e.lint;
    c.rint = e.rint;
    c.gain = cgain;
    c.default_left = ch == 0 ? 1 : 0;
  }
  if (nd == 1 && m.missing == 2) c.default_left = 0;
  c.gain *= m.penalty;
  c.splittable = sp;
  c.missing = m.missing;
  if (lane == 0) store_cand(J, p, si, leaf, f, c);
}

// FindBestThresholdInt for one (leaf, feature): feature_histogram.rs:673-830, scans :839-1142.
// Three barriers: the prefix scan (with the most-frequent-bin fix and the forward scan's start
// folded in), the stop / prefilter summaries, and the arg-max.
template <bool PLAIN, int NW>
__device__ void search_int(const Job& J, const Params& p, const SearchIn& si, const DevFeature& m, int side,
                           int32_t f, int32_t leaf, SearchSmemT<NW>& sm) {
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const LeafConst& C = si.C;
  const int64_t s_int = si.S0.int_sum;
  const int64_t l_int = side ? C.ls.int_sum : s_int;
  const size_t slot_stride = (size_t)p.T * p.B * TILE;
  const size_t feat_off = (size_t)(f / TILE) * p.B * TILE + (f % TILE);
  int64_t* pool = reinterpret_cast<int64_t*>(J.pool);
  int64_t* hs = pool + (size_t)si.sslot * slot_stride + feat_off;  // group bin 0 of the feature
  int64_t* hl = pool + (size_t)(side ? si.lslot : si.sslot) * slot_stride + feat_off;
  const bool fix = m.mfb > 0;  // offset 0: the slice holds every bin and the most frequent one is empty
  const bool in = t < m.len;
  // the smaller leaf's most-frequent entry is rewritten by its side-0 CTA; side 1 never reads it
  const IntPool pv = si.pre ? IntPool{si.sv, si.lv} : int_pool(J, p, m, side, f, si.sslot, si.lslot);
  const int64_t sv = pv.sv, lv = pv.lv;
  const ScanGeom G = scan_geom(m);
  if (t < 2) sm.qn[t] = 0;
  const bool skip_t = G.skip && t + G.off == m.default_bin;
  const bool acc_t = !skip_t && t <= G.tf_r;  // bin t is accumulated by the scans
  const int64_t v0 = side ? lv - sv : sv;     // before the most-frequent bin's fix
  // barrier 1: the packed prefix sums of the accumulated bins, plus the sum that fixes the
  // most-frequent bin (fix) or starts the forward scan outside the slice (fwd_rest; never both:
  // fix needs offset 0, fwd_rest offset 1). Packed arithmetic is exact componentwise.
  int64_t w = acc_t ? v0 : 0;
  int64_t P = warp_incl_scan(w, lane);
  const int64_t aux = warp_sum(fix ? sv : v0);
  if (lane == 31) sm.wi[0][warp] = P;
  if (lane == 0) sm.wi[1][warp] = aux;
  __syncthreads();
  int64_t T = 0, AUX = 0;
#pragma unroll
  for (int i = 0; i < NW; ++i) {
    const int64_t y = sm.wi[0][i];
    if (i < warp) P += y;
    T += y;
    AUX += sm.wi[1][i];
  }
  int64_t v = v0;
  if (fix) {
    const int64_t fixed = s_int - AUX;  // FixHistogram: the leaf total minus every other bin
    const int64_t delta = side ? -fixed : fixed;
    if (t == m.mfb) {
      v = v0 + delta;
      if (side == 0) hs[(size_t)(t + 1) * TILE] = fixed;
    }
    if (m.mfb <= G.tf_r && !(G.skip && m.mfb + G.off == m.default_bin)) {
      T += delta;
      if (t >= m.mfb) P += delta;
      if (t == m.mfb) w += delta;
    }
  }
  if (side && in) hl[(size_t)(t + 1) * TILE] = v;
  const int64_t base_f = G.fwd_rest ? l_int - AUX : 0;
  const int64_t tg = unpack_g(l_int), th = unpack_h(l_int);
  // reverse position t: right side = bins t .. tf_r; forward position t: left side = base_f plus
  // bins 0 .. t; the last thread also holds forward position -1 (left side = base_f)
  const int64_t right = T - (P - w);
  const int64_t left = base_f + P;
  const bool xpos = G.fwd_rest && t == 32 * NW - 1;
  const bool first0 = t >= 1 - G.off && acc_t && unpack_h(right) >= C.first_x;
  const bool brk0 = first0 && unpack_h(right) >= C.brk_x;
  const bool first1 = G.two && t <= G.t_end && !skip_t && unpack_h(left) >= C.first_x;
  const bool brk1 = first1 && unpack_h(left) >= C.brk_x;
  const bool firstx = xpos && unpack_h(base_f) >= C.first_x;
  const bool brkx = firstx && unpack_h(base_f) >= C.brk_x;
  const int64_t lg[2] = {tg - unpack_g(right), xpos ? unpack_g(base_f) : unpack_g(left)};
  const int64_t lh[2] = {th - unpack_h(right), xpos ? unpack_h(base_f) : unpack_h(left)};
  // barrier 2: stops and prefilter summaries
  Filt fl[2];
#pragma unroll
  for (int d = 0; d < 2; ++d) {
    const bool cand = d == 0 ? first0 : (first1 || firstx);
    Bound b{-CUDART_INF_F, CUDART_INF_F};
    if (PLAIN && cand)
      b = bound_int(d == 0 ? l_int - right : (xpos ? base_f : left), (int32_t)tg, (int32_t)th, C, __fmul_rn(C.gsf, C.hsf));
    fl[d] = Filt{cand && b.up > C.d_dn, false, float_key(cand ? b.lo : -CUDART_INF_F), float_key(b.up)};
  }
  publish_dir<PLAIN, NW>(sm, 0, brk0, t, fl[0], lane, warp);
  {
    Filt nat = fl[1];
    if (xpos) nat.lo = float_key(-CUDART_INF_F);  // the natural position 255 is never a candidate
    publish_dir<PLAIN, NW>(sm, 1, brk1, t, nat, lane, warp);
  }
  if (xpos) {
    WarpFilt x;
    x.lb = brkx ? -1 : kNoneHi;
    x.ma = x.mb = fl[1].lo;
    sm.xf = x;
  }
  __syncthreads();
  int S[2];
  int32_t M[2];
  resolve_dir<PLAIN, NW>(sm, 0, false, &S[0], &M[0]);
  resolve_dir<PLAIN, NW>(sm, 1, G.fwd_rest, &S[1], &M[1]);
  const bool valid[2] = {first0 && t > S[0], xpos ? (firstx && S[1] != -1) : (first1 && t < S[1])};
  DirBest r[2];
  int rs[2] = {0, 0};
  if (PLAIN) {
    // a position whose bin adds nothing repeats its scan predecessor (t + 1 reverse, t - 1 forward)
    const bool rep[2] = {w == 0 && t + 1 <= G.tf_r && !(G.skip && t + 1 + G.off == m.default_bin),
                         !xpos && w == 0 && ((t >= 1 && !(G.skip && t - 1 + G.off == m.default_bin)) ||
                                             (t == 0 && G.fwd_rest))};
    // barrier 3: the few positions that need their f64 gain; barrier 4: evaluated on the eight warps
#pragma unroll
    for (int d = 0; d < 2; ++d) {
      const bool exact = valid[d] && !rep[d] && (fl[d].unc || (fl[d].mp && fl[d].up >= M[d]));
      queue_push(sm, d, exact, QEnt{lg[d], lh[d], 0, (int16_t)(d == 0 || !xpos ? t : -1), (int16_t)d}, lane);
    }
    __syncthreads();
    const double gs = C.gs, hsc = C.hs;
    eval_queues(
        sm, warp, lane, C.mgs,
        [&](const QEnt& e, int role) { return int_side(p, e.a, e.b, tg, th, gs, hsc, C.cnt_factor, role); }, r, rs);
    if (warp != 0) return;
  } else {
    // every valid position evaluates its own f64 gain; barrier 3: the arg-max
    double gain[2];
    bool split[2], elig[2];
#pragma unroll
    for (int d = 0; d < 2; ++d) {
      gain[d] = -CUDART_INF;
      if (valid[d])
        gain[d] = int_split_gain(p, lg[d], lh[d], tg, th, C.gs, C.hs, C.cnt_factor, C.parent, false);
      const bool passed = valid[d] && gain_passes(gain[d], C.mgs);
      split[d] = passed;
      elig[d] = passed && !dnan(gain[d]) && !is_neg_inf(gain[d]);  // NaN never wins
    }
    warp_best(0, elig[0], gain[0], t, lg[0], lh[0], 0, lane, &sm.wb[0][warp]);
    warp_best(1, elig[1], gain[1], xpos ? -1 : t, lg[1], lh[1], 0, lane, &sm.wb[1][warp]);
#pragma unroll
    for (int d = 0; d < 2; ++d) {
      const int ws = __any_sync(FULL, split[d]);
      if (lane == 0) sm.spl[d][warp] = ws;
    }
    __syncthreads();
    if (warp != 0) return;
    combine_best(sm, lane, r, rs);
  }
  // FindBestThresholdInt's combination of the directions (feature_histogram.rs:700-830)
  finish_cand(J, p, m, si, leaf, f, G, C.mgs, r, rs, lane, [&](const DirBest& b, int d) {
    (void)d;
    if (PLAIN) {  // evaluated with the gain
      Eval v = b.ev;
      v.lint = (int64_t)(((uint64_t)b.a << 32) | ((uint64_t)b.b & 0xffffffffull));
      v.rint = (int64_t)(((uint64_t)(tg - b.a) << 32) | ((uint64_t)(th - b.b) & 0xffffffffull));
      return v;
    }
    return eval_int(p, b.a, b.b, tg, th, C.gs, C.hs, C.cnt_factor, C.parent, b.ev.gain, lane);
  });
}

// FindBestThreshold (float) for one (leaf, feature): feature_histogram.rs:219-357, scans
// :363-663. f64 (grad, hess) sums and row counts estimated per bin as round_int(hess *
// cnt_factor); the forward scan uses prefix sums, the reverse scan suffix sums (accumulated from
// the top bin down, not derived by subtraction).
template <bool PLAIN, int NW>
__device__ void search_float(const Job& J, const Params& p, const SearchIn& si, const DevFeature& m, int side,
                             int32_t f, int32_t leaf, SearchSmemT<NW>& sm) {
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const LeafConst& C = si.C;
  const LeafSum& S0 = si.S0;
  const int32_t num_data = side ? C.ls.num_data : S0.num_data;
  const size_t slot_stride = (size_t)p.T * p.B * TILE;
  const size_t feat_off = (size_t)(f / TILE) * p.B * TILE + (f % TILE);
  double2* pool = reinterpret_cast<double2*>(J.pool);
  double2* hs = pool + (size_t)si.sslot * slot_stride + feat_off;
  double2* hl = pool + (size_t)(side ? si.lslot : si.sslot) * slot_stride + feat_off;
  const double2 zero = make_double2(0.0, 0.0);
  const bool fix = m.mfb > 0;
  const bool in = t < m.len;
  double2 sv = (in && !(fix && t == m.mfb)) ? hs[(size_t)(t + 1) * TILE] : zero;
  const double2 lv = (side && in) ? pool[(size_t)si.lslot * slot_stride + feat_off + (size_t)(t + 1) * TILE] : zero;
  const ScanGeom G = scan_geom(m);
  if (t < 2) sm.qn[t] = 0;
  const double sum_g = C.sum_g, sum_h = C.sum_h;
  if (fix) {  // one barrier for both sums
    const double ag = warp_sum(sv.x), ah = warp_sum(sv.y);
    if (lane == 0) {
      sm.wd[0][warp] = ag;
      sm.wd[1][warp] = ah;
    }
    __syncthreads();
    double tg = 0.0, th = 0.0;
#pragma unroll
    for (int i = 0; i < NW; ++i) {
      tg += sm.wd[0][i];
      th += sm.wd[1][i];
    }
    if (t == m.mfb) {
      sv = make_double2(S0.sg - tg, S0.sh - th);
      if (side == 0) hs[(size_t)(t + 1) * TILE] = sv;
    }
  }
  const double2 v = side ? make_double2(lv.x - sv.x, lv.y - sv.y) : sv;
  if (side && in) hl[(size_t)(t + 1) * TILE] = v;
  const int32_t cn = in ? round_int(v.y * C.cnt_factor) : 0;
  // barrier: prefix sums (forward), suffix sums over bins <= tf_r (reverse) and, when the forward
  // scan starts outside the slice, the slice totals
  const bool skip_t = G.skip && t + G.off == m.default_bin;
  const double wg = skip_t ? 0.0 : v.x, wh = skip_t ? 0.0 : v.y;
  const int32_t wc = skip_t ? 0 : cn;
  const bool rin = t <= G.tf_r;
  double pg = warp_incl_scan(wg, lane), ph = warp_incl_scan(wh, lane);
  int32_t pc = warp_incl_scan(wc, lane);
  double rg = warp_incl_scan_down(rin ? wg : 0.0, lane), rh = warp_incl_scan_down(rin ? wh : 0.0, lane);
  int32_t rc = warp_incl_scan_down(rin ? wc : 0, lane);
  if (lane == 31) {
    sm.wd[2][warp] = pg;
    sm.wd[3][warp] = ph;
    sm.wc[0][warp] = pc;
  }
  if (lane == 0) {
    sm.wd[4][warp] = rg;
    sm.wd[5][warp] = rh;
    sm.wc[1][warp] = rc;
  }
  if (G.fwd_rest) {
    const double ug = warp_sum(v.x), uh = warp_sum(v.y);
    const int32_t uc = warp_sum(cn);
    if (lane == 0) {
      sm.wd[6][warp] = ug;
      sm.wd[7][warp] = uh;
      sm.wc[2][warp] = uc;
    }
  }
  __syncthreads();
  // forward scan start: nothing (with kEpsilon hessian) or everything outside the slice
  double bg = 0.0, bh = BK_EPS;
  int32_t bc = 0;
  {
    double og = 0.0, oh = 0.0, sg_ = 0.0, sh_ = 0.0, ug = 0.0, uh = 0.0;
    int32_t oc = 0, sc = 0, uc = 0;
#pragma unroll
    for (int i = 0; i < NW; ++i) {
      if (i < warp) {
        og += sm.wd[2][i];
        oh += sm.wd[3][i];
        oc += sm.wc[0][i];
      }
    }
#pragma unroll
    for (int i = NW - 1; i >= 0; --i) {
      if (i > warp) {
        sg_ += sm.wd[4][i];
        sh_ += sm.wd[5][i];
        sc += sm.wc[1][i];
      }
    }
    if (G.fwd_rest) {
#pragma unroll
      for (int i = 0; i < NW; ++i) {
        ug += sm.wd[6][i];
        uh += sm.wd[7][i];
        uc += sm.wc[2][i];
      }
      bg = sum_g - ug;
      bh = (sum_h - BK_EPS) - uh;
      bc = num_data - uc;
    }
    pg = bg + (pg + og);
    ph = bh + (ph + oh);
    pc = bc + (pc + oc);
    rg = rg + sg_;
    rh = BK_EPS + (rh + sh_);
    rc = rc + sc;
  }
  // reverse position t: right side (rg, rh, rc); forward position t: left side (pg, ph, pc); the
  // last thread holds forward position -1 when the scan starts outside the slice
  const bool xpos = G.fwd_rest && t == 32 * NW - 1;
  const bool first0 = t >= 1 - G.off && rin && !skip_t && !(rc < p.min_data || rh < p.min_hess);
  const bool brk0 = first0 && (num_data - rc < p.min_data || sum_h - rh < p.min_hess);
  const bool first1 = G.two && t <= G.t_end && !skip_t && !(pc < p.min_data || ph < p.min_hess);
  const bool brk1 = first1 && (num_data - pc < p.min_data || sum_h - ph < p.min_hess);
  const bool firstx = xpos && !(bc < p.min_data || bh < p.min_hess);
  const bool brkx = firstx && (num_data - bc < p.min_data || sum_h - bh < p.min_hess);
  const double fg = xpos ? bg : pg, fh = xpos ? bh : ph;
  const int32_t fc = xpos ? bc : pc;
  // left / right sums of both positions
  const double slg[2] = {sum_g - rg, fg}, slh[2] = {sum_h - rh, fh};
  const double srg[2] = {rg, sum_g - fg}, srh[2] = {rh, sum_h - fh};
  const int32_t lc[2] = {num_data - rc, fc}, rcn[2] = {rc, num_data - fc};
  Filt fl[2];
#pragma unroll
  for (int d = 0; d < 2; ++d) {
    const bool cand = d == 0 ? first0 : (first1 || firstx);
    Approx a{0.f, 0.f, true};
    if (PLAIN && cand)
      a = approx_from((float)slg[d], __fadd_rn((float)slh[d], C.l2f), (float)srg[d], __fadd_rn((float)srh[d], C.l2f));
    fl[d] = filt_of(cand, a, C);
  }
  publish_dir<PLAIN, NW>(sm, 0, brk0, t, fl[0], lane, warp);
  {
    Filt nat = fl[1];
    if (xpos) nat.lo = float_key(-CUDART_INF_F);
    publish_dir<PLAIN, NW>(sm, 1, brk1, t, nat, lane, warp);
  }
  if (xpos) {
    WarpFilt x;
    x.lb = brkx ? -1 : kNoneHi;
    x.ma = x.mb = fl[1].lo;
    sm.xf = x;
  }
  __syncthreads();
  int S[2];
  int32_t M[2];
  resolve_dir<PLAIN, NW>(sm, 0, false, &S[0], &M[0]);
  resolve_dir<PLAIN, NW>(sm, 1, G.fwd_rest, &S[1], &M[1]);
  const bool valid[2] = {first0 && t > S[0], xpos ? (firstx && S[1] != -1) : (first1 && t < S[1])};
  DirBest r[2];
  int rs[2] = {0, 0};
  // carried per position: the accumulated side's sums (reverse: right, forward: left)
  const int64_t ca[2] = {__double_as_longlong(rg), __double_as_longlong(fg)};
  const int64_t cb[2] = {__double_as_longlong(rh), __double_as_longlong(fh)};
  const int32_t cc[2] = {rc, fc};
  auto gain_of = [&](const QEnt& e) {
    const double ag = __longlong_as_double(e.a), ah = __longlong_as_double(e.b);
    if (e.d == 0)  // reverse: (ag, ah, c) is the right side
      return split_gains(p, sum_g - ag, sum_h - ah, ag, ah, num_data - e.c, e.c, C.parent);
    return split_gains(p, ag, ah, sum_g - ag, sum_h - ah, e.c, num_data - e.c, C.parent);
  };
  if (PLAIN) {
    // a position whose bin adds nothing repeats its scan predecessor (t + 1 reverse, t - 1 forward)
    const bool empty = wg == 0.0 && wh == 0.0 && wc == 0;
    const bool rep[2] = {empty && t + 1 <= G.tf_r && !(G.skip && t + 1 + G.off == m.default_bin),
                         !xpos && empty && ((t >= 1 && !(G.skip && t - 1 + G.off == m.default_bin)) ||
                                            (t == 0 && G.fwd_rest))};
    // barrier 3: the few positions that need their f64 gain; barrier 4: evaluated on the eight warps
#pragma unroll
    for (int d = 0; d < 2; ++d) {
      const bool exact = valid[d] && !rep[d] && (fl[d].unc || (fl[d].mp && fl[d].up >= M[d]));
      queue_push(sm, d, exact, QEnt{ca[d], cb[d], cc[d], (int16_t)(d == 0 || !xpos ? t : -1), (int16_t)d}, lane);
    }
    __syncthreads();
    eval_queues(
        sm, warp, lane, C.mgs,
        [&](const QEnt& e, int role) {
          return float_side(p, e.d, __longlong_as_double(e.a), __longlong_as_double(e.b), e.c, sum_g, sum_h,
                            num_data, role);
        },
        r, rs);
    if (warp != 0) return;
  } else {
    double gain[2];
    bool split[2], elig[2];
#pragma unroll
    for (int d = 0; d < 2; ++d) {
      gain[d] = -CUDART_INF;
      if (valid[d]) gain[d] = split_gains(p, slg[d], slh[d], srg[d], srh[d], lc[d], rcn[d], C.parent);
      const bool passed = valid[d] && gain_passes(gain[d], C.mgs);
      split[d] = passed;
      elig[d] = passed && !dnan(gain[d]) && !is_neg_inf(gain[d]);
    }
    warp_best(0, elig[0], gain[0], t, ca[0], cb[0], cc[0], lane, &sm.wb[0][warp]);
    warp_best(1, elig[1], gain[1], xpos ? -1 : t, ca[1], cb[1], cc[1], lane, &sm.wb[1][warp]);
#pragma unroll
    for (int d = 0; d < 2; ++d) {
      const int ws = __any_sync(FULL, split[d]);
      if (lane == 0) sm.spl[d][warp] = ws;
    }
    __syncthreads();
    if (warp != 0) return;
    combine_best(sm, lane, r, rs);
  }
  // FindBestThreshold's combination of the directions (feature_histogram.rs:240-357)
  finish_cand(J, p, m, si, leaf, f, G, C.mgs, r, rs, lane, [&](const DirBest& b, int d) {
    if (PLAIN) return b.ev;  // evaluated with the gain
    return eval_float(p, d, __longlong_as_double(b.a), __longlong_as_double(b.b), b.c, sum_g, sum_h, num_data,
                      C.parent, b.ev.gain, lane);
  });
}

// The bounds on d (bk_search_warp.cuh: a threshold's gain minus the leaf-wide s0) of a plain float
// threshold. With H2 = h + 2 l2 and yl, yr = hl + l2, hr + l2, d = t^2 H2 / (yl yr) where
// t = gl - (g / H2) yl, the left gradients centred on the leaf's mean: one f64 multiply-add keeps what
// cancels. Its f64 error is below 2^-50 (|gl| + |g / H2| yl); the fp32 rest, truncations of 2^-23
// included, errs less than the 44 u of LeafConst::bk1. The gain itself is taken from f64 sums, which
// round: by up to off_g, off_h (LeafConst), whatever the sums come to, so where large bins of both signs
// cancel that is far more than 2^-50 of them. One side's sum is the leaf's minus the other's, so t moves
// by at most off_g + |g / H2| off_h, and 1 / (yl yr) by a factor of up to 1 + 2 (off_h / yl + off_h / yr)
// = 1 + 2 off_h q while off_h q <= 1/4.
struct FloatLeaf {
  float r2f;  // g / H2
  int g_exp, h_exp;
};
__device__ __forceinline__ Approx bound_float(const Params& p, const Fixed& gl, const Fixed& hl, const Fixed& hr,
                                              const FloatLeaf& K, const LeafConst& C) {
  const double g = fixed_to_double(gl.lo, gl.mid, gl.hi, K.g_exp);
  double yl = fixed_to_double(hl.lo, hl.mid, hl.hi, K.h_exp);
  if (C.l2f != 0.f) yl += p.l2;  // uniform
  const float t = double_to_float(fma(-C.r2, yl, g)), ylf = double_to_float(yl);
  const float yrf = __fadd_rn(fixed_to_float(hr, K.h_exp), C.l2f);
  const float q = __fdividef(C.hs2, __fmul_rn(ylf, yrf));
  const float hq = __fmul_rn(C.off_h, q);
  float off = __fmul_rn(fmaf(fabsf(K.r2f), ylf, fabsf(double_to_float(g))), 1.7763568e-15f);  // 2^-49
  off = __fadd_rn(off, fmaf(fabsf(K.r2f), C.off_h, C.off_g));
  Approx a;
  a.g = __fmul_rn(__fmul_rn(t, t), q);
  a.e = fmaf(__fmul_rn(off, fmaf(2.0f, fabsf(t), off)), q, fmaf(a.g, fmaf(2.0f, hq, C.bk1), C.bk0));
  a.uncertain = !(__fadd_rn(a.g, a.e) < 1e30f) || C.bk1 < 0.f || !(hq <= 0.25f);
  return a;
}
__device__ __forceinline__ Filt filt_of_d(bool cand, const Approx& a, const LeafConst& C) {
  Filt f;
  f.unc = a.uncertain;
  f.mp = cand && (a.uncertain || __fadd_rn(a.g, a.e) > C.d_dn);
  f.lo = (cand && !a.uncertain) ? float_key(__fsub_rn(a.g, a.e)) : float_key(-CUDART_INF_F);
  f.up = a.uncertain ? 0 : float_key(__fadd_rn(a.g, a.e));
  return f;
}

// search_float for plain gains of a tree with fixed-point histograms (JobState::fix_ok). The bins' doubles
// are multiples of the tree's units, so one prefix scan of 96-bit integers gives the exact sums of both
// directions (the reverse side is the total minus a prefix); the validity tests compare integers, and the
// bounds come from them. The queued positions' gains are taken from f64 sums added in search_float's
// order: around an empty bin whose sum is rounding (the most frequent bin of a column without zeros gets
// the leaf's total minus the others) two thresholds are equal but for those roundings, and the choice
// should not depend on the form of the search. That leaves about 45 f64 instructions a bin, where there were
// about 110 (32 leaves x 100 features of 255 bins: 100 -> 45 us a round; 37 with exact sums throughout).
template <int NW>
__device__ void search_float_fixed(const Job& J, const Params& p, const SearchIn& si, const DevFeature& m, int side,
                                   int32_t f, int32_t leaf, SearchSmemT<NW>& sm) {
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const LeafConst& C = si.C;
  const LeafSum& S0 = si.S0;
  const int32_t num_data = side ? C.ls.num_data : S0.num_data;
  const size_t slot_stride = (size_t)p.T * p.B * TILE;
  const size_t feat_off = (size_t)(f / TILE) * p.B * TILE + (f % TILE);
  double2* pool = reinterpret_cast<double2*>(J.pool);
  double2* hs = pool + (size_t)si.sslot * slot_stride + feat_off;
  double2* hl = pool + (size_t)(side ? si.lslot : si.sslot) * slot_stride + feat_off;
  const double2 zero = make_double2(0.0, 0.0);
  const Fixed none{0u, 0u, 0u};
  const bool fix = m.mfb > 0;
  const bool in = t < m.len;
  double2 sv = (in && !(fix && t == m.mfb)) ? hs[(size_t)(t + 1) * TILE] : zero;
  const double2 lv = (side && in) ? pool[(size_t)si.lslot * slot_stride + feat_off + (size_t)(t + 1) * TILE] : zero;
  const ScanGeom G = scan_geom(m);
  FloatLeaf K;
  K.g_exp = fixed_unit(p, J.st->red_maxg);
  K.h_exp = fixed_unit(p, J.st->red_maxh);
  K.r2f = double_to_float(C.r2);
  if (t < 2) sm.qn[t] = 0;
  const double sum_g = C.sum_g, sum_h = C.sum_h;
  if (fix) {  // FixHistogram: the smaller leaf's most frequent bin is its total minus every other bin
    const double ag = warp_sum(sv.x), ah = warp_sum(sv.y);
    if (lane == 0) {
      sm.wd[0][warp] = ag;
      sm.wd[1][warp] = ah;
    }
    __syncthreads();
    if (t == m.mfb) {
      double a = 0.0, b = 0.0;
#pragma unroll 1
      for (int i = 0; i < NW; ++i) {
        a += sm.wd[0][i];
        b += sm.wd[1][i];
      }
      sv = make_double2(S0.sg - a, S0.sh - b);
      if (side == 0) hs[(size_t)(t + 1) * TILE] = sv;
    }
  }
  const double2 v = side ? make_double2(lv.x - sv.x, lv.y - sv.y) : sv;
  if (side && in) hl[(size_t)(t + 1) * TILE] = v;
  const int32_t cn = in ? round_int(v.y * C.cnt_factor) : 0;
  const bool skip_t = G.skip && t + G.off == m.default_bin, rin = t <= G.tf_r;
  const Fixed vg = double_to_fixed(v.x, K.g_exp), vh = double_to_fixed(v.y, K.h_exp);
  // one scan: the bins that the reverse scan accumulates, which are also those of every forward prefix
  const bool acc = rin && !skip_t;
  const Fixed wg = acc ? vg : none, wh = acc ? vh : none;
  const int32_t wc = acc ? cn : 0;
  Fixed pg = wg, ph = wh;
  int32_t pc = wc;
#pragma unroll 1
  for (int o = 1; o < 32; o <<= 1) {
    const Fixed a = shfl_up_fixed(pg, o, 32), b = shfl_up_fixed(ph, o, 32);
    const int32_t c = __shfl_up_sync(FULL, pc, o);
    if (lane >= o) {
      pg = pg + a;
      ph = ph + b;
      pc += c;
    }
  }
  // the f64 sums that a queued position's gain is taken from, as search_float adds them
  double qg[2] = {acc ? v.x : 0.0, 0.0}, qh[2] = {acc ? v.y : 0.0, 0.0};
  if (G.two) {  // uniform
    qg[1] = warp_incl_scan(skip_t ? 0.0 : v.x, lane);
    qh[1] = warp_incl_scan(skip_t ? 0.0 : v.y, lane);
    if (lane == 31) {
      sm.wd[2][warp] = qg[1];
      sm.wd[3][warp] = qh[1];
    }
    if (G.fwd_rest) {
      const double ug = warp_sum(v.x), uh = warp_sum(v.y);
      if (lane == 0) {
        sm.wd[6][warp] = ug;
        sm.wd[7][warp] = uh;
      }
    }
  }
  qg[0] = warp_incl_scan_down(qg[0], lane);
  qh[0] = warp_incl_scan_down(qh[0], lane);
  if (lane == 0) {
    sm.wd[4][warp] = qg[0];
    sm.wd[5][warp] = qh[0];
  }
  if (lane == 31) {
    sm.fx[0][warp] = pg;
    sm.fx[1][warp] = ph;
    sm.fx[2][warp] = Fixed{(uint32_t)pc, 0u, 0u};
  }
  if (G.fwd_rest && t == G.tf_r + 1) {  // the NaN bin: with the scanned ones, the whole slice
    sm.top[0] = vg;
    sm.top[1] = vh;
    sm.top[2] = Fixed{(uint32_t)cn, 0u, 0u};
  }
  __syncthreads();
  // lane 8 q + w: the prefix of quantity q over warps 0 .. w
  Fixed tg, th;
  int32_t tc;
  {
    const int q = lane >> 3, w = lane & 7;
    Fixed x = (q < 3 && w < NW) ? sm.fx[q][w] : none;
#pragma unroll 1
    for (int o = 1; o < 8; o <<= 1) {
      const Fixed y = shfl_up_fixed(x, o, 8);
      if (w >= o) x = x + y;
    }
    tg = shfl_fixed(x, 7);
    th = shfl_fixed(x, 15);
    tc = (int32_t)__shfl_sync(FULL, x.lo, 23);
    const int before = max(warp - 1, 0);
    const Fixed a = shfl_fixed(x, before), b = shfl_fixed(x, 8 + before);
    const int32_t c = (int32_t)__shfl_sync(FULL, x.lo, 16 + before);
    if (warp > 0) {
      pg = pg + a;
      ph = ph + b;
      pc += c;
    }
  }
  // right sums of reverse position t, left sums of forward position t (and of the forward position -1,
  // held by the last thread), the hessians without their kEpsilon
  const Fixed lg = double_to_fixed(sum_g, K.g_exp), lh = double_to_fixed(C.ls.sh, K.h_exp);
  const Fixed need = double_to_fixed(p.min_hess - BK_EPS, K.h_exp);
  const Fixed rg = tg - (pg - wg), rh = th - (ph - wh);
  const int32_t rc = tc - (pc - wc);
  Fixed fg = pg, fh = ph, bh = none;
  int32_t fc = pc, bc = 0;
  const bool xpos = G.fwd_rest && t == 32 * NW - 1;
  if (G.fwd_rest) {  // the forward scan starts with everything outside the slice
    const Fixed bg = lg - (tg + sm.top[0]);
    bh = lh - (th + sm.top[1]);
    bc = num_data - (tc + (int32_t)sm.top[2].lo);
    fg = xpos ? bg : bg + pg;
    fh = xpos ? bh : bh + ph;
    fc = xpos ? bc : bc + pc;
  }
  const bool first0 = t >= 1 - G.off && rin && !skip_t && !(rc < p.min_data || rh < need);
  const bool brk0 = first0 && (num_data - rc < p.min_data || lh - rh < need);
  const bool fok = !(fc < p.min_data || fh < need);
  const bool first1 = G.two && !xpos && t <= G.t_end && !skip_t && fok;
  const bool firstx = xpos && fok;
  const bool brkf = num_data - fc < p.min_data || lh - fh < need;
  const bool brk1 = first1 && brkf, brkx = firstx && brkf;
  Filt fl[2];
  {
    Approx a{0.f, 0.f, true};
    if (first0) a = bound_float(p, lg - rg, lh - rh, rh, K, C);
    fl[0] = filt_of_d(first0, a, C);
  }
  publish_dir<true, NW>(sm, 0, brk0, t, fl[0], lane, warp);
  {
    Approx a{0.f, 0.f, true};
    if (first1 || firstx) a = bound_float(p, fg, fh, lh - fh, K, C);
    fl[1] = filt_of_d(first1 || firstx, a, C);
    Filt nat = fl[1];
    if (xpos) nat.lo = float_key(-CUDART_INF_F);
    publish_dir<true, NW>(sm, 1, brk1, t, nat, lane, warp);
  }
  if (xpos) {
    WarpFilt x;
    x.lb = brkx ? -1 : kNoneHi;
    x.ma = x.mb = fl[1].lo;
    sm.xf = x;
  }
  __syncthreads();
  int S[2];
  int32_t M[2];
  resolve_dir<true, NW>(sm, 0, false, &S[0], &M[0]);
  resolve_dir<true, NW>(sm, 1, G.fwd_rest, &S[1], &M[1]);
  const bool valid[2] = {first0 && t > S[0], xpos ? (firstx && S[1] != -1) : (first1 && t < S[1])};
  // a position whose bin adds nothing repeats its scan predecessor (t + 1 reverse, t - 1 forward)
  const bool empty = (wg.lo | wg.mid | wg.hi | wh.lo | wh.mid | wh.hi) == 0u && wc == 0;
  const bool rep[2] = {empty && t + 1 <= G.tf_r && !(G.skip && t + 1 + G.off == m.default_bin),
                       !xpos && empty && ((t >= 1 && !(G.skip && t - 1 + G.off == m.default_bin)) ||
                                          (t == 0 && G.fwd_rest))};
#pragma unroll
  for (int d = 0; d < 2; ++d) {
    const bool exact = valid[d] && !rep[d] && (fl[d].unc || (fl[d].mp && fl[d].up >= M[d]));
    QEnt e{0, 0, 0, 0, 0};
    if (exact) {  // the accumulated side (reverse: right, forward: left): the other warps' part
      double ag = 0.0, ah = 0.0;
      if (d == 0) {
#pragma unroll 1
        for (int i = NW - 1; i > warp; --i) {
          ag += sm.wd[4][i];
          ah += sm.wd[5][i];
        }
        ag = qg[0] + ag;
        ah = BK_EPS + (qh[0] + ah);
      } else {
#pragma unroll 1
        for (int i = 0; i < warp; ++i) {
          ag += sm.wd[2][i];
          ah += sm.wd[3][i];
        }
        double bg = 0.0, bhd = BK_EPS;
        if (G.fwd_rest) {
          double ug = 0.0, uh = 0.0;
#pragma unroll 1
          for (int i = 0; i < NW; ++i) {
            ug += sm.wd[6][i];
            uh += sm.wd[7][i];
          }
          bg = sum_g - ug;
          bhd = (sum_h - BK_EPS) - uh;
        }
        ag = xpos ? bg : bg + (qg[1] + ag);
        ah = xpos ? bhd : bhd + (qh[1] + ah);
      }
      e.a = __double_as_longlong(ag);
      e.b = __double_as_longlong(ah);
      e.c = d == 0 ? rc : fc;
      e.t = (int16_t)(d == 0 || !xpos ? t : -1);
      e.d = (int16_t)d;
    }
    queue_push(sm, d, exact, e, lane);
  }
  __syncthreads();
  DirBest r[2];
  int rs[2] = {0, 0};
  eval_queues(
      sm, warp, lane, C.mgs,
      [&](const QEnt& e, int role) {
        return float_side(p, e.d, __longlong_as_double(e.a), __longlong_as_double(e.b), e.c, sum_g, sum_h, num_data,
                          role);
      },
      r, rs);
  if (warp != 0) return;
  finish_cand(J, p, m, si, leaf, f, G, C.mgs, r, rs, lane, [&](const DirBest& b, int) { return b.ev; });
}

// The float search of one (leaf, feature).
template <bool PLAIN, int NW>
__device__ __forceinline__ void search_float_any(const Job& J, const Params& p, const SearchIn& si, const DevFeature& m,
                                                 int side, int32_t f, int32_t leaf, SearchSmemT<NW>& sm) {
  if constexpr (PLAIN) {
    if (J.st->fix_ok) {  // uniform
      search_float_fixed<NW>(J, p, si, m, side, f, leaf, sm);
      return;
    }
  }
  search_float<PLAIN, NW>(J, p, si, m, side, f, leaf, sm);
}

// ---- categorical features (feature_histogram.rs:1328-1886) ----
// One CTA per (leaf side, feature) as for numerical features; thread t holds slice index t. The
// histogram slice is loaded, fixed and (larger side) derived by subtraction exactly as the
// numerical searches do, so the pool holds the same values afterwards. Then:
//   one-hot (num_bin <= max_cat_to_onehot): every category's split against the rest is evaluated
//     by its own thread; the first best in category order wins;
//   sorted: the categories with enough data are ranked by grad / (hess + cat_smooth) (a stable
//     rank over order-preserving integer keys, ties by category), one thread per direction walks
//     the reference's sequential scan (its sums, counts, skips and breaks do not depend on the
//     gains) and queues the positions that need a gain, which the CTA then evaluates in parallel;
//     the first best in scan order (ascending direction first) wins.
// Gains and outputs use lambda_l2 + cat_l2 in the sorted form, as the reference does.
constexpr int kCatQueue = kSearchThreads / 2;  // queued positions per direction: max_num_cat <= 128

// The categorical search's shared memory, overlaid on the numerical search's (a CTA runs one or
// the other). V: int64_t (quantized, integer sums) or double (float path).
template <typename V>
struct CatSmem {
  V a[kSearchThreads], b[kSearchThreads];  // per-bin gradient / hessian sums
  int32_t cnt[kSearchThreads];
  long long key[kSearchThreads];
  int16_t sorted[kSearchThreads];
  V qa[2][kCatQueue], qb[2][kCatQueue];    // queued positions: the accumulated left side's sums
  int32_t qlc[2][kCatQueue], qi[2][kCatQueue];
  int32_t qn[2];
  long long wk[kSearchWarps];
  int32_t wo[kSearchWarps], wsp[kSearchWarps];
  int64_t wi[kSearchWarps];
  double wd[2][kSearchWarps];
  double best_gain;
};

__device__ __forceinline__ long long cat_block_max(long long v, long long* w, int lane, int warp) {
  v = warp_max64(v);
  if (lane == 0) w[warp] = v;
  __syncthreads();
  long long r = w[0];
#pragma unroll
  for (int i = 1; i < kSearchWarps; ++i) r = w[i] > r ? w[i] : r;
  __syncthreads();
  return r;
}

__device__ __forceinline__ int32_t cat_block_min(int32_t v, int32_t* w, int lane, int warp) {
  v = __reduce_min_sync(FULL, v);
  if (lane == 0) w[warp] = v;
  __syncthreads();
  int32_t r = w[0];
#pragma unroll
  for (int i = 1; i < kSearchWarps; ++i) r = w[i] < r ? w[i] : r;
  __syncthreads();
  return r;
}

__device__ __forceinline__ int32_t cat_block_or(int32_t v, int32_t* w, int lane, int warp) {
  v = (int32_t)__reduce_or_sync(FULL, (unsigned)v);
  if (lane == 0) w[warp] = v;
  __syncthreads();
  int32_t r = 0;
#pragma unroll
  for (int i = 0; i < kSearchWarps; ++i) r |= w[i];
  __syncthreads();
  return r;
}

// The scan of one direction on one warp (feature_histogram.rs:1666-1760): the positions whose gain is
// needed. Sums and counts only grow along the scan, so the positions before the first that has enough
// data on its left are skipped and the scan ends at the first whose right side has too little; between
// them a position is taken when min_data_per_group rows have come since the last one taken. (One thread
// walking it took 5 of a search's 28 us: a chain of f64 conversions and comparisons.)
__device__ __forceinline__ void cat_scan_int(const Params& p, CatSmem<int64_t>& cs, int d, int32_t used_bin,
                                             int32_t max_num_cat, int32_t num_data, int64_t thi, double hsc, int lane) {
  int64_t g0 = 0, h0 = 0;
  int32_t c0 = 0, taken = 0, q = 0;
  const int32_t n = min(used_bin, max_num_cat);
  for (int32_t i0 = 0; i0 < n; i0 += 32) {
    const int32_t i = i0 + lane;
    int64_t g = 0, h = 0;
    int32_t c = 0;
    if (i < n) {
      const int32_t b = cs.sorted[d == 0 ? i : used_bin - 1 - i];
      g = cs.a[b];
      h = cs.b[b];
      c = cs.cnt[b];
    }
    const int32_t own = c;
    g = g0 + warp_incl_scan(g, lane);
    h = h0 + warp_incl_scan(h, lane);
    c = c0 + warp_incl_scan(c, lane);
    const bool enough = i < n && !(c < p.min_data || (double)h * hsc < p.min_hess);
    const int32_t rc = num_data - c;
    const bool stop = enough && (rc < p.min_data || rc < p.min_data_per_group || (double)(thi - h) * hsc < p.min_hess);
    const unsigned stops = __ballot_sync(FULL, stop);
    const unsigned open = __ballot_sync(FULL, enough) & (stops ? (stops & (0u - stops)) - 1u : FULL);
    // every open position is taken where each brings enough rows by itself
    unsigned take = open;
    if (__any_sync(FULL, ((open >> lane) & 1u) && own < p.min_data_per_group)) {
      take = 0u;
      int32_t last = taken;
      for (unsigned left = open; left;) {
        const unsigned ready = __ballot_sync(FULL, ((left >> lane) & 1u) && c - last >= p.min_data_per_group);
        if (!ready) break;
        const int k = __ffs(ready) - 1;
        take |= 1u << k;
        last = __shfl_sync(FULL, c, k);
        left = k == 31 ? 0u : left & ~((2u << k) - 1u);
      }
    }
    if ((take >> lane) & 1u) {
      const int32_t at = q + __popc(take & ((1u << lane) - 1u));
      if (at < kCatQueue) {
        cs.qa[d][at] = g;
        cs.qb[d][at] = h;
        cs.qlc[d][at] = c;
        cs.qi[d][at] = i;
      }
    }
    if (take) taken = __shfl_sync(FULL, c, 31 - __clz((int)take));
    q += __popc(take);
    if (stops) break;
    g0 = __shfl_sync(FULL, g, 31);
    h0 = __shfl_sync(FULL, h, 31);
    c0 = __shfl_sync(FULL, c, 31);
  }
  if (lane == 0) cs.qn[d] = min(q, kCatQueue);
}

template <bool QUANT>
__device__ void search_cat(const Job& J, const Params& p, const SearchIn& si, const DevFeature& m, int side,
                           int32_t f, int32_t leaf, SearchSmem& sm) {
  using V = typename std::conditional<QUANT, int64_t, double>::type;
  static_assert(sizeof(CatSmem<V>) <= sizeof(SearchSmem), "the categorical search fits the search's shared memory");
  CatSmem<V>& cs = *reinterpret_cast<CatSmem<V>*>(&sm);
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const LeafConst& C = si.C;
  const LeafSum& S0 = si.S0;
  const LeafSum& SL = C.ls;
  const int32_t num_data = SL.num_data;
  const size_t slot_stride = (size_t)p.T * p.B * TILE;
  const size_t feat_off = (size_t)(f / TILE) * p.B * TILE + (f % TILE);
  const bool fix = m.mfb > 0;
  const bool in = t < m.len;
  // -- the slice: FixHistogram of the smaller leaf, the larger as parent minus smaller (serial.rs:
  //    1407-1437, 2205-2238), written back exactly as the numerical searches write it --
  if (QUANT) {
    int64_t* pool = reinterpret_cast<int64_t*>(J.pool);
    int64_t* hs = pool + (size_t)si.sslot * slot_stride + feat_off;
    int64_t* hl = pool + (size_t)(side ? si.lslot : si.sslot) * slot_stride + feat_off;
    const int64_t sv = (in && !(fix && t == m.mfb)) ? hs[(size_t)(t + 1) * TILE] : 0;
    const int64_t lv = (side && in) ? pool[(size_t)si.lslot * slot_stride + feat_off + (size_t)(t + 1) * TILE] : 0;
    int64_t v = side ? lv - sv : sv;
    if (fix) {
      const int64_t a = warp_sum(sv);
      if (lane == 0) cs.wi[warp] = a;
      __syncthreads();
      int64_t aux = 0;
#pragma unroll
      for (int i = 0; i < kSearchWarps; ++i) aux += cs.wi[i];
      const int64_t fixed = S0.int_sum - aux;  // the leaf total minus every other bin
      if (t == m.mfb) {
        v += side ? -fixed : fixed;
        if (side == 0) hs[(size_t)(t + 1) * TILE] = fixed;
      }
    }
    if (side && in) hl[(size_t)(t + 1) * TILE] = v;
    cs.a[t] = in ? unpack_g(v) : 0;
    cs.b[t] = in ? unpack_h(v) : 0;
    cs.cnt[t] = in ? round_int((double)unpack_h(v) * C.cnt_factor) : 0;
  } else {
    double2* pool = reinterpret_cast<double2*>(J.pool);
    double2* hs = pool + (size_t)si.sslot * slot_stride + feat_off;
    double2* hl = pool + (size_t)(side ? si.lslot : si.sslot) * slot_stride + feat_off;
    const double2 zero = make_double2(0.0, 0.0);
    double2 sv = (in && !(fix && t == m.mfb)) ? hs[(size_t)(t + 1) * TILE] : zero;
    const double2 lv = (side && in) ? pool[(size_t)si.lslot * slot_stride + feat_off + (size_t)(t + 1) * TILE] : zero;
    if (fix) {
      const double ag = warp_sum(sv.x), ah = warp_sum(sv.y);
      if (lane == 0) {
        cs.wd[0][warp] = ag;
        cs.wd[1][warp] = ah;
      }
      __syncthreads();
      double tg = 0.0, th = 0.0;
#pragma unroll
      for (int i = 0; i < kSearchWarps; ++i) {
        tg += cs.wd[0][i];
        th += cs.wd[1][i];
      }
      if (t == m.mfb) {
        sv = make_double2(S0.sg - tg, S0.sh - th);
        if (side == 0) hs[(size_t)(t + 1) * TILE] = sv;
      }
    }
    const double2 v = side ? make_double2(lv.x - sv.x, lv.y - sv.y) : sv;
    if (side && in) hl[(size_t)(t + 1) * TILE] = v;
    cs.a[t] = in ? v.x : 0.0;
    cs.b[t] = in ? v.y : 0.0;
    cs.cnt[t] = in ? round_int(v.y * C.cnt_factor) : 0;
  }
  if (t < 2) cs.qn[t] = 0;
  __syncthreads();
  // -- the leaf's totals and min_gain_shift (feature_histogram.rs:1347-1386, :1614-1665) --
  const int64_t l_int = side ? SL.int_sum : S0.int_sum;
  const int64_t tgi = unpack_g(l_int), thi = unpack_h(l_int);
  const double gs = C.gs, hsc = C.hs;
  const double sum_g = C.sum_g, sum_h = C.sum_h;  // float path: sum_h includes 2 kEpsilon
  const double mgs =
      p.use_smooth ? leaf_gain_given_output(p.use_l1, sum_g, sum_h, p, C.parent) + p.min_gain : C.mgs;
  const int32_t bin_start = 1 - m.offset, bin_end = m.num_bin - m.offset;
  const bool onehot = m.num_bin <= p.max_cat_to_onehot;
  Params pl = p;
  int32_t best_dir = 0, best_i = -1, used_bin = 0, sp = 0;
  double best_gain = -CUDART_INF;
  // the chosen position's left side
  double blg = 0.0, blh = 0.0;
  int64_t big = 0, bih = 0;
  int32_t blc = 0;
  if (onehot) {
    // -- one category against the rest, thread t = category t --
    bool pass = false;
    double gain = -CUDART_INF;
    if (t >= bin_start && t < bin_end) {
      const int32_t cnt = cs.cnt[t];
      if (QUANT) {
        const int64_t ig = (int64_t)cs.a[t], ih = (int64_t)cs.b[t];
        const double h = (double)ih * hsc;
        const int32_t other_cnt = num_data - cnt;
        const double other_h = (double)(thi - ih) * hsc;
        if (!(cnt < p.min_data || h < p.min_hess) && other_cnt >= p.min_data && !(other_h < p.min_hess)) {
          const double g = (double)ig * gs, other_g = (double)(tgi - ig) * gs;
          gain = split_gains(pl, other_g, other_h, g, h, other_cnt, cnt, C.parent);
          pass = gain > mgs;
        }
      } else {
        const double g = (double)cs.a[t], h = (double)cs.b[t];
        const int32_t other_cnt = num_data - cnt;
        const double other_h = sum_h - h - BK_EPS;
        if (!(cnt < p.min_data || h < p.min_hess) && other_cnt >= p.min_data && !(other_h < p.min_hess)) {
          const double other_g = sum_g - g;
          gain = split_gains(pl, other_g, other_h, g, h + BK_EPS, other_cnt, cnt, C.parent);
          pass = gain > mgs;
        }
      }
    }
    sp = cat_block_or(pass ? 1 : 0, cs.wsp, lane, warp);
    const long long k = cat_block_max(pass ? dkey(gain) : kNoKey, cs.wk, lane, warp);
    if (k != kNoKey) {
      // the first category (in order) with the best gain
      const int32_t first = cat_block_min(pass && dkey(gain) == k ? t : 0x7fffffff, cs.wo, lane, warp);
      if (t == first) cs.best_gain = gain;
      __syncthreads();
      best_gain = cs.best_gain;
      best_i = first;
      blc = cs.cnt[first];
      if (QUANT) {
        big = (int64_t)cs.a[first];
        bih = (int64_t)cs.b[first];
      } else {
        blg = (double)cs.a[first];
        blh = (double)cs.b[first] + BK_EPS;
      }
    }
    if (warp != 0) return;
  } else {
    // -- the categories with enough data, ranked by grad / (hess + cat_smooth) --
    const bool elig = t >= bin_start && t < bin_end && (double)cs.cnt[t] >= p.cat_smooth;
    double ctr = 0.0;
    if (elig) {
      if (QUANT) ctr = ((double)cs.a[t] * gs) / ((double)cs.b[t] * hsc + p.cat_smooth);
      else ctr = (double)cs.a[t] / ((double)cs.b[t] + p.cat_smooth);
    }
    cs.key[t] = elig ? dkey(ctr) : kNoKey;
    const int32_t ne = __popc(__ballot_sync(FULL, elig));
    if (lane == 0) cs.wo[warp] = ne;
    __syncthreads();
    used_bin = 0;
#pragma unroll
    for (int i = 0; i < kSearchWarps; ++i) used_bin += cs.wo[i];
    if (elig) {
      const long long kt = cs.key[t];
      int32_t rank = 0;
#pragma unroll 4
      for (int u = 0; u < m.len; ++u) {  // no category past the slice is eligible
        const long long ku = cs.key[u];
        rank += (ku != kNoKey && (ku < kt || (ku == kt && u < t))) ? 1 : 0;
      }
      cs.sorted[rank] = (int16_t)t;
    }
    pl.l2 = p.l2 + p.cat_l2;
    __syncthreads();
    const int32_t max_num_cat = min(p.max_cat_threshold, (used_bin + 1) / 2);
    // -- the sequential scans: one warp per direction (warp 0 ascending, warp 1 descending), integer
    //    sums by prefix scans; f64 sums one thread per direction, in order --
    if constexpr (QUANT) {
      if (warp < 2) cat_scan_int(p, cs, warp, used_bin, max_num_cat, num_data, thi, hsc, lane);
    } else if ((t == 0 || t == 32) && used_bin > 0) {
      const int d = t == 0 ? 0 : 1;
      const int dir = d == 0 ? 1 : -1;
      int32_t pos = d == 0 ? 0 : used_bin - 1, cnt_group = 0, left_cnt = 0, q = 0;
      double lg = 0.0, lh = BK_EPS;
      for (int32_t i = 0; i < used_bin && i < max_num_cat; ++i) {
        const int32_t c = cs.sorted[pos];
        pos += dir;
        const int32_t cnt = cs.cnt[c];
        left_cnt += cnt;
        cnt_group += cnt;
        lg += (double)cs.a[c];
        lh += (double)cs.b[c];
        if (left_cnt < p.min_data || lh < p.min_hess) continue;
        const int32_t right_cnt = num_data - left_cnt;
        if (right_cnt < p.min_data || right_cnt < p.min_data_per_group) break;
        if (sum_h - lh < p.min_hess) break;
        if (cnt_group < p.min_data_per_group) continue;
        cnt_group = 0;
        if (q < kCatQueue) {
          cs.qa[d][q] = (V)lg;
          cs.qb[d][q] = (V)lh;
          cs.qlc[d][q] = left_cnt;
          cs.qi[d][q] = i;
          ++q;
        }
      }
      cs.qn[d] = q;
    }
    __syncthreads();
    // -- the queued gains, one thread each: direction 0 on threads 0..127, direction 1 on 128..255 --
    const int d = t >> 7, j = t & 127;
    bool pass = false;
    double gain = -CUDART_INF;
    if (j < cs.qn[d]) {
      const int32_t lc = cs.qlc[d][j], rc = num_data - lc;
      if (QUANT) {
        const int64_t lig = (int64_t)cs.qa[d][j], lih = (int64_t)cs.qb[d][j];
        const double lg = (double)lig * gs, lh = (double)lih * hsc;
        const double rg = (double)(tgi - lig) * gs, rh = (double)(thi - lih) * hsc;
        gain = split_gains(pl, lg, lh, rg, rh, lc, rc, C.parent);
      } else {
        const double lg = (double)cs.qa[d][j], lh = (double)cs.qb[d][j];
        gain = split_gains(pl, lg, lh, sum_g - lg, sum_h - lh, lc, rc, C.parent);
      }
      pass = gain > mgs;
    }
    sp = cat_block_or(pass ? 1 : 0, cs.wsp, lane, warp);
    const long long k = cat_block_max(pass ? dkey(gain) : kNoKey, cs.wk, lane, warp);
    if (k != kNoKey) {
      // scan order: direction 0 before direction 1, then the position
      const int32_t first = cat_block_min(pass && dkey(gain) == k ? t : 0x7fffffff, cs.wo, lane, warp);
      best_dir = first >> 7;
      const int32_t bj = first & 127;
      best_i = cs.qi[best_dir][bj];
      if (QUANT) {
        big = (int64_t)cs.qa[best_dir][bj];
        bih = (int64_t)cs.qb[best_dir][bj];
      } else {
        blg = (double)cs.qa[best_dir][bj];
        blh = (double)cs.qb[best_dir][bj];
      }
      blc = cs.qlc[best_dir][bj];
      if (t == first) cs.best_gain = gain;
      __syncthreads();
      best_gain = cs.best_gain;
    }
    if (warp != 0) return;
  }
  // -- warp 0: the SplitInfo of the chosen position (feature_histogram.rs:1537-1598, :1828-1886) --
  Cand c;
  cand_reset(&c, m.real, f);
  c.default_left = 0;
  c.categorical = 1;
  uint32_t word = 0u;  // lane w: word w of the left bins' bitset
  if (sp && best_i >= 0) {
    if (QUANT) {
      const double lg = (double)big * gs, lh = (double)bih * hsc;
      const int64_t rig = tgi - big, rih = thi - bih;
      const double rg = (double)rig * gs, rh = (double)rih * hsc;
      const int32_t lc = round_int((double)bih * C.cnt_factor), rc = round_int((double)rih * C.cnt_factor);
      c.left_output = split_output(pl, lg, lh, lc, C.parent);
      c.right_output = split_output(pl, rg, rh, rc, C.parent);
      c.left_count = lc;
      c.right_count = rc;
      c.lsg = lg;
      c.lsh = lh;
      c.rsg = rg;
      c.rsh = rh;
      c.lint = (int64_t)(((uint64_t)big << 32) | ((uint64_t)bih & 0xffffffffULL));
      c.rint = (int64_t)(((uint64_t)rig << 32) | ((uint64_t)rih & 0xffffffffULL));
    } else {
      c.left_output = split_output(pl, blg, blh, blc, C.parent);
      c.right_output = split_output(pl, sum_g - blg, sum_h - blh, num_data - blc, C.parent);
      c.left_count = blc;
      c.right_count = num_data - blc;
      c.lsg = blg;
      c.lsh = blh - BK_EPS;
      c.rsg = sum_g - blg;
      c.rsh = sum_h - blh - BK_EPS;
    }
    c.gain = best_gain - mgs;
    // the bins that go left: the category itself (one-hot) or the first best_i + 1 categories of
    // the chosen scan direction; lane w collects word w of the bitset
    if (onehot) {
      const uint32_t b = (uint32_t)(best_i + m.offset);
      if ((int)(b >> 5) == lane) word |= 1u << (b & 31);
    } else {
      for (int32_t i0 = 0; i0 <= best_i; i0 += 32) {  // 32 categories at a time
        const int32_t i = i0 + lane, pos = best_dir == 0 ? i : used_bin - 1 - i;
        const uint32_t b = i <= best_i ? (uint32_t)(cs.sorted[pos] + m.offset) : 0xffffffffu;
#pragma unroll
        for (uint32_t w = 0; w < 8; ++w) {
          const uint32_t bits = __reduce_or_sync(FULL, (b >> 5) == w ? 1u << (b & 31u) : 0u);
          if ((int)w == lane) word |= bits;
        }
      }
    }
  }
  c.gain *= m.penalty;
  c.splittable = sp;
  c.missing = m.missing;
  if (lane == 0) store_cand(J, p, si, leaf, f, c);
  if (lane < 8) cand_cat_bits(J, p, leaf, f)[lane] = word;
}

// One CTA per (feature, side): blockIdx.x = 2 * feature + side (0 = smaller leaf). With `decide`,
// the last CTA to finish runs the fold / arg-max and records the split; otherwise the single-pass
// partition that follows decides it.
// NW warps per CTA: 8 for features of up to 256 group bins; 2 (64 threads) when every feature
// has at most 64, so a CTA holds what a small-bin feature needs and four times as many CTAs fit
// on an SM. Only NW = 8 takes categorical features and the stable path's last-CTA decision
// (both use 256 threads); the host picks NW accordingly.
// post: the histogram launch before this one applied a single-pass split's bookkeeping.
template <bool PLAIN, bool QUANT, int NW>
__global__ void __launch_bounds__(32 * NW) k_search(const JobTable jobs, Params p,
                                                    const DevFeature* __restrict__ feats, int clear_par,
                                                    int decide, int post) {
  __shared__ SearchSmemT<NW> sm;
  __shared__ int last;
  __shared__ Decision dec;
  const int side = (int)(blockIdx.x & 1u);
  const int f = (int)(blockIdx.x >> 1);
  const DevFeature m = feats[f];  // static: loaded while the histogram launch finishes
  const Job& J = jobs.job[blockIdx.z];
  JobState* st = J.st;
  // The two leaves' pool slots, read while the histogram launch finishes: this launch starts only
  // after every histogram CTA has passed its own wait, so the launches before that one are
  // complete. After a single-pass split the smaller child takes the slot the decision recorded
  // and the larger one keeps its parent's (split_pslot); otherwise the state's slots were written
  // before the histogram launch started. The state's own slots, read after the wait, confirm them
  // (a mismatch reloads); clamped, an early slot only ever addresses the pool.
  int32_t pre_s = -1, pre_l = -1;
  if (QUANT && !m.cat) {
    pre_s = __ldcg(post ? &st->split_sslot : &st->smaller_slot);
    pre_l = __ldcg(post ? &st->split_pslot : &st->larger_slot);
  }
  griddep_wait();
  // the partition may be scheduled now: its CTAs read their static data while this search runs,
  // and wait for its completion before reading anything it writes
  griddep_launch();
  if (clear_par >= 0 && blockIdx.x == 0 && threadIdx.x < 2) {
    // the single-pass partition counter pair of the split after next: its last reader, the
    // histogram launch before this one, has finished
    st->pcnt[clear_par][threadIdx.x] = 0;
  }
  // one round of independent loads: the state, the feature's flag, both leaves' constants and
  // (integer search) this thread's pool entries at the early slots
  const int32_t stop = st->stop, do_search = st->do_search;
  const int32_t leaf = side ? st->larger_leaf : st->smaller_leaf;
  const uint8_t used = J.used[f];
  SearchIn si;
  si.sslot = st->smaller_slot;
  si.lslot = st->larger_slot;
  si.group = -1;
  si.crow = side;
  si.C = J.lconst[side];
  si.S0 = side ? J.lconst[0].ls : si.C.ls;
  si.pre = false;
  if (QUANT && !m.cat) {
    const bool ok_s = (unsigned)pre_s < (unsigned)p.num_leaves, ok_l = (unsigned)pre_l < (unsigned)p.num_leaves;
    const IntPool pv = int_pool(J, p, m, side, f, ok_s ? pre_s : 0, ok_l ? pre_l : 0);
    si.sv = pv.sv;
    si.lv = pv.lv;
    si.pre = ok_s && pre_s == si.sslot && (side == 0 || (ok_l && pre_l == si.lslot));
  }
  if (stop) return;  // uniform over the grid
  if (do_search && used && leaf >= 0) {  // uniform over the CTA
    if constexpr (NW == kSearchWarps) {
      if (m.cat) {
        search_cat<QUANT>(J, p, si, m, side, f, leaf, sm);
      } else if (QUANT) {
        search_int<PLAIN>(J, p, si, m, side, f, leaf, sm);
      } else {
        search_float_any<PLAIN>(J, p, si, m, side, f, leaf, sm);
      }
    } else {
      if (QUANT) search_int<PLAIN>(J, p, si, m, side, f, leaf, sm);
      else search_float_any<PLAIN>(J, p, si, m, side, f, leaf, sm);
    }
  }
  if constexpr (NW != kSearchWarps) return;  // the host gives the decision to a 256-thread launch
  if (!decide) return;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    unsigned c = atomicAdd(&st->search_done, 1u);
    last = c == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  decide_split(J, p, feats, true, &dec);
  if (threadIdx.x == 0) st->search_done = 0u;
}

// The search of a grow round (bk_rounds.cuh): blockIdx.x = 2 * feature group + side, blockIdx.y = the
// expansion. The expansion and, on the quantized path, the parent's bins are read while the histogram
// launch finishes: both were written before it.
// WARP: groups of kWarpFeatures numerical features, a warp each (bk_search_warp.cuh), then one
// categorical feature per CTA; otherwise one feature per CTA in the form of k_search.
struct RoundSearch {
  const RoundHdr* hdr;
  RoundExp c;
  int32_t stop;
  bool active;
};

__device__ __forceinline__ RoundSearch round_search_load(const Job& J, const Params& p, int q, int e) {
  const RoundView v = round_view(J, p);
  RoundSearch r;
  r.hdr = v.hdr + q;
  const int32_t n_cur = __ldcg(&r.hdr->n_cur);
  r.stop = __ldcg(&r.hdr->stop);
  r.active = e < n_cur;
  r.c.x = -1;
  r.c.node = r.c.slot = r.c.sslot = 0;
  if (r.active) r.c = v.cur[q * kMaxRoundW + e];
  return r;
}

// Whether feature f is searched for the expansion's children.
__device__ __forceinline__ bool round_used(const Job& J, const Params& p, const RoundExp& c, int f) {
  return J.tree_mask[f] && (c.x < 0 || __ldcg(&J.splittable[(size_t)c.node * p.F + f]));
}

// After the wait, first thing: the row counters of the expansions that this round's partition is
// given (their last reader, the histogram launch of the round before, has finished).
__device__ __forceinline__ void round_clear_counters(const Job& J, const Params& p, const RoundSearch& r, int q) {
  if (!r.stop && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x < 2 * kMaxRoundW)
    round_view(J, p).pcnt[(size_t)(q ^ 1) * 2 * kMaxRoundW + threadIdx.x] = 0;
}

// One feature on the whole CTA (k_search's forms).
template <bool PLAIN, bool QUANT, int NW>
__device__ __forceinline__ void round_search_cta(const Job& J, const Params& p, const RoundExp& c, const DevFeature& m,
                                                 int f, int g, int e, int side, bool used, SearchSmemT<NW>& sm) {
  SearchIn si;
  si.group = g;
  si.crow = 2 * e + side;
  si.C = J.lconst[si.crow];
  si.S0 = side ? J.lconst[2 * e].ls : si.C.ls;
  if (!si.C.go) return;  // not searched (uniform over the expansion's side): no candidates
  const int32_t node = c.x < 0 ? 0 : 2 * c.x + si.C.go;
  si.sslot = c.x < 0 ? c.slot : c.sslot;
  si.lslot = c.slot;
  si.pre = false;
  si.sv = si.lv = 0;
  if (!used) {  // uniform over the CTA
    if (threadIdx.x == 0) {
      round_view(J, p).cand[(size_t)si.crow * p.n_groups + g] = RoundCand{kNoKey, 0u, 0x7fffffff};
      J.splittable[(size_t)node * p.F + f] = 0;
    }
    return;
  }
  if constexpr (NW == kSearchWarps) {
    if (m.cat) {
      search_cat<QUANT>(J, p, si, m, side, f, node, sm);
      return;
    }
  }
  if constexpr (QUANT) search_int<PLAIN>(J, p, si, m, side, f, node, sm);
  else search_float_any<PLAIN>(J, p, si, m, side, f, node, sm);
}

template <bool PLAIN, bool QUANT, int NW, int CTAS = 1>
__global__ void __launch_bounds__(32 * NW, CTAS) k_search_round(const JobTable jobs, Params p,
                                                          const DevFeature* __restrict__ feats, int q) {
  __shared__ SearchSmemT<NW> sm;
  const int side = (int)(blockIdx.x & 1u), e = (int)blockIdx.y, f = (int)(blockIdx.x >> 1);
  const DevFeature m = feats[f];  // static: loaded while the histogram launch finishes
  const Job& J = jobs.job[blockIdx.z];
  const RoundSearch r = round_search_load(J, p, q, e);
  const bool used = r.active && round_used(J, p, r.c, f);
  griddep_wait();
  // the partition may be scheduled now: its CTAs read the round's state while this search runs
  griddep_launch();
  round_clear_counters(J, p, r, q);
  if (r.active) round_search_cta<PLAIN, QUANT, NW>(J, p, r.c, m, f, f, e, side, used, sm);
}

// CAT: the learner has categorical features (their search's registers and code stay out otherwise).
template <bool CAT>
__global__ void __launch_bounds__(32 * kWarpFeatures, 3)
    k_search_round_warp(const JobTable jobs, Params p, const DevFeature* __restrict__ feats, int q) {
  union Smem {
    WarpSearchSmem w;
    typename std::conditional<CAT, SearchSmem, int>::type c;
    __device__ Smem() {}
  };
  __shared__ Smem sm;
  const int side = (int)(blockIdx.x & 1u), e = (int)blockIdx.y, g = (int)(blockIdx.x >> 1);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n_num_groups = (p.n_numeric + kWarpFeatures - 1) / kWarpFeatures;
  const bool numeric = !CAT || g < n_num_groups;
  // the warp's feature (the CTA's, for a categorical one)
  const int oi = numeric ? g * kWarpFeatures + warp : p.n_numeric + (g - n_num_groups);
  const int f = (!numeric || oi < p.n_numeric) ? p.order[oi] : -1;
  DevFeature m{};
  if (f >= 0) m = feats[f];  // static: loaded while the histogram launch finishes
  // the group's bins are moved with thread = (bin t0 + 32 i, feature fj of the group): eight adjacent
  // features' bins are 64 consecutive bytes of the pool
  const int j = threadIdx.x & (kWarpFeatures - 1), t0 = (int)threadIdx.x / kWarpFeatures;
  const int oj = g * kWarpFeatures + j;
  const int fj = (numeric && oj < p.n_numeric) ? p.order[oj] : -1;
  int lenj = 0, mfbj = -1;
  if (fj >= 0) {
    lenj = feats[fj].len;
    mfbj = feats[fj].mfb > 0 ? feats[fj].mfb : -1;
  }
  const Job& J = jobs.job[blockIdx.z];
  const RoundSearch r = round_search_load(J, p, q, e);
  const RoundExp c = r.c;
  const bool used = r.active && f >= 0 && round_used(J, p, c, f);
  const size_t slot_stride = (size_t)p.T * p.B * TILE;
  int64_t* pool = reinterpret_cast<int64_t*>(J.pool);
  const size_t offj = fj >= 0 ? (size_t)(fj / TILE) * p.B * TILE + (fj % TILE) + TILE : 0;  // its bin 1
  int64_t lv[8];
  bool usedj = false;
  if (r.active && side && c.x >= 0 && fj >= 0) {
    const int64_t* parent = pool + (size_t)c.slot * slot_stride + offj;
    usedj = round_used(J, p, c, fj);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int t = t0 + 32 * i;
      lv[i] = t < lenj ? parent[(size_t)t * TILE] : 0;
    }
  }
  griddep_wait();
  // the partition may be scheduled now: its CTAs read the round's state while this search runs
  griddep_launch();
  round_clear_counters(J, p, r, q);
  if (!r.active) return;
  if constexpr (CAT) {
    if (!numeric) {
      round_search_cta<true, true, kSearchWarps>(J, p, c, m, f, g, e, side, used, sm.c);
      return;
    }
  }
  const int crow = 2 * e + side;
  const LeafConst& C = J.lconst[crow];
  if (!C.go) return;  // uniform over the CTA
  const int32_t node = c.x < 0 ? 0 : 2 * c.x + C.go;
  if (fj >= 0) {
    // the larger leaf: parent minus smaller, in place (its most frequent bin is fixed below)
    const int64_t* hs = pool + (size_t)(c.x < 0 ? c.slot : c.sslot) * slot_stride + offj;
    int64_t* hl = pool + (size_t)c.slot * slot_stride + offj;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int t = t0 + 32 * i;
      int64_t v = 0;
      if (t < lenj && t != mfbj && (!side || usedj)) {
        v = hs[(size_t)t * TILE];
        if (side) {
          v = lv[i] - v;
          hl[(size_t)t * TILE] = v;
        }
      }
      sm.w.w[j].e[slice_at(t)] = v;
    }
  }
  __syncthreads();
  int64_t* own = pool + (size_t)(side || c.x < 0 ? c.slot : c.sslot) * slot_stride +
                 (f >= 0 ? (size_t)(f / TILE) * p.B * TILE + (f % TILE) : 0);
  const ScanGeom G = scan_geom(m);
  WarpSlice& ws = sm.w.w[warp];
  WarpSearch sr;
  const int nb = m.len > 63 ? 8 : 2;
  int32_t M = float_key(-CUDART_INF_F);
  if (used) M = sr.bounds(m, G, C, own, ws, nb, lane);
  if (lane == 0) sm.w.m[warp] = M;
  __syncthreads();
  if (p.unit_penalty) {
#pragma unroll
    for (int w = 0; w < kWarpFeatures; ++w) M = max(M, sm.w.m[w]);
  }
  long long key = kNoKey;
  Cand cd;
  if (used) {
    ExactBest r2[2];
    sr.queue(C, M, ws, nb, lane);
    int split = sr.certain;
    exact_batches(p, ws, sr.n, sr.T, sr.base_f, C, lane, r2);
    split |= r2[0].split | (G.two ? r2[1].split : 0);
    cd = warp_cand(m, G, f, C, r2, split);
    key = dnan(cd.gain) ? kNoKey : dkey(cd.gain);
  }
  if (lane == 0) {
    sm.w.key[warp] = key;
    sm.w.real[warp] = f >= 0 ? m.real : 0x7fffffff;
    if (f >= 0) J.splittable[(size_t)node * p.F + f] = used ? (uint8_t)cd.splittable : (uint8_t)0;
  }
  __syncthreads();
  // the group's candidate: the highest gain, then the smaller real feature
  int best = 0;
#pragma unroll
  for (int w = 1; w < kWarpFeatures; ++w)
    if (sm.w.key[w] > sm.w.key[best] || (sm.w.key[w] == sm.w.key[best] && sm.w.real[w] < sm.w.real[best])) best = w;
  if (warp != best || lane != 0) return;
  RoundCand rc{kNoKey, 0u, 0x7fffffff};
  if (key != kNoKey) {
    J.cand[(size_t)node * p.F + f] = cd;
    rc.key = key;
    rc.pk = ((uint32_t)f << 9) | ((uint32_t)(cd.default_left != 0) << 8) | cd.threshold;
    rc.real = cd.feature;
  }
  round_view(J, p).cand[(size_t)crow * p.n_groups + g] = rc;
}

// The bookkeeping of a tree's last split when it was partitioned in one pass (no histogram launch
// follows it to apply it).
__global__ void __launch_bounds__(32) k_apply_split(const JobTable jobs, Params p, int par) {
  const Job& J = jobs.job[blockIdx.z];
  JobState* st = J.st;
  if (st->stop) return;
  const SplitOutcome o = split_outcome(p, st, __ldcg(&st->pcnt[par][0]) & 0xffffffffLL);
  post_split_writes(J, p, o, (int)threadIdx.x);
}

// The rounds' state at the root of a tree: one leaf, the root the first round's only expansion.
__device__ __forceinline__ void rounds_begin(const Job& J, const Params& p) {
  const RoundView v = round_view(J, p);
  const int t = threadIdx.x;
  if (t < 2 * 2 * kMaxRoundW) v.pcnt[t] = 0;
  if (t == 0) {
    const int32_t count = (int32_t)J.st->root_count;
    RoundHdr h{};
    h.leaves = 1;
    h.last_x = -1;
    v.hdr[1] = h;
    h.n_cur = 1;
    v.hdr[0] = h;
    LeafEnt e{};
    e.key = dkey(-CUDART_INF);
    e.pay = (long long)-1 * 4294967296LL;
    e.feat = -1;
    e.out = -1;
    e.count = count;
    v.leaf[0] = e;
    RoundExp c{};
    c.x = -1;
    c.out = -1;
    c.count = count;
    v.cur[0] = c;
  }
}

// The finished tree: leaf arrays from the final leaves, split records from the committed splits
// (the arguments of Tree::split_numerical / split_categorical, serial.rs:1685-1876).
__global__ void __launch_bounds__(256) k_rounds_finish(const JobTable jobs, Params p) {
  const Job& J = jobs.job[blockIdx.z];
  const JobState* st = J.st;
  if (!st->stop) return;
  const RoundView v = round_view(J, p);
  const int32_t leaves = st->tree_leaves;
  const RoundHdr h = v.hdr[st->fin_q];  // the copy of the state that the last decision wrote
  const LeafEnt* ent = v.leaf + (size_t)st->fin_q * p.num_leaves;
  const int i = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  // the tree's last split, when it was taken before its rows were partitioned
  const int32_t last_L = h.last_x >= 0 ? (int32_t)(v.pcnt[(size_t)h.last_par * 2 * kMaxRoundW] & 0xffffffffLL) : 0;
  if (i < leaves) {
    const LeafEnt e = ent[i];
    int32_t begin = e.begin, count = e.count, slot = e.slot, rest = -1;
    if (h.last_x >= 0 && e.node > 2 * h.last_x) {  // one of its children (no later nodes exist)
      const bool left = e.node == 1 + 2 * h.last_x;
      const int32_t R = count - last_L, pslot = ent[v.commit[leaves - 2].leaf].slot;
      const bool go = !(p.max_depth > 0 && (e.depth_buf >> 1) >= p.max_depth) &&
                      !(R < p.min_data * 2 && last_L < p.min_data * 2);
      slot = !go ? (left ? pslot : -1) : (left == (last_L < R) ? round_sslot(h.last_x) : pslot);
      begin = left ? begin : begin + last_L;
      count = left ? last_L : R;
    } else if (e.out >= 0) {  // expanded, not split: its slot holds its larger child's histogram by now
      const OutEnt o = v.out[st->fin_q * kMaxRoundOut + e.out];
      if (o.slot[1] >= 0) rest = round_sslot(o.x);
    }
    // a root that was not searched (round_go) has no histogram
    if (leaves == 1 && ((p.max_depth > 0 && (e.depth_buf >> 1) >= p.max_depth) || count < p.min_data * 2)) slot = -1;
    J.leaf_begin[i] = begin;
    J.leaf_count[i] = count;
    J.leaf_buf[i] = e.depth_buf & 1;
    J.leaf_slot[i] = slot;
    J.leaf_slot[p.num_leaves + i] = rest;
    J.leaf_slot[2 * p.num_leaves + i] = e.node;
    J.leaf_depth[i] = e.depth_buf >> 1;
    if (e.node > 0) {  // a tree of one leaf keeps the root's output
      const int2 xi = v.xinfo[(e.node - 1) >> 1];
      const Cand& info = J.cand[(size_t)xi.x * p.F + xi.y];
      const double o = (e.node & 1) ? info.left_output : info.right_output;
      J.leaf_value[i] = isnan(o) ? 0.0 : o;
    }
  }
  if (i < leaves - 1) {
    const Commit c = v.commit[i];
    const int2 xi = v.xinfo[c.x];
    const Cand info = J.cand[(size_t)xi.x * p.F + xi.y];
    const int32_t L = c.L >= 0 ? c.L : last_L;
    int32_t count = c.count;
    bk_split& r = J.records[i];
    r.leaf = c.leaf;
    r.right_leaf = i + 1;
    r.inner_feature = info.inner;
    r.real_feature = info.feature;
    r.threshold = info.threshold;
    r.default_left = info.default_left;
    r.missing_type = info.missing;
    r.left_count = L;
    r.right_count = count - L;
    r.left_output = info.left_output;
    r.right_output = info.right_output;
    r.left_sum_gradient = info.lsg;
    r.left_sum_hessian = info.lsh;
    r.right_sum_gradient = info.rsg;
    r.right_sum_hessian = info.rsh;
    r.gain = info.gain;
    r.left_int_sum = info.lint;
    r.right_int_sum = info.rint;
    r.categorical = info.categorical;
    r._pad = 0;
    for (int w = 0; w < 8; ++w) r.cat_bins[w] = info.categorical ? cand_cat_bits(J, p, xi.x, xi.y)[w] : 0u;
  }
}

// Root of a tree (serial.rs:658-776 after the root sums, then :580-586 and the first
// BeforeFindBestSplit). leaf_sum[0] and root_count are already set.
__global__ void __launch_bounds__(256) k_tree_begin(const Job* __restrict__ jobs, Params p, int rounds) {
  const Job& J = jobs[blockIdx.z];
  JobState* st = J.st;
  for (int i = threadIdx.x; i < p.num_leaves; i += blockDim.x) {
    J.leaf_begin[i] = 0;
    J.leaf_count[i] = i == 0 ? st->root_count : 0;
    J.leaf_buf[i] = 0;
    J.leaf_depth[i] = 0;
    J.leaf_slot[i] = J.leaf_slot[p.num_leaves + i] = -1;
    J.leaf_value[i] = 0.0;
    J.bgain[i] = -CUDART_INF;
    J.bfeat[i] = -1;
    J.bsplit[i] = (int64_t)-1 * 4294967296LL;
  }
  if (p.n_icons > 0) {  // serial.rs:660-662: every leaf's path starts empty
    uint32_t* paths = leaf_path_bits(J, p, 0);
    for (int i = threadIdx.x; i < p.num_leaves * p.path_words; i += blockDim.x) paths[i] = 0u;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    if (lane == 0) {
      st->stop = 0;
      st->tree_leaves = 1;
      st->next_free = 0;
      st->pcnt[0][0] = st->pcnt[0][1] = st->pcnt[1][0] = st->pcnt[1][1] = 0;
      const LeafSum r = J.leaf_sum[0];
      double root = leaf_output_root(p, r.sg, r.sh, r.num_data);
      st->root_output = round_to_zero(root);
      J.leaf_value[0] = st->root_output;
    }
    __syncwarp();
    if (!rounds) before_find_best_split(J, p, st, 0, -1, lane);
  }
  if (rounds) rounds_begin(J, p);
}

}  // namespace

void launch_search(const Job* h_jobs, int num_jobs, const Params& p, const DevFeature* feats, int clear_par,
                   bool decide, int post, cudaStream_t s) {
  const bool plain = !p.use_l1 && !p.use_max && !p.use_smooth;
  // 64-thread CTAs when every feature's slice fits in 63 bins (thread 63 holds the forward scan's
  // position -1), no feature is categorical and no CTA has to run the 256-thread decision
  const bool narrow = plain && p.search_narrow && !decide;
  const int dec = decide ? 1 : 0;
  for_job_groups(h_jobs, num_jobs, [&](const JobTable& t, int nz) {
    dim3 grid((unsigned)(2 * p.F), 1, nz);
    if (narrow) {
      const dim3 block(64);
      if (p.quant) (void)launch_kernel(k_search<true, true, 2>, grid, block, 0, s, p.pdl, t, p, feats, clear_par, dec, post);
      else (void)launch_kernel(k_search<true, false, 2>, grid, block, 0, s, p.pdl, t, p, feats, clear_par, dec, post);
      return;
    }
    const dim3 block(kSearchThreads);
    if (p.quant) {
      if (plain) (void)launch_kernel(k_search<true, true, 8>, grid, block, 0, s, p.pdl, t, p, feats, clear_par, dec, post);
      else (void)launch_kernel(k_search<false, true, 8>, grid, block, 0, s, p.pdl, t, p, feats, clear_par, dec, post);
    } else {
      if (plain) (void)launch_kernel(k_search<true, false, 8>, grid, block, 0, s, p.pdl, t, p, feats, clear_par, dec, post);
      else (void)launch_kernel(k_search<false, false, 8>, grid, block, 0, s, p.pdl, t, p, feats, clear_par, dec, post);
    }
  });
}

void launch_apply_split(const Job* h_jobs, int num_jobs, const Params& p, int par, cudaStream_t s) {
  for_job_groups(h_jobs, num_jobs, [&](const JobTable& t, int nz) {
    k_apply_split<<<dim3(1, 1, nz), 32, 0, s>>>(t, p, par);
  });
}

// The warp form takes the quantized, plain searches of rounds that would not fit the chip at once with a
// CTA per feature (by their registers two of 256 threads per SM). Both forms on 20k and 300k rows, 6 to 200
// features, 15 to 127 leaves, time of a tree with a CTA per feature over that with warps, by the round's
// CTAs: 255 bins 0.83 at 304, 0.88 at 608, 1.0 at 912, 1.17 at 1600, 1.84 at 6400; 63 bins 0.94 at 304, 0.95
// at 912, 1.0 at 1600, 1.17 at 6400. The line lies below the crossing for the sake of learners that train
// side by side, whose warps share an SM better: twelve in a group took 1.6% longer with the line at 912,
// and a learner with categorical features (300k x 40) 2%.
static bool search_round_warp(const Params& p) {
  return p.quant && !p.use_l1 && !p.use_max && !p.use_smooth && 2 * p.F * p.round_w * p.search_jobs > 2 * 152;
}

int rounds_groups(const Params& p) {
  if (!search_round_warp(p)) return p.F;
  return (p.n_numeric + kWarpFeatures - 1) / kWarpFeatures + (p.F - p.n_numeric);
}

// The float search's registers allow two CTAs per SM; four with some spilled are faster once there are
// several waves of them. Time of a tree with two over that with four, the shapes above, by the round's CTAs:
// 0.88 at 304, 0.92 at 608, 0.97 at 1024, 1.05 at 1280 (80 features; 0.99 at 1408 with 44), 1.09 at 1600,
// 1.15 at 3200, 1.22 at 6400.
constexpr int64_t kManySearches = 8 * 152;

void launch_search_round(const Job* h_jobs, int num_jobs, const Params& p, const DevFeature* feats, int q,
                         cudaStream_t s) {
  const bool plain = !p.use_l1 && !p.use_max && !p.use_smooth;
  const bool narrow = plain && p.search_narrow;  // as in launch_search
  for_job_groups(h_jobs, num_jobs, [&](const JobTable& t, int nz) {
    const dim3 grid((unsigned)(2 * p.n_groups), p.round_w, nz);
    auto go = [&](auto kern, int threads) {
      (void)launch_kernel(kern, grid, dim3(threads), 0, s, p.pdl, t, p, feats, q);
    };
    if (search_round_warp(p) && p.n_numeric < p.F) go(k_search_round_warp<true>, 32 * kWarpFeatures);
    else if (search_round_warp(p)) go(k_search_round_warp<false>, 32 * kWarpFeatures);
    else if (p.quant && narrow) go(k_search_round<true, true, 2>, 64);
    else if (p.quant && plain) go(k_search_round<true, true, 8>, kSearchThreads);
    else if (p.quant) go(k_search_round<false, true, 8>, kSearchThreads);
    else if (narrow) go(k_search_round<true, false, 2>, 64);
    else if (plain && (int64_t)grid.x * grid.y * nz > kManySearches) go(k_search_round<true, false, 8, 4>, kSearchThreads);
    else if (plain) go(k_search_round<true, false, 8>, kSearchThreads);
    else go(k_search_round<false, false, 8>, kSearchThreads);
  });
}

void launch_tree_begin(const Job* d_jobs, int num_jobs, const Params& p, bool rounds, cudaStream_t s) {
  k_tree_begin<<<dim3(1, 1, num_jobs), 256, 0, s>>>(d_jobs, p, rounds ? 1 : 0);
}

void launch_rounds_finish(const Job* h_jobs, int num_jobs, const Params& p, cudaStream_t s) {
  for_job_groups(h_jobs, num_jobs, [&](const JobTable& t, int nz) {
    k_rounds_finish<<<dim3((p.num_leaves + 255) / 256, 1, nz), 256, 0, s>>>(t, p);
  });
}

size_t rounds_state_bytes(int num_leaves, int max_exp, int F) {
  return round_view(nullptr, num_leaves, max_exp, F).bytes;
}

}  // namespace bk
