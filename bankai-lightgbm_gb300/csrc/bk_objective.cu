// Built-in objective gradients on the device, written into the learner's gradient buffers, and
// the training loss, so one boosting iteration (gradients, K trees, score update) stays in HBM:
//   L2         objective/regression.rs:240-248   g = (score - label) as f32, h = 1
//              weighted, regression.rs:321-329   g = ((score - label) as f32) * w, h = w
//   binary     objective/binary.rs:71-90         response = -label*s / (1 + exp(label*s*score)),
//                                                times the label weight of the row's class
//                                                (binary.rs:33-52) and the row weight
//   multiclass objective/multiclass.rs:68-90     softmax over the K class scores of a row, times
//                                                the row weight
// Operation order follows the reference. Row weights (`w`, device f32 [n], or null) and the
// binary label weights are set on the learner (bk_learner_set_objective_weights). `exp` is CUDA's double-precision exp, which can differ
// from the host libm's in the last bit, so binary / multiclass gradients may differ from a host
// computation by one f32 ulp; the learner's parity is checked on given gradients.
//
// A multiclass label outside [0, K) (or NaN) is not a class: the softmax gradient treats the row
// as belonging to no class and the loss skips the row, and both count it in `bad_label`, which the
// host turns into an error (a label is never used as an index without this check).
#include <math_constants.h>

#include <cmath>

#include "bk_common.cuh"
#include "bk_pair.cuh"

namespace bk {

namespace {

// The gradients end as fp32, so they are computed as fp32 pairs and, where a pair's error could move
// the rounding, in f64 (bk_pair.cuh): the same fp32 numbers without the f64 pipe. `rel` is the bound on
// a pair's relative error, plus what the f64 evaluation itself rounds away. Measured, 10M rows: L2 60
// -> 48 us (HBM), binary 637 -> 89 us; softmax of ten classes on 2M rows 1277 -> 262 us (issue).
__host__ __device__ constexpr float kTwo(int e) { return e >= 0 ? (float)(1ull << e) : 1.0f / (float)(1ull << -e); }

__global__ void __launch_bounds__(256) k_grad_l2(const double* __restrict__ score, const float* __restrict__ label,
                                                 int64_t n, const float* __restrict__ w, float* __restrict__ g,
                                                 float* __restrict__ h) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const double s = score[i];
    const float l = label[i];
    bool ok;
    const Pair sp = pair_of(s, &ok);
    Pair d = two_sum(sp.hi, -l);
    d = quick_two_sum(d.hi, __fadd_rn(d.lo, sp.lo));
    const float rel = __fdividef(__fmul_rn(kTwo(-46), fabsf(sp.hi)), fabsf(d.hi)) + kTwo(-50);
    float v;
    if (!pair_round(d, rel, &v) || !ok) v = (float)(s - (double)l);
    if (w) {
      const float wi = w[i];
      g[i] = __fmul_rn(v, wi);
      h[i] = wi;
    } else {
      g[i] = v;
      h[i] = 1.0f;
    }
  }
}

// The reference's arithmetic of one binary row in f64 (zs = sigmoid * score; the factors with the label's sign
// and label weights of 1 change nothing but signs).
__device__ __noinline__ float2 binary_row(double zs, bool pos, double sigmoid, double lw, bool unit, const float* wi) {
  const double e = exp(pos ? zs : -zs);
  const double ar = sigmoid / (1.0 + e);
  double r = ar, q = ar * (sigmoid - ar);
  if (!unit) r *= lw, q *= lw;
  if (wi) r *= (double)*wi, q *= (double)*wi;
  return make_float2((float)(pos ? -r : r), (float)q);
}

__global__ void __launch_bounds__(256) k_grad_binary(const double* __restrict__ score, const float* __restrict__ label,
                                                     int64_t n, double sigmoid, const float* __restrict__ w,
                                                     double lw_neg, double lw_pos, const ExpTable T,
                                                     float* __restrict__ g, float* __restrict__ h) {
  __shared__ ExpTable st;
  if (threadIdx.x < 32) {
    st.hi[threadIdx.x] = T.hi[threadIdx.x];
    st.lo[threadIdx.x] = T.lo[threadIdx.x];
  }
  __syncthreads();
  bool ok_s, ok_n, ok_p;
  const Pair sg = pair_of(sigmoid, &ok_s), ln = pair_of(lw_neg, &ok_n), lp = pair_of(lw_pos, &ok_p);
  const bool unit = lw_neg == 1.0 && lw_pos == 1.0, one = sigmoid == 1.0;
  const bool ok_c = ok_s && ok_n && ok_p;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const double s = score[i];
    const bool pos = label[i] > 0.0f;
    bool ok;
    const double zs = one ? s : sigmoid * s;
    Pair z = pair_of<true>(zs, &ok);  // exp(z) and 1 + exp(z): absolute errors count
    if (!pos) z = pair_neg(z);
    ok = ok && ok_c && fabsf(z.hi) <= 60.0f;
    // a warp with a row for f64 takes all of them there: the f64 instructions cost the same
    ok = __all_sync(__activemask(), ok);
    float gv = 0.f, hv = 0.f;
    if (ok) {
      // response = -label s / (1 + e), hessian |response| (s - |response|) = s^2 e / (1 + e)^2
      const Pair e = pair_exp(z, st);
      const Pair d = e.hi > 1.0f ? pair_add(e, Pair{1.f, 0.f}) : pair_add(Pair{1.f, 0.f}, e);
      Pair r = pair_div(sg, d);
      const Pair c = pair_mul(r, e);  // s - |response|
      Pair q = pair_mul(r, c);
      const float rel_h = kTwo(-39) + __fdividef(__fmul_rn(kTwo(-50), sg.hi), c.hi);
      if (!unit) {
        const Pair lw = pos ? lp : ln;
        r = pair_mul(r, lw);
        q = pair_mul(q, lw);
      }
      if (w) {
        const Pair wi{w[i], 0.f};
        r = pair_mul(r, wi);
        q = pair_mul(q, wi);
      }
      const bool a = pair_round(r, kTwo(-40), &gv), b = pair_round(q, rel_h, &hv);
      ok = (a && b) || (w && w[i] == 0.f);  // a row of no weight: zeros
      if (pos) gv = -gv;
    }
    if (!ok) {
      const float2 v = binary_row(zs, pos, sigmoid, pos ? lw_pos : lw_neg, unit, w ? w + i : nullptr);
      gv = v.x;
      hv = v.y;
    }
    g[i] = gv;
    h[i] = hv;
  }
}

// The class of a multiclass label, or -1 (counted in *bad_label) when it is not in [0, K).
__device__ __forceinline__ int class_of(float lf, int K, int32_t* bad_label) {
  if (lf >= 0.0f && lf < (float)K) return (int)lf;
  atomicAdd(bad_label, 1);
  return -1;
}

// The reference's arithmetic of one softmax row in f64.
__device__ __noinline__ void softmax_row(const double* __restrict__ score, int64_t n, int64_t i, int K, int lab,
                                         const float* __restrict__ w, float* __restrict__ g, float* __restrict__ h) {
  const double factor = (double)K / ((double)K - 1.0);
  double rec[32];
  double wmax = score[i];
  for (int k = 1; k < K; ++k) wmax = fmax(score[(size_t)k * n + i], wmax);
  double wsum = 0.0;
  for (int k = 0; k < K; ++k) {
    rec[k] = exp(score[(size_t)k * n + i] - wmax);
    wsum += rec[k];
  }
  const double wi = w ? (double)w[i] : 1.0;
  for (int k = 0; k < K; ++k) {
    double p = rec[k] / wsum;
    double gi = lab == k ? p - 1.0 : p;
    double hi = factor * p;
    hi = hi * (1.0 - p);
    g[(size_t)k * n + i] = (float)(w ? gi * wi : gi);
    h[(size_t)k * n + i] = (float)(w ? hi * wi : hi);
  }
}

// The classes' exponentials of a thread's row stay in shared memory ([K][128] pairs) between the sum
// and the gradients. Scores up to 64 in magnitude take pairs.
constexpr int kSoftmaxThreads = 128;
__global__ void __launch_bounds__(kSoftmaxThreads)
    k_grad_softmax(const double* __restrict__ score, const float* __restrict__ label, int64_t n, int K,
                   const float* __restrict__ w, const ExpTable T, float* __restrict__ g, float* __restrict__ h,
                   int32_t* __restrict__ bad_label) {
  extern __shared__ float2 s_e[];
  __shared__ ExpTable st;
  if (threadIdx.x < 32) {
    st.hi[threadIdx.x] = T.hi[threadIdx.x];
    st.lo[threadIdx.x] = T.lo[threadIdx.x];
  }
  __syncthreads();
  bool ok_f;
  const Pair factor = pair_of((double)K / ((double)K - 1.0), &ok_f);
  float2* mine = s_e + threadIdx.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int lab = class_of(label[i], K, bad_label);
    // the scores as pairs, whose differences' absolute errors count; their maximum (pairs compare like the
    // scores up to 2^-53, which the bound allows)
    bool ok = ok_f;
    Pair top{-CUDART_INF_F, 0.f};
    float least = CUDART_INF_F;
    for (int k = 0; k < K; ++k) {
      bool o;
      const Pair x = pair_of<true>(score[(size_t)k * n + i], &o);
      ok = ok && o && fabsf(x.hi) <= 64.0f;
      mine[k * kSoftmaxThreads] = make_float2(x.hi, x.lo);
      if (x.hi > top.hi || (x.hi == top.hi && x.lo > top.lo)) top = x;
      least = fminf(least, x.hi);
    }
    // as in k_grad_binary; the exponents reach down to the lowest score's
    ok = ok && __fsub_rn(least, top.hi) >= -59.0f;
    if (!__all_sync(__activemask(), ok)) {
      softmax_row(score, n, i, K, lab, w, g, h);
      continue;
    }
    // two classes at a time: the chains of a class alone leave the schedulers idle
    Pair sum{0.f, 0.f}, others{0.f, 0.f};
    top = pair_neg(top);
#pragma unroll 2
    for (int k = 0; k < K; ++k) {
      const float2 x = mine[k * kSoftmaxThreads];
      const Pair z = pair_add(Pair{x.x, x.y}, top);
      const Pair e = pair_exp(z, st);
      sum = pair_add(sum, e);
      if (k != lab) others = pair_add(others, e);
      mine[k * kSoftmaxThreads] = make_float2(e.hi, e.lo);
    }
    const Pair wi{w ? w[i] : 1.0f, 0.f};
    const Pair per = pair_div(Pair{1.f, 0.f}, sum);
#pragma unroll 2
    for (int k = 0; k < K; ++k) {
      const float2 x = mine[k * kSoftmaxThreads];
      const Pair e{x.x, x.y};
      const Pair p = pair_mul(e, per);
      const Pair rest = k == lab ? others : pair_add(sum, pair_neg(e));
      const Pair np = pair_mul(rest, per);  // 1 - p
      const float inv = __fdividef(1.0f, np.hi);
      Pair gp = k == lab ? np : p, hp = pair_mul(pair_mul(factor, p), np);
      const float rel_g = kTwo(-38) + (k == lab ? __fmul_rn(kTwo(-51), inv) : 0.f);
      const float rel_h = kTwo(-37) + __fmul_rn(k == lab ? kTwo(-51) : kTwo(-40), inv);
      if (w) {
        gp = pair_mul(gp, wi);
        hp = pair_mul(hp, wi);
      }
      float gv, hv;
      const bool a = pair_round(gp, rel_g, &gv), b = pair_round(hp, rel_h, &hv);
      ok = ok && ((a && b) || wi.hi == 0.f);  // a row of no weight: zeros
      g[(size_t)k * n + i] = k == lab ? -gv : gv;
      h[(size_t)k * n + i] = hv;
    }
    if (!ok) softmax_row(score, n, i, K, lab, w, g, h);
  }
}

// 2^(j / 32), from the host's f64 exp2.
ExpTable exp_table() {
  ExpTable t;
  for (int j = 0; j < 32; ++j) {
    const double v = std::exp2((double)j / 32.0);
    t.hi[j] = (float)v;
    t.lo[j] = (float)(v - (double)t.hi[j]);
  }
  return t;
}

// Per-CTA partial losses (mean squared error / log loss / multiclass log loss).
__global__ void k_loss(int kind, const double* __restrict__ score, const float* __restrict__ label, int64_t n, int K,
                       double* __restrict__ partial, int32_t* __restrict__ bad_label) {
  double acc = 0.0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    if (kind == 0) {
      double d = score[i] - (double)label[i];
      acc += d * d;
    } else if (kind == 1) {
      double p = 1.0 / (1.0 + exp(-score[i]));
      p = fmin(fmax(p, 1e-15), 1.0 - 1e-15);
      acc += label[i] > 0.0f ? -log(p) : -log(1.0 - p);
    } else {
      double wmax = score[i];
      for (int k = 1; k < K; ++k) wmax = fmax(score[(size_t)k * n + i], wmax);
      double wsum = 0.0;
      for (int k = 0; k < K; ++k) wsum += exp(score[(size_t)k * n + i] - wmax);
      const int lab = class_of(label[i], K, bad_label);
      if (lab >= 0) acc += -(score[(size_t)lab * n + i] - wmax - log(wsum));
    }
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  __shared__ double sh[32];
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += sh[w];
    partial[blockIdx.x] = s;
  }
}

}  // namespace

cudaError_t objective_gradients(int kind, const double* score, const float* label, int64_t n, int K, double sigmoid,
                                const ObjectiveWeights& ow, float* g, float* h, int32_t* bad_label, cudaStream_t s) {
  const int grid = 1216, threads = 256;  // eight CTAs per SM
  static const ExpTable table = exp_table();
  if (kind == 0) k_grad_l2<<<grid, threads, 0, s>>>(score, label, n, ow.row, g, h);
  else if (kind == 1)
    k_grad_binary<<<grid, threads, 0, s>>>(score, label, n, sigmoid, ow.row, ow.label_neg, ow.label_pos, table, g, h);
  else
    k_grad_softmax<<<grid, kSoftmaxThreads, (size_t)K * kSoftmaxThreads * sizeof(float2), s>>>(
        score, label, n, K, ow.row, table, g, h, bad_label);
  return cudaGetLastError();
}

cudaError_t objective_loss(int kind, const double* score, const float* label, int64_t n, int K, double* partial,
                           int grid, int32_t* bad_label, cudaStream_t s) {
  k_loss<<<grid, 256, 0, s>>>(kind, score, label, n, K, partial, bad_label);
  return cudaGetLastError();
}

}  // namespace bk
