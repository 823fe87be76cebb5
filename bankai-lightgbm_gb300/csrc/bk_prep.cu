// Per-tree preparation and finishing kernels of the GB300 learner:
//   - row-index initialisation (DataPartition::init / init_with, data_partition.rs:90-107);
//   - gradient discretization (GradientDiscretizer, gradient_discretizer/mod.rs:116-201) with the
//     per-tree stochastic-rounding rotation drawn on the device from a std::mt19937 state
//     (mt19937.rs:32-128), so every draw happens exactly when the reference draws;
//   - root leaf sums (serial.rs:705-775);
//   - score update and leaf lookup over the final partition (serial.rs:1974-1990).
#include <math_constants.h>

#include <algorithm>
#include <cstddef>

#include "bk_math.cuh"

namespace bk {

namespace {

constexpr unsigned FULL = 0xffffffffu;

// What a train call sets in the job states (a launch; a copy per field and job took 3 us each).
__global__ void __launch_bounds__(32) k_job_begin(const Job* __restrict__ jobs, int num_jobs, int use_rows,
                                                  int64_t root_count) {
  for (int j = threadIdx.x; j < num_jobs; j += 32) {
    JobState* s = jobs[j].st;
    s->use_rows = use_rows;
    s->root_count = root_count;
    s->hist_rows_direct = s->hist_rows_gather = s->hist_builds = 0;
  }
}

// What a train call returns, written to the host's pinned memory: the results (a multiple of 16 bytes) and
// each job's state without its random engine. Two copies took longer, and a stream that ends in a copy
// shares half as many of the device's queues in the next calls: 32 learners of 2000 x 10 in one batch call
// 2290 us with copies, 1488 with this.
__global__ void __launch_bounds__(256) k_results(const uint4* __restrict__ results, uint4* __restrict__ h_results, int n16,
                                                 const JobState* __restrict__ states, JobState* __restrict__ h_states,
                                                 int num_jobs) {
  static_assert(offsetof(JobState, mt) % 4 == 0, "the state is written in words");
  constexpr int kWords = (int)(offsetof(JobState, mt) / 4);
  const int step = gridDim.x * blockDim.x, t = blockIdx.x * blockDim.x + threadIdx.x;
  for (int i = t; i < n16; i += step) h_results[i] = results[i];
  for (int i = t; i < num_jobs * kWords; i += step) {
    const int j = i / kWords, w = i % kWords;
    reinterpret_cast<uint32_t*>(h_states + j)[w] = reinterpret_cast<const uint32_t*>(states + j)[w];
  }
}

// The root's row indices. Without bagging they are the identity, which the grow rounds (and every
// reader of a leaf of all rows) derive instead of reading: `bagged_only` skips those 4 bytes a row.
__global__ void k_init_rows(const Job* __restrict__ jobs, Params p, const int32_t* __restrict__ rows, int bagged_only) {
  const Job& J = jobs[blockIdx.z];
  const int64_t cnt = J.st->root_count;
  if (bagged_only && !J.st->use_rows) return;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < cnt; i += (int64_t)gridDim.x * blockDim.x)
    J.idx0[i] = J.st->use_rows ? rows[i] : (int32_t)i;
}

// ---- std::mt19937 on the device (one thread per job) ----
__device__ void mt_twist(uint32_t* st) {
  for (int i = 0; i < 624; ++i) {
    uint32_t y = (st[i] & 0x80000000u) | (st[(i + 1) % 624] & 0x7fffffffu);
    uint32_t nx = st[(i + 397) % 624] ^ (y >> 1);
    if (y & 1u) nx ^= 0x9908b0dfu;
    st[i] = nx;
  }
}

__device__ uint32_t mt_next(JobState* s) {
  if (s->mt_idx >= 624) {
    mt_twist(s->mt);
    s->mt_idx = 0;
  }
  uint32_t y = s->mt[s->mt_idx++];
  y ^= y >> 11;
  y ^= (y << 7) & 0x9d2c5680u;
  y ^= (y << 15) & 0xefc60000u;
  y ^= y >> 18;
  return y;
}

// libc++ uniform_int_distribution<int>(0, n) (mt19937.rs:109-128).
__device__ uint32_t mt_uniform_int_inclusive(JobState* s, uint32_t n) {
  uint32_t rp = n + 1u;
  if (rp == 1u) return 0u;
  if (rp == 0u) return mt_next(s);
  uint32_t w = 32u - (uint32_t)__clz(rp) - 1u;
  if (rp & (0xffffffffu >> (32u - w))) w += 1u;
  uint32_t mask = w >= 32u ? 0xffffffffu : ((1u << w) - 1u);
  for (int guard = 0; guard < 1 << 20; ++guard) {  // rejection succeeds with probability >= 1/2
    uint32_t u = mt_next(s) & mask;
    if (u < rp) return u;
  }
  return 0u;
}

__global__ void k_mt_seed(const Job* __restrict__ jobs, uint32_t seed) {
  JobState* s = jobs[blockIdx.z].st;
  s->mt[0] = seed;
  for (int i = 1; i < 624; ++i) s->mt[i] = 1812433253u * (s->mt[i - 1] ^ (s->mt[i - 1] >> 30)) + (uint32_t)i;
  s->mt_idx = 624;
}

// ---- discretization ----
__global__ void k_disc_reset(const Job* __restrict__ jobs) {
  JobState* s = jobs[blockIdx.z].st;
  s->red_maxg = 0u;
  s->red_maxh = 0u;
  s->red_flags = 0u;
}

// max |g| and max h over all rows (order-free), and the refused cases (mod.rs:134-155). HBM-bound:
// 16-byte loads, four rows a thread and step (10M rows: 28 -> 22 us).
__global__ void __launch_bounds__(256) k_disc_reduce(const Job* __restrict__ jobs, Params p) {
  const Job& J = jobs[blockIdx.z];
  float mg = 0.f, mh = 0.f;
  uint32_t bad = 0;
  auto take = [&](float g, float h) {
    if (!isfinite(g) || !isfinite(h) || h < 0.f) bad = 1u;
    mg = fmaxf(mg, fabsf(g));
    mh = fmaxf(mh, h);
  };
  const int64_t step = (int64_t)gridDim.x * blockDim.x, t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  // a job's rows start at a multiple of n floats: 16-byte loads where that is aligned
  const bool vec = ((reinterpret_cast<uintptr_t>(J.g) | reinterpret_cast<uintptr_t>(J.h)) & 15u) == 0u;
  const int64_t n4 = vec ? p.n / 4 : 0;
  for (int64_t i = t; i < n4; i += step) {
    const float4 g = reinterpret_cast<const float4*>(J.g)[i], h = reinterpret_cast<const float4*>(J.h)[i];
    take(g.x, h.x);
    take(g.y, h.y);
    take(g.z, h.z);
    take(g.w, h.w);
  }
  for (int64_t i = 4 * n4 + t; i < p.n; i += step) take(J.g[i], J.h[i]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    mg = fmaxf(mg, __shfl_xor_sync(FULL, mg, o));
    mh = fmaxf(mh, __shfl_xor_sync(FULL, mh, o));
    bad |= __shfl_xor_sync(FULL, bad, o);
  }
  if ((threadIdx.x & 31) == 0) {
    // non-negative floats order like their bit patterns
    atomicMax(&J.st->red_maxg, __float_as_uint(mg));
    atomicMax(&J.st->red_maxh, __float_as_uint(mh));
    if (bad) atomicOr(&J.st->red_flags, 1u);
  }
}

// The scales of every job on a thread each; then one thread in job order: the K class trees of an
// iteration share one discretizer, so their rotation offsets are consecutive draws of one engine
// (held by job 0).
__global__ void __launch_bounds__(32) k_disc_setup(const Job* __restrict__ jobs, int num_jobs, Params p) {
  for (int j = threadIdx.x; j < num_jobs; j += 32) {
    JobState* s = jobs[j].st;
    float max_g = __uint_as_float(s->red_maxg), max_h = __uint_as_float(s->red_maxh);
    bool ok = s->red_flags == 0u && max_g != 0.f && (p.const_hess || max_h != 0.f);
    s->disc_ok = ok ? 1 : 0;
    if (!ok) continue;  // the reference warns and keeps the previous discretization (serial.rs:692-703)
    s->gscale = (double)max_g / (double)(p.quant_bins / 2);
    s->hscale = p.const_hess ? (double)max_h : (double)max_h / (double)p.quant_bins;
    s->inv_g = 1.0 / s->gscale;
    s->inv_h = 1.0 / s->hscale;
  }
  __syncwarp();
  if (threadIdx.x != 0 || !p.stochastic) return;
  JobState* eng = jobs[0].st;
  for (int j = 0; j < num_jobs; ++j)
    if (jobs[j].st->disc_ok) jobs[j].st->start_pos = mt_uniform_int_inclusive(eng, (uint32_t)p.n);
}

__device__ __forceinline__ int32_t sat_i8(double v) {  // Rust `f64 as i8`
  if (isnan(v)) return 0;
  if (v >= 127.0) return 127;
  if (v <= -128.0) return -128;
  return (int32_t)trunc(v);
}

// trunc(v * scale + noise) saturated to int8, as f64 arithmetic gives it. f64 costs 64 cycles of a
// scheduler's pipe per warp instruction on this part, so the value is computed in fp32 first: its
// error is at most 4u (|x| + 1) (u = 2^-24: the scale's and the noise's rounding, the product, the
// sum), so a result further than twice that from every whole number truncates to the same one; the
// others (about one row in 400,000) are evaluated in f64.
__device__ __forceinline__ int32_t disc_value(float v, float scale_f, float noise_f, double scale, const double* noise,
                                              double off, bool fused) {
  const float x = fmaf(v, scale_f, v >= 0.f ? noise_f : -noise_f);
  const float w = rintf(x);
  if (fabsf(x - w) > 8.0f * 5.9604645e-08f * (fabsf(x) + 1.0f) && fabsf(x) < 126.0f) return (int32_t)x;
  const double nv = noise ? *noise : off, dv = (double)v;
  return sat_i8(madd(dv, scale, dv >= 0.0 ? nv : -nv, fused));
}

// Four rows a thread; also the root's integer sums when the root is all rows (k_root_partial then has
// nothing to do). HBM-bound: 4 bytes each of gradient (hessian), fp32 noise, 2 of result a row (10M
// rows, constant hessian: 181 -> 25 us; with hessians 336 -> 44; the f64 form was bound by the f64 pipe).
__global__ void __launch_bounds__(256) k_discretize(const Job* __restrict__ jobs, Params p,
                                                    const double* __restrict__ noise_g,
                                                    const double* __restrict__ noise_h,
                                                    const float* __restrict__ noise_gf,
                                                    const float* __restrict__ noise_hf) {
  __shared__ long long sg_s[8], sh_s[8];
  const Job& J = jobs[blockIdx.z];
  const JobState* s = J.st;
  if (!s->disc_ok) return;
  const double ig = s->inv_g, ih = s->inv_h;
  const float igf = (float)ig, ihf = (float)ih;
  const bool fused = p.fused != 0;
  const uint32_t n = (uint32_t)p.n, start = s->start_pos;
  long long sg = 0, sh = 0;
  auto one = [&](uint32_t i, float g, float h) -> uint32_t {
    uint32_t pos = i + start;  // both at most n < 2^31
    if (pos >= n) pos -= n;
    int32_t gi, hi = 1;
    if (p.stochastic) {
      gi = disc_value(g, igf, noise_gf ? noise_gf[pos] : (float)noise_g[pos], ig, noise_g + pos, 0.0, fused);
      if (!p.const_hess)
        hi = disc_value(h, ihf, noise_hf ? noise_hf[pos] : (float)noise_h[pos], ih, noise_h + pos, 0.0, fused);
    } else {
      gi = disc_value(g, igf, 0.5f, ig, nullptr, 0.5, fused);
      if (!p.const_hess) hi = disc_value(h, ihf, 0.5f, ih, nullptr, 0.5, fused);
    }
    sg += gi;
    sh += hi & 0xff;
    return (uint32_t)((gi * 256) | (hi & 0xff)) & 0xffffu;
  };
  const uint32_t step = gridDim.x * blockDim.x, t = blockIdx.x * blockDim.x + threadIdx.x;
  const bool vec = (((reinterpret_cast<uintptr_t>(J.g) | reinterpret_cast<uintptr_t>(J.h)) & 15u) |
                    (reinterpret_cast<uintptr_t>(J.packed) & 7u)) == 0u;
  const uint32_t n4 = vec ? n / 4u : 0u;
  for (uint32_t k = t; k < n4; k += step) {
    const float4 g = reinterpret_cast<const float4*>(J.g)[k];
    const float4 h = p.const_hess ? make_float4(0.f, 0.f, 0.f, 0.f) : reinterpret_cast<const float4*>(J.h)[k];
    const uint32_t a = one(4u * k, g.x, h.x), b = one(4u * k + 1u, g.y, h.y);
    const uint32_t c = one(4u * k + 2u, g.z, h.z), d = one(4u * k + 3u, g.w, h.w);
    reinterpret_cast<uint2*>(J.packed)[k] = make_uint2(a | (b << 16), c | (d << 16));
  }
  for (uint32_t i = 4u * n4 + t; i < n; i += step) J.packed[i] = (int16_t)one(i, J.g[i], p.const_hess ? 0.f : J.h[i]);
  if (s->use_rows) return;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    sg += __shfl_xor_sync(FULL, sg, o);
    sh += __shfl_xor_sync(FULL, sh, o);
  }
  if ((threadIdx.x & 31) == 0) {
    sg_s[threadIdx.x >> 5] = sg;
    sh_s[threadIdx.x >> 5] = sh;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) {
      sg += sg_s[w];
      sh += sh_s[w];
    }
    J.ired[2 * blockIdx.x] = sg;
    J.ired[2 * blockIdx.x + 1] = sh;
  }
}

__global__ void k_noise_f32(const double* __restrict__ a, float* __restrict__ b, int64_t n) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    b[i] = (float)a[i];
}

// ---- root sums ----
// Float path: Σg, Σh in f64 over the root rows; per-CTA partials summed in CTA order.
// Quantized path: exact integer sums; the f64 sums Σ(int · scale) are the integer sum times the
// scale whenever every partial sum is exactly representable (power-of-two bin counts and fewer
// than 2^29 units), which is then bit-identical to the reference's sequential sum; otherwise a
// single warp sums sequentially in row order like the reference.
// The float path also finds the largest and the smallest non-zero magnitude of the gradients and
// hessians (their bits, max << 32 | min), for the histograms' unit.
__device__ __forceinline__ int64_t join_range(int64_t a, int64_t b) {
  const uint32_t lo = min((uint32_t)a, (uint32_t)b), hi = max((uint32_t)(a >> 32), (uint32_t)(b >> 32));
  return (int64_t)(((uint64_t)hi << 32) | lo);
}

// Whether every value of the range is a 24-bit multiple of a unit below 2^bits of them, and its
// largest biased exponent.
__device__ __forceinline__ bool fixed_fits(int64_t range, int bits, uint32_t* emax) {
  const uint32_t hi = (uint32_t)(range >> 32), lo = min((uint32_t)range, hi);
  *emax = max(hi >> 23, 1u);
  return hi < 0x7f800000u && (int)*emax - (int)max(lo >> 23, 1u) <= bits - 24;
}

__global__ void __launch_bounds__(256) k_root_partial(const Job* __restrict__ jobs, Params p) {
  __shared__ double sg_s[8], sh_s[8];
  __shared__ long long ig_s[8], ih_s[8];
  const Job& J = jobs[blockIdx.z];
  const int64_t cnt = J.st->root_count;
  const bool bagged = J.st->use_rows != 0;
  if (p.quant && !bagged && J.st->disc_ok) return;  // the discretization has left its sums
  double sg = 0.0, sh = 0.0;
  long long ig = 0, ih = 0;
  // float path: the largest and the smallest non-zero magnitude's bits
  uint32_t max_g = 0, min_g = 0x7fffffffu, max_h = 0, min_h = 0x7fffffffu;
  auto range = [](float v, uint32_t& hi, uint32_t& lo) {
    const uint32_t a = __float_as_uint(v) & 0x7fffffffu;
    hi = max(hi, a);
    if (a) lo = min(lo, a);
  };
  const int64_t step = (int64_t)gridDim.x * blockDim.x;
  int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p.quant) {
    for (; k < cnt; k += step) {
      int32_t pk = J.packed[bagged ? J.idx0[k] : k];
      ig += (int8_t)(pk >> 8);
      ih += pk & 0xff;
    }
  } else {
    // four rows' values on their way at a time, added in order
    for (; k < cnt; k += 4 * step) {
      float g[4], h[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int64_t at = k + u * step;
        g[u] = h[u] = 0.f;
        if (at < cnt) {
          const int64_t i = bagged ? J.idx0[at] : at;
          g[u] = J.g[i];
          h[u] = J.h[i];
        }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (k + u * step < cnt) {
          sg += (double)g[u];
          sh += (double)h[u];
        }
        range(g[u], max_g, min_g);
        range(h[u], max_h, min_h);
      }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    sg += __shfl_xor_sync(FULL, sg, o);
    sh += __shfl_xor_sync(FULL, sh, o);
    ig += __shfl_xor_sync(FULL, ig, o);
    ih += __shfl_xor_sync(FULL, ih, o);
    if (!p.quant) {
      max_g = max(max_g, __shfl_xor_sync(FULL, max_g, o));
      min_g = min(min_g, __shfl_xor_sync(FULL, min_g, o));
      max_h = max(max_h, __shfl_xor_sync(FULL, max_h, o));
      min_h = min(min_h, __shfl_xor_sync(FULL, min_h, o));
    }
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (!p.quant) {
    ig = (long long)(((unsigned long long)max_g << 32) | min_g);
    ih = (long long)(((unsigned long long)max_h << 32) | min_h);
  }
  if (lane == 0) {
    sg_s[warp] = sg;
    sh_s[warp] = sh;
    ig_s[warp] = ig;
    ih_s[warp] = ih;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double a = 0.0, b = 0.0;
    long long c = 0, d = 0;
    for (int w = 0; w < 8; ++w) {
      a += sg_s[w];
      b += sh_s[w];
      if (p.quant) {
        c += ig_s[w];
        d += ih_s[w];
      } else {
        c = join_range(w ? c : ig_s[w], ig_s[w]);
        d = join_range(w ? d : ih_s[w], ih_s[w]);
      }
    }
    J.red[2 * blockIdx.x] = a;
    J.red[2 * blockIdx.x + 1] = b;
    J.ired[2 * blockIdx.x] = c;
    J.ired[2 * blockIdx.x + 1] = d;
  }
}

// One warp: the partials, on the quantized path lane l taking CTAs l, l + 32, ... and a tree over the
// lanes (one lane over all of them took 45 us).
__global__ void __launch_bounds__(32) k_root_finish(const Job* __restrict__ jobs, Params p, int exact_quant_root) {
  const Job& J = jobs[blockIdx.z];
  JobState* s = J.st;
  const int lane = threadIdx.x;
  double sg = 0.0, sh = 0.0;
  int64_t ig = 0, ih = 0;
  static_assert(kRootGrid % 32 == 0, "whole rounds of the warp");
  if (p.quant) {
#pragma unroll 4
    for (int b = 0; b < kRootGrid; b += 32) {
      ig += J.ired[2 * (b + lane)];
      ih += J.ired[2 * (b + lane) + 1];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      ig += __shfl_xor_sync(FULL, ig, o);
      ih += __shfl_xor_sync(FULL, ih, o);
    }
  } else {
    // CTA after CTA, as a column whose most frequent bin holds no rows (the bin of zero) gets this sum's
    // rounding for that bin, which decides between the two equal thresholds around it: the order is part
    // of the result. Even lanes add the gradients, odd lanes the hessians.
    double pg[kFloatRootGrid / 32], ph[kFloatRootGrid / 32], sum = 0.0;
#pragma unroll
    for (int r = 0; r < kFloatRootGrid / 32; ++r) {
      pg[r] = J.red[2 * (32 * r + lane)];
      ph[r] = J.red[2 * (32 * r + lane) + 1];
      ig = join_range(r ? ig : J.ired[2 * lane], J.ired[2 * (32 * r + lane)]);
      ih = join_range(r ? ih : J.ired[2 * lane + 1], J.ired[2 * (32 * r + lane) + 1]);
    }
#pragma unroll
    for (int r = 0; r < kFloatRootGrid / 32; ++r)
#pragma unroll 4
      for (int l = 0; l < 32; ++l) {
        const double a = __shfl_sync(FULL, pg[r], l), b = __shfl_sync(FULL, ph[r], l);
        sum += (lane & 1) ? b : a;
      }
    sg = __shfl_sync(FULL, sum, 0);
    sh = __shfl_sync(FULL, sum, 1);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      ig = join_range(ig, __shfl_xor_sync(FULL, ig, o));
      ih = join_range(ih, __shfl_xor_sync(FULL, ih, o));
    }
    if (lane == 0) {
      const bool g_ok = fixed_fits(ig, p.fix_bits, &s->red_maxg);
      const bool h_ok = fixed_fits(ih, p.fix_bits, &s->red_maxh);
      s->fix_ok = g_ok && h_ok ? 1 : 0;
    }
  }
  if (p.quant && !exact_quant_root) {
    // sequential f64 sum of int * scale in root row order (serial.rs:717-739): even lanes the gradients, odd
    // lanes the hessians, a batch of rows on its way while the one before is added
    const int64_t cnt = s->root_count;
    const bool bagged = s->use_rows != 0;
    const int16_t* packed = J.packed;
    const int32_t* idx = J.idx0;
    const double scale = (lane & 1) ? s->hscale : s->gscale;
    auto load = [&](int64_t base) -> int32_t {
      const int64_t k = base + lane;
      return k < cnt ? packed[bagged ? idx[k] : (int32_t)k] : 0;
    };
    double sum = 0.0;
    int32_t next = load(0);
    for (int64_t base = 0; base < cnt; base += 32) {
      const int32_t pk = next;
      next = load(base + 32);
      const int jn = (int)min((int64_t)32, cnt - base);
#pragma unroll 4
      for (int j = 0; j < jn; ++j) {
        const int32_t x = __shfl_sync(FULL, pk, j);
        sum += (double)((lane & 1) ? x & 0xff : (int32_t)(int8_t)(x >> 8)) * scale;
      }
    }
    const double a = __shfl_sync(FULL, sum, 0), b = __shfl_sync(FULL, sum, 1);
    sg = a;
    sh = b;
  } else if (p.quant) {
    sg = (double)ig * s->gscale;
    sh = (double)ih * s->hscale;
  }
  if (lane == 0) {
    LeafSum r;
    r.sg = sg;
    r.sh = sh;
    r.weight = 0.0;
    r.int_sum = p.quant ? (int64_t)((uint64_t)ig * 4294967296ull + (uint64_t)ih) : 0;
    r.num_data = (int32_t)s->root_count;
    r._pad = 0;
    J.leaf_sum[0] = r;
  }
}

// ---- score update / leaf lookup over the final partition ----
// The leaves' row ranges tile the positions 0 .. root count of the index buffers, so every CTA takes
// the same number of positions (`per`), whatever the leaves' sizes: it lists the leaves that overlap
// them (one thread per leaf), then walks those parts, four positions a thread in flight. (A grid over
// leaves left the chip to the largest ones: the score update of ten 63-leaf trees on 2M rows took 515
// us, now 132.) Bound by the scattered 8-byte updates: 10M rows, whose score outgrows L2, 167 us.
constexpr int kLeafParts = 256;  // leaves looked at per pass

// Calls f(leaf, rows[4]) for this CTA's rows (-1: none). All 256 threads call it.
template <typename F>
__device__ __forceinline__ void for_leaf_rows(const Job& J, const Params& p, int per, F f) {
  __shared__ int32_t s_leaf[kLeafParts], s_n;
  const int32_t leaves = J.st->tree_leaves;
  const int64_t q0 = (int64_t)blockIdx.x * per, q1 = q0 + per;
  for (int32_t l0 = 0; l0 < leaves; l0 += kLeafParts) {
    if (threadIdx.x == 0) s_n = 0;
    __syncthreads();
    const int32_t l = l0 + (int32_t)threadIdx.x;
    static_assert(kLeafParts == 256, "one leaf per thread");
    if (l < leaves) {
      const int64_t b = J.leaf_begin[l], c = J.leaf_count[l];
      if (b < q1 && b + c > q0) s_leaf[atomicAdd(&s_n, 1)] = l;
    }
    __syncthreads();
    for (int k = 0; k < s_n; ++k) {
      const int32_t leaf = s_leaf[k];
      const int64_t b = J.leaf_begin[leaf], c = J.leaf_count[leaf];
      const int32_t* idx = leaf_idx(J, J.leaf_buf[leaf]);
      const bool all = c == p.n;  // every row, in order
      const int64_t e0 = max(b, q0), e1 = min(b + c, q1);
      for (int64_t i = e0 + threadIdx.x; i < e1; i += 4 * 256) {
        int32_t row[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) row[u] = i + u * 256 < e1 ? (all ? (int32_t)(i + u * 256) : idx[i + u * 256]) : -1;
        f(leaf, row);
      }
    }
    __syncthreads();
  }
}

__device__ __forceinline__ void add_rows(double* __restrict__ sc, const int32_t (&row)[4], double v) {
  double x[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) x[u] = row[u] >= 0 ? sc[row[u]] : 0.0;
#pragma unroll
  for (int u = 0; u < 4; ++u)
    if (row[u] >= 0) sc[row[u]] = x[u] + v;
}

__global__ void __launch_bounds__(256) k_add_score(const Job* __restrict__ jobs, Params p, int per,
                                                   const double* __restrict__ vals, double* __restrict__ score) {
  const Job& J = jobs[blockIdx.z];
  if (J.st->tree_leaves <= 1) return;
  const double* v = vals + (size_t)blockIdx.z * p.num_leaves;
  double* sc = score + (size_t)blockIdx.z * p.n;
  for_leaf_rows(J, p, per, [&](int32_t leaf, const int32_t (&row)[4]) { add_rows(sc, row, v[leaf]); });
}

// The same update with the tree's own leaf outputs from the device, shrunk as Tree::apply_shrinkage
// does (tree.rs:446-463): score += round_to_zero(leaf_value * rate). A one-leaf tree adds nothing
// (train.rs:776-795 turns it into a constant tree instead).
__global__ void __launch_bounds__(256) k_add_score_own(const Job* __restrict__ jobs, Params p, int per, double rate,
                                                       double* __restrict__ score, int need_stop) {
  const Job& J = jobs[blockIdx.z];
  for (int j = 0; need_stop && j < (int)gridDim.z; ++j)
    if (!jobs[j].st->stop) return;  // the trees need more rounds: the update comes after those
  if (J.st->tree_leaves <= 1) return;
  double* sc = score + (size_t)blockIdx.z * p.n;
  for_leaf_rows(J, p, per, [&](int32_t leaf, const int32_t (&row)[4]) {
    double v = __dmul_rn(J.leaf_value[leaf], rate);
    if (v >= -BK_ZERO_THRESHOLD && v <= BK_ZERO_THRESHOLD) v = 0.0;
    add_rows(sc, row, v);
  });
}

__global__ void __launch_bounds__(256) k_row_leaf(const Job* __restrict__ jobs, Params p, int per,
                                                  int32_t* __restrict__ out, int need_stop) {
  const Job& J = jobs[blockIdx.z];
  if (need_stop && !J.st->stop) return;
  int32_t* o = out + (size_t)blockIdx.z * p.n;
  for_leaf_rows(J, p, per, [&](int32_t leaf, const int32_t (&row)[4]) {
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (row[u] >= 0) o[row[u]] = leaf;
  });
}

// Positions per CTA: about eight CTAs per SM, 256 to 4096.
static int leaf_rows_per(const Params& p) {
  const int64_t per = ceil_div64(ceil_div64(p.n, 1216), 256) * 256;
  return (int)std::min<int64_t>(std::max<int64_t>(per, 256), 4096);
}
static dim3 leaf_rows_grid(const Params& p, int num_jobs) {
  return dim3((unsigned)ceil_div64(p.n, leaf_rows_per(p)), 1, num_jobs);
}

__global__ void k_zero_pool(uint4* __restrict__ pool, size_t per_job, size_t n) {
  uint4* z = pool + (size_t)blockIdx.z * per_job;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    z[i] = make_uint4(0, 0, 0, 0);
}

}  // namespace

void launch_job_begin(const Job* d_jobs, int num_jobs, bool use_rows, int64_t root_count, cudaStream_t s) {
  k_job_begin<<<1, 32, 0, s>>>(d_jobs, num_jobs, use_rows ? 1 : 0, root_count);
}

void launch_results(const void* results, void* h_results, size_t bytes, const JobState* states, JobState* h_states,
                    int num_jobs, cudaStream_t s) {
  const int n16 = (int)(bytes / 16), grid = std::min(32, 1 + n16 / 256);
  k_results<<<grid, 256, 0, s>>>(static_cast<const uint4*>(results), static_cast<uint4*>(h_results), n16, states, h_states,
                                 num_jobs);
}

void launch_init_rows(const Job* d_jobs, int num_jobs, const Params& p, const int32_t* rows, bool bagged_only,
                      cudaStream_t s) {
  k_init_rows<<<dim3(1024, 1, num_jobs), 256, 0, s>>>(d_jobs, p, rows, bagged_only ? 1 : 0);
}

void launch_mt_seed(const Job* d_jobs, int num_jobs, uint32_t seed, cudaStream_t s) {
  (void)num_jobs;  // one engine, held by job 0
  k_mt_seed<<<1, 1, 0, s>>>(d_jobs, seed);
}

void launch_noise_f32(const double* a, float* b, int64_t n, cudaStream_t s) { k_noise_f32<<<1024, 256, 0, s>>>(a, b, n); }

void launch_discretize(const Job* d_jobs, int num_jobs, const Params& p, const double* noise_g, const double* noise_h,
                       const float* noise_gf, const float* noise_hf, cudaStream_t s) {
  k_disc_reset<<<dim3(1, 1, num_jobs), 1, 0, s>>>(d_jobs);
  const unsigned grid = (unsigned)std::min<int64_t>(ceil_div64(p.n, 1024), 1216);
  k_disc_reduce<<<dim3(grid, 1, num_jobs), 256, 0, s>>>(d_jobs, p);
  k_disc_setup<<<1, 32, 0, s>>>(d_jobs, num_jobs, p);
  k_discretize<<<dim3(kRootGrid, 1, num_jobs), 256, 0, s>>>(d_jobs, p, noise_g, noise_h, noise_gf, noise_hf);
}

void launch_root_sums(const Job* d_jobs, int num_jobs, const Params& p, int exact_quant_root, cudaStream_t s) {
  k_root_partial<<<dim3(p.quant ? kRootGrid : kFloatRootGrid, 1, num_jobs), 256, 0, s>>>(d_jobs, p);
  k_root_finish<<<dim3(1, 1, num_jobs), 32, 0, s>>>(d_jobs, p, exact_quant_root);
}

void launch_add_score(const Job* d_jobs, int num_jobs, const Params& p, const double* leaf_vals, double* score,
                      cudaStream_t s) {
  k_add_score<<<leaf_rows_grid(p, num_jobs), 256, 0, s>>>(d_jobs, p, leaf_rows_per(p), leaf_vals, score);
}

void launch_add_score_own(const Job* d_jobs, int num_jobs, const Params& p, double rate, double* score, int need_stop,
                          cudaStream_t s) {
  k_add_score_own<<<leaf_rows_grid(p, num_jobs), 256, 0, s>>>(d_jobs, p, leaf_rows_per(p), rate, score, need_stop);
}

void launch_zero_pool(void* pool, size_t bytes_per_job, size_t bytes, int num_jobs, cudaStream_t s) {
  k_zero_pool<<<dim3(1024, 1, num_jobs), 256, 0, s>>>(reinterpret_cast<uint4*>(pool), bytes_per_job / 16, bytes / 16);
}

void launch_row_leaf(const Job* d_jobs, int num_jobs, const Params& p, int32_t* out, int need_stop, cudaStream_t s) {
  k_row_leaf<<<leaf_rows_grid(p, num_jobs), 256, 0, s>>>(d_jobs, p, leaf_rows_per(p), out, need_stop);
}

}  // namespace bk
