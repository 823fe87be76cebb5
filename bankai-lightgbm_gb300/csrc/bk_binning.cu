// Dense bin construction on the device: the O(rows x features) part of Dataset::from_dense and
// Dataset::from_dense_reference (io/dataset.rs:633-685 fill_dense, io/dataset.rs:987-1003), with
// BinMapper::value_to_bin (io/bin.rs:558-589) per value. The bin mappers themselves (upper bounds,
// missing type, most frequent bin) come from the host's BinMapper::find_bin over a row sample, as
// in the reference; this file turns a device-resident value matrix into the learner's stored-bin
// columns.
//
// Layout: the values are row-major [num_data][num_columns], f64 or f32. A CTA owns 16 used
// features and a run of rows; the flat grid runs feature groups fastest, so the CTAs that read the
// same rows' lines run side by side. It walks its rows in tiles of 256: a tile's values go to shared
// memory feature by feature while the next tile's are on their way; then a warp bins 256 rows of one
// feature, eight rows per lane at a time, and each feature's 256 stored bins leave as 4-byte words.
//
// The number of bounds below a value is value_to_bin's binary-search result for sorted bounds. A value
// first finds its bucket among 512 by a function that never decreases (one multiply-add in f32, clamped),
// the same function of the bounds: the bounds of lower buckets are below the value, those of higher
// ones above it, so the search covers the bounds of one bucket only, with as many steps as the
// feature's fullest bucket needs (two for the 254 quantiles of a normal distribution, eight at worst).
// Instructions and shared-memory wavefronts (a warp's random reads of a table cost about three) bound
// the kernel, and every step takes four of the former. 3M rows x 100 features, f32: 1900 us a call with
// eight steps over the sorted bounds, 1090 with eight over a tree laid out by levels, 730 so (f64: 4150
// -> 1270). Searching in the layout of the loads, 16 features to a warp, saves the values' way through
// shared memory but not time: its reads conflict more.
//
// GB300 issues one warp f64 instruction per 64 cycles per SM sub-partition, so no f64 arithmetic
// runs per value: f64 searches compare order-preserving integer keys built from the bits (-0.0 folded
// into +0.0, as the f64 comparison treats them). An f32 value is compared in f32 against its bound
// rounded down to f32, which is exact: a float v satisfies v <= ub exactly when v <= the largest float
// not above ub.
#include <cuda_runtime.h>
#include <math_constants.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <mutex>
#include <vector>

#include "bk_common.cuh"
#include "bkgpu.h"

namespace bk {

namespace {

constexpr int kBinRows = 256;     // rows per tile
constexpr int kBinTiles = 16;     // tiles per CTA at most
constexpr int kBinFeatures = 16;  // used features per CTA
constexpr int kBinThreads = 256;
constexpr int kBinCtas = 1216;    // CTAs to spread the rows over before a CTA takes more tiles

struct BinFeature {
  int32_t real, num_bin, missing, mfb, ub_off;
};

// A feature's search: the bucket function and the steps of the search within a bucket.
struct BinSearch {
  float a, b;
  int32_t steps, _pad;
};
constexpr int kBuckets = 512;

// In [2^23, 2^24) a float's last bit is 1: the addend's 2^23 makes the sum's low bits the bucket. The
// rounding, the clamps (which a NaN sum passes as the lower one) and the mask never decrease.
__device__ __forceinline__ uint32_t bucket_of(float v, float a, float b) {
  const float u = fminf(fmaxf(fmaf(v, a, b), 8388608.0f), 8388608.0f + (kBuckets - 1));
  return __float_as_uint(u) & (kBuckets - 1);
}

// What the search compares: f32 values themselves, int64 keys of f64 values whose signed order is the
// order of the non-NaN values. `pitch`: the distance of two features' rows in shared memory, so that
// storing 16 features of one or two rows hits different banks.
template <typename T>
struct KeyOf;
template <>
struct KeyOf<double> {
  using K = long long;
  static constexpr int kPitch = kBinRows + 1;
  static constexpr K kNan = (K)0x8000000000000000ULL;  // below every value's key
  __device__ static K key(double v) {
    long long b = __double_as_longlong(v);
    if ((b << 1) == 0) b = 0;  // -0.0
    return b ^ ((b >> 63) & 0x7fffffffffffffffLL);
  }
  __device__ static K bound(double ub) { return key(ub); }
  __device__ static bool nan(double v) { return (__double_as_longlong(v) & 0x7fffffffffffffffLL) > 0x7ff0000000000000LL; }
  __device__ static bool is_nan(K k) { return k == kNan; }
  __device__ static K nan_key() { return kNan; }
  // the value of a key, truncated to a float's precision and range (which never decreases)
  __device__ static float approx(K k) {
    const unsigned long long b = (unsigned long long)(k ^ ((k >> 63) & 0x7fffffffffffffffLL));
    const uint32_t hi = (uint32_t)(b >> 32), abs_hi = hi & 0x7fffffffu;
    uint32_t f = __funnelshift_l((uint32_t)b, abs_hi - (896u << 20), 3);
    if (abs_hi < (897u << 20)) f = 0u;
    if (abs_hi >= (1151u << 20)) f = 0x7f7fffffu;
    return __uint_as_float(f | (hi & 0x80000000u));
  }
};
template <>
struct KeyOf<float> {
  using K = float;
  static constexpr int kPitch = kBinRows + 2;
  __device__ static K key(float v) { return v; }
  __device__ static K bound(double ub) { return __double2float_rd(ub); }
  __device__ static bool nan(float v) { return isnan(v); }
  __device__ static bool is_nan(K k) { return isnan(k); }
  __device__ static K nan_key() { return CUDART_NAN_F; }
  __device__ static float approx(K k) { return k; }
};

// The searched bounds of a feature.
__device__ __forceinline__ int searched_bounds(const BinFeature& m) { return m.num_bin - 1 - (m.missing == 2 ? 1 : 0); }

// One CTA per feature: its bounds' keys (+inf past the searched ones), its bucket function, and for each
// bucket the number of bounds in lower ones, where its search starts (at most 256 - 2^steps, so that
// the steps stay inside the keys; starting lower changes nothing, those bounds are below the value).
template <typename T>
__global__ void __launch_bounds__(256)
    k_bin_tables(const BinFeature* __restrict__ feats, const double* __restrict__ ub, typename KeyOf<T>::K* __restrict__ keys,
                 uint8_t* __restrict__ starts, BinSearch* __restrict__ search) {
  using KO = KeyOf<T>;
  __shared__ uint32_t bucket[256];
  __shared__ int32_t start[kBuckets + 1], most;
  const BinFeature m = feats[blockIdx.x];
  const int i = (int)threadIdx.x, rr = max(searched_bounds(m), 0);
  const typename KO::K key = KO::bound(i < rr ? ub[m.ub_off + i] : CUDART_INF);
  keys[(size_t)blockIdx.x * 256 + i] = key;
  BinSearch s{0.f, 8388608.0f, 0, 0};
  if (rr > 1) {
    const float first = KO::approx(KO::bound(ub[m.ub_off])), last = KO::approx(KO::bound(ub[m.ub_off + rr - 1]));
    const float a = (kBuckets - 1) / (last - first), b = fmaf(-first, a, 8388608.0f);
    if (a > 0.f && a < 1e30f && fabsf(b) < 1e30f) s.a = a, s.b = b;
  }
  bucket[i] = bucket_of(KO::approx(key), s.a, s.b);
  for (int k = i; k <= kBuckets; k += 256) start[k] = 0;  // bounds out of order would leave gaps
  if (i == 0) most = 0;
  __syncthreads();
  // the buckets after bound i - 1's and up to bound i's start at i
  if (i <= rr) {
    const int from = i == 0 ? 0 : (int)bucket[i - 1] + 1, to = i == rr ? kBuckets : (int)bucket[i];
    for (int k = from; k <= to; ++k) start[k] = i;
  }
  __syncthreads();
  for (int k = i; k < kBuckets; k += 256) atomicMax(&most, start[k + 1] - start[k]);
  __syncthreads();
  s.steps = most > 0 ? min(32 - __clz(most), 8) : 0;
  for (int k = i; k < kBuckets; k += 256)
    starts[(size_t)blockIdx.x * kBuckets + k] = (uint8_t)min(start[k], 256 - (1 << s.steps));
  if (i == 0) search[blockIdx.x] = s;
}

template <typename K, int PITCH>
struct BinSmem {
  K keys[kBinFeatures][256];
  K xs[kBinFeatures * PITCH];
  uint8_t starts[kBinFeatures][kBuckets];
  uint8_t stage[kBinFeatures][kBinRows + 16];
  BinSearch ss[kBinFeatures];
  BinFeature sf[kBinFeatures];
};

template <typename T>
__global__ void __launch_bounds__(kBinThreads, sizeof(T) == 4 ? 4 : 2)
    k_bin_dense(const T* __restrict__ X, int64_t n, int32_t ncol, const BinFeature* __restrict__ feats, int32_t F,
                const typename KeyOf<T>::K* __restrict__ keys, const uint8_t* __restrict__ starts,
                const BinSearch* __restrict__ search, int tiles, uint8_t* __restrict__ out) {
  using KO = KeyOf<T>;
  using K = typename KO::K;
  constexpr int kPerThread = kBinRows * kBinFeatures / kBinThreads, kRowStep = kBinThreads / kBinFeatures;
  extern __shared__ __align__(16) unsigned char bin_smem[];
  using Smem = BinSmem<K, KO::kPitch>;
  Smem& S = *reinterpret_cast<Smem*>(bin_smem);
  const int ngroups = (F + kBinFeatures - 1) / kBinFeatures;
  const int g0 = (int)(blockIdx.x % (unsigned)ngroups) * kBinFeatures;
  const int64_t row0 = (int64_t)(blockIdx.x / (unsigned)ngroups) * tiles * kBinRows;
  const int gf = min(kBinFeatures, F - g0);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // a thread reads one feature's values, rows tr, tr + 16, ... of the tile
  const int tf = threadIdx.x & (kBinFeatures - 1), tr = threadIdx.x / kBinFeatures;
  BinFeature mine{};
  if (tf < gf) mine = feats[g0 + tf];
  const T* src = X + (row0 + tr) * (int64_t)ncol + mine.real;
  const int64_t step = (int64_t)kRowStep * ncol;
  const bool whole = gf == kBinFeatures;
  T v[kPerThread];
  auto fetch = [&](int64_t r0) {
    const T* q = src;
    if (whole && r0 + kBinRows <= n) {
#pragma unroll
      for (int k = 0; k < kPerThread; ++k, q += step) v[k] = *q;
    } else {
#pragma unroll
      for (int k = 0; k < kPerThread; ++k, q += step) v[k] = (tf < gf && r0 + tr + k * kRowStep < n) ? *q : (T)0;
    }
    src += (int64_t)kBinRows * ncol;
  };
  fetch(row0);
  if (threadIdx.x < gf) {
    S.sf[threadIdx.x] = feats[g0 + threadIdx.x];
    S.ss[threadIdx.x] = search[g0 + threadIdx.x];
  }
  {
    const uint4* ks = reinterpret_cast<const uint4*>(keys + (size_t)g0 * 256);
    uint4* kd = reinterpret_cast<uint4*>(&S.keys[0][0]);
    for (int e = threadIdx.x; e < gf * 256 * (int)sizeof(K) / 16; e += kBinThreads) kd[e] = ks[e];
    const uint4* bs = reinterpret_cast<const uint4*>(starts + (size_t)g0 * kBuckets);
    uint4* bd = reinterpret_cast<uint4*>(&S.starts[0][0]);
    for (int e = threadIdx.x; e < gf * kBuckets / 16; e += kBinThreads) bd[e] = bs[e];
  }
  // value_to_bin's NaN: its own bin (missing NaN) or the value 0.0
  const K nan_as = mine.missing == 2 ? KO::nan_key() : KO::key((T)0);
  for (int tile = 0; tile < tiles; ++tile) {
    const int64_t r0 = row0 + (int64_t)tile * kBinRows;
    if (r0 >= n) break;  // uniform
    const int rows = (int)min((int64_t)kBinRows, n - r0);
#pragma unroll
    for (int k = 0; k < kPerThread; ++k)
      S.xs[tf * KO::kPitch + tr + k * kRowStep] = KO::nan(v[k]) ? nan_as : KO::key(v[k]);
    if (tile + 1 < tiles) fetch(r0 + kBinRows);
    __syncthreads();  // the tile's values (and, the first time, the tables) are complete
    for (int fi = warp; fi < gf; fi += kBinThreads / 32) {
      const BinFeature m = S.sf[fi];
      const BinSearch bs = S.ss[fi];
      const unsigned char* kb = reinterpret_cast<const unsigned char*>(&S.keys[fi][0]);
      K x[kBinRows / 32];
      uint32_t at[kBinRows / 32];  // byte offset of the first key not known to be below
#pragma unroll
      for (int k = 0; k < kBinRows / 32; ++k) {
        x[k] = S.xs[fi * KO::kPitch + lane + 32 * k];
        at[k] = S.starts[fi][bucket_of(KO::approx(x[k]), bs.a, bs.b)] * (uint32_t)sizeof(K);
      }
#pragma unroll 1
      for (uint32_t st = (uint32_t)sizeof(K) << bs.steps >> 1; st >= (uint32_t)sizeof(K); st >>= 1) {
#pragma unroll
        for (int k = 0; k < kBinRows / 32; ++k)
          if (*reinterpret_cast<const K*>(kb + at[k] + st - sizeof(K)) < x[k]) at[k] += st;
      }
      // fill_dense: the most frequent bin is stored as 0, the others shift past it
      const uint32_t shift = m.mfb == 0 ? 0u : 1u, zero = (uint32_t)m.mfb + shift;
      const uint32_t nan_bin = (uint32_t)m.num_bin - 1u + shift;
#pragma unroll
      for (int k = 0; k < kBinRows / 32; ++k) {
        uint32_t b = at[k] / (uint32_t)sizeof(K) + shift;
        if (KO::is_nan(x[k])) b = nan_bin;
        S.stage[fi][lane + 32 * k] = (uint8_t)(b == zero ? 0u : b);
      }
      __syncwarp();
      // the feature's bins, 4 bytes at a time from the first aligned address on
      uint8_t* dst = out + (size_t)(g0 + fi) * (size_t)n + (size_t)r0;
      const int head = min(rows, (int)((0u - (uint32_t)reinterpret_cast<uintptr_t>(dst)) & 3u)), words = (rows - head) / 4;
      const uint32_t* st = reinterpret_cast<const uint32_t*>(&S.stage[fi][0]);
      for (int w = lane; w < words; w += 32)
        reinterpret_cast<uint32_t*>(dst + head)[w] = __funnelshift_r(st[w], st[w + 1], 8 * head);
      if (lane < head) dst[lane] = S.stage[fi][lane];
      const int tail = head + 4 * words + lane;
      if (lane < 4 && tail < rows) dst[tail] = S.stage[fi][tail];
    }
    __syncthreads();  // the values are done with
  }
}

// The smallest flat index (feature * n + row) whose stored bin is outside its feature's
// [0, gbins), or INT64_MAX: the reference's BinsCheck (histogram.rs:50-65) over device columns.
__global__ void __launch_bounds__(256)
    k_check_bins(const uint8_t* __restrict__ bins, int64_t n, const DevFeature* __restrict__ feats,
                 unsigned long long* first_bad) {
  const int f = blockIdx.y;
  const uint32_t gb = (uint32_t)feats[f].gbins;
  const uint8_t* col = bins + (size_t)f * (size_t)n;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    if ((uint32_t)col[i] >= gb) atomicMin(first_bad, (unsigned long long)((int64_t)f * n + i));
}

}  // namespace

cudaError_t check_bins_device(const uint8_t* bins, int64_t n, int32_t F, const DevFeature* d_feat,
                              int64_t* first_bad, cudaStream_t s) {
  unsigned long long* d_bad = nullptr;
  cudaError_t e = cudaMalloc(&d_bad, sizeof(unsigned long long));
  if (e != cudaSuccess) return e;
  const unsigned long long none = ~0ull;
  e = cudaMemcpyAsync(d_bad, &none, sizeof(none), cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) {
    const int gx = (int)std::min<int64_t>(ceil_div64(n, 256), 64);
    k_check_bins<<<dim3(gx, F), 256, 0, s>>>(bins, n, d_feat, d_bad);
    e = cudaGetLastError();
  }
  unsigned long long h = none;
  if (e == cudaSuccess) e = cudaMemcpyAsync(&h, d_bad, sizeof(h), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  cudaFree(d_bad);
  *first_bad = h == none ? INT64_MAX : (int64_t)h;
  return e;
}

}  // namespace bk

using namespace bk;

namespace {

void bin_error(const char* msg) { bk_set_last_error(msg); }

template <typename A0, typename... A>
void bin_error(const char* fmt, A0 a0, A... a) {
  char buf[256];
  snprintf(buf, sizeof(buf), fmt, a0, a...);
  bk_set_last_error(buf);
}

// A call's tables (keys, searches, buckets' starts, bounds, features) come from a stream-ordered pool of
// the device that keeps at most 64 MB between calls (it grows by 32): cudaMalloc and cudaFree took 200
// of a small call's 250 us. Without a pool, cudaMalloc.
constexpr uint64_t kPoolKeep = 64ull << 20;

cudaMemPool_t bin_pool() {
  constexpr int kMaxDevices = 64;
  static std::mutex m;
  static cudaMemPool_t pools[kMaxDevices] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return nullptr;
  std::lock_guard<std::mutex> g(m);
  if (!pools[dev]) {
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t pool = nullptr;
    uint64_t keep = kPoolKeep;
    if (cudaMemPoolCreate(&pool, &props) == cudaSuccess &&
        cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep) == cudaSuccess)
      pools[dev] = pool;
  }
  return pools[dev];
}

template <typename T>
cudaError_t bin_launch(const T* values, int64_t n, int32_t ncol, const BinFeature* h_f, int32_t F, const double* ub,
                       size_t nub, int tiles, unsigned blocks, uint8_t* out, cudaStream_t s) {
  using K = typename KeyOf<T>::K;
  const size_t keys = 0, search = keys + (size_t)F * 256 * sizeof(K), starts = search + (size_t)F * sizeof(BinSearch),
               bounds = starts + (size_t)F * kBuckets, feats = bounds + nub * sizeof(double),
               bytes = feats + (size_t)F * sizeof(BinFeature);
  unsigned char* d = nullptr;
  cudaMemPool_t pool = bin_pool();
  cudaError_t e = pool ? cudaMallocFromPoolAsync(&d, bytes, pool, s) : cudaErrorNotSupported;
  const bool pooled = e == cudaSuccess;
  if (!pooled) {
    (void)cudaGetLastError();
    e = cudaMalloc(&d, bytes);
  }
  if (e != cudaSuccess) return e;
  const int smem = (int)sizeof(BinSmem<K, KeyOf<T>::kPitch>);
  e = cudaFuncSetAttribute(k_bin_dense<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e == cudaSuccess) e = cudaMemcpyAsync(d + feats, h_f, (size_t)F * sizeof(BinFeature), cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(d + bounds, ub, nub * sizeof(double), cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) {
    const BinFeature* d_f = reinterpret_cast<const BinFeature*>(d + feats);
    K* d_keys = reinterpret_cast<K*>(d + keys);
    BinSearch* d_search = reinterpret_cast<BinSearch*>(d + search);
    k_bin_tables<T><<<F, 256, 0, s>>>(d_f, reinterpret_cast<const double*>(d + bounds), d_keys, d + starts, d_search);
    k_bin_dense<T><<<blocks, kBinThreads, smem, s>>>(values, n, ncol, d_f, F, d_keys, d + starts, d_search, tiles, out);
    e = cudaGetLastError();
  }
  if (pooled) (void)cudaFreeAsync(d, s);
  const cudaError_t done = cudaStreamSynchronize(s);
  if (e == cudaSuccess) e = done;
  if (!pooled) (void)cudaFree(d);
  return e;
}

}  // namespace

extern "C" int bk_bin_dense_device(const void* values, int32_t value_type, int64_t num_data, int32_t num_columns,
                                   const bk_feature* features, int32_t num_features, const double* upper_bounds,
                                   const int32_t* bound_offsets, uint8_t* out, void* stream) {
  if (!values || !features || !upper_bounds || !bound_offsets || !out || num_data <= 0 || num_columns <= 0 ||
      num_features <= 0 || (value_type != 0 && value_type != 1)) {
    bin_error("bk_bin_dense_device: invalid arguments");
    return -1;
  }
  std::vector<BinFeature> hf((size_t)num_features);
  for (int f = 0; f < num_features; ++f) {
    const bk_feature& x = features[f];
    const int32_t nb = x.num_bin, off = x.most_freq_bin == 0 ? 1 : 0;
    if (x.bin_type != 0) {
      bin_error("bk_bin_dense_device: feature %d is categorical; device binning takes numerical features", f);
      return -1;
    }
    if (x.real_feature < 0 || x.real_feature >= num_columns || nb < 1 || 1 + nb - off > 256 ||
        x.missing_type < 0 || x.missing_type > 2 || x.most_freq_bin < 0 || x.most_freq_bin >= nb ||
        bound_offsets[f] < 0 || bound_offsets[f + 1] - bound_offsets[f] != nb) {
      bin_error("bk_bin_dense_device: feature %d: bad bin mapper", f);
      return -1;
    }
    hf[(size_t)f] = BinFeature{x.real_feature, nb, x.missing_type, x.most_freq_bin, bound_offsets[f]};
  }
  const size_t nub = (size_t)bound_offsets[num_features];
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // one flat grid, feature groups fastest: the CTAs reading the same rows' lines run side by side
  const int64_t groups = ceil_div64(num_features, kBinFeatures), all_tiles = ceil_div64(num_data, (int64_t)kBinRows);
  const int tiles = (int)std::min<int64_t>(kBinTiles, std::max<int64_t>(1, all_tiles * groups / kBinCtas));
  const int64_t blocks = groups * ceil_div64(all_tiles, (int64_t)tiles);
  if (blocks > INT32_MAX) {
    bin_error("bk_bin_dense_device: too many rows x features for one launch");
    return -1;
  }
  const cudaError_t e =
      value_type == 0 ? bin_launch(static_cast<const double*>(values), num_data, num_columns, hf.data(), num_features,
                                   upper_bounds, nub, tiles, (unsigned)blocks, out, s)
                      : bin_launch(static_cast<const float*>(values), num_data, num_columns, hf.data(), num_features,
                                   upper_bounds, nub, tiles, (unsigned)blocks, out, s);
  if (e != cudaSuccess) {
    bin_error("bk_bin_dense_device: %s", cudaGetErrorString(e));
    return -1;
  }
  return 0;
}
