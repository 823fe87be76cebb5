// Quantized leaf renewal (quant_train_renew_leaf, serial.rs:634-655): every leaf's output from its rows'
// original gradients and hessians, whose f64 sums the reference takes one row after the other in leaf
// row order (the stable compaction's: the root's row order within a leaf).
//
// A sequential f64 sum costs an addition's latency a row (40 ns: 2.4 ms for a leaf of 60,000 rows, half
// of a 500k-row iteration). But while a sum stays below 2^53 multiples of the lowest bit seen, no
// addition rounds, and its value is the exact sum, in any order. So the rows are cut into chunks of 256
// per leaf; a warp sums up each chunk in integers (total, largest and smallest partial sum, as multiples
// of the chunk's lowest bit), and one warp per leaf joins the chunks in order: where every partial
// sum is representable the total is added exactly, otherwise the chunk's rows are added one by one, as
// the reference does. Gradients round for values near zero only: of 500k rows a handful of chunks take
// that way (2414 us -> 13 for the chunks and 24 for joining them).
//
// Grow rounds leave a leaf's rows in no particular order, so they are first grouped by leaf in the
// root's order (a counting sort: counts per 2048 rows and leaf, their prefix sums, a stable scatter; 22
// us for 500k rows, where growing one split at a time with a stable partition took 1850 us for the 62
// splits that the rounds grow in 350).
#include <algorithm>

#include "bk_math.cuh"

namespace bk {

namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr int kChunk = 256;       // rows per chunk: eight per lane
constexpr int kGroupRows = 2048;  // rows per CTA of the grouping
constexpr int kNoBit = 0x7fff;    // lowest bit of zero

// A chunk's partial sums of one quantity, multiples of 2^(low - 150).
struct __align__(16) ChunkSum {
  long long total, most, least;
  int32_t low, bad;  // bad: not finite, or too wide for 64 bits
};

struct RenewView {
  const int32_t* idx;  // the leaf's rows in order, or null: every row
  int64_t cnt;
};

__device__ __forceinline__ RenewView renew_view(const Job& J, const Params& p, int32_t leaf, const int32_t* order) {
  RenewView v;
  v.cnt = J.leaf_count[leaf];
  const int64_t begin = J.leaf_begin[leaf];
  v.idx = v.cnt == p.n ? nullptr : (order ? order + (size_t)blockIdx.z * p.n : leaf_idx(J, J.leaf_buf[leaf])) + begin;
  return v;
}

// The place of a leaf's first chunk: the chunks of the leaves before it. Every thread calls it.
__device__ __forceinline__ int64_t first_chunk(const Job& J, int32_t leaf, int nthreads) {
  __shared__ int64_t part[8];
  int64_t s = 0;
  for (int32_t l = (int32_t)threadIdx.x; l < leaf; l += nthreads) s += ceil_div64(J.leaf_count[l], kChunk);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(FULL, s, o);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
  __syncthreads();
  s = 0;
  for (int w = 0; w < nthreads / 32; ++w) s += part[w];
  return s;
}

// The lowest bit of a non-zero finite value and its biased exponent (at least 1).
__device__ __forceinline__ void bits_of(float v, uint32_t* m, int* e) {
  const uint32_t u = __float_as_uint(v) & 0x7fffffffu;
  *e = max((int)(u >> 23), 1);
  *m = (u & 0x7fffffu) | ((u >> 23) ? 0x800000u : 0u);
}

// One warp: the summary of eight values a lane, in lane order.
__device__ __forceinline__ ChunkSum sum_chunk(const float (&v)[8], int lane) {
  int low = kNoBit, high = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    uint32_t m;
    int e;
    bits_of(v[i], &m, &e);
    if (m) {
      low = min(low, e + __ffs((int)m) - 1);
      high = max(high, e);
    }
  }
  low = __reduce_min_sync(FULL, low);
  high = __reduce_max_sync(FULL, high);
  ChunkSum c;
  c.total = c.most = c.least = 0;
  c.low = low;
  c.bad = high >= 255 || high + 24 - low > 52;  // 256 values below 2^52: below 2^60
  if (low == kNoBit) c.bad = 0;
  if (low == kNoBit || c.bad) return c;
  long long s = 0, most = 0, least = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    uint32_t m;
    int e;
    bits_of(v[i], &m, &e);
    const long long x = !m ? 0 : (e >= low ? (long long)m << (e - low) : (long long)(m >> (low - e)));
    s += v[i] < 0.f ? -x : x;
    most = max(most, s);
    least = min(least, s);
  }
  long long incl = s;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const long long u = __shfl_up_sync(FULL, incl, o);
    if (lane >= o) incl += u;
  }
  most += incl - s;
  least += incl - s;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    most = max(most, (long long)__shfl_xor_sync(FULL, most, o));
    least = min(least, (long long)__shfl_xor_sync(FULL, least, o));
  }
  c.total = __shfl_sync(FULL, incl, 31);
  c.most = most;
  c.least = least;
  return c;
}

__global__ void __launch_bounds__(256) k_renew_chunks(const Job* __restrict__ jobs, Params p,
                                                      const int32_t* __restrict__ order, ChunkSum* __restrict__ sums,
                                                      int64_t slots, int need_stop) {
  const Job& J = jobs[blockIdx.z];
  const int32_t leaf = (int32_t)blockIdx.x;
  if ((need_stop && !J.st->stop) || leaf >= J.st->tree_leaves) return;
  const RenewView v = renew_view(J, p, leaf, order);
  const int64_t chunks = ceil_div64(v.cnt, kChunk);
  if ((int64_t)blockIdx.y * 8 >= chunks) return;
  ChunkSum* out = sums + 2 * ((size_t)blockIdx.z * slots + first_chunk(J, leaf, 256));
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int64_t c = (int64_t)blockIdx.y * 8 + warp; c < chunks; c += (int64_t)gridDim.y * 8) {
    float g[8], h[8];
    int32_t row[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int64_t k = c * kChunk + lane * 8 + i;
      row[i] = k < v.cnt ? (v.idx ? v.idx[k] : (int32_t)k) : -1;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      g[i] = row[i] >= 0 ? J.g[row[i]] : 0.f;
      h[i] = row[i] >= 0 ? J.h[row[i]] : 0.f;
    }
    const ChunkSum a = sum_chunk(g, lane), b = sum_chunk(h, lane);
    if (lane == 0) {
      out[2 * c] = a;
      out[2 * c + 1] = b;
    }
  }
}

// A double as an odd multiple of 2^(low - 150), or zero; false when it is not finite.
struct ExactSum {
  long long s;
  int low;
};
__device__ __forceinline__ bool split_double(double x, ExactSum* r) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x), a = b & 0x7fffffffffffffffULL;
  const int e = max((int)(a >> 52), 1);
  if ((a >> 52) == 0x7ff) return false;
  const long long m = (long long)((a & 0xfffffffffffffULL) | ((a >> 52) ? 0x10000000000000ULL : 0));
  r->s = 0;
  r->low = kNoBit;
  if (m) {
    const int z = __ffsll(m) - 1;
    r->s = (b >> 63) ? -(m >> z) : m >> z;
    r->low = e - 1075 + 150 + z;
  }
  return true;
}
__device__ __forceinline__ double join_double(const ExactSum& x) {  // |s| <= 2^53
  return x.s == 0 ? 0.0 : (double)x.s * __longlong_as_double((long long)(x.low - 150 + 1023) << 52);
}

// x plus a chunk, if no partial sum rounds.
__device__ __forceinline__ bool add_chunk(ExactSum* x, const ChunkSum& c) {
  if (c.bad) return false;
  if (c.low == kNoBit) return true;
  const int low = x->s ? min(x->low, c.low) : c.low;
  const int ds = x->s ? x->low - low : 0, dc = c.low - low;
  const unsigned long long as = (unsigned long long)llabs(x->s), ac = (unsigned long long)max(llabs(c.most), llabs(c.least));
  if ((as && 64 - __clzll((long long)as) + ds > 61) || (ac && 64 - __clzll((long long)ac) + dc > 61)) return false;
  const long long s = x->s << ds;
  if (ac && (s + (c.most << dc) > (1LL << 53) || s + (c.least << dc) < -(1LL << 53))) return false;
  x->s = s + (c.total ? c.total << dc : 0);
  x->low = low;
  if (x->s) {  // keep it odd
    const int z = __ffsll(x->s) - 1;
    x->s >>= z;
    x->low += z;
  }
  return true;
}

// One warp per leaf: even lanes the gradient sum, odd lanes the hessian sum.
__global__ void __launch_bounds__(32) k_renew_join(const Job* __restrict__ jobs, Params p,
                                                   const int32_t* __restrict__ order, const ChunkSum* __restrict__ sums,
                                                   int64_t slots, int need_stop) {
  const Job& J = jobs[blockIdx.z];
  const int32_t leaf = (int32_t)blockIdx.x;
  if ((need_stop && !J.st->stop) || leaf >= J.st->tree_leaves) return;
  const RenewView v = renew_view(J, p, leaf, order);
  const int64_t chunks = ceil_div64(v.cnt, kChunk);
  const ChunkSum* in = sums + 2 * ((size_t)blockIdx.z * slots + first_chunk(J, leaf, 32));
  const int lane = threadIdx.x, what = lane & 1;
  ExactSum x{0, kNoBit};
  double wide = 0.0;
  bool finite = true;
  for (int64_t c0 = 0; c0 < chunks; c0 += 16) {
    ChunkSum mine{};
    mine.low = kNoBit;
    if (2 * c0 + lane < 2 * chunks) mine = in[2 * c0 + lane];
    const int n = (int)min((int64_t)16, chunks - c0);
    for (int j = 0; j < n; ++j) {
      const int from = 2 * j + what;
      ChunkSum c;
      c.total = __shfl_sync(FULL, mine.total, from);
      c.most = __shfl_sync(FULL, mine.most, from);
      c.least = __shfl_sync(FULL, mine.least, from);
      c.low = __shfl_sync(FULL, mine.low, from);
      c.bad = __shfl_sync(FULL, mine.bad, from);
      ExactSum y = x;
      const bool ok = finite && add_chunk(&y, c);
      if (__all_sync(FULL, ok)) {
        x = y;
        continue;
      }
      // the chunk's rows one after the other
      if (finite) wide = join_double(x);
      const int64_t k0 = (c0 + j) * kChunk;
      for (int64_t b = k0; b < min(k0 + kChunk, v.cnt); b += 32) {
        float gv = 0.f, hv = 0.f;
        if (b + lane < v.cnt) {
          const int32_t r = v.idx ? v.idx[b + lane] : (int32_t)(b + lane);
          gv = J.g[r];
          hv = J.h[r];
        }
        const int m = (int)min((int64_t)32, v.cnt - b);
        for (int i = 0; i < m; ++i) {
          const float a = __shfl_sync(FULL, gv, i), h = __shfl_sync(FULL, hv, i);
          wide += (double)(what ? h : a);
        }
      }
      finite = split_double(wide, &x);
    }
  }
  if (finite) wide = join_double(x);
  const double s1 = __shfl_sync(FULL, wide, 0), s2 = __shfl_sync(FULL, wide, 1);
  if (lane == 0) J.leaf_value[leaf] = round_to_zero(leaf_output(true, true, false, s1, s2, p, (int32_t)v.cnt, 0.0));
}

// ---- the rows grouped by leaf in the root's order ----
// counts[leaf][CTA]: how many of the CTA's rows are in the leaf. At most 512 leaves (grow rounds).
__device__ __forceinline__ int32_t group_row(const Job& J, const int32_t* rows, int64_t k) {
  return J.st->use_rows ? rows[k] : (int32_t)k;
}

__global__ void __launch_bounds__(256) k_group_count(const Job* __restrict__ jobs, Params p,
                                                     const int32_t* __restrict__ rows, const int32_t* __restrict__ row_leaf,
                                                     int32_t* __restrict__ counts) {
  __shared__ int32_t cnt[kMaxRoundLeaves];
  const Job& J = jobs[blockIdx.z];
  if (!J.st->stop) return;
  const int32_t leaves = J.st->tree_leaves;
  for (int l = threadIdx.x; l < leaves; l += 256) cnt[l] = 0;
  __syncthreads();
  const int64_t k0 = (int64_t)blockIdx.x * kGroupRows, k1 = min(k0 + kGroupRows, J.st->root_count);
  for (int64_t k = k0 + threadIdx.x; k < k1; k += 256)
    atomicAdd(&cnt[row_leaf[(size_t)blockIdx.z * p.n + group_row(J, rows, k)]], 1);
  __syncthreads();
  int32_t* out = counts + (size_t)blockIdx.z * p.num_leaves * gridDim.x;
  for (int l = threadIdx.x; l < leaves; l += 256) out[(size_t)l * gridDim.x + blockIdx.x] = cnt[l];
}

// One warp per leaf: exclusive prefix sums over the CTAs, from the leaf's first position on.
__global__ void __launch_bounds__(32) k_group_scan(const Job* __restrict__ jobs, Params p, int32_t* __restrict__ counts,
                                                   int ctas) {
  const Job& J = jobs[blockIdx.z];
  const int32_t leaf = (int32_t)blockIdx.x;
  if (!J.st->stop || leaf >= J.st->tree_leaves) return;
  int32_t* c = counts + ((size_t)blockIdx.z * p.num_leaves + leaf) * ctas;
  const int lane = threadIdx.x;
  int32_t base = (int32_t)J.leaf_begin[leaf];
  for (int b = 0; b < ctas; b += 32) {
    const int32_t x = b + lane < ctas ? c[b + lane] : 0;
    int32_t incl = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int32_t u = __shfl_up_sync(FULL, incl, o);
      if (lane >= o) incl += u;
    }
    if (b + lane < ctas) c[b + lane] = base + incl - x;
    base += __shfl_sync(FULL, incl, 31);
  }
}

// Each warp places 256 consecutive rows of its CTA's, 32 at a time: a row's place is its leaf's next one
// plus the rows of the same leaf in lower lanes.
__global__ void __launch_bounds__(256) k_group_scatter(const Job* __restrict__ jobs, Params p,
                                                       const int32_t* __restrict__ rows,
                                                       const int32_t* __restrict__ row_leaf,
                                                       const int32_t* __restrict__ starts, int32_t* __restrict__ order) {
  __shared__ int32_t next[8][kMaxRoundLeaves];  // counts per warp, then the warps' next places
  const Job& J = jobs[blockIdx.z];
  if (!J.st->stop) return;
  const int32_t leaves = J.st->tree_leaves;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int e = threadIdx.x; e < 8 * kMaxRoundLeaves; e += 256) next[e / kMaxRoundLeaves][e % kMaxRoundLeaves] = 0;
  const int64_t k0 = (int64_t)blockIdx.x * kGroupRows + warp * (kGroupRows / 8);
  int32_t row[kGroupRows / 256], leaf[kGroupRows / 256];
#pragma unroll
  for (int i = 0; i < kGroupRows / 256; ++i) {
    const int64_t k = k0 + 32 * i + lane;
    row[i] = k < J.st->root_count ? group_row(J, rows, k) : -1;
    leaf[i] = row[i] >= 0 ? row_leaf[(size_t)blockIdx.z * p.n + row[i]] : -1;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kGroupRows / 256; ++i)
    if (leaf[i] >= 0) atomicAdd(&next[warp][leaf[i]], 1);
  __syncthreads();
  const int32_t* start = starts + (size_t)blockIdx.z * p.num_leaves * gridDim.x;
  for (int l = threadIdx.x; l < leaves; l += 256) {
    int32_t at = start[(size_t)l * gridDim.x + blockIdx.x];
    for (int w = 0; w < 8; ++w) {
      const int32_t c = next[w][l];
      next[w][l] = at;
      at += c;
    }
  }
  __syncthreads();
  int32_t* out = order + (size_t)blockIdx.z * p.n;
#pragma unroll
  for (int i = 0; i < kGroupRows / 256; ++i) {
    const unsigned same = __match_any_sync(FULL, leaf[i]);
    const int32_t at = leaf[i] >= 0 ? next[warp][leaf[i]] + __popc(same & ((1u << lane) - 1u)) : 0;
    __syncwarp();
    if (leaf[i] >= 0) {
      out[at] = row[i];
      if ((same >> lane) == 1u) next[warp][leaf[i]] = at + 1;  // the highest lane of the leaf
    }
    __syncwarp();
  }
}

}  // namespace

RenewSizes renew_sizes(const Params& p, bool grouped) {
  RenewSizes r;
  r.slots = ceil_div64(p.n, kChunk) + p.num_leaves;
  r.sums = 2 * (size_t)r.slots * sizeof(ChunkSum);
  r.counts = grouped ? (size_t)p.num_leaves * ceil_div64(p.n, kGroupRows) : 0;
  r.rows = grouped ? (size_t)p.n : 0;
  return r;
}

void launch_group_rows(const Job* d_jobs, int num_jobs, const Params& p, const int32_t* d_rows, const RenewBuffers& b,
                       cudaStream_t s) {
  launch_row_leaf(d_jobs, num_jobs, p, b.row_leaf, 1, s);
  const int ctas = (int)ceil_div64(p.n, kGroupRows);
  k_group_count<<<dim3(ctas, 1, num_jobs), 256, 0, s>>>(d_jobs, p, d_rows, b.row_leaf, b.counts);
  k_group_scan<<<dim3(p.num_leaves, 1, num_jobs), 32, 0, s>>>(d_jobs, p, b.counts, ctas);
  k_group_scatter<<<dim3(ctas, 1, num_jobs), 256, 0, s>>>(d_jobs, p, d_rows, b.row_leaf, b.counts, b.order);
}

void launch_renew(const Job* d_jobs, int num_jobs, const Params& p, const RenewBuffers& b, bool grouped, cudaStream_t s) {
  const int32_t* order = grouped ? b.order : nullptr;
  ChunkSum* sums = static_cast<ChunkSum*>(b.sums);
  // a leaf's share of a few CTAs per SM
  const int gy = (int)std::max<int64_t>(1, std::min<int64_t>(ceil_div64(p.n, 8 * kChunk), 2432 / (p.num_leaves * num_jobs)));
  k_renew_chunks<<<dim3(p.num_leaves, gy, num_jobs), 256, 0, s>>>(d_jobs, p, order, sums, b.slots, grouped ? 1 : 0);
  k_renew_join<<<dim3(p.num_leaves, 1, num_jobs), 32, 0, s>>>(d_jobs, p, order, sums, b.slots, grouped ? 1 : 0);
}

}  // namespace bk
