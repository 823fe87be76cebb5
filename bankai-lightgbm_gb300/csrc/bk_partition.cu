// DataPartition::Split (data_partition.rs:124-174), GB300 form: a stable partition of the
// split leaf's row-index range into the left rows (kept in leaf order) followed by the right
// rows (kept in leaf order), written into the other index buffer. The batched grow loop uses a
// single-pass form instead, which keeps no order (k_part_onepass, k_part_round, below): only leaf
// renewal depends on it, and after grow rounds it groups the rows in order again.
//
// The reference routes each row through SplitRule::route_bin; here every CTA evaluates that rule
// once per stored bin into a 256-entry shared route table, so routing a row is one byte read of
// the split feature's column-major bins plus one shared-memory lookup. Two kernels on a fixed grid
// (so the step can be captured in a CUDA graph while the leaf size varies): count the left rows
// of each CTA's contiguous chunk; then scatter, each CTA summing the counts of the chunks before
// its own (at most a few hundred) and ordering its rows with block-wide scans.
#include "bk_decide.cuh"
#include "bk_grow.cuh"
#include "bk_launch.cuh"
#include "bk_rounds.cuh"

namespace bk {

namespace {

constexpr int kThreads = 256;
constexpr int kItems = 8;

struct PartRange {
  int64_t begin, count, r0, r1;
  int active;  // CTAs with rows: ceil(count / chunk)
  const int32_t* src;
  int32_t* dst;
  const uint8_t* col;
  // quantized path: the packed values move with the row indices; the root's are read by row
  const int16_t* pk_src;
  int16_t* pk_dst;
  bool pk_row;
  bool all;  // every row in order: the row of position e is e
};

__device__ __forceinline__ int32_t part_pk(const PartRange& R, int64_t e, int32_t row) {
  return R.pk_row ? R.pk_src[row] : R.pk_src[e];
}

// The split recorded in the job state (the search launch decided it).
__device__ __forceinline__ Decision recorded_decision(const JobState* st) {
  Decision d;
  d.stop = st->stop;
  d.leaf = st->split_leaf;
  d.inner = st->split_inner;
  d.thr = st->split_thr;
  d.begin = st->split_begin;
  d.count = st->split_count;
  d.buf = st->split_buf;
  d.depth = st->split_depth;
  d.sslot = st->split_sslot;
  d.new_leaf = st->new_leaf;
  d.pslot = st->split_pslot;
  return d;
}

__device__ __forceinline__ void part_range(const Job& J, const Params& p, const uint8_t* bins_cm, const Decision& d,
                                           PartRange* r) {
  r->begin = d.begin;
  r->count = d.count;
  const int32_t buf = d.buf;
  r->src = leaf_idx(J, buf) + r->begin;
  r->dst = leaf_idx_w(J, 1 - buf) + r->begin;
  r->col = bins_cm + (size_t)d.inner * (size_t)p.n;
  r->all = false;
  r->pk_row = d.new_leaf == 1;  // the root (one leaf when decided): no leaf-ordered copy yet
  r->pk_src = p.quant ? (r->pk_row ? J.packed : leaf_pk(J, buf) + r->begin) : nullptr;
  r->pk_dst = p.quant ? leaf_pk(J, 1 - buf) + r->begin : nullptr;
  // rows per CTA in multiples of one row per thread: a small leaf spreads over as many CTAs as
  // it fills, so each CTA's gather of the split column is short
  int64_t chunk = ceil_div64(r->count, p.part_grid);
  chunk = (chunk + kThreads - 1) / kThreads * kThreads;
  if (chunk < kThreads) chunk = kThreads;
  r->r0 = min((int64_t)blockIdx.x * chunk, r->count);
  r->r1 = min(r->r0 + chunk, r->count);
  r->active = (int)ceil_div64(r->count, chunk);
}

template <typename T>
__device__ __forceinline__ T block_excl_scan(T v, T* total, T* sh) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  T x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    T u = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += u;
  }
  if (lane == 31) sh[warp] = x;
  __syncthreads();
  if (warp == 0) {
    T w = lane < (int)(blockDim.x >> 5) ? sh[lane] : (T)0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      T u = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += u;
    }
    if (lane < (int)(blockDim.x >> 5)) sh[lane] = w;
  }
  __syncthreads();
  T warp_prefix = warp > 0 ? sh[warp - 1] : (T)0;
  *total = sh[(blockDim.x >> 5) - 1];
  T excl = warp_prefix + x - v;
  __syncthreads();
  return excl;
}

// The route of every stored bin of the chosen split (data_partition.rs:299-410), one per thread,
// from the split feature's metadata `m` (gbins, default_bin, mfb, missing, cat, offset).
// A categorical split routes by the bitset of its left bins, kept in the chosen leaf's candidate
// (data_partition.rs:264-300 and route_bin :367-377): group bin 0 (the most frequent bin's rows)
// goes left when the most frequent bin is not 0 and is in the bitset; stored bin b looks up bit
// b - 1 + offset.
__device__ __forceinline__ void build_route_of(const Job& J, const Params& p, const Decision& d, const DevFeature m,
                                               uint8_t* lut) {
  const uint32_t b = threadIdx.x;
  if (m.cat) {
    const uint32_t* bits = cand_cat_bits(J, p, d.leaf, d.inner);
    const uint32_t pos = b == 0 ? (uint32_t)m.mfb : b - 1 + (uint32_t)m.offset;
    const bool set = pos < 256u && ((__ldcg(bits + (pos >> 5)) >> (pos & 31)) & 1u) != 0u;
    lut[b] = ((int)b < m.gbins && set && (b != 0 || m.mfb > 0)) ? 1 : 0;
    return;
  }
  const uint32_t th = d.thr;
  lut[b] = (int)b < m.gbins ? route_bin(m, th & 0x7fffffffu, (th >> 31) != 0, b) : 0;
}

__device__ __forceinline__ void build_route(const Job& J, const Params& p, const Decision& d,
                                            const DevFeature* feats, uint8_t* lut) {
  build_route_of(J, p, d, feats[d.inner], lut);
}

// What build_route needs of a feature, packed in 8 bytes so a CTA can hold every feature's in
// shared memory before the split is known: x = gbins | default_bin << 16, y = mfb | missing << 16 |
// cat << 20 | offset << 21.
constexpr int kRoutePrefetch = 1024;  // features whose descriptors a partition CTA keeps

__device__ __forceinline__ uint2 route_desc(const DevFeature& m) {
  return make_uint2((uint32_t)m.gbins | ((uint32_t)m.default_bin << 16),
                    (uint32_t)m.mfb | ((uint32_t)m.missing << 16) | ((uint32_t)(m.cat != 0) << 20) |
                        ((uint32_t)m.offset << 21));
}

__device__ __forceinline__ DevFeature route_feature(uint2 q) {
  DevFeature m{};
  m.gbins = (int32_t)(q.x & 0xffffu);
  m.default_bin = (int32_t)(q.x >> 16);
  m.mfb = (int32_t)(q.y & 0xffffu);
  m.missing = (int32_t)((q.y >> 16) & 15u);
  m.cat = (int32_t)((q.y >> 20) & 1u);
  m.offset = (int32_t)((q.y >> 21) & 1u);
  return m;
}

__global__ void __launch_bounds__(kThreads) k_part_count(const JobTable jobs, Params p,
                                                         const uint8_t* __restrict__ bins_cm,
                                                         const DevFeature* __restrict__ feats) {
  __shared__ uint8_t lut[256];
  __shared__ int64_t sh[32];
  griddep_wait();
  const Job& J = jobs.job[blockIdx.z];
  if (J.st->stop) return;
  const Decision dec = recorded_decision(J.st);
  PartRange R;
  part_range(J, p, bins_cm, dec, &R);  // its loads are in flight with the route table's
  build_route(J, p, dec, feats, lut);
  __syncthreads();
  if ((int)blockIdx.x >= R.active) {  // no rows: the scatter reads only active CTAs' counts
    griddep_launch();
    return;
  }
  // per tile: every row index first, then every bin byte, so a tile costs two memory round trips
  int64_t local = 0;
  for (int64_t base = R.r0; base < R.r1; base += kThreads * kItems) {
    int32_t rows[kItems];
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
      const int64_t e = base + (int64_t)k * kThreads + threadIdx.x;
      rows[k] = e < R.r1 ? __ldg(R.src + e) : -1;
    }
#pragma unroll
    for (int k = 0; k < kItems; ++k)
      if (rows[k] >= 0) local += lut[__ldg(R.col + rows[k])];
  }
  griddep_launch();
  int64_t total;
  block_excl_scan<int64_t>(local, &total, sh);
  if (threadIdx.x == 0) J.part_cnt[blockIdx.x] = total;
}

__global__ void __launch_bounds__(kThreads) k_part_scatter(const JobTable jobs, Params p,
                                                           const uint8_t* __restrict__ bins_cm,
                                                           const DevFeature* __restrict__ feats) {
  __shared__ uint8_t lut[256];
  __shared__ int32_t sh[32];
  griddep_wait();
  const Job& J = jobs.job[blockIdx.z];
  if (J.st->stop) return;
  __shared__ int64_t sh64[32];
  const Decision dec = recorded_decision(J.st);
  PartRange R;
  part_range(J, p, bins_cm, dec, &R);  // its loads are in flight with the route table's
  build_route(J, p, dec, feats, lut);
  __syncthreads();
  // left rows before this chunk, and in total
  int64_t before = 0, all = 0;
  const bool active = (int)blockIdx.x < R.active;
  for (int i = threadIdx.x; active && i < R.active; i += kThreads) {
    int64_t c = J.part_cnt[i];
    all += c;
    if (i < (int)blockIdx.x) before += c;
  }
  int64_t total_left = 0, running = 0;
  if (active) {
    block_excl_scan<int64_t>(all, &total_left, sh64);
    block_excl_scan<int64_t>(before, &running, sh64);
    if (blockIdx.x == 0 && threadIdx.x == 0) J.st->total_left = total_left;
  }
  for (int64_t base = R.r0; base < R.r1; base += kThreads * kItems) {
    int64_t e0 = base + (int64_t)threadIdx.x * kItems;
    int32_t rows[kItems];
    uint32_t flags = 0;
    int32_t cnt = 0;
#pragma unroll
    for (int k = 0; k < kItems; ++k) rows[k] = e0 + k < R.r1 ? __ldg(R.src + e0 + k) : -1;
#pragma unroll
    for (int k = 0; k < kItems; ++k)
      if (rows[k] >= 0 && lut[__ldg(R.col + rows[k])]) {
        flags |= 1u << k;
        ++cnt;
      }
    int32_t tile_total;
    int32_t pre = block_excl_scan<int32_t>(cnt, &tile_total, sh);
    int64_t left_before = running + pre;
    int32_t pkv[kItems];
#pragma unroll
    for (int k = 0; k < kItems; ++k) pkv[k] = (p.quant && rows[k] >= 0) ? part_pk(R, e0 + k, rows[k]) : 0;
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
      int64_t e = e0 + k;
      if (e < R.r1) {
        const int64_t slot = (flags & (1u << k)) ? left_before++ : total_left + (e - left_before);
        R.dst[slot] = rows[k];
        if (p.quant) R.pk_dst[slot] = (int16_t)pkv[k];
      }
    }
    running += tile_total;
  }
  griddep_launch();  // only the last CTA's bookkeeping is left: the next histogram may be scheduled
  // the last CTA of the launch applies the split to the leaf records (bk_grow.cuh)
  __shared__ int last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    unsigned t = atomicAdd(&J.st->part_done, 1u);
    last = t == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  if (threadIdx.x < 32) post_split_body(J, p, feats);
  if (threadIdx.x == 0) J.st->part_done = 0u;
}

// Rows [r0, r1) of a single-pass partition, in tiles of kTileRows. A tile claims the slots of its
// left rows from the front of the leaf's range and those of its right rows from the back with one
// atomic on `counter` (left rows in the low half, right rows in the high half); inside a tile the rows
// keep their leaf order. The tiles are pipelined: a tile is claimed while the one before it is
// written, the next one's bins and the one after's rows are on their way, so a tile costs its issue
// and two barriers instead of four memory round trips in a row (10M-row root: 61 -> 48 us on two
// CTAs per SM).
constexpr int kTileItems = 4;
constexpr int kTileRows = kThreads * kTileItems;
struct TileSmem {
  int32_t pre[3][kTileItems][kThreads / 32];  // left rows before each (item, warp) group, by tile mod 3
  unsigned long long off[3];
  int32_t left[3];
};

__device__ __forceinline__ void onepass_rows(const PartRange& R, bool quant, const uint8_t* lut,
                                             unsigned long long* counter, TileSmem& sm) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned lanes_below = (1u << lane) - 1u;
  // a tile's element j = k * kThreads + threadIdx.x (item k of this thread): every load and store
  // instruction covers 32 consecutive elements
  struct Rows {
    int32_t row[kTileItems], pk[kTileItems];
  };
  auto load = [&](int64_t base) {
    Rows r;
#pragma unroll
    for (int k = 0; k < kTileItems; ++k) {
      const int64_t e = base + k * kThreads + threadIdx.x;
      r.row[k] = e < R.r1 ? (R.all ? (int32_t)e : __ldg(R.src + e)) : -1;
    }
#pragma unroll
    for (int k = 0; k < kTileItems; ++k) {
      const int64_t e = base + k * kThreads + threadIdx.x;
      // the root's packed values go by row: for an unbagged root by position, else after the row
      r.pk[k] = (quant && e < R.r1 && (!R.pk_row || R.all)) ? R.pk_src[e] : 0;
    }
    return r;
  };
  uint32_t bin[kTileItems];
  auto gather = [&](Rows& r) {
#pragma unroll
    for (int k = 0; k < kTileItems; ++k) bin[k] = r.row[k] >= 0 ? __ldg(R.col + r.row[k]) : 0u;
    if (quant && R.pk_row && !R.all) {
#pragma unroll
      for (int k = 0; k < kTileItems; ++k) r.pk[k] = r.row[k] >= 0 ? R.pk_src[r.row[k]] : 0;
    }
  };
  Rows cur = load(R.r0), nxt = load(R.r0 + kTileRows), old{};
  gather(cur);
  // the tile before (old): its flags and each element's place in its warp
  uint32_t old_flags = 0;
  int32_t old_in[kTileItems] = {};
  unsigned long long claim = 0;  // warp 0, lane 31: the claim of the tile before, still in flight
  auto write = [&](int64_t base, int ob) {
    const int32_t n = (int32_t)min((int64_t)kTileRows, R.r1 - base);
    // left rows fill [lo, lo + tile_left); right rows fill the tile's slots ending at count - ro
    const int32_t tile_left = sm.left[ob];
    const unsigned long long off = sm.off[ob];
    const int64_t lo = (int64_t)(uint32_t)off;
    const int64_t ro = R.count - (int64_t)(off >> 32) - (n - tile_left);
#pragma unroll
    for (int k = 0; k < kTileItems; ++k) {
      const int32_t j = k * kThreads + (int32_t)threadIdx.x;
      if (j < n) {
        const int32_t left_before = sm.pre[ob][k][warp] + old_in[k];
        const int64_t slot = ((old_flags >> k) & 1u) ? lo + left_before : ro + (j - left_before);
        R.dst[slot] = old.row[k];
        if (quant) R.pk_dst[slot] = (int16_t)old.pk[k];
      }
    }
  };
  int buf = 0, ob = 2;
  int64_t base = R.r0;
  for (; base < R.r1; base += kTileRows) {
    uint32_t flags = 0;
#pragma unroll
    for (int k = 0; k < kTileItems; ++k)
      if (cur.row[k] >= 0 && lut[bin[k]]) flags |= 1u << k;
    // left rows before each element of the tile, in element order: within the warp's 32 elements of
    // item k by ballot, across (item, warp) groups by one scan of a warp
    int32_t in_warp[kTileItems];
#pragma unroll
    for (int k = 0; k < kTileItems; ++k) {
      const unsigned b = __ballot_sync(FULL, (flags >> k) & 1u);
      in_warp[k] = __popc(b & lanes_below);
      if (lane == 0) sm.pre[buf][k][warp] = __popc(b);
    }
    __syncthreads();
    if (warp == 0) {
      static_assert(kTileItems * (kThreads / 32) == 32, "one (item, warp) group per lane");
      const int32_t n = (int32_t)min((int64_t)kTileRows, R.r1 - base);
      int32_t* flat = &sm.pre[buf][0][0];
      const int32_t c = flat[lane];
      int32_t x = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int32_t y = __shfl_up_sync(FULL, x, o);
        if (lane >= o) x += y;
      }
      __syncwarp();
      flat[lane] = x - c;
      if (lane == 31) {
        sm.left[buf] = x;
        sm.off[ob] = claim;
        claim = atomicAdd(counter, (unsigned long long)(uint32_t)x | ((unsigned long long)(uint32_t)(n - x) << 32));
      }
    }
    const Rows nn = load(base + 2 * kTileRows);
    gather(nxt);
    __syncthreads();
    if (base > R.r0) write(base - kTileRows, ob);
    old = cur;
    old_flags = flags;
#pragma unroll
    for (int k = 0; k < kTileItems; ++k) old_in[k] = in_warp[k];
    cur = nxt;
    nxt = nn;
    ob = buf;
    buf = buf == 2 ? 0 : buf + 1;
  }
  if (warp == 0 && lane == 31) sm.off[ob] = claim;
  __syncthreads();
  if (base > R.r0) write(base - kTileRows, ob);
  __syncthreads();  // the caller may go on to another leaf
}

// Single-pass partition, for when the order of a child's rows inside its range cannot change any
// result (no leaf renewal: integer histograms, the score update and the row -> leaf map do not
// depend on it): onepass_rows on the counter of this split's parity. No count pass and no serial
// tail: the histogram launch that follows reads the left total and applies the split's bookkeeping
// (bk_grow.cuh), and the search after it clears the counter for the split after next.
__global__ void __launch_bounds__(kThreads) k_part_onepass(const JobTable jobs, Params p,
                                                           const uint8_t* __restrict__ bins_cm,
                                                           const DevFeature* __restrict__ feats, int par,
                                                           int decide) {
  static_assert(kThreads == kDecideThreads, "the partition CTA runs the split decision");
  __shared__ uint8_t lut[256];
  __shared__ Decision dec;
  __shared__ uint2 s_route[kRoutePrefetch];
  __shared__ DecideSmem ds;
  // static: every feature's route descriptor, read while the search finishes
  const bool prefetched = p.F <= kRoutePrefetch;
  if (prefetched)
    for (int f = threadIdx.x; f < p.F; f += kThreads) s_route[f] = route_desc(feats[f]);
  // the leaf arg-max over the leaves the search does not cover, while the search runs (their
  // records come from the histogram launch of this step and earlier, complete by the time the
  // search lets this launch start)
  const Job& Jpre = jobs.job[blockIdx.z];
  if (decide) decide_leaves(Jpre, p, ds);
  griddep_wait();
  // the next histogram launch may be scheduled now: its CTAs zero their shared histograms while
  // this partition runs, and wait for its completion before reading anything it writes
  griddep_launch();
  const Job& J = jobs.job[blockIdx.z];
  JobState* st = J.st;
  if (decide) {
    // every CTA decides the split from the search's records (a stopped tree included: the stop
    // flag comes with part one's loads); CTA 0 records it
    __syncthreads();
    decide_finish(J, p, feats, blockIdx.x == 0, &dec, ds);
  } else if (threadIdx.x == 0) {
    dec = recorded_decision(st);
  }
  __syncthreads();
  if (dec.stop) return;
  PartRange R;
  part_range(J, p, bins_cm, dec, &R);
  if ((int)blockIdx.x >= R.active) return;  // CTAs past the leaf's rows leave at once
  if (prefetched) build_route_of(J, p, dec, route_feature(s_route[dec.inner]), lut);
  else build_route(J, p, dec, feats, lut);
  __syncthreads();
  __shared__ TileSmem ts;
  onepass_rows(R, p.quant != 0, lut, reinterpret_cast<unsigned long long*>(&st->pcnt[par][0]), ts);
}

// The partition of a grow round (bk_rounds.cuh): every CTA takes the round's decision, then moves its
// share of the chosen leaves' rows in one pass (round_cut: equal intervals of whole 256-row blocks); a
// CTA whose interval crosses into the next leaf builds that leaf's route table there.
__global__ void __launch_bounds__(kThreads) k_part_round(const JobTable jobs, Params p,
                                                         const uint8_t* __restrict__ bins_cm,
                                                         const DevFeature* __restrict__ feats, int q) {
  __shared__ uint8_t lut[256];
  __shared__ TileSmem ts;
  __shared__ RoundSmem rs;
  const Job& J = jobs.job[blockIdx.z];
  decide_round_load(J, p, q, rs);
  __syncthreads();
  decide_round_open(rs);
  griddep_wait();
  // the next histogram launch may be scheduled now: its CTAs zero their shared histograms while
  // this partition runs
  griddep_launch();
  if (rs.hdr.stop) {  // the tree is finished: only keep the other copy of the state saying so
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      RoundHdr* h = round_view(J, p).hdr + (q ^ 1);
      h->stop = 1;
      h->n_cur = 0;
    }
    return;
  }
  decide_round_fold(J, p, rs);
  __syncthreads();
  if (threadIdx.x < 32) decide_round_commit(J, p, blockIdx.x == 0, rs);
  __syncthreads();
  decide_round_choose(J, p, q, blockIdx.x == 0, rs);
  if (blockIdx.x == 0) decide_round_store(J, p, q, rs);
  const int n = rs.hdr.n_cur;
  if (n == 0) return;
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    int64_t off;
    const RoundCut cut = round_cut(lane < n ? rs.nxt[lane].count : 0, n, (int)gridDim.x, kThreads, kThreads,
                                   4 * kThreads, lane, &off);
    if (lane < n) rs.off[lane] = off;
    if (lane == 0) rs.cut = cut;
  }
  __syncthreads();
  const int64_t q0 = (int64_t)blockIdx.x * rs.cut.per, q1 = q0 + rs.cut.per;
  unsigned long long* pcnt =
      reinterpret_cast<unsigned long long*>(round_view(J, p).pcnt) + (size_t)(q ^ 1) * 2 * kMaxRoundW;
  for (int e = 0; e < n; ++e) {
    const RoundExp& c = rs.nxt[e];
    const int64_t off = rs.off[e];
    const int64_t a = max(q0, off), b = min(q1, off + c.count);
    if (a < b) {
      Decision d;
      d.leaf = c.node;
      d.inner = c.inner;
      d.thr = c.thr;
      PartRange R;
      const int buf = c.depth_buf & 1;
      R.begin = c.begin;
      R.count = c.count;
      R.r0 = a - off;
      R.r1 = b - off;
      R.src = leaf_idx(J, buf) + R.begin;
      R.dst = leaf_idx_w(J, 1 - buf) + R.begin;
      R.col = bins_cm + (size_t)d.inner * (size_t)p.n;
      R.pk_row = c.node == 0;  // the root: no leaf-ordered copy yet
      R.all = c.node == 0 && c.count == p.n;  // an unbagged root: the identity
      R.pk_src = p.quant ? (R.pk_row ? J.packed : leaf_pk(J, buf) + R.begin) : nullptr;
      R.pk_dst = p.quant ? leaf_pk(J, 1 - buf) + R.begin : nullptr;
      build_route(J, p, d, feats, lut);
      __syncthreads();
      onepass_rows(R, p.quant != 0, lut, pcnt + 2 * e, ts);
      if (rs.cut.apart) break;
    }
  }
}

}  // namespace

void launch_partition_round(const Job* h_jobs, int num_jobs, const Params& p, const uint8_t* bins_cm,
                            const DevFeature* feats, int q, cudaStream_t s) {
  for_job_groups(h_jobs, num_jobs, [&](const JobTable& t, int nz) {
    (void)launch_kernel(k_part_round, dim3(p.part_grid, 1, nz), dim3(kThreads), 0, s, p.pdl, t, p, bins_cm, feats, q);
  });
}

void launch_partition(const Job* h_jobs, int num_jobs, const Params& p, const uint8_t* bins_cm,
                      const DevFeature* feats, bool stable, int par, bool decide, cudaStream_t s) {
  for_job_groups(h_jobs, num_jobs, [&](const JobTable& t, int nz) {
    dim3 grid(p.part_grid, 1, nz);
    if (stable) {
      (void)launch_kernel(k_part_count, grid, dim3(kThreads), 0, s, p.pdl, t, p, bins_cm, feats);
      (void)launch_kernel(k_part_scatter, grid, dim3(kThreads), 0, s, p.pdl, t, p, bins_cm, feats);
    } else {
      (void)launch_kernel(k_part_onepass, grid, dim3(kThreads), 0, s, p.pdl, t, p, bins_cm, feats, par,
                          decide ? 1 : 0);
    }
  });
}

}  // namespace bk
