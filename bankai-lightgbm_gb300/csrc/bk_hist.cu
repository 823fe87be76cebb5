// ConstructHistograms for the smaller leaf (serial.rs:891-1164), GB300 form.
//
// Grid: (blocks_per_tile, T, jobs), or the CTAs of a grow round split over the tiles. Each CTA owns one
// 32-feature tile and one contiguous chunk of the leaf's rows (in a round: of the leaves' rows). A warp takes 32 rows at a time: every lane fetches its row's run of the
// tile (32 bytes of 8-bit bins, or 16 bytes of 4-bit bins) with 128-bit loads. The CTA-private
// shared histogram keeps feature f's counters of every bin in bank f. Every lane adds its own
// row feature by feature, lane l taking feature k ^ l at step k: the 32 lanes of each shared
// atomic hit 32 different features, 32 different banks, so they never conflict and never
// collide, and no row passes through shared memory. At the end the CTA adds its non-zero bins to
// the leaf's slot in the histogram pool with global atomics (the pool slot is zeroed when the
// tree starts). Only the tile's own bins (its largest feature's group bins) are zeroed and
// flushed.
//
// A quantized CTA with few rows (at most `direct_rows`) skips the shared histogram: it stages
// each warp's 32 rows in shared memory and adds every (row, feature) to the pool slot with one
// global 64-bit atomic, lane = feature, so each atomic instruction covers 32 consecutive pool
// entries. That saves the CTA's zeroing, barrier and flush pass (with so few rows nearly every
// bin would be flushed anyway). Integer sums do not depend on the order, so both forms give the
// same slot.
//
// Quantized path: the packed int8 gradient / uint8 hessian of a row is added as one 32-bit
// value (grad << shift) + hess into a "hot" histogram, which is folded into 32-bit
// grad/hess "cold" counters before either half can overflow, and finally into the int64
// (grad << 32) + hess pool slot. Integer sums are exact, so the result equals the reference's
// sequential i64 histogram bit for bit.
//
// Float path: gradients and hessians are summed as 96-bit integer multiples of a unit of their own,
// chosen per tree so that every value is a multiple (24 mantissa bits and the distance from the
// largest exponent to the smallest non-zero one) and no sum overflows: exact, in any order. The pool
// slot receives each CTA's sum, rounded to a double, via f64 global atomics. A shared-memory integer
// atomic costs 1.2 cycles of the SM a warp (1.7 with its old value), an fp32 one is a compare-and-swap
// loop of 6.3, so the two top words cost 2.9 against a pair's 12.6 (the low word is zero for
// all but the smallest values, and a warp whose rows have none skips it): 4M rows x 100 features,
// constant hessian: 6203 -> 1746 us of histograms in a 255-leaf tree, 250 of them the root's. When the
// exponents span too much (or a value is not finite) the tree uses fp32 (hi, lo) pairs instead: hi is
// updated with atomicAdd, which returns the previous value, and the exact rounding error of that addition
// (Knuth's TwoSum on old and addend) is added to lo, which carries a sum to about 2^-48 of its rows'
// magnitudes. With a constant hessian the hessian slot counts rows and is scaled by hessians[0] at the
// flush (serial.rs:980-988), which is exact.
//
// The last CTA of tile 0 also computes the per-leaf constants of the search that follows
// (bk_leaf.cuh) before its own rows.
#include <algorithm>
#include <mutex>

#include "bk_fixed.cuh"
#include "bk_launch.cuh"
#include "bk_leaf.cuh"

namespace bk {

namespace {

__device__ __forceinline__ float two_sum_err(float a, float b, float s) {
  float bb = __fsub_rn(s, a);
  float e1 = __fsub_rn(a, __fsub_rn(s, bb));
  float e2 = __fsub_rn(b, bb);
  return __fadd_rn(e1, e2);
}

struct Range {
  int64_t r0, r1, count;
  const int32_t* idx;
  const int16_t* pk;  // packed values: by row for the root, else in leaf order
  int32_t slot;       // the pool slot the histogram goes to
  bool direct, pk_row;
  int hot_shift;      // Params::hot_shift
};

// The smaller leaf's rows for this CTA: 1 with rows, 2 without rows for this CTA (r->slot set),
// 0 when the job builds no histogram in this launch (the same for every CTA of the job). With
// `post`, the previous split's single-pass partition left its bookkeeping to this launch: the
// range comes from the split's outcome (bk_grow.cuh), and the side CTA writes the bookkeeping and
// the leaf constants. Otherwise it comes from the job state and the side CTA computes the
// constants.
__device__ __forceinline__ int cta_range(const Job& J, const Params& p, int blocks_per_tile, int post, int par,
                                         Range* r) {
  const JobState* st = J.st;
  // the stop flag is loaded with the rest of the state (one round of independent loads)
  const int32_t stop = st->stop;
  int64_t begin, count;
  int32_t buf;
  if (post) {
    const SplitOutcome o = split_outcome(p, st, __ldcg(&st->pcnt[par][0]) & 0xffffffffLL);
    if (stop) return 0;
    hist_apply_split(J, p, o);
    if (!o.go) return 0;
    begin = o.hist_begin();
    count = o.hist_count();
    buf = o.nbuf;
    r->slot = o.sslot;
    r->pk_row = false;
  } else {
    const int32_t do_search = st->do_search, slot = st->smaller_slot, leaves = st->tree_leaves;
    begin = st->hist_begin;
    count = st->hist_count;
    buf = st->hist_buf;
    if (stop) return 0;
    hist_leaf_constants(J, p);
    if (!do_search) return 0;
    r->slot = slot;
    r->pk_row = leaves == 1;  // the root: no leaf-ordered copy yet
  }
  // at least p.hist_min_rows rows per CTA (256 by default, eight warps' worth): small leaves spread
  // over as many SMs as they can fill, since a CTA's rows cost its SM's load and shared-atomic
  // pipes, not a DRAM share. Tile 0 leaves its last CTA, the side CTA, without rows (when it has
  // others), so the side work (bookkeeping, leaf constants) runs beside the rows, not before them.
  const int row_ctas = (blockIdx.y == 0 && blocks_per_tile > 1) ? blocks_per_tile - 1 : blocks_per_tile;
  int64_t chunk = ceil_div64(count, row_ctas);
  if (chunk < p.hist_min_rows) chunk = p.hist_min_rows;
  chunk = (chunk + 31) / 32 * 32;
  r->r0 = (int64_t)blockIdx.x * chunk;
  if (r->r0 >= count) return 2;
  r->r1 = min(count, r->r0 + chunk);
  r->count = count;
  r->idx = leaf_idx(J, buf) + begin;
  r->direct = (count == p.n);  // all rows in order: the index buffer is the identity
  r->pk = r->pk_row ? J.packed : (J.pk0 ? leaf_pk(J, buf) + begin : nullptr);
  r->hot_shift = p.hot_shift;
  return 1;
}

// The rows of a warp's round are fetched in two stages, each one round ahead of its use: the row
// index (a coalesced load of the leaf's index range, two rounds ahead) and then the row's 32-byte
// tile sector and packed value (one round ahead), so no gather waits on an index load.

struct RoundLoad {
  uint4 a, b;
  int32_t v;
};

// A tile of 17 to 32 features takes 32 steps, one per feature. One of at most 16 takes `steps` = 16, 8
// or 4 (the least that covers its features): the 32 columns of the shared histogram then hold
// 32 / steps copies of its features, feature f in columns f, f + steps, ..., and the lanes with the
// same high bits share a copy. At step k lane l adds to column k ^ l either way. Features past the
// tile's last one (padding, bin 0) add to columns of their own, which the flush skips: that is cheaper
// than a test per step (4M rows: 20 features 86 -> 47 us, 4 features 55 -> 37 us).
__device__ __forceinline__ int tile_steps(int nf) { return nf > 16 ? 32 : (nf > 8 ? 16 : (nf > 4 ? 8 : 4)); }

// Positions are 32-bit: a leaf has fewer than 2^31 rows, and a lookahead position past the
// leaf's end stays below 2^32. `swap` (0 or 1) exchanges the two 16-byte halves of a 32-byte run
// as they are loaded.
__device__ __forceinline__ int32_t round_row32(const Range& R, uint32_t i, uint32_t r1) {
  if (i >= r1) return -1;
  return R.direct ? (int32_t)i : __ldg(R.idx + i);
}

__device__ __forceinline__ RoundLoad load_round_int(const uint8_t* tb, uint32_t rs, const Range& R, uint32_t i,
                                                    int32_t row, bool wide, bool half, uint32_t swap) {
  RoundLoad L;
  L.a = make_uint4(0, 0, 0, 0);
  L.b = make_uint4(0, 0, 0, 0);
  L.v = 0;
  if (row >= 0) {
    const uint4* src = reinterpret_cast<const uint4*>(tb + (size_t)(uint32_t)row * rs);
    L.a = __ldg(src + swap);
    if (!half) L.b = __ldg(src + (swap ^ 1u));
    int32_t pk = R.pk[R.pk_row ? (uint32_t)row : i];
    int32_t gi = (int32_t)(int8_t)(pk >> 8);
    int32_t hi = pk & 0xff;
    L.v = wide ? ((gi & 0xffff) | (hi << 16)) : (int32_t)(((uint32_t)gi << R.hot_shift) + (uint32_t)hi);
  }
  return L;
}

// The two halves of a hot counter, (grad << shift) + hess with hess in [0, 2^shift).
__device__ __forceinline__ int32_t hot_h(uint32_t s, int shift) { return (int32_t)(s & ((1u << shift) - 1u)); }
__device__ __forceinline__ int32_t hot_g(uint32_t s, int shift) { return ((int32_t)s - hot_h(s, shift)) >> shift; }

// Lane f's stored bin of staged row j: byte f of the row's 32-byte run, or the nibble f of its
// 16-byte run (low nibble for even f).
template <bool NIBBLE>
__device__ __forceinline__ uint32_t staged_bin(const uint8_t* sb, int j, int lane) {
  if (!NIBBLE) return sb[j * 32 + lane];
  return (sb[j * 32 + (lane >> 1)] >> ((lane & 1) << 2)) & 15u;
}

// The (grad << 32) + hess pool value of a row's packed statistics as the kernel carries them.
template <bool WIDE>
__device__ __forceinline__ unsigned long long pool_value(int32_t v, int shift) {
  const int32_t g = WIDE ? (int32_t)(int16_t)(v & 0xffff) : hot_g((uint32_t)v, shift);
  const int32_t h = WIDE ? (v >> 16) : hot_h((uint32_t)v, shift);
  return (unsigned long long)((int64_t)g * 4294967296LL + (int64_t)h);
}

// Shared memory of the integer kernel. Hot form: one 256-byte row per bin holding the tile's 32
// 16:16 hot counters and then its 32 cold (32-bit) gradient counters, followed by the cold
// hessian counters [bin][32]. Wide form (no hot counters): the cold gradient counters
// [bin][32], then the cold hessian ones. Feature f's counters sit in bank f either way. A CTA
// that adds straight to the pool slot (direct) uses none of them and stages its rows over the
// same bytes instead: 64 uint4 per warp, then 32 packed values per warp.
template <bool WIDE>
struct IntHist {
  static constexpr int GS = WIDE ? TILE : 2 * TILE;  // words from one bin's counters to the next
  unsigned char* base;
  int Bt;
  __device__ uint32_t* hot() const { return reinterpret_cast<uint32_t*>(base); }
  __device__ int32_t* cold_g() const { return reinterpret_cast<int32_t*>(base) + (WIDE ? 0 : TILE); }
  __device__ int32_t* cold_h() const { return reinterpret_cast<int32_t*>(base) + (size_t)Bt * GS; }
};

// Adds a row's packed value to the (bin, feature) counters of the wide form.
__device__ __forceinline__ void add_wide(const IntHist<true>& H, uint32_t bin, int32_t v, uint32_t f) {
  atomicAdd(&H.cold_g()[bin * TILE + f], (int32_t)(int16_t)(v & 0xffff));
  atomicAdd(&H.cold_h()[bin * TILE + f], v >> 16);
}

// Adds a row's packed value to the hot counter at shared address `at` (the histogram's start plus
// (bin << 8) | 4 f).
__device__ __forceinline__ void add_hot(uint32_t at, int32_t v) {
  asm volatile("red.shared.add.u32 [%0], %1;" ::"r"(at), "r"(v) : "memory");
}

// w[i] <- w[i ^ (q & (2 TOP - 1))] (N a power of two, TOP <= N / 2): one select per word and bit.
template <int N, int TOP = N / 2>
__device__ __forceinline__ void xor_permute(uint32_t (&w)[N], uint32_t q) {
#pragma unroll
  for (int bit = TOP; bit >= 1; bit >>= 1) {
    const bool s = (q & (uint32_t)bit) != 0u;
    uint32_t t[N];
#pragma unroll
    for (int i = 0; i < N; ++i) t[i] = s ? w[i ^ bit] : w[i];
#pragma unroll
    for (int i = 0; i < N; ++i) w[i] = t[i];
  }
}

// The bins of a lane's row as counter offsets, for 8-bit bins. At step k lane l takes feature
// (k ^ l) mod steps and adds to column k ^ l, so the 32 lanes of each atomic hit 32 different columns,
// 32 different banks, whatever their bins; no row is staged through shared memory or broadcast. The
// run's words are permuted by the lane's high feature bits (a word index that varies by lane cannot be
// a register index); within a word, step j takes byte j ^ (l & 3). One byte permute then makes the hot
// counter's byte offset (bin << 8) | 4 column: byte 1 from the run's word, byte 0 from a word of the
// four columns' offsets (all below 128, so their sign fills bytes 2 and 3 with zeros); `sel[j]`
// selects the bytes of step j. The loop is bound by the ALU pipe, so one instruction per step instead
// of two (and none to permute the bytes) is what counts: 4M rows x 96 features 123 -> 107 us.
struct ColumnPerm {
  uint32_t sel[4], col0, base;  // base: the histogram's shared address
  __device__ __forceinline__ ColumnPerm(uint32_t lane, const unsigned char* smem) {
    base = (uint32_t)__cvta_generic_to_shared(smem);
#pragma unroll
    for (uint32_t j = 0; j < 4; ++j) {
      const uint32_t b = j ^ (lane & 3u);
      sel[j] = (b << 4) | (4u + b) | ((12u + b) << 8) | ((12u + b) << 12);
    }
    // byte b: 4 times the column of byte b of the first word after the permutation
    col0 = (lane & ~3u) * 0x04040404u + 0x0c080400u;
  }
};
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t r;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
  return r;
}

template <bool WIDE, int W>
__device__ __forceinline__ void add_words8(const IntHist<WIDE>& H, const uint32_t (&w)[W], int32_t v, const ColumnPerm& cp) {
#pragma unroll
  for (int i = 0; i < W; ++i) {
    const uint32_t col = cp.col0 ^ ((uint32_t)i * 0x10101010u);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t off = prmt(w[i], col, cp.sel[j]);
      if constexpr (WIDE) add_wide(H, off >> 8, v, (off & 255u) >> 2);
      else add_hot(cp.base + off, v);
    }
  }
}

// 4-bit bins: feature f at bits 4 (f & 7) of word f >> 3
template <bool WIDE, int W>
__device__ __forceinline__ void add_words4(const IntHist<WIDE>& H, const uint32_t (&w)[W], int32_t v, uint32_t lane,
                                           int steps, uint32_t base) {
#pragma unroll
  for (int k = 0; k < 8 * W; ++k) {
    if (W == 1 && k >= steps) break;  // four or eight steps
    const uint32_t f = (uint32_t)k ^ lane;
    const uint32_t bin = (w[k >> 3] >> ((((uint32_t)k ^ lane) & (steps == 4 ? 3u : 7u)) << 2)) & 15u;
    if constexpr (WIDE) add_wide(H, bin, v, f);
    else add_hot(base + ((bin << 8) | (f << 2)), v);
  }
}

template <bool WIDE, bool NIBBLE>
__device__ __forceinline__ void add_own_row(const IntHist<WIDE>& H, const RoundLoad& L, uint32_t lane, int steps,
                                            const ColumnPerm& cp) {
  const int32_t v = L.v;
  if (NIBBLE) {
    if (steps == 32) {
      uint32_t w[4] = {L.a.x, L.a.y, L.a.z, L.a.w};
      xor_permute<4>(w, (lane >> 3) & 3u);
      add_words4<WIDE, 4>(H, w, v, lane, 32, cp.base);
    } else if (steps == 16) {
      uint32_t w[2] = {L.a.x, L.a.y};
      xor_permute<2>(w, (lane >> 3) & 1u);
      add_words4<WIDE, 2>(H, w, v, lane, 16, cp.base);
    } else {
      uint32_t w[1] = {L.a.x};
      add_words4<WIDE, 1>(H, w, v, lane, steps, cp.base);
    }
    return;
  }
  if (steps == 32) {
    // 32 features in eight words, feature f in byte f & 3 of word f >> 2; the full run arrives with its
    // halves already exchanged for lanes 16-31 (bit 2 of the word permutation)
    uint32_t w[8] = {L.a.x, L.a.y, L.a.z, L.a.w, L.b.x, L.b.y, L.b.z, L.b.w};
    xor_permute<8, 2>(w, lane >> 2);
    add_words8<WIDE, 8>(H, w, v, cp);
  } else if (steps == 16) {
    uint32_t w[4] = {L.a.x, L.a.y, L.a.z, L.a.w};
    xor_permute<4>(w, (lane >> 2) & 3u);
    add_words8<WIDE, 4>(H, w, v, cp);
  } else if (steps == 8) {
    uint32_t w[2] = {L.a.x, L.a.y};
    xor_permute<2>(w, (lane >> 2) & 1u);
    add_words8<WIDE, 2>(H, w, v, cp);
  } else {
    uint32_t w[1] = {L.a.x};
    add_words8<WIDE, 1>(H, w, v, cp);
  }
}

// Folds the hot counters into the cold ones and clears them. Every thread of the CTA calls it
// between barriers. A leaf's hessians fit 32 unsigned bits (checked when the learner is created), so the
// cold hessian counters are read as such.
__device__ __forceinline__ void fold_hot(const IntHist<false>& H, int shift) {
  uint4* row4 = reinterpret_cast<uint4*>(H.base);   // 16 per bin: 8 hot, then 8 cold gradient
  int4* h4 = reinterpret_cast<int4*>(H.cold_h());  // 8 per bin
  for (int e = threadIdx.x; e < H.Bt * (TILE / 4); e += blockDim.x) {
    const int b = e >> 3, q = e & 7;
    uint4* hp = row4 + b * 16 + q;
    const uint4 s = *hp;
    if (s.x | s.y | s.z | s.w) {
      int4* gp = reinterpret_cast<int4*>(hp + 8);
      int4 g = *gp, h = h4[e];
      g.x += hot_g(s.x, shift);
      g.y += hot_g(s.y, shift);
      g.z += hot_g(s.z, shift);
      g.w += hot_g(s.w, shift);
      h.x += hot_h(s.x, shift);
      h.y += hot_h(s.y, shift);
      h.z += hot_h(s.z, shift);
      h.w += hot_h(s.w, shift);
      *gp = g;
      h4[e] = h;
      *hp = make_uint4(0, 0, 0, 0);
    }
  }
}

// The row loop of an integer-histogram CTA that adds to its shared histogram (the hot counters folded
// into the cold ones every `flush_rounds` rounds, before either half can overflow; the last round's
// are folded by the flush). Software pipeline: the next round's runs and the round after's row indices
// are in flight while this round is added up; two rounds per iteration, so the buffers change roles
// without moves.
template <bool WIDE, bool NIBBLE>
__device__ __forceinline__ void hist_int_loop(const Params& p, const Range& R, const TileGeom& geo, int tile,
                                              const uint8_t* tb, size_t rs, int flush_rounds, unsigned char* smem) {
  const int Bt = geo.bins;
  const bool half = geo.width == 16;  // one 16-byte run per row
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const IntHist<WIDE> H{smem, Bt};
  const int steps = tile_steps(min(TILE, p.F - tile * TILE));
  const ColumnPerm cp((uint32_t)lane, smem);
  const uint32_t r0 = (uint32_t)R.r0, r1 = (uint32_t)R.r1;
  const uint32_t per_round = (uint32_t)(TILE * nwarps);
  const uint32_t rounds = (r1 - r0 + per_round - 1u) / per_round;
  const uint32_t rs32 = (uint32_t)rs;
  // the full 8-bit path loads lanes 16-31's runs with their halves exchanged
  const uint32_t swap = (!NIBBLE && !half) ? ((uint32_t)lane >> 4) & 1u : 0u;
  uint32_t pos = r0 + (uint32_t)(warp * TILE + lane);  // this lane's row position in the current round
  RoundLoad a = load_round_int(tb, rs32, R, pos, round_row32(R, pos, r1), WIDE, half, swap), b;
  int32_t row_nxt = round_row32(R, pos + per_round, r1);
  int until_flush = flush_rounds;
  uint32_t left = rounds;
  auto step = [&](RoundLoad& cur, RoundLoad& nxt) {
    const int32_t row_nn = round_row32(R, pos + 2u * per_round, r1);
    nxt = load_round_int(tb, rs32, R, pos + per_round, row_nxt, WIDE, half, swap);
    row_nxt = row_nn;
    if (pos - (uint32_t)lane < r1) add_own_row<WIDE, NIBBLE>(H, cur, (uint32_t)lane, steps, cp);
    pos += per_round;
    --left;
    if constexpr (!WIDE) {
      if (--until_flush == 0 && left != 0u) {
        until_flush = flush_rounds;
        __syncthreads();
        fold_hot(H, p.hot_shift);
        __syncthreads();
      }
    }
  };
  while (left > 1u) {
    step(a, b);
    step(b, a);
  }
  if (left) step(a, b);
}

// The row loop of a CTA with few rows: every (row, feature) goes to the pool slot by a global atomic.
// The round's rows are staged so that each atomic covers one row's 32 features, 32 consecutive pool
// entries.
template <bool WIDE, bool NIBBLE>
__device__ __forceinline__ void hist_int_direct(const Params& p, const Range& R, const TileGeom& geo, int tile,
                                                const uint8_t* tb, size_t rs, unsigned long long* slot, unsigned char* smem) {
  const bool half = geo.width == 16;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  uint4* my_stage = reinterpret_cast<uint4*>(smem) + warp * 64;
  int32_t* my_v = reinterpret_cast<int32_t*>(reinterpret_cast<uint4*>(smem) + nwarps * 64) + warp * 32;
  const uint8_t* sb = reinterpret_cast<const uint8_t*>(my_stage);
  // lanes past the last feature of the last tile (padding) add nothing
  const bool feat_lane = lane < p.F - tile * TILE;
  const uint32_t r1 = (uint32_t)R.r1, per_round = (uint32_t)(TILE * nwarps);
  for (uint32_t base = (uint32_t)R.r0 + (uint32_t)(warp * TILE); base < r1; base += per_round) {
    const uint32_t pos = base + (uint32_t)lane;
    const RoundLoad cur = load_round_int(tb, (uint32_t)rs, R, pos, round_row32(R, pos, r1), WIDE, half, 0u);
    my_stage[lane * 2] = cur.a;
    if (!half) my_stage[lane * 2 + 1] = cur.b;
    my_v[lane] = cur.v;
    __syncwarp();
    const int jn = (int)min(32u, r1 - base);  // warp-uniform
    for (int j = 0; j < jn; ++j) {
      const uint32_t b0 = staged_bin<NIBBLE>(sb, j, lane);
      const int32_t v0 = my_v[j];
      if (feat_lane) atomicAdd(slot + b0 * TILE + lane, pool_value<WIDE>(v0, p.hot_shift));
    }
    __syncwarp();
  }
}

// The rows and flush of one integer-histogram CTA, its range known (NIBBLE: the tile holds
// 4-bit bins).
template <bool WIDE, bool NIBBLE>
__device__ __forceinline__ void hist_int_rows(const Job& J, const Params& p, const Range& R, const TileGeom& geo, int tile,
                                              const uint8_t* __restrict__ bins_rt, const uint8_t* __restrict__ bins_tm,
                                              int flush_rounds, int direct_rows, bool in_cluster, unsigned char* smem,
                                              bool more = false) {
  const int Bt = geo.bins;
  const IntHist<WIDE> H{smem, Bt};
  unsigned long long* slot = reinterpret_cast<unsigned long long*>(J.pool) +
                             ((size_t)R.slot * p.T + tile) * (size_t)p.B * TILE;
  // uniform over the CTA; a CTA of a cluster always adds through its shared histogram
  const bool direct = !in_cluster && R.r1 - R.r0 <= (int64_t)direct_rows;
  __syncthreads();
  // the tile's run of row 0 and the row stride, in the copy that suits the leaf's density
  const bool dense = R.count * 4 >= p.n;
  const uint8_t* tb = dense ? bins_tm + geo.tm_off : bins_rt + geo.rt_off;
  const size_t rs = dense ? (size_t)tile_width(geo) : (size_t)p.rt_stride;
  if (direct) {
    hist_int_direct<WIDE, NIBBLE>(p, R, geo, tile, tb, rs, slot, smem);
    return;
  }
  hist_int_loop<WIDE, NIBBLE>(p, R, geo, tile, tb, rs, flush_rounds, smem);
  if (in_cluster) return;  // a cluster flushes its CTAs' histograms together
  __syncthreads();
  const int nf = min(TILE, p.F - tile * TILE), steps = tile_steps(nf);
  for (int e = threadIdx.x; e < Bt * TILE; e += blockDim.x) {
    const int bin = e >> 5, col = e & (TILE - 1);
    const int gi = bin * IntHist<WIDE>::GS + col;  // (bin, column) in the row layout
    int32_t gg = H.cold_g()[gi], hh = H.cold_h()[e];
    if (!WIDE) {
      const uint32_t s = H.hot()[gi];
      gg += hot_g(s, p.hot_shift);
      hh += hot_h(s, p.hot_shift);
    }
    if (more) {  // the CTA's next rows belong to another leaf
      H.cold_g()[gi] = 0;
      H.cold_h()[e] = 0;
      if (!WIDE) H.hot()[gi] = 0u;
    }
    // the feature's copies sit in the warp's lanes
    for (int o = steps; o < TILE; o <<= 1) {
      gg += __shfl_xor_sync(0xffffffffu, gg, o);
      hh += __shfl_xor_sync(0xffffffffu, hh, o);
    }
    if ((gg | hh) && col < nf) {
      int64_t pk = (int64_t)gg * 4294967296LL + (int64_t)(uint32_t)hh;
      atomicAdd(slot + e, (unsigned long long)pk);
    }
  }
}

// The flush of a thread-block cluster of `ncta` CTAs of one feature tile: every CTA folds its
// 16:16 counters into its 32-bit ones, then (after a cluster barrier) CTA `rank` adds up its
// 1/ncta share of the tile's bins over every CTA's shared histogram through distributed shared
// memory and adds the non-zero sums to the pool slot — ncta times fewer global atomics than a
// flush per CTA. A second cluster barrier keeps every CTA's shared memory alive until the others
// have read it. Every CTA of the cluster calls it, with or without rows of its own (a CTA without
// rows contributes its zeroed histogram). Integer sums: the slot gets the same values.
template <bool WIDE>
__device__ __forceinline__ void hist_cluster_flush(const Params& p, const TileGeom& geo, unsigned long long* slot,
                                                   uint32_t ncta, unsigned char* smem) {
  const int Bt = geo.bins;
  const IntHist<WIDE> H{smem, Bt};
  const int nf = min(TILE, p.F - (int)blockIdx.y * TILE), steps = tile_steps(nf);
  const int n4 = Bt * TILE / 4;  // int4 groups of the tile's bins: a multiple of 64 (Bt a multiple of 8)
  __syncthreads();
  if constexpr (!WIDE) fold_hot(H, p.hot_shift);
  cluster_sync_all();
  const uint32_t rank = cluster_ctarank();
  const int per = n4 / (int)ncta;
  for (int e = (int)rank * per + threadIdx.x; e < ((int)rank + 1) * per; e += blockDim.x) {
    int4 g = make_int4(0, 0, 0, 0), h = make_int4(0, 0, 0, 0);
    for (uint32_t q = 0; q < ncta; ++q) {
      // int4 group e = (bin e >> 3, features 4 (e & 7) ..)
      const int4 a = ld_dsmem_v4(H.cold_g() + (e >> 3) * IntHist<WIDE>::GS + 4 * (e & 7), q);
      const int4 b = ld_dsmem_v4(H.cold_h() + 4 * e, q);
      g.x += a.x;
      g.y += a.y;
      g.z += a.z;
      g.w += a.w;
      h.x += b.x;
      h.y += b.y;
      h.z += b.z;
      h.w += b.w;
    }
    const int32_t gg[4] = {g.x, g.y, g.z, g.w}, hh[4] = {h.x, h.y, h.z, h.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int f = (4 * (e & 7) + k) & (steps - 1);  // a column holds a copy of feature column mod steps
      if ((gg[k] | hh[k]) && f < nf)
        atomicAdd(slot + (e >> 3) * TILE + f, (unsigned long long)((int64_t)gg[k] * 4294967296LL + (int64_t)(uint32_t)hh[k]));
    }
  }
  cluster_sync_all();
}

template <bool WIDE>
__global__ void __launch_bounds__(1024, 1)
    k_hist_int(const JobTable jobs, Params p, const uint8_t* __restrict__ bins_rt, const uint8_t* __restrict__ bins_tm,
               int blocks_per_tile, int flush_rounds, int direct_rows, int post, int par) {
  extern __shared__ __align__(16) unsigned char smem[];
  const TileGeom geo = p.tiles[blockIdx.y];  // static: loaded while the previous kernel finishes
  // the shared histogram is zeroed while the previous kernel of the grow loop finishes
  {
    uint4* z = reinterpret_cast<uint4*>(smem);
    const int n16 = (WIDE ? 2 : 3) * geo.bins * TILE / 4;
    for (int e = threadIdx.x; e < n16; e += blockDim.x) z[e] = make_uint4(0, 0, 0, 0);
  }
  griddep_wait();
  // the search may be scheduled now: its CTAs read their static data while this launch runs, and
  // wait for its completion before reading anything it writes
  griddep_launch();
  const Job& J = jobs.job[blockIdx.z];
  Range R;
  // a cluster's CTAs belong to one job and tile, so code 0 is the same for all of them; every
  // other CTA of a cluster reaches both cluster barriers of the flush
  const uint32_t ncta = cluster_nctarank();
  const int rc = cta_range(J, p, blocks_per_tile, post, par, &R);
  if (rc == 0 || (rc == 2 && ncta == 1)) return;
  if (rc == 1) {
    if (geo.nibble)
      hist_int_rows<WIDE, true>(J, p, R, geo, blockIdx.y, bins_rt, bins_tm, flush_rounds, direct_rows, ncta > 1, smem);
    else
      hist_int_rows<WIDE, false>(J, p, R, geo, blockIdx.y, bins_rt, bins_tm, flush_rounds, direct_rows, ncta > 1, smem);
  }
  if (ncta > 1) {
    unsigned long long* slot = reinterpret_cast<unsigned long long*>(J.pool) +
                               ((size_t)R.slot * p.T + blockIdx.y) * (size_t)p.B * TILE;
    hist_cluster_flush<WIDE>(p, geo, slot, ncta, smem);
  }
}

// ---- grow rounds (bk_rounds.cuh): the smaller children of up to kMaxRoundW expansions ----
// The children's rows, one after the other, are cut into an interval for each CTA of a tile (at least
// hist_min_rows rows each), so every CTA of a tile takes the same number of rows whatever the
// leaves' sizes; a CTA whose interval crosses from one leaf into the next flushes and clears its
// shared histogram there. round_cut() starts every leaf at an interval of its own where that costs
// little (small rounds): a second leaf costs its CTA a pass of its own.
struct RoundRows {
  int64_t off[kMaxRoundW];  // where expansion e's rows start among all
  int32_t begin[kMaxRoundW], count[kMaxRoundW], buf[kMaxRoundW], slot[kMaxRoundW];
  int32_t n, root;
  RoundCut cut;
};

// A CTA's tile, its place among the tile's CTAs and their number (hist_split_ctas): the first
// cta_extra full tiles have cta_full + 1 CTAs, the others cta_full; a narrow last tile has cta_last.
__device__ __forceinline__ int3 round_cta(const Params& p) {
  const int b = (int)blockIdx.x, c1 = p.cta_full + 1, full = p.T - (p.cta_last ? 1 : 0);
  const int n1 = p.cta_extra * c1, n2 = n1 + (full - p.cta_extra) * p.cta_full;
  if (b < n1) return make_int3(b / c1, b % c1, c1);
  if (b < n2) return make_int3(p.cta_extra + (b - n1) / p.cta_full, (b - n1) % p.cta_full, p.cta_full);
  return make_int3(full, b - n2, p.cta_last);
}

// Every thread calls it, between the launch's wait and its rows; ends with a barrier. The search
// constants of expansion e are computed by the last two warps of one CTA per expansion, spread over
// the grid from its end (whose CTAs are the ones without rows when there are few), before the rows
// of those warps.
__device__ __forceinline__ void round_rows(const Job& J, const Params& p, int q, int ctas, RoundRows* s) {
  const RoundView v = round_view(J, p);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  if (warp == 0) {
    const int n_cur = __ldcg(&v.hdr[q].n_cur);
    int32_t rows = 0;
    if (lane < kMaxRoundW) {  // loaded with the count (stale past it), not after it
      const RoundExp c = v.cur[q * kMaxRoundW + lane];
      const int32_t L = (int32_t)__ldcg(v.pcnt + ((size_t)q * kMaxRoundW + lane) * 2);
      const HistPart h = round_hist_part(p, c, L);
      if (lane < n_cur) {
        rows = h.go ? h.count : 0;
        s->begin[lane] = h.begin;
        s->count[lane] = rows;
        s->buf[lane] = h.buf;
        s->slot[lane] = h.slot;
        if (lane == 0) s->root = c.x < 0;
      }
    }
    int64_t off;
    const RoundCut cut = round_cut(rows, n_cur, ctas, p.hist_min_rows, 32, 2048, lane, &off);
    if (lane < n_cur) s->off[lane] = off;
    if (lane == 0) {
      s->n = n_cur;
      s->cut = cut;
    }
  } else if (warp >= nwarps - 2) {
    const int from_end = (int)(gridDim.x - 1 - blockIdx.x);
    if (from_end < kMaxRoundW) {
      const int n_cur = __ldcg(&v.hdr[q].n_cur);
      for (int e = from_end; e < n_cur; e += (int)gridDim.x) {
        const RoundExp c = v.cur[q * kMaxRoundW + e];
        const int32_t L = (int32_t)__ldcg(v.pcnt + ((size_t)q * kMaxRoundW + e) * 2);
        round_leaf_constants(J, p, c, L, e, warp - (nwarps - 2), lane);
      }
    }
  }
}

// The part of this CTA's interval that lies in expansion e: false when it has no row of it. `last`:
// no later leaf has rows in the interval.
__device__ __forceinline__ bool round_segment(const Job& J, const Params& p, const RoundRows& s, int cta, int e,
                                              Range* r, bool* single, bool* last) {
  const int64_t q0 = (int64_t)cta * s.cut.per, q1 = q0 + s.cut.per;
  const int64_t off = s.off[e];
  const int64_t a = max(q0, off), b = min(q1, off + s.count[e]);
  if (a >= b) return false;
  r->r0 = a - off;
  r->r1 = b - off;
  r->count = s.count[e];
  r->idx = leaf_idx(J, s.buf[e]) + s.begin[e];
  r->direct = r->count == p.n;  // all rows in order: the index buffer is the identity
  r->pk_row = s.root != 0;      // the root: no leaf-ordered copy yet
  r->pk = r->pk_row ? J.packed : (J.pk0 ? leaf_pk(J, s.buf[e]) + s.begin[e] : nullptr);
  r->slot = s.slot[e];
  r->hot_shift = p.hot_shift;
  *last = s.cut.apart || b == q1 || e == s.n - 1;
  *single = *last && a == q0;
  return true;
}

template <bool WIDE>
__global__ void __launch_bounds__(1024, 1)
    k_hist_int_round(const JobTable jobs, Params p, const uint8_t* __restrict__ bins_rt,
                     const uint8_t* __restrict__ bins_tm, int flush_rounds, int direct_rows, int q) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ RoundRows rows;
  const int3 m = round_cta(p);
  const TileGeom geo = p.tiles[m.x];  // static: loaded while the previous kernel finishes
  {
    uint4* z = reinterpret_cast<uint4*>(smem);
    const int n16 = (WIDE ? 2 : 3) * geo.bins * TILE / 4;
    for (int e = threadIdx.x; e < n16; e += blockDim.x) z[e] = make_uint4(0, 0, 0, 0);
  }
  griddep_wait();
  griddep_launch();
  const Job& J = jobs.job[blockIdx.z];
  round_rows(J, p, q, m.z, &rows);
  __syncthreads();
  for (int e = 0; e < rows.n; ++e) {
    Range R;
    bool single, last;
    if (!round_segment(J, p, rows, m.y, e, &R, &single, &last)) continue;
    // a CTA that adds straight to the pool slot stages its rows over the shared histogram, so it
    // takes rows of one leaf only
    const int direct = single ? direct_rows : -1;
    if (geo.nibble)
      hist_int_rows<WIDE, true>(J, p, R, geo, m.x, bins_rt, bins_tm, flush_rounds, direct, false, smem, !last);
    else
      hist_int_rows<WIDE, false>(J, p, R, geo, m.x, bins_rt, bins_tm, flush_rounds, direct, false, smem, !last);
    if (last) break;
  }
}

// Shared memory of the float kernel: regions of one 256-byte row per bin, two planes of 32 columns each
// (so that a byte permute makes the offset, as in the integer kernel). Region 0: the gradient's middle
// and high words; region 1: with a constant hessian the row counts and the gradient's low words, else
// the hessian's middle and high words; region 2 (varying hessians): both low words. The pair form
// uses the first four planes as gradient hi, lo, hessian hi (or counts), lo.
struct FloatHist {
  unsigned char* base;
  uint32_t addr;    // its shared address
  uint32_t region;  // bytes of a region
  __device__ uint32_t* word(int r, int plane, int e) const {  // entry e = (bin, column)
    return reinterpret_cast<uint32_t*>(base + (size_t)r * region) + ((e >> 5) * 64 + plane * 32 + (e & 31));
  }
};

// Adds (hi:mid) to the two words at shared address `at` (mid) and at + 128 (hi). The addition to mid
// returns the word before it, which gives the carry: exact whatever the order of the rows.
__device__ __forceinline__ void add_top(uint32_t at, uint32_t mid, uint32_t hi) {
  uint32_t old;
  asm volatile("atom.shared.add.u32 %0, [%1], %2;" : "=r"(old) : "r"(at), "r"(mid) : "memory");
  asm volatile("red.shared.add.u32 [%0], %1;" ::"r"(at + 128u), "r"(hi + (old + mid < mid ? 1u : 0u)) : "memory");
}

// Adds `lo` to the low word at shared address `low`; a carry goes to the words at `at`.
__device__ __forceinline__ void add_low(uint32_t low, uint32_t lo, uint32_t at) {
  uint32_t old;
  asm volatile("atom.shared.add.u32 %0, [%1], %2;" : "=r"(old) : "r"(low), "r"(lo) : "memory");
  if (old + lo < lo) add_top(at, 1u, 0u);
}

// Adds v to the fp32 pair at `hi`, `hi + 32`: hi takes the value by atomicAdd, which returns the
// previous sum, and lo the exact rounding error of that addition (TwoSum).
__device__ __forceinline__ void add_pair(float* hi, float v) {
  const float old = atomicAdd(hi, v);
  const float err = two_sum_err(old, v, __fadd_rn(old, v));
  if (err != 0.f) atomicAdd(hi + 32, err);
}

// Calls add(offset of the (bin, column) entry in a region) for every step of this lane's row: the same
// steps and columns as the integer kernel's add_own_row.
template <int W, class Add>
__device__ __forceinline__ void words8_steps(const uint32_t (&w)[W], const ColumnPerm& cp, const Add& add) {
#pragma unroll
  for (int i = 0; i < W; ++i) {
    const uint32_t col = cp.col0 ^ ((uint32_t)i * 0x10101010u);
#pragma unroll
    for (int j = 0; j < 4; ++j) add(prmt(w[i], col, cp.sel[j]));
  }
}

template <bool NIBBLE, class Add>
__device__ __forceinline__ void row_steps(const uint4& a, const uint4& b, uint32_t lane, int steps, const ColumnPerm& cp,
                                          const Add& add) {
  if (NIBBLE) {
    // feature f at bits 4 (f & 7) of word f >> 3
    uint32_t w[4] = {a.x, a.y, a.z, a.w};
    if (steps == 32) xor_permute<4>(w, (lane >> 3) & 3u);
    else if (steps == 16 && (lane & 8u)) w[0] = a.y, w[1] = a.x;
    const uint32_t m = steps == 4 ? 3u : 7u;
#pragma unroll
    for (int k = 0; k < 32; ++k) {
      if (k >= steps) break;
      const uint32_t f = (uint32_t)k ^ lane;
      add((((w[k >> 3] >> ((f & m) << 2)) & 15u) << 8) | (f << 2));
    }
    return;
  }
  if (steps == 32) {
    uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    xor_permute<8, 2>(w, lane >> 2);
    words8_steps<8>(w, cp, add);
  } else if (steps == 16) {
    uint32_t w[4] = {a.x, a.y, a.z, a.w};
    xor_permute<4>(w, (lane >> 2) & 3u);
    words8_steps<4>(w, cp, add);
  } else if (steps == 8) {
    uint32_t w[2] = {a.x, a.y};
    xor_permute<2>(w, (lane >> 2) & 1u);
    words8_steps<2>(w, cp, add);
  } else {
    uint32_t w[1] = {a.x};
    words8_steps<1>(w, cp, add);
  }
}

// The rows and flush of one float-histogram CTA, its range known (NIBBLE: the tile holds 4-bit
// bins; FIXED: fixed-point sums, else fp32 pairs).
template <bool CONST_HESS, bool NIBBLE, bool FIXED>
__device__ __forceinline__ void hist_float_rows(const Job& J, const Params& p, const Range& R, const TileGeom& geo, int tile,
                                                const uint8_t* __restrict__ bins_rt,
                                                const uint8_t* __restrict__ bins_tm, unsigned char* smem, bool more) {
  const int B = geo.bins;
  const bool half = geo.width == 16;  // one 16-byte run per row
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const uint32_t region = (uint32_t)B * 256u;
  const ColumnPerm cp((uint32_t)lane, smem);
  const FloatHist H{smem, cp.base, region};
  __syncthreads();
  // the tile's run of row 0 and the row stride, in the copy that suits the leaf's density
  const bool dense = R.count * 4 >= p.n;
  const uint8_t* tb = dense ? bins_tm + geo.tm_off : bins_rt + geo.rt_off;
  const uint32_t rs = dense ? (uint32_t)tile_width(geo) : (uint32_t)p.rt_stride;
  const int nf = min(TILE, p.F - tile * TILE), steps = tile_steps(nf);
  const float* G = J.g;
  const float* Hs = J.h;
  // the shifts of biased exponent 0: the largest exponent's values end at bit p.fix_bits
  const int g_shift0 = p.fix_bits - 24 - (int)J.st->red_maxg, h_shift0 = p.fix_bits - 24 - (int)J.st->red_maxh;
  const uint32_t r0 = (uint32_t)R.r0, r1 = (uint32_t)R.r1;
  const uint32_t per_round = (uint32_t)(TILE * nwarps);
  // the full 8-bit path loads lanes 16-31's runs with their halves exchanged
  const uint32_t swap = (!NIBBLE && !half) ? ((uint32_t)lane >> 4) & 1u : 0u;
  // the same two-stage software pipeline as the integer kernel
  auto load = [&](int32_t row, uint4& a, uint4& b, float2& v) {
    a = make_uint4(0, 0, 0, 0);
    b = make_uint4(0, 0, 0, 0);
    v = make_float2(0.f, 0.f);
    if (row >= 0) {
      const uint4* src = reinterpret_cast<const uint4*>(tb + (size_t)(uint32_t)row * rs);
      a = __ldg(src + swap);
      if (!half) b = __ldg(src + (swap ^ 1u));
      v.x = G[row];
      if (!CONST_HESS) v.y = Hs[row];
    }
  };
  uint32_t pos = r0 + (uint32_t)(warp * TILE + lane);
  uint4 ca, cb;
  float2 cv;
  load(round_row32(R, pos, r1), ca, cb, cv);
  int32_t row_nxt = round_row32(R, pos + per_round, r1);
  for (; pos - (uint32_t)lane < r1; pos += per_round) {
    const int32_t row_nn = round_row32(R, pos + 2u * per_round, r1);
    uint4 na, nb;
    float2 nv;
    load(row_nxt, na, nb, nv);
    row_nxt = row_nn;
    if constexpr (FIXED) {
      // a lane without a row adds zeros
      const Fixed g = to_fixed(cv.x, g_shift0);
      if constexpr (CONST_HESS) {
        const uint32_t one = pos < r1 ? 1u : 0u;
        row_steps<NIBBLE>(ca, cb, (uint32_t)lane, steps, cp, [&](uint32_t off) {
          const uint32_t at = H.addr + off;
          add_top(at, g.mid, g.hi);
          asm volatile("red.shared.add.u32 [%0], %1;" ::"r"(at + region), "r"(one) : "memory");
        });
        if (__any_sync(0xffffffffu, g.lo != 0u))
          row_steps<NIBBLE>(ca, cb, (uint32_t)lane, steps, cp,
                            [&](uint32_t off) { add_low(H.addr + region + 128u + off, g.lo, H.addr + off); });
      } else {
        const Fixed h = to_fixed(cv.y, h_shift0);
        row_steps<NIBBLE>(ca, cb, (uint32_t)lane, steps, cp, [&](uint32_t off) {
          add_top(H.addr + off, g.mid, g.hi);
          add_top(H.addr + region + off, h.mid, h.hi);
        });
        if (__any_sync(0xffffffffu, (g.lo | h.lo) != 0u))
          row_steps<NIBBLE>(ca, cb, (uint32_t)lane, steps, cp, [&](uint32_t off) {
            add_low(H.addr + 2u * region + off, g.lo, H.addr + off);
            add_low(H.addr + 2u * region + 128u + off, h.lo, H.addr + region + off);
          });
      }
    } else {
      if (pos < r1)
        row_steps<NIBBLE>(ca, cb, (uint32_t)lane, steps, cp, [&](uint32_t off) {
          add_pair(reinterpret_cast<float*>(smem + off), cv.x);
          if constexpr (CONST_HESS) atomicAdd(reinterpret_cast<uint32_t*>(smem + region + off), 1u);
          else add_pair(reinterpret_cast<float*>(smem + region + off), cv.y);
        });
    }
    ca = na;
    cb = nb;
    cv = nv;
  }
  __syncthreads();
  double2* slot = reinterpret_cast<double2*>(J.pool) + ((size_t)R.slot * p.T + tile) * (size_t)p.B * TILE;
  const float h0 = CONST_HESS ? Hs[0] : 0.f;
  const uint32_t h0_bits = __float_as_uint(h0) & 0x7fffffffu, h0_e = h0_bits >> 23;
  const uint32_t h0_m = (h0_bits & 0x7fffffu) | (h0_e ? 0x800000u : 0u);
  const int h0_exp = (int)max(h0_e, 1u) - 150;
  // the units' exponents: the value at shift 0 of biased exponent e has weight 2^(e - 150)
  const int g_exp = -150 - g_shift0, h_exp = -150 - h_shift0;
  for (int e = threadIdx.x; e < B * TILE; e += blockDim.x) {
    uint32_t* g0 = H.word(0, 0, e);  // planes: 32 words apart
    uint32_t* h1 = H.word(1, 0, e);
    uint32_t* low = H.word(CONST_HESS ? 1 : 2, CONST_HESS ? 1 : 0, e);
    double gs = 0.0, hs = 0.0;
    bool touched;
    if constexpr (FIXED) {
      Fixed g{low[0], g0[0], g0[32]}, h{0u, 0u, 0u};
      uint32_t cnt = 0;
      if constexpr (CONST_HESS) cnt = h1[0];
      else h = Fixed{low[32], h1[0], h1[32]};
      for (int o = steps; o < TILE; o <<= 1) {  // the feature's copies sit in the warp's lanes
        auto join = [&](Fixed& x) {
          const uint32_t l = __shfl_xor_sync(0xffffffffu, x.lo, o), m = __shfl_xor_sync(0xffffffffu, x.mid, o),
                         t = __shfl_xor_sync(0xffffffffu, x.hi, o);
          x.lo += l;
          const uint64_t top = (((uint64_t)x.hi << 32) | x.mid) + (((uint64_t)t << 32) | m) + (x.lo < l ? 1u : 0u);
          x.mid = (uint32_t)top;
          x.hi = (uint32_t)(top >> 32);
        };
        join(g);
        if constexpr (CONST_HESS) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
        else join(h);
      }
      touched = (g.lo | g.mid | g.hi | h.lo | h.mid | h.hi | cnt) != 0u;
      if (touched && (e & (TILE - 1)) < nf) {
        gs = fixed_to_double(g.lo, g.mid, g.hi, g_exp);
        if constexpr (CONST_HESS) {
          const uint64_t c = (uint64_t)cnt * h0_m;  // at most 31 and 24 bits
          hs = copysign(fixed_to_double((uint32_t)c, (uint32_t)(c >> 32), 0u, h0_exp), (double)h0);
        } else {
          hs = fixed_to_double(h.lo, h.mid, h.hi, h_exp);
        }
      }
    } else {
      gs = (double)__uint_as_float(g0[0]) + (double)__uint_as_float(g0[32]);
      hs = CONST_HESS ? (double)h1[0] * (double)h0 : (double)__uint_as_float(h1[0]) + (double)__uint_as_float(h1[32]);
      touched = CONST_HESS ? h1[0] != 0u : ((g0[0] | g0[32] | h1[0] | h1[32]) << 1) != 0u;
      for (int o = steps; o < TILE; o <<= 1) {
        gs += __shfl_xor_sync(0xffffffffu, gs, o);
        hs += __shfl_xor_sync(0xffffffffu, hs, o);
        touched = __shfl_xor_sync(0xffffffffu, (int)touched, o) || touched;
      }
    }
    if (touched && (e & (TILE - 1)) < nf) {
      atomicAdd(&slot[e].x, gs);
      atomicAdd(&slot[e].y, hs);
    }
    if (more) {  // the CTA's next rows belong to another leaf
      g0[0] = g0[32] = h1[0] = 0u;
      if (!CONST_HESS) h1[32] = low[32] = 0u;
      low[0] = 0u;
    }
  }
}

template <bool CONST_HESS>
__device__ __forceinline__ void hist_float_range(const Job& J, const Params& p, const Range& R, const TileGeom& geo, int tile,
                                                 const uint8_t* bins_rt, const uint8_t* bins_tm, unsigned char* smem,
                                                 bool more) {
  if (J.st->fix_ok) {
    if (geo.nibble) hist_float_rows<CONST_HESS, true, true>(J, p, R, geo, tile, bins_rt, bins_tm, smem, more);
    else hist_float_rows<CONST_HESS, false, true>(J, p, R, geo, tile, bins_rt, bins_tm, smem, more);
  } else {
    if (geo.nibble) hist_float_rows<CONST_HESS, true, false>(J, p, R, geo, tile, bins_rt, bins_tm, smem, more);
    else hist_float_rows<CONST_HESS, false, false>(J, p, R, geo, tile, bins_rt, bins_tm, smem, more);
  }
}

template <bool CONST_HESS>
__global__ void __launch_bounds__(1024, 1)
    k_hist_float_round(const JobTable jobs, Params p, const uint8_t* __restrict__ bins_rt,
                       const uint8_t* __restrict__ bins_tm, int q) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ RoundRows rows;
  const int3 m = round_cta(p);
  const TileGeom geo = p.tiles[m.x];  // static: loaded while the previous kernel finishes
  {
    uint4* z = reinterpret_cast<uint4*>(smem);
    const int n16 = (CONST_HESS ? 4 : 6) * geo.bins * TILE / 4;
    for (int e = threadIdx.x; e < n16; e += blockDim.x) z[e] = make_uint4(0, 0, 0, 0);
  }
  griddep_wait();
  griddep_launch();
  const Job& J = jobs.job[blockIdx.z];
  round_rows(J, p, q, m.z, &rows);
  __syncthreads();
  for (int e = 0; e < rows.n; ++e) {
    Range R;
    bool single, last;
    if (!round_segment(J, p, rows, m.y, e, &R, &single, &last)) continue;
    hist_float_range<CONST_HESS>(J, p, R, geo, m.x, bins_rt, bins_tm, smem, !last);
    if (last) break;
  }
}

template <bool CONST_HESS>
__global__ void __launch_bounds__(1024, 1)
    k_hist_float(const JobTable jobs, Params p, const uint8_t* __restrict__ bins_rt, const uint8_t* __restrict__ bins_tm,
                 int blocks_per_tile, int post, int par) {
  extern __shared__ __align__(16) unsigned char smem[];
  const TileGeom geo = p.tiles[blockIdx.y];  // static: loaded while the previous kernel finishes
  {
    uint4* z = reinterpret_cast<uint4*>(smem);
    const int n16 = (CONST_HESS ? 4 : 6) * geo.bins * TILE / 4;
    for (int e = threadIdx.x; e < n16; e += blockDim.x) z[e] = make_uint4(0, 0, 0, 0);
  }
  griddep_wait();
  // the search may be scheduled now: its CTAs read their static data while this launch runs, and
  // wait for its completion before reading anything it writes
  griddep_launch();
  const Job& J = jobs.job[blockIdx.z];
  Range R;
  if (cta_range(J, p, blocks_per_tile, post, par, &R) != 1) return;
  hist_float_range<CONST_HESS>(J, p, R, geo, blockIdx.y, bins_rt, bins_tm, smem, false);
}

}  // namespace

size_t hist_smem_bytes(const Params& p, int threads, bool quant, bool wide) {
  size_t warps = (size_t)threads / 32;
  size_t stage = warps * 64 * sizeof(uint4);
  size_t bins = (size_t)p.B * TILE;
  // the integer kernel's direct CTAs stage their rows over the (unused) shared histogram
  if (quant) return std::max((wide ? 0 : bins * 4) + bins * 8, stage + warps * 32 * 4);
  return bins * (p.const_hess ? 16 : 24);
}

void launch_hist(const Job* h_jobs, int num_jobs, const Params& p, const uint8_t* bins_rt, const uint8_t* bins_tm,
                 const HistLaunch& hl, int post, int par, cudaStream_t s) {
  for_job_groups(h_jobs, num_jobs, [&](const JobTable& t, int nz) {
    dim3 grid(hl.blocks_per_tile, p.T, nz);
    if (p.quant) {
      if (hl.flush_rounds > 0)
        (void)launch_kernel_cluster(k_hist_int<false>, grid, dim3(hl.threads), hl.smem, s, p.pdl, hl.cluster, t, p,
                                    bins_rt, bins_tm, hl.blocks_per_tile, hl.flush_rounds, hl.direct_rows, post, par);
      else
        (void)launch_kernel_cluster(k_hist_int<true>, grid, dim3(hl.threads), hl.smem, s, p.pdl, hl.cluster, t, p,
                                    bins_rt, bins_tm, hl.blocks_per_tile, 1, hl.direct_rows, post, par);
    } else if (p.const_hess) {
      (void)launch_kernel(k_hist_float<true>, grid, dim3(hl.threads), hl.smem, s, p.pdl, t, p, bins_rt, bins_tm,
                          hl.blocks_per_tile, post, par);
    } else {
      (void)launch_kernel(k_hist_float<false>, grid, dim3(hl.threads), hl.smem, s, p.pdl, t, p, bins_rt, bins_tm,
                          hl.blocks_per_tile, post, par);
    }
  });
}

void launch_hist_round(const Job* h_jobs, int num_jobs, const Params& p, const uint8_t* bins_rt,
                       const uint8_t* bins_tm, const HistLaunch& hl, int q, cudaStream_t s) {
  for_job_groups(h_jobs, num_jobs, [&](const JobTable& t, int nz) {
    const dim3 grid(hl.round_ctas, 1, nz), block(hl.threads);
    if (p.quant) {
      if (hl.flush_rounds > 0)
        (void)launch_kernel(k_hist_int_round<false>, grid, block, hl.smem, s, p.pdl, t, p, bins_rt, bins_tm,
                            hl.flush_rounds, hl.direct_rows, q);
      else
        (void)launch_kernel(k_hist_int_round<true>, grid, block, hl.smem, s, p.pdl, t, p, bins_rt, bins_tm, 1,
                            hl.direct_rows, q);
    } else if (p.const_hess) {
      (void)launch_kernel(k_hist_float_round<true>, grid, block, hl.smem, s, p.pdl, t, p, bins_rt, bins_tm, q);
    } else {
      (void)launch_kernel(k_hist_float_round<false>, grid, block, hl.smem, s, p.pdl, t, p, bins_rt, bins_tm, q);
    }
  });
}

void hist_split_ctas(Params& p, int total) {
  // a row costs a narrow tile's CTA about three quarters of what it costs a full one's (4M rows: 29
  // against 39 us above the launch's fixed part)
  const bool narrow = p.F % TILE != 0 && p.F % TILE <= 16;
  const int full = p.T - (narrow ? 1 : 0);
  total = std::max(total, p.T);
  p.cta_last = !narrow ? 0 : (full == 0 ? total : std::max(1, std::min(total - full, (int)(total * 0.75 / (full + 0.75)))));
  p.cta_full = full ? (total - p.cta_last) / full : 0;
  p.cta_extra = full ? (total - p.cta_last) % full : 0;
}

cudaError_t hist_set_smem_attrs(size_t smem) {
  // The attribute belongs to the kernel on the current device: remember the largest value set on
  // each device and only ever raise it, so learners created earlier with larger tiles keep working.
  constexpr int kMaxDevices = 64;
  static std::mutex m;
  static size_t current[kMaxDevices] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> g(m);
  if (smem <= current[dev]) return cudaSuccess;
  int v = (int)smem;
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_hist_int<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, v);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_hist_int<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, v);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_hist_float<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, v);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_hist_float<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, v);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_hist_int_round<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, v);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_hist_int_round<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, v);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_hist_float_round<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, v);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_hist_float_round<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, v);
  if (e == cudaSuccess) current[dev] = smem;
  return e;
}

}  // namespace bk
