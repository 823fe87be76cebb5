// Grow rounds: leaf-wise growth (serial.rs:578-628) with several leaves expanded at once.
//
// The reference splits the leaf with the best gain, searches its two children and repeats:
// num_leaves - 1 dependent steps. Which leaf comes next depends on the children's gains, but the
// children of any leaf do not depend on the order: they are the same whenever the leaf is split. So
// a round expands — partitions, builds the smaller child's histogram of, searches both children
// of — up to `round_w` leaves with the highest gains at once, and the splits are then committed in
// the reference's order from what is already known: while the best leaf of the tree so far is
// expanded, its split is taken, its children replace it and compete with the rest; the first best
// leaf that is not expanded ends the round and heads the next one. Only leaves that the remaining
// splits could reach are expanded (the `left` best of the tree, `left` splits remaining), so with
// round_w 16 a tree of 255 leaves takes about 22 rounds and, in practice, no work that the
// one-by-one loop does not do; the records, leaf numbers, values and partitions are the same.
// What bounds the one-by-one loop is its chain of 3 dependent launches per split (25 us, most of it
// latency); a round is the same three launches (25 us for 4 small leaves, 80 us for 16 of 40,000
// rows) for up to 16 splits, and its launches have enough rows and slices to fill the chip. A boosting
// iteration before rounds and now, other changes included: 10M x 100, 255 leaves 9.58 -> 3.75 ms; 10M x
// 200 12.1 -> 6.06 ms; 4M x 100 float 16.9 -> 4.21 ms; 300k x 40 with categories 2.51 -> 0.77 ms; 100k x 28
// float, 31 leaves 1.64 -> 0.50 ms; 5k x 20, 31 leaves 0.71 -> 0.44 ms; 12 jobs in one graph 2.90 -> 1.84 ms.
//
// An expanded leaf that is not split yet keeps its rows: they stay in its own index buffer (the
// children are written to the other one, and are expanded only after the commit). Its pool slot goes
// to its larger child, whose histogram is the leaf's minus the smaller child's, as when one leaf is
// split at a time; its own is both children's together, should anyone ask for it. So a tree of L
// leaves has 1 + max_exp slots, 287 of 255 leaves (573 with two new ones for every expansion).
//
// Every partition CTA takes the round's decision from the same records (decide_round), CTA 0
// writes it down. The state it reads and the state it writes are two copies that swap roles every
// round, so a CTA that is late still reads the old one.
#pragma once
#include "bk_decide.cuh"

namespace bk {

// A leaf of the tree so far.
struct alignas(16) LeafEnt {
  long long key, pay;   // dkey of its best gain; inner feature << 32 | threshold | default_left << 31
  int32_t feat, node;   // real feature of its best split; node (0 the root, 1 + 2x / 2 + 2x the left /
                        // right child of expansion x)
  int32_t out;          // its entry in the table of expanded leaves (-1: not expanded)
  int32_t begin, count, slot;
  int32_t depth_buf;    // depth << 1 | index buffer
  int32_t _pad;
};

// An expanded leaf whose split is not taken yet: what its children would be.
struct alignas(16) OutEnt {
  long long key[2], pay[2];  // left, right
  int32_t feat[2];
  int32_t slot[2];
  int32_t x, L;              // the expansion, its left row count
  int32_t leaf, _pad;        // the leaf
};

// An expansion of the current round.
struct alignas(16) RoundExp {
  int32_t x;             // -1: the root, before any split
  int32_t out, node, inner;
  uint32_t thr;          // threshold | default_left << 31
  int32_t begin, count, depth_buf;
  int32_t slot, sslot;   // pool slots: the leaf's, which its larger child gets, and its smaller child's
  int32_t leaf, _pad;
};

// The best candidate of one group of features (or of one feature) of a searched leaf.
struct alignas(16) RoundCand {
  long long key;  // dkey of its gain, kNoKey when there is none
  uint32_t pk;    // inner feature << 9 | default_left << 8 | threshold
  int32_t real;   // real feature
};

// A split as it was taken: expansion x at leaf `leaf`; the right child becomes leaf (index + 1).
struct Commit {
  int32_t x, leaf, L;  // L -1: the tree's last split, whose left count is still in the counters
  int32_t count;       // rows of the leaf
};

struct alignas(16) RoundHdr {
  int32_t leaves, n_cur, n_x, stop;
  unsigned int out_mask;
  int32_t last_x, last_par, _pad;  // the tree's last split when its count was not known yet (else -1)
};

__host__ __device__ __forceinline__ size_t round_align(size_t x) { return (x + 15) / 16 * 16; }

// A job's rounds state, laid out in one allocation.
struct RoundView {
  RoundHdr* hdr;     // [2]
  RoundExp* cur;     // [2][kMaxRoundW]
  OutEnt* out;       // [2][kMaxRoundOut]
  long long* pcnt;   // [2][kMaxRoundW][2] rows the partition placed from the front (low half) and the back (high)
  LeafEnt* leaf;     // [2][num_leaves]
  Commit* commit;    // [num_leaves]
  int2* xinfo;       // [max_exp] node and inner feature of every expansion
  RoundCand* cand;   // [2 kMaxRoundW][feature groups] the search's candidates, row 2 e + side
  size_t bytes;
};

__host__ __device__ __forceinline__ RoundView round_view(uint8_t* base, int num_leaves, int max_exp, int F) {
  RoundView v;
  size_t o = 0;
  v.hdr = reinterpret_cast<RoundHdr*>(base + o);
  o += round_align(2 * sizeof(RoundHdr));
  v.cur = reinterpret_cast<RoundExp*>(base + o);
  o += round_align(2 * kMaxRoundW * sizeof(RoundExp));
  v.out = reinterpret_cast<OutEnt*>(base + o);
  o += round_align(2 * kMaxRoundOut * sizeof(OutEnt));
  v.pcnt = reinterpret_cast<long long*>(base + o);
  o += round_align(2 * kMaxRoundW * 2 * sizeof(long long));
  v.leaf = reinterpret_cast<LeafEnt*>(base + o);
  o += round_align(2 * (size_t)num_leaves * sizeof(LeafEnt));
  v.commit = reinterpret_cast<Commit*>(base + o);
  o += round_align((size_t)num_leaves * sizeof(Commit));
  v.xinfo = reinterpret_cast<int2*>(base + o);
  o += round_align((size_t)max_exp * sizeof(int2));
  v.cand = reinterpret_cast<RoundCand*>(base + o);
  o += round_align((size_t)2 * kMaxRoundW * F * sizeof(RoundCand));
  v.bytes = o;
  return v;
}
__device__ __forceinline__ RoundView round_view(const Job& J, const Params& p) {
  return round_view(J.rounds, p.num_leaves, p.max_exp, p.F);
}

// Pool slots: the root's is 0; expansion x's smaller child gets 1 + x (zeroed when the tree starts,
// as histograms are added up in it).
__host__ __device__ __forceinline__ int32_t round_sslot(int32_t x) { return 1 + x; }

// Whether the children of an expansion are searched (serial.rs:779-825: not at max_depth, not when
// both have fewer than 2 min_data_in_leaf rows).
__device__ __forceinline__ bool round_go(const Params& p, const RoundExp& c, int32_t L) {
  if (c.x < 0)
    return !(p.max_depth > 0 && (c.depth_buf >> 1) >= p.max_depth) && !(c.count < p.min_data * 2);
  if (p.max_depth > 0 && (c.depth_buf >> 1) + 1 >= p.max_depth) return false;
  return !(c.count - L < p.min_data * 2 && L < p.min_data * 2);
}

// How a round's leaves, one after the other, are cut into `ctas` equal intervals of whole `unit`s of
// rows, at least min_rows each: interval b is [b per, (b + 1) per). With `apart`, every leaf starts
// at an interval of its own; that is chosen when the intervals grow by at most `slack` rows by it.
// One warp; lane e < n passes leaf e's rows (lanes past it 0) and gets its start in *off.
struct RoundCut {
  int64_t per;
  bool apart;
};
__device__ __forceinline__ RoundCut round_cut(int32_t rows, int n, int ctas, int min_rows, int unit, int slack,
                                              int lane, int64_t* off) {
  auto scan = [&](int64_t x) {
#pragma unroll 1
    for (int o = 1; o < kMaxRoundW; o <<= 1) {
      const int64_t y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    return x;
  };
  const int64_t incl = scan(rows);
  const int64_t total = __shfl_sync(0xffffffffu, incl, kMaxRoundW - 1);
  RoundCut c;
  // 32-bit divisions: a leaf's and a round's rows are fewer than 2^31
  auto per_of = [&](int parts) {
    int64_t per = ((uint32_t)total + (uint32_t)parts - 1u) / (uint32_t)parts;
    if (per < min_rows) per = min_rows;
    return (per + unit - 1) / unit * unit;
  };
  c.per = per_of(ctas);
  c.apart = false;
  *off = incl - rows;
  if (ctas > n) {
    const int64_t apart = per_of(ctas - n);  // sum of ceil(rows / apart) <= (ctas - n) + n
    if (apart <= c.per + slack) {
      c.per = apart;
      c.apart = true;
      const int64_t len = ((uint32_t)rows + (uint32_t)apart - 1u) / (uint32_t)apart * apart;
      *off = scan(len) - len;
    }
  }
  return c;
}

// The rows of an expansion's histogram: the smaller child's (the root's own).
struct HistPart {
  int32_t begin, count, buf, slot;
  bool go, left_smaller;
};
__device__ __forceinline__ HistPart round_hist_part(const Params& p, const RoundExp& c, int32_t L) {
  HistPart h;
  h.go = round_go(p, c, L);
  const int32_t buf = c.depth_buf & 1;
  if (c.x < 0) {
    h.begin = c.begin;
    h.count = c.count;
    h.buf = buf;
    h.slot = c.slot;
    h.left_smaller = true;
  } else {
    const int32_t R = c.count - L;
    h.left_smaller = L < R;
    h.begin = h.left_smaller ? c.begin : c.begin + L;
    h.count = h.left_smaller ? L : R;
    h.buf = 1 - buf;
    h.slot = c.sslot;
  }
  return h;
}

namespace {

// The order of the leaf arg-max (split_info.rs:104-133): the higher gain, then the smaller real
// feature (-1 as the largest), then the smaller leaf index.
struct LeafOrd {
  long long key;
  int32_t feat, i;
};
__device__ __forceinline__ LeafOrd leaf_ord(long long key, int32_t feat, int32_t i) {
  return LeafOrd{key, feat == -1 ? 0x7fffffff : feat, i};
}
__device__ __forceinline__ bool ord_before(const LeafOrd& a, const LeafOrd& b) {
  if (a.key != b.key) return a.key > b.key;
  if (a.feat != b.feat) return a.feat < b.feat;
  return a.i < b.i;
}
// Shared memory of a round's decision.
struct RoundSmem {
  RoundHdr hdr;                      // in; then out
  long long key[kMaxRoundLeaves], pay[kMaxRoundLeaves];
  int32_t feat[kMaxRoundLeaves], node[kMaxRoundLeaves], out[kMaxRoundLeaves];
  int32_t begin[kMaxRoundLeaves], count[kMaxRoundLeaves], slot[kMaxRoundLeaves], depth_buf[kMaxRoundLeaves];
  alignas(16) uint32_t open[kMaxRoundLeaves];  // open_key of the leaves, 0 past the last one
  LeafOrd wopen[kDecideWarps], sorted[32];     // the best open leaf per warp; the expanded leaves in order
  uint8_t perm[32];                            // their table entries
  int32_t leaves, still0, still1;
  int64_t off[kMaxRoundW];                     // the chosen leaves' rows, cut over the partition's CTAs
  RoundCut cut;
  unsigned int mask, got;
  OutEnt ot[kMaxRoundOut];
  RoundExp cur[kMaxRoundW];          // the expansions the search covered
  int32_t curL[kMaxRoundW];
  RoundExp nxt[kMaxRoundW];          // the expansions chosen
  long long fkey[2 * kMaxRoundW], fpay[2 * kMaxRoundW];
  int32_t ffeat[2 * kMaxRoundW];
};

// A leaf's key in 32 bits, order-preserving up to ties: 0 when its gain is not positive or it is
// expanded already, else one more than the key's high word.
__device__ __forceinline__ uint32_t open_key(const RoundSmem& s, int i) {
  return (s.key[i] > 0 && s.out[i] < 0) ? (uint32_t)(s.key[i] >> 32) + 1u : 0u;
}

// Before the search has finished: the round's state and the row counts of its expansions (written
// two launches ago and earlier). Every thread of the CTA calls it; no barrier.
__device__ __forceinline__ void decide_round_load(const Job& J, const Params& p, int q, RoundSmem& s) {
  const RoundView v = round_view(J, p);
  const int t = threadIdx.x;
  if (t == 0) {
    const int4* h = reinterpret_cast<const int4*>(v.hdr + q);
    int4* d = reinterpret_cast<int4*>(&s.hdr);
    d[0] = __ldcg(h);
    d[1] = __ldcg(h + 1);
  }
  for (int i = t; i < p.num_leaves; i += kDecideThreads) {
    const int4* e = reinterpret_cast<const int4*>(v.leaf + (size_t)q * p.num_leaves + i);
    const int4 a = __ldcg(e), b = __ldcg(e + 1), c = __ldcg(e + 2);
    s.key[i] = (long long)(((unsigned long long)(unsigned)a.y << 32) | (unsigned)a.x);
    s.pay[i] = (long long)(((unsigned long long)(unsigned)a.w << 32) | (unsigned)a.z);
    s.feat[i] = b.x;
    s.node[i] = b.y;
    s.out[i] = b.z;
    s.begin[i] = b.w;
    s.count[i] = c.x;
    s.slot[i] = c.y;
    s.depth_buf[i] = c.z;
    s.open[i] = open_key(s, i);
  }
  if (t == 0) s.got = 0u;
  {
    static_assert(sizeof(OutEnt) % 16 == 0 && sizeof(RoundExp) % 16 == 0 && sizeof(LeafEnt) == 48 && sizeof(RoundHdr) == 32,
                  "the records are moved in 16-byte words");
    const int4* o = reinterpret_cast<const int4*>(v.out + q * kMaxRoundOut);
    for (int i = t; i < (int)(kMaxRoundOut * sizeof(OutEnt) / 16); i += kDecideThreads)
      reinterpret_cast<int4*>(s.ot)[i] = __ldcg(o + i);
    const int4* c = reinterpret_cast<const int4*>(v.cur + q * kMaxRoundW);
    for (int i = t; i < (int)(kMaxRoundW * sizeof(RoundExp) / 16); i += kDecideThreads)
      reinterpret_cast<int4*>(s.cur)[i] = __ldcg(c + i);
    if (t < kMaxRoundW) s.curL[t] = (int32_t)__ldcg(v.pcnt + ((size_t)q * kMaxRoundW + t) * 2);
  }
}

// After the search: the fold of every searched leaf's candidates (serial.rs:1523-1558,
// split_info.rs:67-133: the higher gain, then the smaller real feature), eight threads per leaf.
// Barrier before and after.
__device__ __forceinline__ void decide_round_fold(const Job& J, const Params& p, RoundSmem& s) {
  static_assert(kDecideThreads == 8 * 2 * kMaxRoundW, "eight threads per searched leaf");
  const int i = threadIdx.x >> 3, sub = threadIdx.x & 7;
  const int n_cur = s.hdr.n_cur;
  if (i >= ((2 * n_cur + 3) & ~3)) return;  // whole warps: four leaves each
  const int e = i >> 1;
  const bool searched = i < 2 * n_cur && round_go(p, s.cur[e], s.curL[e]) && !(s.cur[e].x < 0 && (i & 1));
  long long key = kNoKey;
  int32_t real = 0x7fffffff;
  uint32_t pk = 0u;
  if (searched) {
    const int4* c = reinterpret_cast<const int4*>(round_view(J, p).cand + (size_t)i * p.n_groups);
#pragma unroll 4
    for (int g = sub; g < p.n_groups; g += 8) {
      const int4 x = __ldcg(c + g);
      const long long k = (long long)(((unsigned long long)(unsigned)x.y << 32) | (unsigned)x.x);
      if (k > key || (k == key && x.w < real)) {
        key = k;
        real = x.w;
        pk = (uint32_t)x.z;
      }
    }
  }
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) {
    const long long k = __shfl_xor_sync(FULL, key, o);
    const int32_t r = __shfl_xor_sync(FULL, real, o);
    const uint32_t q = __shfl_xor_sync(FULL, pk, o);
    if (k > key || (k == key && r < real)) {
      key = k;
      real = r;
      pk = q;
    }
  }
  if (sub == 0 && i < 2 * n_cur) {
    // the fold starts from SplitInfo::default (gain -inf, feature -1) and replaces it only with a
    // better candidate
    const long long none = dkey(-CUDART_INF);
    const bool take = key > none;
    s.fkey[i] = take ? key : none;
    s.ffeat[i] = take ? real : -1;
    s.fpay[i] = take ? (long long)(pk >> 9) * 4294967296LL + (long long)((pk & 255u) | (((pk >> 8) & 1u) << 31))
                     : (long long)-1 * 4294967296LL;
  }
}

__device__ __forceinline__ LeafOrd ord_best_warp(LeafOrd x) {
#pragma unroll 1
  for (int o = 16; o > 0; o >>= 1) {
    const LeafOrd y{__shfl_xor_sync(FULL, x.key, o), __shfl_xor_sync(FULL, x.feat, o), __shfl_xor_sync(FULL, x.i, o)};
    if (ord_before(y, x)) x = y;
  }
  return x;
}

// Before the search has finished, with the state loaded and a barrier passed: the best open leaf.
__device__ __forceinline__ void decide_round_open(RoundSmem& s) {
  LeafOrd x = leaf_ord(kNoKey, -1, 0x7fffffff);
  for (int i = threadIdx.x; i < kMaxRoundLeaves; i += kDecideThreads)
    if (i >= s.hdr.leaves) {
      s.open[i] = 0u;
    } else if (s.open[i] != 0u) {
      const LeafOrd y = leaf_ord(s.key[i], s.feat[i], i);
      if (ord_before(y, x)) x = y;
    }
  x = ord_best_warp(x);
  if ((threadIdx.x & 31) == 0) s.wopen[threadIdx.x >> 5] = x;
}

// Warp 0, after the fold: commits the splits that are known. record: this CTA writes them down.
//
// The one-by-one loop takes the expanded leaves in their order for as long as the next one comes
// before every leaf that is not expanded: the open leaves of the tree and the children of those
// taken before it. So with the expanded leaves sorted (one per lane), an exclusive prefix maximum
// over their children tells how many are taken, all at once.
__device__ __forceinline__ void decide_round_commit(const Job& J, const Params& p, bool record, RoundSmem& s) {
  const RoundView v = round_view(J, p);
  const int lane = threadIdx.x & 31;
  const int n_cur = s.hdr.n_cur;
  const int leaves0 = s.hdr.leaves;
  const unsigned int mask = s.hdr.out_mask;
  const LeafOrd none = leaf_ord(kNoKey, -1, 0x7fffffff);
  // the expanded leaves, one per table entry
  LeafOrd mine = none;
  if ((mask >> lane) & 1u) {
    const int32_t i = s.ot[lane].leaf;
    mine = leaf_ord(s.key[i], s.feat[i], i);
  }
  s.sorted[lane] = mine;
  // what the search found: the root's best, or both children's of every expansion
  if (lane < n_cur) {
    const RoundExp& c = s.cur[lane];
    if (c.x < 0) {
      s.key[0] = s.fkey[0];
      s.pay[0] = s.fpay[0];
      s.feat[0] = s.ffeat[0];
      s.open[0] = open_key(s, 0);
    } else {
      const int32_t L = s.curL[lane];
      const HistPart h = round_hist_part(p, c, L);
      const int il = 2 * lane + (h.left_smaller ? 0 : 1), ir = 2 * lane + (h.left_smaller ? 1 : 0);
      OutEnt& o = s.ot[c.out];
      o.key[0] = s.fkey[il];
      o.pay[0] = s.fpay[il];
      o.feat[0] = s.ffeat[il];
      o.key[1] = s.fkey[ir];
      o.pay[1] = s.fpay[ir];
      o.feat[1] = s.ffeat[ir];
      // children that are not searched: the left one keeps the leaf's slot, the right one has none
      o.slot[0] = !h.go ? c.slot : (h.left_smaller ? c.sslot : c.slot);
      o.slot[1] = !h.go ? -1 : (h.left_smaller ? c.slot : c.sslot);
      o.x = c.x;
      o.L = L;
    }
  }
  __syncwarp();
  // sorted by counting, eight entries' loads in flight at a time
  int rank = 0;
  const int n_tab = 32 - __clz(mask);  // entries are handed out lowest first
#pragma unroll 4
  for (int j = 0; j < n_tab; ++j) rank += ord_before(s.sorted[j], mine) ? 1 : 0;
  const int n_exp = __popc(mask);
  __syncwarp();
  if ((mask >> lane) & 1u) {
    s.sorted[rank] = mine;
    s.perm[rank] = (uint8_t)lane;
  }
  // the best open leaf (the root's first search: the root)
  LeafOrd before = lane < kDecideWarps ? s.wopen[lane] : none;
  if (n_cur > 0 && s.cur[0].x < 0) before = s.open[0] ? leaf_ord(s.key[0], s.feat[0], 0) : none;
  before = ord_best_warp(before);
  __syncwarp();
  const int oi = lane < n_exp ? s.perm[lane] : 0;
  const LeafOrd e = lane < n_exp ? s.sorted[lane] : none;
  const OutEnt& o = s.ot[oi];
  // the better child, with the leaf indices they would get (the left one keeps the leaf's)
  LeafOrd ch = none;
  if (lane < n_exp) {
    const LeafOrd l = leaf_ord(o.key[0], o.feat[0], e.i), r = leaf_ord(o.key[1], o.feat[1], leaves0 + lane);
    ch = ord_before(l, r) ? l : r;
  }
#pragma unroll 1
  for (int k = 1; k < 32; k <<= 1) {
    const LeafOrd y{__shfl_up_sync(FULL, ch.key, k), __shfl_up_sync(FULL, ch.feat, k), __shfl_up_sync(FULL, ch.i, k)};
    if (lane >= k && ord_before(y, ch)) ch = y;
  }
  const LeafOrd prev{__shfl_up_sync(FULL, ch.key, 1), __shfl_up_sync(FULL, ch.feat, 1), __shfl_up_sync(FULL, ch.i, 1)};
  if (lane > 0 && ord_before(prev, before)) before = prev;
  const bool take = lane < n_exp && lane < p.num_leaves - leaves0 && ord_before(e, before);
  const unsigned fail = __ballot_sync(FULL, !take);
  const int n_take = fail ? __ffs(fail) - 1 : 32;
  unsigned int freed = 0u;
  if (lane < n_take) {
    const int at = e.i, nl = leaves0 + lane;
    const int32_t x = o.x, L = o.L, begin = s.begin[at], count = s.count[at];
    const int32_t db = ((s.depth_buf[at] >> 1) + 1) * 2 + (1 - (s.depth_buf[at] & 1));
    if (record) v.commit[nl - 1] = Commit{x, at, L, count};
    s.key[at] = o.key[0];
    s.pay[at] = o.pay[0];
    s.feat[at] = o.feat[0];
    s.node[at] = 1 + 2 * x;
    s.out[at] = -1;
    s.count[at] = L;
    s.slot[at] = o.slot[0];
    s.depth_buf[at] = db;
    s.key[nl] = o.key[1];
    s.pay[nl] = o.pay[1];
    s.feat[nl] = o.feat[1];
    s.node[nl] = 2 + 2 * x;
    s.out[nl] = -1;
    s.begin[nl] = begin + L;
    s.count[nl] = count - L;
    s.slot[nl] = o.slot[1];
    s.depth_buf[nl] = db;
    s.open[at] = open_key(s, at);
    s.open[nl] = open_key(s, nl);
    freed = 1u << oi;
  }
  freed = __reduce_or_sync(FULL, freed);
  if (lane == 0) {
    s.leaves = leaves0 + n_take;
    s.mask = mask & ~freed;
    s.still0 = n_take;  // sorted[still0 .. still1): expanded leaves that are not split yet
    s.still1 = n_exp;
  }
}

// Every thread, after the commit and a barrier: the round's expansions (s.nxt) and the header of the
// coming round — the best open leaves, among the leaves that the remaining splits can reach. The
// best leaf of the tree is open (or there is none: the tree ends, serial.rs:611) and always finds
// room; any other leaves one entry of the table free. Every thread ranks its leaves among the open
// ones by counting. Ends with a barrier.
__device__ __forceinline__ void decide_round_choose(const Job& J, const Params& p, int q, bool record, RoundSmem& s) {
  const RoundView v = round_view(J, p);
  const int leaves = s.leaves, left = p.num_leaves - leaves, used = __popc(s.mask), n_x = s.hdr.n_x;
  const int n4 = (leaves + 3) >> 2;
  int n_new = 0;
  for (int i0 = 0; i0 < leaves; i0 += kDecideThreads) {  // one pass for up to kDecideThreads leaves
    const int i = i0 + (int)threadIdx.x;
    const uint32_t k = i < leaves ? s.open[i] : 0u;
    bool chosen = false;
    int rank = 0;
    if (k != 0u && left > 0) {
      int eq = 0;
      const uint4* o4 = reinterpret_cast<const uint4*>(s.open);
#pragma unroll 4
      for (int j = 0; j < n4; ++j) {
        const uint4 x = o4[j];  // entries past the last leaf are 0
        rank += (x.x > k) + (x.y > k) + (x.z > k) + (x.w > k);
        eq += (x.x == k) + (x.y == k) + (x.z == k) + (x.w == k);
      }
      const LeafOrd me = leaf_ord(s.key[i], s.feat[i], i);
      if (eq > 1)  // equal high words: settled in full
        for (int j = 0; j < leaves; ++j)
          rank += (s.open[j] == k && j != i && ord_before(leaf_ord(s.key[j], s.feat[j], j), me)) ? 1 : 0;
      chosen = rank < p.round_w && (rank == 0 || used + rank < p.round_out - 1);
      if (chosen && rank > 0) {
        int ahead = rank;
        for (int j = s.still0; j < s.still1; ++j) ahead += ord_before(s.sorted[j], me) ? 1 : 0;
        chosen = ahead < left;
      }
    }
    if (chosen) {
      unsigned int z = ~s.mask;
      for (int j = 0; j < rank; ++j) z &= z - 1u;
      const int slot = __ffs(z) - 1;
      const int32_t x = n_x + rank;
      RoundExp c;
      c.x = x;
      c.out = slot;
      c.node = s.node[i];
      c.inner = (int32_t)(s.pay[i] >> 32);
      c.thr = (uint32_t)(s.pay[i] & 0xffffffffLL);
      c.begin = s.begin[i];
      c.count = s.count[i];
      c.depth_buf = s.depth_buf[i];
      c.slot = s.slot[i];
      c.sslot = round_sslot(x);
      c.leaf = i;
      c._pad = 0;
      s.nxt[rank] = c;
      s.ot[slot].leaf = i;
      s.out[i] = slot;
      atomicOr(&s.got, 1u << slot);
      if (record) v.xinfo[x] = make_int2(c.node, c.inner);
    }
    n_new += __syncthreads_count(chosen);
  }
  if (threadIdx.x == 0) {
    const bool last = n_new > 0 && left == 1;
    RoundHdr h;
    h.leaves = leaves + (last ? 1 : 0);
    h.n_cur = n_new;
    h.last_x = last ? n_x : -1;
    h.last_par = q ^ 1;
    h.n_x = n_x + n_new;
    h.stop = (n_new == 0 || last) ? 1 : 0;
    h.out_mask = s.mask | s.got;
    h._pad = 0;
    if (last) {
      // the tree's last split: nothing about its children is searched, so it is taken now; its row
      // counts come from the partition that follows
      const RoundExp c = s.nxt[0];
      const int at = c.leaf;
      if (record) v.commit[leaves - 1] = Commit{c.x, at, -1, c.count};
      const int32_t db = ((c.depth_buf >> 1) + 1) * 2 + (1 - (c.depth_buf & 1));
      s.node[at] = 1 + 2 * c.x;
      s.depth_buf[at] = db;
      s.node[leaves] = 2 + 2 * c.x;
      s.begin[leaves] = c.begin;
      s.count[leaves] = c.count;
      s.slot[leaves] = c.slot;
      s.depth_buf[leaves] = db;
      s.key[leaves] = s.pay[leaves] = 0;
      s.feat[leaves] = s.out[leaves] = -1;
    }
    s.hdr = h;
  }
  __syncthreads();
}

// CTA 0, after the commit and a barrier: the state of the coming round.
__device__ __forceinline__ void decide_round_store(const Job& J, const Params& p, int q, const RoundSmem& s) {
  const RoundView v = round_view(J, p);
  const int t = threadIdx.x, w = q ^ 1;
  if (t == 0) {
    RoundHdr h = s.hdr;
    if (h.stop) h.n_cur = 0;  // no histogram or search follows
    v.hdr[w] = h;
    if (h.stop) {
      J.st->tree_leaves = h.leaves;
      J.st->fin_q = w;
      J.st->stop = 1;
    }
  }
  for (int i = t; i < s.hdr.leaves; i += kDecideThreads) {
    LeafEnt e;
    e.key = s.key[i];
    e.pay = s.pay[i];
    e.feat = s.feat[i];
    e.node = s.node[i];
    e.out = s.out[i];
    e.begin = s.begin[i];
    e.count = s.count[i];
    e.slot = s.slot[i];
    e.depth_buf = s.depth_buf[i];
    e._pad = 0;
    v.leaf[(size_t)w * p.num_leaves + i] = e;
  }
  for (int i = t; i < kMaxRoundOut; i += kDecideThreads) v.out[w * kMaxRoundOut + i] = s.ot[i];
  for (int i = t; i < s.hdr.n_cur; i += kDecideThreads) v.cur[w * kMaxRoundW + i] = s.nxt[i];
}

}  // namespace

}  // namespace bk
