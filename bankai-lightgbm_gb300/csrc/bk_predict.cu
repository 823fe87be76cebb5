// Prediction of binned rows through a trained tree on the device: the replay that
// SerialTreeLearner::add_prediction_for_rows performs for rows outside the training partition
// (serial.rs:2009-2041), with each split's routing rule (data_partition.rs:299-410) evaluated on
// the rows' stored bins. Rows binned with the training bin mappers land in the same leaves as
// the reference's threshold comparisons on raw values (a value is <= the bin's upper bound
// exactly when its bin is <= the threshold bin). A categorical split routes by the bitset of its
// left bins over the feature's bin mapper (data_partition.rs:264-300, route_bin :367-377): stored
// bin 0 holds the most frequent bin's rows and goes left when that bin is not 0 and is in the
// set; stored bin b looks up bit b - 1 + offset.
//
// Two forms. k_predict_staged copies the columns that the tree splits on, a tile of rows at a time,
// into shared memory and walks packed 8-byte nodes there: the columns' bytes move once, 16 at a time,
// and a step of a row's walk is two shared-memory reads. k_predict_tree walks with global loads: a
// step's warp touches up to 32 lines, each a cycle of the SM's L1, behind six dependent loads (2M rows, a
// tree of 255 leaves on 100 features: 125 us, staged 70). It remains for trees that split on more
// columns than the tile holds, or with more leaves than a packed node can name.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>

#include "bk_math.cuh"

namespace bk {

namespace {

constexpr int kPredictRows = 496;   // rows per tile: 31 runs of 16 bytes, one more for the misalignment
constexpr int kPredictPitch = 528;  // bytes from one column's run to the next: four banks on
constexpr int kPredictColumns = 96;   // four CTAs per SM; at 150 columns both forms take the same time
constexpr int kPredictSmem = 227 * 1024;

// The packed tree: the leaf values, the nodes, the columns, the nodes' sets.
struct PredictLayout {
  int32_t nodes, cols, sets, bytes;  // byte offsets; bytes without the sets
};
__host__ __device__ __forceinline__ PredictLayout predict_layout(int32_t num_leaves, int32_t ncols) {
  PredictLayout l;
  l.nodes = 8 * num_leaves;
  l.cols = l.nodes + 8 * (num_leaves - 1);
  l.bytes = l.cols + 4 * ncols;
  l.sets = (l.bytes + 15) / 16 * 16;
  return l;
}

// A node is two words. x: the left and right child, 16 bits each (negative: ~leaf). y, from bit 0: stored
// bin 0 goes left; the special bin goes left; the column's misalignment (4 bits); its place among the
// tree's columns (10); the highest bin of the left side (8); the special bin (8; 0: the node routes by
// its 256-bit set of left bins).
__device__ __forceinline__ int32_t packed_child(uint2 nd, uint32_t bin, const uint32_t* __restrict__ set) {
  const uint32_t special = nd.y >> 24;
  bool left;
  if (special == 0u) left = ((__ldg(set + (bin >> 5)) >> (bin & 31u)) & 1u) != 0u;
  else left = bin == special ? (nd.y & 2u) != 0u : (bin == 0u ? (nd.y & 1u) != 0u : bin <= ((nd.y >> 16) & 255u));
  return left ? (int32_t)(int16_t)(nd.x & 0xffffu) : (int32_t)nd.x >> 16;
}
__device__ __forceinline__ uint32_t packed_column(uint2 nd) {  // byte offset of its run in the tile
  return ((nd.y >> 6) & 0x3ffu) * kPredictPitch + ((nd.y >> 2) & 15u);
}

// Persistent CTAs over tiles of kPredictRows rows. A column's run is copied from its 16-byte boundary on,
// so the copies are aligned whatever the number of rows. Two rows per thread, their walks interleaved.
__global__ void __launch_bounds__(256)
    k_predict_staged(int32_t num_leaves, int32_t ncols, int32_t F, const unsigned char* __restrict__ tree,
                     const uint8_t* __restrict__ bins, int64_t m, double* __restrict__ score) {
  extern __shared__ __align__(16) unsigned char smem[];
  const PredictLayout lay = predict_layout(num_leaves, ncols);
  const int32_t* cols = reinterpret_cast<const int32_t*>(tree + lay.cols);
  const uint32_t* sets = reinterpret_cast<const uint32_t*>(tree + lay.sets);
  unsigned char* tab = smem + (size_t)ncols * kPredictPitch;
  for (int e = threadIdx.x; e < lay.cols / 8; e += blockDim.x)  // the values and the nodes
    reinterpret_cast<uint2*>(tab)[e] = reinterpret_cast<const uint2*>(tree)[e];
  const double* values = reinterpret_cast<const double*>(tab);
  const uint2* nodes = reinterpret_cast<const uint2*>(tab + lay.nodes);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(smem);
  const uintptr_t lo = reinterpret_cast<uintptr_t>(bins), hi = lo + (uintptr_t)F * (uintptr_t)m;
  for (int64_t r0 = (int64_t)blockIdx.x * kPredictRows; r0 < m; r0 += (int64_t)gridDim.x * kPredictRows) {
    const int rows = (int)min((int64_t)kPredictRows, m - r0);
    __syncthreads();  // the tile before is done with
    for (int c = warp; c < ncols; c += nwarps) {
      const uintptr_t col = lo + (uintptr_t)cols[c] * (uintptr_t)m + (uintptr_t)r0;
      const uintptr_t src = (col & ~(uintptr_t)15) + 16u * lane;
      if (src >= col + (uintptr_t)rows) continue;  // past the tile's rows
      const uint32_t at = (uint32_t)c * kPredictPitch + 16u * lane;
      if (src >= lo && src + 16 <= hi) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sbase + at), "l"(src) : "memory");
      } else {  // the two ends of the matrix
        for (int k = 0; k < 16; ++k)
          if (src + k >= lo && src + k < hi) smem[at + k] = *reinterpret_cast<const uint8_t*>(src + k);
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    const int ra = (int)threadIdx.x, rb = ra + 256;
    int32_t na = ra < rows && num_leaves > 1 ? 0 : -1, nb = rb < rows && num_leaves > 1 ? 0 : -1;
    for (int guard = 0; guard < num_leaves && (na >= 0 || nb >= 0); ++guard) {
      const uint2 da = nodes[max(na, 0)], db = nodes[max(nb, 0)];
      const uint32_t bin_a = smem[packed_column(da) + (na >= 0 ? ra : 0)];
      const uint32_t bin_b = smem[packed_column(db) + (nb >= 0 ? rb : 0)];
      if (na >= 0) na = packed_child(da, bin_a, sets + 8 * na);
      if (nb >= 0) nb = packed_child(db, bin_b, sets + 8 * nb);
    }
    if (ra < rows) score[r0 + ra] += values[na < 0 ? ~na : 0];
    if (rb < rows) score[r0 + rb] += values[nb < 0 ? ~nb : 0];
  }
}

__global__ void k_predict_tree(const DevFeature* __restrict__ feats, int32_t num_leaves,
                               const int32_t* __restrict__ tree, const double* __restrict__ leaf_value,
                               const uint8_t* __restrict__ bins, int64_t m, double* __restrict__ score) {
  // tree: [left_child | right_child | split_feature_inner | threshold_in_bin | decision_type],
  // then 8 words of left-bin bitset per node (categorical splits, decision_type bit 0)
  const int32_t ni = num_leaves - 1;
  const int32_t* lc = tree;
  const int32_t* rc = tree + ni;
  const int32_t* sf = tree + 2 * ni;
  const int32_t* th = tree + 3 * ni;
  const int32_t* dt = tree + 4 * ni;
  const uint32_t* cb = reinterpret_cast<const uint32_t*>(tree + 5 * ni);
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x) {
    int32_t node = num_leaves > 1 ? 0 : -1;
    int guard = 0;
    while (node >= 0 && guard++ < num_leaves) {
      const int32_t f = sf[node];
      const uint32_t bin = bins[(size_t)f * (size_t)m + i];
      const DevFeature& fm = feats[f];
      bool left;
      if (dt[node] & 1) {
        const uint32_t pos = bin == 0 ? (uint32_t)fm.mfb : bin - 1 + (uint32_t)fm.offset;
        const bool set = pos < 256u && ((cb[(size_t)node * 8 + (pos >> 5)] >> (pos & 31)) & 1u) != 0u;
        left = (int)bin < fm.gbins && set && (bin != 0 || fm.mfb > 0);
      } else {
        left = route_bin(fm, (uint32_t)th[node], (dt[node] & 2) != 0, bin) != 0;
      }
      node = left ? lc[node] : rc[node];
    }
    score[i] += leaf_value[node < 0 ? ~node : 0];
  }
}

}  // namespace

size_t predict_pack(const DevFeature* h_feat, int32_t num_leaves, const int32_t* left, const int32_t* right,
                    const int32_t* feature, const uint32_t* threshold, const int8_t* type, const uint32_t* cat_bins,
                    const double* leaf_value, const uint8_t* bins, int64_t m, int32_t* column_of, unsigned char* out,
                    int32_t* num_columns) {
  const int32_t ni = num_leaves - 1;
  if (num_leaves > 32768) return 0;
  int32_t ncols = 0;
  for (int32_t i = 0; i < ni; ++i) column_of[feature[i]] = -1;
  for (int32_t i = 0; i < ni; ++i)
    if (column_of[feature[i]] < 0) column_of[feature[i]] = ncols++;
  if (ncols > kPredictColumns || ncols * kPredictPitch + 16 * num_leaves > kPredictSmem) return 0;
  const PredictLayout lay = predict_layout(num_leaves, ncols);
  std::memcpy(out, leaf_value, 8 * (size_t)num_leaves);
  uint32_t* nodes = reinterpret_cast<uint32_t*>(out + lay.nodes);
  int32_t* cols = reinterpret_cast<int32_t*>(out + lay.cols);
  uint32_t* sets = reinterpret_cast<uint32_t*>(out + lay.sets);
  bool any_set = false;
  for (int32_t i = 0; i < ni; ++i) {
    const int32_t f = feature[i];
    const DevFeature& d = h_feat[f];
    cols[column_of[f]] = f;
    const bool dleft = (type[i] & 2) != 0;
    const uint32_t max_bin = (uint32_t)d.gbins - 1;
    uint32_t flags = 0, th = 0, special = 0;
    if ((type[i] & 1) || max_bin < 2) {
      any_set = true;
      for (uint32_t w = 0; w < 8; ++w) {
        uint32_t bits = 0;
        for (uint32_t b = 32 * w; b < 32 * w + 32; ++b) {
          bool l;
          if (type[i] & 1) {
            const uint32_t pos = b == 0 ? (uint32_t)d.mfb : b - 1 + (uint32_t)d.offset;
            const bool set = pos < 256u && ((cat_bins[(size_t)i * 8 + (pos >> 5)] >> (pos & 31)) & 1u) != 0u;
            l = (int)b < d.gbins && set && (b != 0 || d.mfb > 0);
          } else {
            l = route_bin(d, threshold[i], dleft, b) != 0;
          }
          bits |= (uint32_t)l << (b & 31);
        }
        sets[8 * (size_t)i + w] = bits;
      }
    } else {
      // route_bin over more than two stored bins: bin 0, the missing values' bin, and the rest by
      // bin <= threshold; without a missing bin, 255 stands in with the rest's answer
      const uint32_t base = d.mfb == 0 ? 0u : 1u;
      th = std::min(threshold[i] + base, 255u);
      special = 255u;
      if (d.missing == 1 && d.default_bin != d.mfb) special = std::min((uint32_t)d.default_bin + base, 255u);
      if (d.missing == 2 && !(max_bin == (uint32_t)d.mfb + 1 && d.mfb > 0)) special = max_bin;
      flags = (route_bin(d, threshold[i], dleft, 0) ? 1u : 0u) | (route_bin(d, threshold[i], dleft, special) ? 2u : 0u);
    }
    const uint32_t shift = (uint32_t)((reinterpret_cast<uintptr_t>(bins) + (uintptr_t)f * (uintptr_t)m) & 15u);
    nodes[2 * i] = ((uint32_t)left[i] & 0xffffu) | ((uint32_t)right[i] << 16);
    nodes[2 * i + 1] = flags | (shift << 2) | ((uint32_t)column_of[f] << 6) | (th << 16) | (special << 24);
  }
  *num_columns = ncols;
  return any_set ? (size_t)lay.sets + 32 * (size_t)ni : (size_t)lay.bytes;
}

cudaError_t predict_staged(int32_t F, int32_t num_leaves, int32_t num_columns, const unsigned char* d_packed,
                           const uint8_t* bins, int64_t m, double* score, cudaStream_t s) {
  const int smem = num_columns * kPredictPitch + 16 * num_leaves;
  cudaError_t e = cudaFuncSetAttribute(k_predict_staged, cudaFuncAttributeMaxDynamicSharedMemorySize, kPredictSmem);
  if (e != cudaSuccess) return e;
  const int64_t tiles = ceil_div64(m, (int64_t)kPredictRows);
  const int per_sm = std::max(1, std::min(8, kPredictSmem / (smem + 1024)));
  k_predict_staged<<<(unsigned)std::min<int64_t>(tiles, 152 * per_sm), 256, smem, s>>>(num_leaves, num_columns, F, d_packed,
                                                                                     bins, m, score);
  return cudaGetLastError();
}

cudaError_t predict_tree(const DevFeature* feats, int32_t num_leaves, const int32_t* d_tree, const double* d_leaf_value,
                         const uint8_t* bins, int64_t m, double* score, cudaStream_t s) {
  k_predict_tree<<<1024, 256, 0, s>>>(feats, num_leaves, d_tree, d_leaf_value, bins, m, score);
  return cudaGetLastError();
}

}  // namespace bk
