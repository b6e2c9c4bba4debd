// K7, tiled form: a block stages a tile of rows in shared memory once (feature-major, so that the lane that owns a
// row always reads its own bank) and walks it through the whole forest; the trees stream through shared memory in
// chunks of a few trees, double-buffered with asynchronous copies, as 8-byte nodes whose two children sit next to
// each other. The block's threads are (row, tree slice) pairs: kWalks walks in flight per thread, and the slices add warps
// where the shared memory has no room for more rows.
//
// What bounds it: instructions per step of a walk. A node holds everything as ready-made offsets into the block's shared
// memory (feature row, left child) and a leaf is a node that leads to itself - its feature row holds -infinity, which goes
// left everywhere - so a step is shift, mask, load, mask, compare, add, load, without a test for the end.
// Measured: 4M rows x 136 features, 500 trees of 255 leaves, 41.0 -> 24.6 ms against 256 threads with eight walks each and
// nodes of indices; 200k rows x 100 features, 500 trees of 127 leaves with missing values, 3.9 -> 2.1 ms.
//
// Parity: python-package/falcata/basic.py:L5112-5163 (device predict route: raw score, converted score, leaf index),
// include/Falcata/tree.h:L361-439 (numerical decision with missing-value handling). Forests with categorical splits, a tree of
// more than kTiledTreeLeaves leaves, or more than kTiledFeatures used features take the general one-thread-per-row kernel;
// leaf indices of these, and of double rows with more than kTiledFeaturesF64Leaf used features, come from the host.
#include <cuda_fp16.h>
#include <cuda_pipeline.h>
#include <omp.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <limits>
#include <memory>
#include <vector>

#include "engine.h"

namespace fb {

namespace {

// value: threshold of an internal node; output of a leaf (leaf-index prediction: the leaf's index, as bits).
// meta:  bits 16-31 feature slot: the feature's row of the tile, counted in rows from the start of the block's shared memory;
//        bits 3-15 byte offset of the left child in its chunk (a multiple of 8; the right child is the next node, a leaf
//        leads to itself); bits 1-2 missing type (kLeafType: a leaf); bit 0 default-left.
struct PackedNode { float value; unsigned int meta; };
static_assert(sizeof(PackedNode) == 8, "8-byte nodes");

constexpr int kPredictThreads = 512;        // threads of a block = rows of its tile x tree slices
constexpr int kTreeBytes = 32 * 1024;       // a tree and its root word must fit this much; also the smaller chunk size
constexpr int kMaxTreeSplits = kTiledTreeLeaves - 1;
static_assert((2 * kTiledTreeLeaves - 1) * static_cast<int>(sizeof(PackedNode)) + 32 <= kTreeBytes, "the largest tree fits a chunk");
constexpr int kPredictSmem = 220 * 1024;
static_assert(2 * kTreeBytes + (kTiledFeatures + 1) * 32 * 4 + kPredictThreads * 8 <= kPredictSmem, "the widest forest fits a 32-row tile beside two chunks");
constexpr unsigned int kLeafType = 3;
constexpr unsigned int kChildMask = 0xFFF8u;
constexpr int kWalks = 4;                   // tree walks a thread keeps in flight

struct ChunkDesc { long long offset; int bytes; int ntrees; int roots; int cls; int first_tree; int pad; };   // blob offset (16-byte aligned); roots: offset of the trees' root words

template <typename T> __device__ inline float ToF(T v) { return static_cast<float>(v); }
template <> __device__ inline float ToF<__half>(__half v) { return __half2float(v); }

// PLAIN: no node of the forest treats zero or NaN as missing; NaN inputs were replaced by 0 when the tile was staged
// (that is what such nodes do with them), so a step is one comparison.
template <bool PLAIN>
__device__ __forceinline__ bool GoLeft(float v, float thr, unsigned int meta) {
  if (PLAIN) return v <= thr;
  const unsigned int mt = (meta >> 1) & 3u;
  const bool nan = isnan(v);
  if (nan && mt != 2u) v = 0.f;
  const bool use_default = (mt == 1u && fabsf(v) <= 1e-35f) || (mt == 2u && nan);
  return use_default ? (meta & 1u) != 0u : v <= thr;
}

// LEAF: write the leaf index of every (row, tree) instead of summing outputs.
// Shared memory: [2][chunk_bytes] tree ring (chunk_bytes a power of two), [num_used + 1][tile_rows] floats (the last row is the
// leaves' -infinity), [kPredictThreads] doubles. log_rows: log2(tile_rows), 5..8.
template <typename T, bool LEAF, bool PLAIN>
__global__ void __launch_bounds__(kPredictThreads, 1)
PredictTiledKernel(const unsigned char* __restrict__ blob, const ChunkDesc* __restrict__ chunks, int num_chunks, int chunk_bytes, const int* __restrict__ used, int num_used,
                   const T* __restrict__ data, int nrow, int ncol, int row_major, int log_rows, int num_class, int trees_total, float inv_avg, float* __restrict__ out) {
  extern __shared__ __align__(1024) unsigned char smem[];
  const int tile_rows = 1 << log_rows, slices = kPredictThreads >> log_rows;
  unsigned char* ring = smem;
  float* rows_s = reinterpret_cast<float*>(smem + 2 * chunk_bytes);
  double* sums = reinterpret_cast<double*>(smem + 2 * chunk_bytes + (num_used + 1) * tile_rows * 4);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int r = tid & (tile_rows - 1), slice = tid >> log_rows;
  // a slot's byte offset is slot * tile_rows * 4: shift it out of the meta word, the row's own offset fills the low bits
  const unsigned int slot_shift = 16 - (log_rows + 2), slot_mask = ~(static_cast<unsigned int>(tile_rows) * 4u - 1u), row_bytes = r * 4;
  const int num_tiles = (nrow + tile_rows - 1) >> log_rows;
  for (int i = tid; i < tile_rows; i += kPredictThreads) rows_s[num_used * tile_rows + i] = __int_as_float(0xff800000);   // -infinity
  for (int tile = blockIdx.x; tile < num_tiles; tile += gridDim.x) {
    const int row0 = tile << log_rows;
    const int row = row0 + r;
    __syncthreads();   // the previous tile's walks are over before its rows and ring buffers are overwritten
    // ---- stage the tile: rows_s[j][r] = value of used feature j in row row0 + r ----
    if (!row_major) {
      for (int j = slice; j < num_used; j += slices) {
        float v = row < nrow ? ToF<T>(data[static_cast<size_t>(used[j]) * nrow + row]) : 0.f;
        if (PLAIN && isnan(v)) v = 0.f;
        rows_s[j * tile_rows + r] = v;
      }
    } else {
      // 16 rows x 32 features: read with the lanes along the features (coalesced), turn in a padded scratch piece that
      // borrows the still unused ring, write with the lanes along the rows
      float* scratch = reinterpret_cast<float*>(ring) + warp * (16 * 33);
      static_assert(kPredictThreads / 32 * 16 * 33 * 4 <= 2 * kTreeBytes, "the pieces fit the ring");
      const int fpieces = (num_used + 31) / 32;
      for (int piece = warp; piece < fpieces * (tile_rows / 16); piece += kPredictThreads / 32) {
        const int fp = piece % fpieces, rp = piece / fpieces;
        const int j = fp * 32 + lane;
        const int col = j < num_used ? used[j] : -1;
#pragma unroll
        for (int k = 0; k < 16; ++k) {
          const int rr = row0 + rp * 16 + k;
          float v = (col >= 0 && rr < nrow) ? ToF<T>(data[static_cast<size_t>(rr) * ncol + col]) : 0.f;
          if (PLAIN && isnan(v)) v = 0.f;
          scratch[k * 33 + lane] = v;
        }
        __syncwarp();
#pragma unroll
        for (int k = 0; k < 32; k += 2) {
          const int jj = fp * 32 + k + (lane >> 4);
          if (jj < num_used) rows_s[jj * tile_rows + rp * 16 + (lane & 15)] = scratch[(lane & 15) * 33 + k + (lane >> 4)];
        }
        __syncwarp();
      }
    }
    __syncthreads();
    // ---- walk the forest, chunk by chunk ----
    auto fetch = [&](int c) {
      if (c < num_chunks) {
        const ChunkDesc d = chunks[c];
        const uint4* src = reinterpret_cast<const uint4*>(blob + d.offset);
        uint4* dst = reinterpret_cast<uint4*>(ring + (c & 1) * chunk_bytes);
        for (int i = tid; i < d.bytes / 16; i += kPredictThreads) __pipeline_memcpy_async(dst + i, src + i, 16);
      }
      __pipeline_commit();
    };
    // the slices' sums of one class, added in slice order; all threads of the block
    auto finish_class = [&](int cls, double acc) {
      sums[tid] = acc;
      __syncthreads();
      if (slice == 0 && row < nrow) {
        double t = sums[r];
        for (int k = 1; k < slices; ++k) t += sums[(k << log_rows) + r];
        out[static_cast<size_t>(cls) * nrow + row] = static_cast<float>(t * inv_avg);
      }
      __syncthreads();
    };
    fetch(0);
    double acc = 0.0;   // a forest of a thousand trees summed in float would drift from the host's double sums
    int cur_cls = num_chunks > 0 ? chunks[0].cls : 0;
    for (int c = 0; c < num_chunks; ++c) {
      fetch(c + 1);
      __pipeline_wait_prior(1);
      __syncthreads();
      const ChunkDesc d = chunks[c];
      if (!LEAF && d.cls != cur_cls) { finish_class(cur_cls, acc); acc = 0.0; cur_cls = d.cls; }
      const unsigned int buf = (c & 1) * chunk_bytes;
      const int* roots = reinterpret_cast<const int*>(smem + buf + d.roots);   // [ntrees] chunk offset of every tree's root
      for (int t = slice * kWalks; t < d.ntrees; t += slices * kWalks) {
        PackedNode nd[kWalks];
#pragma unroll
        for (int q = 0; q < kWalks; ++q) nd[q] = *reinterpret_cast<const PackedNode*>(smem + buf + roots[min(t + q, d.ntrees - 1)]);   // past the last tree: walked again, not counted
        auto step = [&]() {
          float v[kWalks];
#pragma unroll
          for (int q = 0; q < kWalks; ++q) v[q] = *reinterpret_cast<const float*>(smem + (((nd[q].meta >> slot_shift) & slot_mask) | row_bytes));
#pragma unroll
          for (int q = 0; q < kWalks; ++q) {
            unsigned int next = (nd[q].meta & kChildMask) | buf;
            // a leaf stays where it is: -infinity goes left, and its left child is itself (a NaN leaf: right, and so is its right child)
            if (!GoLeft<PLAIN>(v[q], nd[q].value, nd[q].meta)) next += 8u;
            nd[q] = *reinterpret_cast<const PackedNode*>(smem + next);
          }
        };
        for (;;) {
          unsigned int all = nd[0].meta;
#pragma unroll
          for (int q = 1; q < kWalks; ++q) all &= nd[q].meta;
          if ((all & (kLeafType << 1)) == (kLeafType << 1)) break;   // every walk is at a leaf
          step(); step();
        }
#pragma unroll
        for (int q = 0; q < kWalks; ++q) {
          if (t + q < d.ntrees) {
            if (LEAF) { if (row < nrow) reinterpret_cast<int*>(out)[static_cast<size_t>(row) * trees_total + d.first_tree + (t + q) * num_class] = __float_as_int(nd[q].value); }
            else acc += static_cast<double>(nd[q].value);
          }
        }
      }
      __syncthreads();   // everyone is done with this buffer before the fetch after next refills it
    }
    __pipeline_wait_prior(0);
    if (!LEAF && num_chunks > 0) finish_class(cur_cls, acc);
  }
}

// Nodes of one tree in sibling-adjacent order, root first, then every split's two children next to each other, placed at
// byte `base` of their chunk. slot_base: slot of the tile's first feature row; leaf_slot: slot of the row of -infinity.
// queue: room for the tree's splits (this runs inside a parallel region, which no exception may leave: nothing is allocated here).
struct QueuedSplit { int id, pos; };   // host id, packed position
void PackTree(const Tree& T, const std::vector<int>& slot_of_feature, int slot_base, int leaf_slot, bool leaf_index, int base, QueuedSplit* queue, PackedNode* out) {
  auto offset = [&](int pos) { return static_cast<unsigned int>(base + pos * static_cast<int>(sizeof(PackedNode))); };
  auto place = [&](int id, int pos) {   // host ids: >= 0 split, < 0 leaf ~id
    if (id >= 0) return;
    if (leaf_index) { const int leaf = ~id; std::memcpy(&out[pos].value, &leaf, sizeof(int)); } else out[pos].value = static_cast<float>(T.leaf_value[~id]);
    // -infinity goes left at every value but NaN: a NaN leaf's left child is the node before it, so that its right one is itself
    const bool nan = !leaf_index && std::isnan(T.leaf_value[~id]);
    out[pos].meta = (static_cast<unsigned int>(leaf_slot) << 16) | offset(nan ? pos - 1 : pos) | (kLeafType << 1);
  };
  if (T.num_leaves <= 1) { place(~0, 0); return; }
  int queued = 0, next_free = 1;   // splits in breadth-first order
  queue[queued++] = {0, 0};
  for (int qi = 0; qi < queued; ++qi) {
    const int id = queue[qi].id, left_pos = next_free;
    next_free += 2;
    float thr = static_cast<float>(T.threshold[id]);
    // keep "v <= threshold" exact for float inputs: round the double threshold DOWN to float
    if (static_cast<double>(thr) > T.threshold[id]) thr = std::nextafterf(thr, -std::numeric_limits<float>::infinity());
    PackedNode& nd = out[queue[qi].pos];
    nd.value = thr;
    nd.meta = (static_cast<unsigned int>(slot_base + slot_of_feature[T.split_feature[id]]) << 16) | offset(left_pos) |
              (static_cast<unsigned int>(Tree::MissingTypeOf(T.decision_type[id])) << 1) | ((T.decision_type[id] & kDefaultLeftMask) ? 1u : 0u);
    const int child[2] = {T.left_child[id], T.right_child[id]};
    for (int c = 0; c < 2; ++c) { if (child[c] >= 0) queue[queued++] = {child[c], left_pos + c}; else place(child[c], left_pos + c); }
  }
}

// What the packed form asks of a tree, and what the tree brings: the features it reads and whether it has missing-aware nodes.
// uses: a flag per feature. (Inside a parallel region, like PackTree.)
bool ScanTree(const Tree& T, bool leaf_index, char* uses, int num_features, bool* plain) {
  if (T.is_linear || T.num_leaves > kTiledTreeLeaves) return false;
  if (!leaf_index && T.num_leaves <= 1 && std::isnan(T.leaf_value[0])) return false;   // no node before it to lead to
  for (int s = 0; s < T.num_leaves - 1; ++s) {
    if (T.decision_type[s] & kCategoricalMask) return false;
    if (Tree::MissingTypeOf(T.decision_type[s]) != 0) *plain = false;
    const int f = T.split_feature[s];
    if (f < 0 || f >= num_features) return false;
    uses[f] = 1;
  }
  return true;
}

}  // namespace

// Returns false when the forest or the matrix is outside what the tiled kernel covers (the caller then takes the
// general kernel). predict_type 0/1: out[class][row] sums; 2: out_leaf[row][tree] leaf indices.
bool DevicePredictTiled(const GBDT* gbdt, const void* device_data, int dtype, int32_t nrow, int32_t ncol, bool row_major, int first_tree, int num_trees, int K,
                        bool leaf_index, float inv_avg, float* out_device, cudaStream_t s) {
  if (num_trees <= 0 || nrow <= 0) return false;
  if (dtype != kF32 && dtype != kF64 && dtype != kF16) return false;
  // Packing is host work of every call (a quarter million nodes took 1.8 ms on one core): large forests are scanned and packed
  // by all cores, straight into the one buffer that goes to the device in one copy.
  long long forest_nodes = 0;
  for (int t = first_tree; t < first_tree + num_trees; ++t) forest_nodes += 2LL * gbdt->models_[t]->num_leaves - 1;
  const bool parallel = forest_nodes > (1 << 15);
  // features the forest reads, in ascending order
  const size_t nfeat = std::max(1, gbdt->max_feature_idx_ + 1);
  const int team = parallel ? TeamThreads() : 1;
  std::vector<char> uses(team * nfeat, 0);   // a row per thread
  bool plain = true, covered = true;   // plain: no node with a missing type - NaN reads as 0 everywhere, zero is an ordinary value
#pragma omp parallel for schedule(static) num_threads(team) reduction(&& : plain, covered)
  for (int t = 0; t < num_trees; ++t)
    covered = covered && ScanTree(*gbdt->models_[first_tree + t], leaf_index, uses.data() + omp_get_thread_num() * nfeat, static_cast<int>(nfeat), &plain);
  if (!covered) return false;
  std::vector<int> slot_of_feature(nfeat, -1), used;
  for (int k = 1; k < team; ++k) for (size_t f = 0; f < nfeat; ++f) uses[f] |= uses[k * nfeat + f];
  for (size_t f = 0; f < nfeat; ++f) if (uses[f]) { slot_of_feature[f] = static_cast<int>(used.size()); used.push_back(static_cast<int>(f)); }
  if (used.empty()) used.push_back(0);
  const int nu = static_cast<int>(used.size());
  // the walk compares in fp32, which is exact for fp32 and half rows; the leaf of a double row next to a threshold can differ from
  // the host's, which compares in double: wide forests, which only tiles of fewer rows hold, leave it to the host as they always did
  if (leaf_index && dtype == kF64 && nu > kTiledFeaturesF64Leaf) return false;
  int dev = 0, sms = 0; FB_CUDA(cudaGetDevice(&dev)); FB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  // The tile: as many rows as fit beside two chunks (the forest streams through the ring once per tile), but no more than
  // leave every SM a tile; the threads that rows do not take walk other trees.
  auto smem_of = [&](int log_rows, int chunk) { return 2 * static_cast<size_t>(chunk) + (static_cast<size_t>(nu + 1) << log_rows) * 4 + kPredictThreads * sizeof(double); };
  int log_rows = 8;
  while (log_rows > 5 && (smem_of(log_rows, kTreeBytes) > kPredictSmem || ((nrow + (1 << log_rows) - 1) >> log_rows) < sms)) --log_rows;
  if (smem_of(log_rows, kTreeBytes) > kPredictSmem) return false;
  const int chunk_bytes = smem_of(log_rows, 2 * kTreeBytes) <= kPredictSmem ? 2 * kTreeBytes : kTreeBytes;   // more trees per barrier where there is room
  const size_t smem = smem_of(log_rows, chunk_bytes);
  const int slot_base = (2 * chunk_bytes) >> (log_rows + 2);   // the tile's rows start behind the ring
  if (slot_base + nu > 0xFFFF) return false;
  // chunks: trees of one class in iteration order, as many as fit a ring buffer; the root words behind the nodes
  struct Place { int chunk, base, pos; };   // pos: the tree's number in its chunk
  std::vector<Place> place(num_trees);
  std::vector<ChunkDesc> chunks;
  size_t bytes = 0;
  for (int cls = 0; cls < K; ++cls) {
    ChunkDesc d; d.ntrees = 0; d.roots = 0; d.cls = cls; d.first_tree = 0; d.pad = 0;
    auto close = [&]() {
      if (d.ntrees == 0) return;
      d.offset = static_cast<long long>(bytes); d.bytes = (d.roots + d.ntrees * 4 + 15) & ~15;
      bytes += d.bytes;
      chunks.push_back(d); d.ntrees = 0; d.roots = 0;
    };
    for (int t = cls; t < num_trees; t += K) {
      const int tree = std::max(1, 2 * gbdt->models_[first_tree + t]->num_leaves - 1) * static_cast<int>(sizeof(PackedNode));
      if (d.roots + tree + (d.ntrees + 1) * 4 + 16 > chunk_bytes) close();
      if (d.ntrees == 0) d.first_tree = t;
      place[t] = {static_cast<int>(chunks.size()), d.roots, d.ntrees};
      d.roots += tree; ++d.ntrees;
    }
    close();
  }
  if (chunks.empty()) return false;
  // one buffer, one copy: chunk list, used features, trees
  const size_t chunks_at = 0, used_at = chunks.size() * sizeof(ChunkDesc), blob_at = (used_at + used.size() * sizeof(int) + 15) & ~static_cast<size_t>(15);
  std::vector<unsigned char> staged(blob_at + bytes);
  memcpy(staged.data() + chunks_at, chunks.data(), chunks.size() * sizeof(ChunkDesc));
  memcpy(staged.data() + used_at, used.data(), used.size() * sizeof(int));
  const std::unique_ptr<QueuedSplit[]> queues(new QueuedSplit[static_cast<size_t>(team) * kMaxTreeSplits]);
#pragma omp parallel for schedule(static) num_threads(team)
  for (int t = 0; t < num_trees; ++t) {
    const ChunkDesc& d = chunks[place[t].chunk];
    unsigned char* chunk = staged.data() + blob_at + d.offset;
    PackTree(*gbdt->models_[first_tree + t], slot_of_feature, slot_base, slot_base + nu, leaf_index, place[t].base,
             queues.get() + static_cast<size_t>(omp_get_thread_num()) * kMaxTreeSplits, reinterpret_cast<PackedNode*>(chunk + place[t].base));
    reinterpret_cast<int*>(chunk + d.roots)[place[t].pos] = place[t].base;
  }
  DevBuf<unsigned char> forest;
  forest.Upload(staged.data(), staged.size(), s);
  const unsigned char* d_blob = forest.get() + blob_at;
  const ChunkDesc* d_chunks = reinterpret_cast<const ChunkDesc*>(forest.get() + chunks_at);
  const int* d_used = reinterpret_cast<const int*>(forest.get() + used_at);
  const int tiles = (nrow + (1 << log_rows) - 1) >> log_rows;
  const int grid = std::min(tiles, sms);
  const int nc = static_cast<int>(chunks.size());
#define FB_TILED_P(T, LEAF, PLAIN)                                                                                                 \
  {                                                                                                                                \
    static PerDevice allowed;                                                                                                      \
    AllowSharedMemory(PredictTiledKernel<T, LEAF, PLAIN>, kPredictSmem, &allowed);                                                 \
    PredictTiledKernel<T, LEAF, PLAIN><<<grid, kPredictThreads, smem, s>>>(d_blob, d_chunks, nc, chunk_bytes, d_used, nu, static_cast<const T*>(device_data), nrow, ncol, \
                                                                           row_major ? 1 : 0, log_rows, K, num_trees, inv_avg, out_device);   \
  }
#define FB_TILED(T, LEAF) { if (plain) FB_TILED_P(T, LEAF, true) else FB_TILED_P(T, LEAF, false) }
  if (leaf_index) {
    if (dtype == kF32) FB_TILED(float, true) else if (dtype == kF64) FB_TILED(double, true) else FB_TILED(__half, true)
  } else {
    if (dtype == kF32) FB_TILED(float, false) else if (dtype == kF64) FB_TILED(double, false) else FB_TILED(__half, false)
  }
#undef FB_TILED
#undef FB_TILED_P
  FB_LAUNCHED(); FB_KERNEL_CHECK();
  FB_CUDA(cudaStreamSynchronize(s));   // the packed forest lives in this call's buffers
  return true;
}

}  // namespace fb
