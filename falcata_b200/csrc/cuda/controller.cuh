// K8: the level controller as a device function, shared by its own kernel and by the fused tail of the
// split search (the last block of the search grid runs it, so a level needs no controller launch).
// One block decides, between two levels, which frontier leaves split (all of them, or the highest gains
// when the leaf budget binds; ties: lower leaf id), numbers the new leaves, and writes everything the next
// level's kernels need: partition descriptors, child bookkeeping, the smaller children's construct
// allotments, the search children, the journal entry of every split and the new frontier.
// Parity: src/treelearner/cuda/cuda_hybrid_graph.cu:L220-631 (device controller of the graph loop),
// cuda_single_gpu_tree_learner.cpp:L1355-1478 (CollectSplittableLeaves / ArbitrateLevelBudget),
// L1718-1775 (FinishLevelBookkeeping). The selection rule is the one of the host-driven loop and of
// the host learner's `level` policy, so all three grow identical trees.
#pragma once
#include "kernels.cuh"

namespace fb {

constexpr int kCtrlMaxLeaves = 1024;

// Shared-memory working set of the controller (the caller provides it).
struct CtrlShared {
  int leaf[kCtrlMaxLeaves];               // candidate leaves
  double gain[kCtrlMaxLeaves];            // and their gains
  int rank[kCtrlMaxLeaves];               // leaf-wise growth: evaluated nodes before the candidate (kNotKept: beyond the budget)
  int chosen[kCtrlMaxLeaves];             // chosen leaves in ascending order
  int chunks[kCtrlMaxLeaves], blocks[kCtrlMaxLeaves];   // their exclusive prefixes
  unsigned int kept[kCtrlMaxLeaves / 32];               // chosen leaves as a bit set
  int kept_before[kCtrlMaxLeaves / 32];                 // chosen leaves before each word
  double first[2 * kCtrlMaxLeaves + 2];   // leaf-wise growth: first order-key step of every evaluated node
  int ncand, nkeep, total_chunks, total_blocks;
};

// A record that another block of the SAME launch may have written a moment ago: read through L2, in 16- or 8-byte pieces
// where the type allows it (the loads of one record are independent and issue back to back).
template <typename T>
__device__ inline T LoadWords(const T* p) {
  static_assert(sizeof(T) % 4 == 0, "word-sized records only");
  T v;
  if constexpr (sizeof(T) % 16 == 0 && alignof(T) >= 16) {
    const uint4* s = reinterpret_cast<const uint4*>(p);
    uint4* d = reinterpret_cast<uint4*>(&v);
#pragma unroll
    for (int w = 0; w < static_cast<int>(sizeof(T) / 16); ++w) d[w] = __ldcg(s + w);
  } else if constexpr (sizeof(T) % 8 == 0 && alignof(T) >= 8) {
    const unsigned long long* s = reinterpret_cast<const unsigned long long*>(p);
    unsigned long long* d = reinterpret_cast<unsigned long long*>(&v);
#pragma unroll
    for (int w = 0; w < static_cast<int>(sizeof(T) / 8); ++w) d[w] = __ldcg(s + w);
  } else {
    const unsigned int* s = reinterpret_cast<const unsigned int*>(p);
    unsigned int* d = reinterpret_cast<unsigned int*>(&v);
#pragma unroll
    for (int w = 0; w < static_cast<int>(sizeof(T) / 4); ++w) d[w] = __ldcg(s + w);
  }
  return v;
}

// Call with all threads of one block (whole warps). Reads the level record `a.cur`, writes the next level's into `a.nxt`.
// listed: the caller has filled S.leaf / S.gain / S.ncand with the frontier leaves that have a usable split.
__device__ inline void ControllerBody(const CtrlArgs& a, CtrlShared& S, bool listed) {
  constexpr int kNotKept = 0x7fffffff;
  const int T = blockDim.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = T >> 5;
  // the level record is read whole before anything is written: `cur` and `nxt` may be the same object
  const LevelCtrl c0 = LoadWords(a.cur);
  int num_eval_out = c0.num_eval;
  LevelCtrl* c = a.nxt;
  if (!listed) {
    if (threadIdx.x == 0) S.ncand = 0;
    __syncthreads();
    // 1. candidates: frontier leaves with a usable split
    const int nfront = c0.done ? 0 : c0.frontier_count;
    for (int i = threadIdx.x; i < nfront; i += T) {
      const int l = a.frontier[i];
      const int feature = LoadWords(&a.best[l].feature); const double gain = LoadWords(&a.best[l].gain);
      if (feature >= 0 && gain > 0.0) { const int p = atomicAdd(&S.ncand, 1); S.leaf[p] = l; S.gain[p] = gain; }
    }
  }
  for (int w = threadIdx.x; w < kCtrlMaxLeaves / 32; w += T) S.kept[w] = 0u;
  __syncthreads();
  const int ncand = S.ncand;
  const int budget = a.max_leaves - c0.num_leaves;
  if (a.leafwise_budget > 0) {
    // 2'. leaf-wise: record the order keys of the newly evaluated nodes, then keep the candidates with fewer than
    //     leafwise_budget evaluated nodes strictly before them; if the growth cap binds, the best of those by rank
    const int base_eval = c0.num_eval, total = base_eval + ncand;
    // first key step of every evaluated node in shared memory: it decides nearly every comparison
    for (int j = threadIdx.x; j < base_eval; j += T) S.first[j] = a.eval_key[static_cast<size_t>(j) * 4];
    for (int i = threadIdx.x; i < ncand; i += T) {
      double key[4];
      LeafwiseChildKey(LoadWords(a.leaves + S.leaf[i]).pkey, S.gain[i], key);
      for (int k = 0; k < 4; ++k) a.eval_key[static_cast<size_t>(base_eval + i) * 4 + k] = key[k];
      S.first[base_eval + i] = key[0];
    }
    __syncthreads();
    // one warp per candidate, the lanes stride over the evaluated nodes
    for (int i = warp; i < ncand; i += warps) {
      double ki[4]; for (int k = 0; k < 4; ++k) ki[k] = a.eval_key[static_cast<size_t>(base_eval + i) * 4 + k];
      int cnt = 0;
#pragma unroll 4
      for (int j = lane; j < total; j += 32) {
        const double pj = S.first[j];
        bool before = pj > ki[0];
        if (pj == ki[0]) before = LeafwiseKeyBefore(a.eval_key + static_cast<size_t>(j) * 4, ki);
        cnt += before ? 1 : 0;
      }
      cnt = __reduce_add_sync(0xffffffffu, cnt);
      if (lane == 0) S.rank[i] = cnt < a.leafwise_budget ? cnt : kNotKept;
    }
    num_eval_out = total;
    __syncthreads();
  }
  // 2. rank when the budget binds: by gain (ties: lower leaf id), or by the leaf-wise rank; the kept ones as a bit set
  for (int i = warp; i < ncand; i += warps) {
    const int li = S.leaf[i];
    bool keep = a.leafwise_budget <= 0 || S.rank[i] != kNotKept;
    if (keep && ncand > budget) {
      int better = 0;
      for (int j = lane; j < ncand; j += 32) {
        const int lj = S.leaf[j];
        if (a.leafwise_budget > 0) better += (S.rank[j] < S.rank[i]) || (S.rank[j] == S.rank[i] && lj < li);
        else better += (S.gain[j] > S.gain[i]) || (S.gain[j] == S.gain[i] && lj < li);
      }
      keep = __reduce_add_sync(0xffffffffu, better) < budget;
    }
    if (keep && lane == 0) atomicOr(&S.kept[li >> 5], 1u << (li & 31));
  }
  __syncthreads();
  // 3. the kept leaves by leaf id
  if (warp == 0) {
    static_assert(kCtrlMaxLeaves / 32 == 32, "a word per lane");
    const int n = __popc(S.kept[lane]);
    int incl = n;
    for (int o = 1; o < 32; o <<= 1) { const int y = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += y; }
    S.kept_before[lane] = incl - n;
    if (lane == 31) S.nkeep = incl;
  }
  __syncthreads();
  const int NS = S.nkeep;
  for (int i = threadIdx.x; i < ncand; i += T) {
    const int li = S.leaf[i];
    const unsigned int word = S.kept[li >> 5], bit = 1u << (li & 31);
    if (!(word & bit)) continue;
    const int s = S.kept_before[li >> 5] + __popc(word & (bit - 1u));
    S.chosen[s] = li;
    // 4. local allotments: chunks of the partition (at least one: the chunk block of a split also sets up its children), blocks of the construct
    const int cnt = LoadWords(&a.leaves[li].count);
    S.chunks[s] = max(1, (cnt + kPartChunk - 1) / kPartChunk);
    S.blocks[s] = max(1, (cnt + a.rows_per_block - 1) / a.rows_per_block);
  }
  __syncthreads();
  if (warp == 0) {
    int ac = 0, ab = 0;
    for (int s0 = 0; s0 < NS; s0 += 32) {
      const int s = s0 + lane;
      const int vc = s < NS ? S.chunks[s] : 0, vb = s < NS ? S.blocks[s] : 0;
      int ic = vc, ib = vb;
      for (int o = 1; o < 32; o <<= 1) { const int yc = __shfl_up_sync(0xffffffffu, ic, o), yb = __shfl_up_sync(0xffffffffu, ib, o); if (lane >= o) { ic += yc; ib += yb; } }
      if (s < NS) { S.chunks[s] = ac + ic - vc; S.blocks[s] = ab + ib - vb; }
      ac += __shfl_sync(0xffffffffu, ic, 31); ab += __shfl_sync(0xffffffffu, ib, 31);
    }
    if (lane == 0) { S.total_chunks = ac; S.total_blocks = ab; }
  }
  __syncthreads();
  // 5. descriptors
  const int base_leaf = c0.num_leaves, base_slot = c0.next_slot, base_journal = c0.journal_count;
  for (int s = threadIdx.x; s < NS; s += T) {
    const int l = S.chosen[s];
    const int right = base_leaf + s;
    const LeafInfo P = LoadWords(a.leaves + l);
    const SplitRecord b = LoadWords(a.best + l);
    const FeatureMeta m = a.meta[b.feature];
    PartSplit q;
    q.leaf = l; q.right_leaf = right; q.begin = P.begin; q.count = P.count; q.buffer = P.buffer; q.group = m.group; q.bundled = m.bundled; q.group_offset = m.group_offset;
    q.num_bin = m.num_bin; q.most_freq_bin = m.most_freq_bin; q.threshold = b.threshold; q.default_left = b.default_left; q.missing_type = m.missing_type;
    q.default_bin = m.default_bin; q.is_categorical = b.is_categorical; for (int w = 0; w < 8; ++w) q.cat_bitset[w] = b.cat_bitset[w];
    q.chunk_begin = S.chunks[s]; q.num_chunks = max(1, (P.count + kPartChunk - 1) / kPartChunk); q.pad_[0] = q.pad_[1] = 0;
    q.owner = a.bin_owner != nullptr ? a.bin_owner[m.hist_offset] : 0;
    a.splits[s] = q;
    ChildInit ci;
    ci.smaller_is_left = b.left_cnt <= b.right_cnt ? 1 : 0;
    const int fresh = base_slot + s;
    ci.left_slot = ci.smaller_is_left ? fresh : P.hist_slot; ci.right_slot = ci.smaller_is_left ? P.hist_slot : fresh;
    ci.left_g = b.left_g; ci.left_h = b.left_h; ci.right_g = b.right_g; ci.right_h = b.right_h; ci.left_out = b.left_out; ci.right_out = b.right_out;
    ci.left_gi = b.left_gi; ci.left_hi = b.left_hi; ci.right_gi = P.sum_gi - b.left_gi; ci.right_hi = P.sum_hi - b.left_hi;
    ci.hist_block_begin = S.blocks[s]; ci.hist_num_blocks = max(1, (P.count + a.rows_per_block - 1) / a.rows_per_block);
    ci.monotone = b.monotone; ci.pad_ = 0; LeafwiseChildKey(P.pkey, b.gain, ci.pkey);
    a.child_init[s] = ci;
    FindChild fl, fr;
    fl.leaf = l; fl.slot = ci.left_slot; fl.other_slot = ci.right_slot; fl.is_larger = ci.smaller_is_left ? 0 : 1; fl.split = s; fl.is_left = 1; fl.parent_global = P.num_data_global; fl.task = s;
    fr.leaf = right; fr.slot = ci.right_slot; fr.other_slot = ci.left_slot; fr.is_larger = ci.smaller_is_left ? 1 : 0; fr.split = s; fr.is_left = 0; fr.parent_global = P.num_data_global; fr.task = s;
    a.children[2 * s] = fl; a.children[2 * s + 1] = fr;
    SplitJournal j; j.leaf = l; j.right_leaf = right; j.parent_global = P.num_data_global; j.pad = 0; j.rec = b;
    j.begin = P.begin; j.count = P.count; j.buffer = P.buffer; j.depth = P.depth;
    a.journal[base_journal + s] = j;
  }
  // 6. new frontier (children in split order) and the level record
  for (int s = threadIdx.x; s < NS; s += T) { a.frontier[2 * s] = S.chosen[s]; a.frontier[2 * s + 1] = base_leaf + s; }
  if (threadIdx.x == 0) {
    LevelCtrl o = c0;
    o.num_leaves = base_leaf + NS; o.next_slot = base_slot + NS; o.journal_count = base_journal + NS; o.level = c0.level + 1; o.num_eval = num_eval_out;
    // A level that uses up the leaf budget ends the tree: its children are partitioned (the score update and the
    // leaf counts need their windows) but neither constructed nor searched.
    const bool last = base_leaf + NS >= a.max_leaves;
    o.num_splits = NS; o.num_children = 2 * NS; o.total_chunks = S.total_chunks; o.total_blocks = last ? 0 : S.total_blocks;
    o.skip_search = last ? 1 : 0;
    o.frontier_count = last ? 0 : 2 * NS;
    if (NS == 0) o.done = 1; else o.pad0 = o.level;   // pad0: last level that applied a split
    *c = o;
  }
}

}  // namespace fb
