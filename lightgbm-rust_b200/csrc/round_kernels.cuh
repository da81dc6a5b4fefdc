// Growth of a tree in rounds. The reference splits one leaf at a time: the
// leaf of largest gain (learner/mod.rs:653-706), until num_leaves leaves or
// no positive gain. One split per step leaves the GPU idle: a step is three
// dependent launches of a few microseconds whatever its rows, so a 255-leaf
// tree cost 254 x about 20 us. But the splits of the finished tree are known
// in advance up to their order: a node is split exactly when the smallest
// gain on its path from the root is among the num_leaves - 1 largest such
// values of all nodes. So a round expands many nodes at once (partition, histogram, scan
// of every expanded node's children in one launch each), the likely ones
// first, and the reference's order is replayed over the gains found so far
// (k_round_decide): the replay splits the leaf of largest gain as long as
// that leaf has been expanded, with the reference's tie rules, and the node
// it waits for is always part of the next round. The tree is therefore the
// reference's, split by split; an expansion the replay never reaches is
// wasted work (about half as many again on a 255-leaf tree, but of small
// leaves: 8% more rows) and leaves no trace.
//
// A 255-leaf tree takes 16 (the first of a run, whose gains fall with depth) to
// 30 rounds instead of 254 steps.
//
// Included by learner_kernels.cu, whose histogram, scan and partition bodies
// the round kernels share.
#pragma once

// Overhead of a histogram segment (its cells cleared and flushed) in rows,
// for the split of a round's work over the CTAs.
constexpr int kHistSegmentRows = 512;

// ---- partition: every expanded node's rows, in one launch --------------------------

struct RoundPartShared {
  alignas(16) RItem item[kMaxRoundItems];
  alignas(16) uint8_t lut[kMaxBins];
  int32_t warp_tot[32];
  int32_t tile, prefix;
};

// The children of expansion e (one thread): their rows, sums, smaller /
// larger choice (learner/mod.rs:1200-1208), histogram buffers
// (HistogramPool::Move: the larger child takes the parent's, the smaller one
// the item's fresh one) and before_find_best_split (learner/mod.rs:712-731). A child
// without rows cannot be searched; the tree fails only if the replay splits
// the parent (k_round_emit).
__device__ void round_children(const DCtx& c, const DSlot& s, int32_t e, const RItem& it, int32_t nl, bool last_split) {
  const DRounds& r = s.r;
  const DParams& p = c.p;
  const RNode up = r.node[it.node];
  const DSplit& info = r.best[it.node];
  const int32_t nr = it.count - nl;
  RNode a = up, b = up;
  a.parent = b.parent = it.node;
  a.count = nl;
  b.begin = up.begin + nl;
  b.count = nr;
  a.side = b.side = 1 - up.side;
  a.depth = b.depth = up.depth + 1;
  b.desc = 1 - up.desc;
  const bool left_smaller = nl < nr;
  a.buf = left_smaller ? it.buf : up.buf;
  b.buf = left_smaller ? up.buf : it.buf;
  bool need = (left_smaller ? nl : nr) > 0;
  if (p.max_depth > 0 && up.depth + 1 >= p.max_depth) need = false;
  else if (nr < p.min_data_in_leaf * 2 && nl < p.min_data_in_leaf * 2) need = false;
  else if (last_split) need = false;  // the tree's: its children are not searched
  a.need = b.need = need ? 1 : 0;
  a.ls = DLeafSplits{0, nl, info.left_sum_gradient, info.left_sum_hessian, info.left_sum_gh, info.left_output};
  b.ls = DLeafSplits{0, nr, info.right_sum_gradient, info.right_sum_hessian, info.right_sum_gh, info.right_output};
  // basic monotone constraints (constraints.rs:467-480)
  if (p.use_monotone && c.feats[it.inner].bin_type == 0) {
    const double mid = (info.left_output + info.right_output) / 2.0;
    if (info.monotone_type < 0) {
      a.cmin = mid < a.cmin ? a.cmin : mid;
      b.cmax = b.cmax < mid ? b.cmax : mid;
    } else if (info.monotone_type > 0) {
      a.cmax = a.cmax < mid ? a.cmax : mid;
      b.cmin = mid < b.cmin ? b.cmin : mid;
    }
  }
  const int32_t L = 2 * e + 1, R = 2 * e + 2;
  r.node[L] = a;
  r.node[R] = b;
  r.gain[L] = r.gain[R] = -INFINITY;
  r.feat[L] = r.feat[R] = -1;
  r.exp[L] = r.exp[R] = -1;
}

// Grid (G, 1, slots), kPartThreads threads. The row tiles of the round's
// items are claimed in order over all items; a tile chains only to its own
// item's earlier tiles, which running CTAs hold, so any G makes progress.
__global__ void __launch_bounds__(kPartThreads) k_round_part(const __grid_constant__ DCtx c) {
  __shared__ RoundPartShared ps;
  constexpr int kItems = kPartTileRows / kPartThreads;
  const DSlot& s = c.slots[blockIdx.z];
  RoundState* rs = s.r.st;
  const int tid = threadIdx.x;
  const int32_t nb = rs->nb, e0 = rs->e0, ntiles = rs->ntiles;
  const uint32_t epoch = rs->epoch;
  const bool last_split = rs->popped + 2 >= c.p.num_leaves;
  if (nb == 0) return;
  int32_t next = -1;
  if (tid == 0) next = atomicAdd(&rs->ticket, 1);
  for (int i = tid; i < nb * (int)(sizeof(RItem) / 16); i += kPartThreads)
    reinterpret_cast<uint4*>(ps.item)[i] = reinterpret_cast<const uint4*>(s.r.item)[i];
  __syncthreads();
  {  // the smaller children's histogram buffers
    const uint32_t cells = (uint32_t)c.total_bins * (c.hist_mode == LGBM_B200_HIST_QUANT ? 1 : 2);
    for (uint32_t i = blockIdx.x * kPartThreads + tid; i < cells; i += gridDim.x * kPartThreads)
      for (int k = 0; k < nb; ++k) reinterpret_cast<double*>(s.hist)[(size_t)ps.item[k].buf * cells + i] = 0.0;
  }
  int32_t cur = -1;
  while (true) {
    __syncthreads();
    if (tid == 0) ps.tile = next;
    __syncthreads();
    const int32_t gtile = ps.tile;
    if (gtile >= ntiles) break;
    if (tid == 0) next = atomicAdd(&rs->ticket, 1);
    int lo = 0, hi = nb - 1;  // the item of this tile
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (ps.item[mid].tile0 <= gtile) lo = mid;
      else hi = mid - 1;
    }
    const RItem it = ps.item[lo];
    const int32_t tile = gtile - it.tile0, cnt = it.count, t0 = tile * kPartTileRows;
    const uint32_t* in = s.idx[it.side] + it.begin;
    uint32_t* out = s.idx[1 - it.side] + it.begin;
    const uint8_t* col = c.colbins + (size_t)it.inner * (size_t)c.num_data;
    uint32_t rows[kItems], raws[kItems];
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
      const int32_t pos = t0 + tid * kItems + k;
      rows[k] = pos < cnt ? __ldcg(in + pos) : 0u;
    }
    if (lo != cur) {
      build_partition_lut(c.feats[it.inner], s.r.best[it.node], ps.lut, tid, kPartThreads);
      cur = lo;
    }
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
      const int32_t pos = t0 + tid * kItems + k;
      raws[k] = pos < cnt ? (uint32_t)col[rows[k]] : 0u;
    }
    __syncthreads();  // the table
    uint32_t flags = 0;
    int32_t nleft = 0;
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
      const int32_t pos = t0 + tid * kItems + k;
      if (pos < cnt && ps.lut[raws[k]]) {
        flags |= 1u << k;
        ++nleft;
      }
    }
    const int32_t lefts = tile_scatter<kItems>(s.st, ps, s.r.status + it.tile0, tile, epoch, t0, cnt, rows, flags,
                                               nleft, out);
    if (tid == 0 && t0 + kPartTileRows >= cnt) {
      atomicAdd(reinterpret_cast<unsigned long long*>(&s.st->part_rows), (unsigned long long)cnt);
      round_children(c, s, e0 + lo, it, lefts, last_split);
    }
  }
}

// ---- histogram: every smaller child, in one launch ---------------------------------

// Sum over the CTA's kThreads threads before this one, and the total.
template <int kThreads, class T>
__device__ __forceinline__ T block_prefix(T v, T* warp_sums, T& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  T incl = v;
  for (int o = 1; o < 32; o <<= 1) {
    const T u = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += u;
  }
  if (lane == 31) warp_sums[warp] = incl;
  __syncthreads();
  T base = 0;
  total = 0;
  for (int w = 0; w < kThreads / 32; ++w) {
    const T u = warp_sums[w];
    if (w < warp) base += u;
    total += u;
  }
  __syncthreads();
  return base + incl - v;
}

// Grid (G, feature tiles, slots), kHistThreads threads. The rows of the
// round's smaller children form one sequence, in which each child first
// counts kHistSegmentRows for its cells' clearing and flush; the CTAs take
// equal shares of it, so a round of one large leaf and one of many small ones
// both spread evenly. A share that spans several children is accumulated and
// flushed child by child.
template <int kMode, int kNG>
__global__ void __launch_bounds__(kHistThreads, 2)
    k_round_hist(const __grid_constant__ DCtx c, DTileTable tt, int32_t sub_rows) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ long long start[kMaxRoundItems + 1];
  __shared__ int32_t begin[kMaxRoundItems], buf[kMaxRoundItems];
  __shared__ long long warp_sums[kHistThreads / 32];
  static_assert(kMaxRoundItems <= kHistThreads, "one item per thread");
  const DSlot& s = c.slots[blockIdx.z];
  const DRounds& r = s.r;
  const int tid = threadIdx.x;
  const bool root = r.st->root != 0;
  const int32_t nb = root ? 1 : r.st->nb, e0 = r.st->e0;
  const DFixed fx = s.st->fx;
  long long w = 0;
  if (tid < nb) {
    int32_t id = 0;
    if (!root) {
      const int32_t l = 2 * (e0 + tid) + 1;
      id = r.node[l].count < r.node[l + 1].count ? l : l + 1;
    }
    const RNode& nd = r.node[id];
    begin[tid] = nd.begin;
    buf[tid] = nd.buf | (nd.side << 30);
    w = nd.need && nd.count > 0 ? (long long)nd.count + kHistSegmentRows : 0;
  }
  long long total;
  const long long before = block_prefix<kHistThreads>(w, warp_sums, total);
  if (tid < nb) start[tid] = before;
  if (tid == 0) start[nb] = total;
  const int live = __syncthreads_count(w > 0);
  if (total == 0) return;
  const long long active = min((long long)gridDim.x, (total + c.rows_per_block - 1) / c.rows_per_block);
  if ((long long)blockIdx.x >= active) return;
  if (blockIdx.x == 0 && blockIdx.y == 0 && tid == 0)
    s.st->hist_rows += total - (long long)live * kHistSegmentRows;
  const long long lo = total * blockIdx.x / active, hi = total * (blockIdx.x + 1) / active;
  int i = 0, last = nb - 1;  // the last child that starts at or before lo
  while (i < last) {
    const int mid = (i + last + 1) >> 1;
    if (start[mid] <= lo) i = mid;
    else last = mid - 1;
  }
  for (; i < nb && start[i] < hi; ++i) {
    const long long s0 = start[i] + kHistSegmentRows;
    const long long r0 = max(0LL, max(lo, start[i]) - s0), r1 = min(hi, start[i + 1]) - s0;
    if (r1 <= r0) continue;
    LeafRows lr;
    lr.begin = begin[i];
    lr.count = start[i + 1] - s0;
    lr.buf = buf[i] & 0x3FFFFFFF;
    lr.idx = s.idx[buf[i] >> 30 & 1];
    if constexpr (kMode != 2) {
      if (fx.ok) {
        hist_body_fixed(c, s, fx, tt, blockIdx.y, lr, r0, r1, smem_raw);
        continue;
      }
    }
    hist_body<kMode, kNG, 1>(c, s, tt, blockIdx.y, lr, r0, r1, sub_rows, smem_raw);
  }
}

size_t round_hist_smem(int mode, int ng) {
  const size_t b = hist_smem_bytes(mode, ng);
  return mode == 2 ? b : std::max(b, kFixedSmem);
}

#define LGBM_B200_ROUND_HIST_INST(M, G) \
  template __global__ void k_round_hist<M, G>(const __grid_constant__ DCtx, DTileTable, int32_t);
LGBM_B200_ROUND_HIST_INST(0, 1)
LGBM_B200_ROUND_HIST_INST(1, 1)
LGBM_B200_ROUND_HIST_INST(2, 1)
LGBM_B200_ROUND_HIST_INST(2, 2)
LGBM_B200_ROUND_HIST_INST(2, 3)
LGBM_B200_ROUND_HIST_INST(2, 4)
#undef LGBM_B200_ROUND_HIST_INST

const void* round_hist_kernel(int mode, int ng) {
  if (mode == 0) return reinterpret_cast<const void*>(&k_round_hist<0, 1>);
  if (mode == 1) return reinterpret_cast<const void*>(&k_round_hist<1, 1>);
  switch (ng) {
    case 1: return reinterpret_cast<const void*>(&k_round_hist<2, 1>);
    case 2: return reinterpret_cast<const void*>(&k_round_hist<2, 2>);
    case 3: return reinterpret_cast<const void*>(&k_round_hist<2, 3>);
    default: return reinterpret_cast<const void*>(&k_round_hist<2, 4>);
  }
}

cudaError_t launch_round_hist(int mode, int ng, dim3 grid, size_t smem, cudaStream_t st, const DCtx& c,
                              const DTileTable& tt, int32_t sub_rows) {
  void* args[] = {const_cast<DCtx*>(&c), const_cast<DTileTable*>(&tt), &sub_rows};
  return cudaLaunchKernel(round_hist_kernel(mode, ng), grid, dim3(kHistThreads), args, smem, st);
}

#include "round_scan.cuh"

// ---- the decision between rounds ----------------------------------------------------

// Leaves (of trees of more than 256, groups of leaves) the replay keeps in a lane's registers.
constexpr int kReplaySlots = 8;

// The explored nodes as the replay and the ranking read them, in shared
// memory when they fit.
struct NodeFacts {
  const double* gain;
  const int32_t* feat;
  int32_t* exp;
  const int32_t* exp_node;
};
size_t round_decide_smem(int num_leaves) {
  // the replayed tree's leaves, then the nodes' facts
  const size_t leaves = ((size_t)num_leaves * sizeof(int32_t) + 15) / 16 * 16;
  return leaves + (size_t)kDecideSmemNodes * (sizeof(double) + 2 * sizeof(int32_t)) + kDecideSmemNodes / 2 * sizeof(int32_t);
}

// A double as an unsigned integer of the same order (no NaN reaches it).
__device__ __forceinline__ unsigned long long order_key(double v) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v);
  return (b >> 63) ? ~b : b | (1ull << 63);
}

// The reference's order of splits (learner/mod.rs:653-706) replayed by one
// warp over the gains found so far, from `popped` splits on: the leaf of
// largest gain (then smallest feature, then smallest leaf) is split as long
// as it has been expanded. ln: the node of each leaf of the replayed tree. Returns the node the replay waits for, or -1 when the
// tree is finished. Lane l owns leaves l, l + 32, ...; up to 256 leaves their
// gains stay in registers, of larger trees the best of each of 8 groups.
template <bool kRegs>
__device__ int32_t replay(const DRounds& r, const NodeFacts& nd, int32_t* ln, int32_t need, int32_t& popped) {
  const int lane = threadIdx.x & 31;
  // kRegs: the order keys of this lane's leaves; else, of each group of `per`
  // of them, the largest and its leaf (with all of a lane's leaves looked
  // through at every split an iteration of 200k rows x 28 took 242 ms at 8000
  // leaves and 45 at 4095; 59 and 18)
  unsigned long long own[kReplaySlots];
  int32_t own_leaf[kReplaySlots];
  unsigned long long best = 0;  // the largest, 0: none
  int32_t bl = INT32_MAX;       // and its leaf
  const int32_t per = (need / 32 + kReplaySlots) / kReplaySlots;
  auto better = [&](unsigned long long k, int32_t l, unsigned long long than, int32_t of) {
    return k > than || (k == than && of != INT32_MAX && l != INT32_MAX && better_than(0.0, nd.feat[ln[l]], 0.0, nd.feat[ln[of]]));
  };
  auto group_best = [&](int32_t g, int32_t leaves, unsigned long long& key, int32_t& leaf) {
    key = 0;
    leaf = INT32_MAX;
    for (int32_t l = lane + 32 * per * g; l < min(leaves, 32 * per * (g + 1)); l += 32) {
      const unsigned long long k = order_key(nd.gain[ln[l]]);
      if (better(k, l, key, leaf)) {
        key = k;
        leaf = l;
      }
    }
  };
  auto own_best = [&](int32_t leaves) {
    best = 0;
    bl = INT32_MAX;
#pragma unroll
    for (int k = 0; k < kReplaySlots; ++k) {
      const int32_t l = kRegs ? lane + 32 * k : own_leaf[k];
      if ((!kRegs || l < leaves) && better(own[k], l, best, bl)) {
        best = own[k];
        bl = l;
      }
    }
  };
#pragma unroll
  for (int k = 0; k < kReplaySlots; ++k) {
    if constexpr (kRegs) own[k] = lane + 32 * k <= popped ? order_key(nd.gain[ln[lane + 32 * k]]) : 0ull;
    else group_best(k, popped + 1, own[k], own_leaf[k]);
  }
  own_best(popped + 1);
  const unsigned long long zero = order_key(0.0);
  while (true) {
    if (popped >= need) return -1;
    const uint32_t hi = __reduce_max_sync(0xffffffffu, (uint32_t)(best >> 32));
    bool in = (uint32_t)(best >> 32) == hi;
    unsigned who = __ballot_sync(0xffffffffu, in);
    if (who & (who - 1)) {
      const uint32_t lo = __reduce_max_sync(0xffffffffu, in ? (uint32_t)best : 0u);
      in = in && (uint32_t)best == lo;
      who = __ballot_sync(0xffffffffu, in);
      if (who & (who - 1)) {  // equal gains: the smallest feature, then the smallest leaf
        const int32_t feat = in && bl != INT32_MAX ? nd.feat[ln[bl]] : -1;
        const uint32_t fe = !in ? 0xffffffffu : feat == -1 ? (uint32_t)INT32_MAX : (uint32_t)feat;
        const uint32_t mf = __reduce_min_sync(0xffffffffu, fe);
        in = in && fe == mf;
        const uint32_t ml = __reduce_min_sync(0xffffffffu, in ? (uint32_t)bl : 0xffffffffu);
        who = __ballot_sync(0xffffffffu, in && (uint32_t)bl == ml);
      }
    }
    const int src = __ffs(who) - 1;
    const int32_t l = __shfl_sync(0xffffffffu, bl, src);
    const bool positive = __shfl_sync(0xffffffffu, (int)(best > zero), src);
    if (l == INT32_MAX || !positive) return -1;
    const int32_t v = ln[l], e = nd.exp[v];
    if (e < 0) return v;
    const int32_t R = popped + 1, a = 2 * e + 1, b = 2 * e + 2;
    const unsigned long long ka = order_key(nd.gain[a]), kb = order_key(nd.gain[b]);
    __syncwarp();
    if (lane == 0) {
      nd.exp[v] = e | kReplayed;
      r.exp[v] = e | kReplayed;
      r.pop_node[popped] = v;
      ln[l] = a;
      ln[R] = b;
    }
    __syncwarp();
    ++popped;
    if constexpr (kRegs) {
#pragma unroll
      for (int k = 0; k < kReplaySlots; ++k) {
        if (l == lane + 32 * k) own[k] = ka;
        if (R == lane + 32 * k) own[k] = kb;
      }
    } else {
#pragma unroll 1
      for (int side = 0; side < 2; ++side) {  // the groups of the two leaves
        const int32_t x = side ? R : l;
        if (lane != (x & 31)) continue;
        const int32_t g = (x >> 5) / per;
        unsigned long long key;
        int32_t leaf;
        group_best(g, popped + 1, key, leaf);
#pragma unroll
        for (int k = 0; k < kReplaySlots; ++k)
          if (k == g) {
            own[k] = key;
            own_leaf[k] = leaf;
          }
      }
    }
    if (lane == (l & 31) || lane == (R & 31)) own_best(popped + 1);
  }
}

// Grid (1, 1, slots), kDecideThreads threads: the replay as far as it goes,
// then the nodes the next round expands, or that the tree is finished.
//
// A node's key is the smallest gain on its path from the replayed tree's leaf
// above it (in FP32: rounding keeps the order). Of two nodes the replay has
// not reached, it splits the one of larger key first: when it splits the
// node that holds the smaller one's minimum, the larger one's path offers a
// leaf of larger gain until that one is split. Nodes are ranked by their keys'
// place in kRoundBins steps between the best and the worst candidate's.
//   - A candidate ranked past as many known nodes as there are splits to come
//     can never be split. It is dropped and its histogram buffer is free again.
//   - Expanded next are the node the replay waits for and the best-ranked
//     candidates, at most a share of the splits still to come (DRounds): fewer
//     take more rounds, more expand what is not needed (at a quarter 1.6 times
//     the splits on early trees, 2 to 3 times on late ones, whose gains hardly
//     fall with depth). Nodes of many rows are expanded
//     ahead of need only up to kRoundRows rows a round, whose partition and
//     histogram take as long as a few rounds.
//   - A split needs one buffer and one expansion, and as many as there are
//     splits to come are always left.
__global__ void __launch_bounds__(kDecideThreads) k_round_decide(const __grid_constant__ DCtx c, int32_t* ctrl,
                                                                 cudaGraphConditionalHandle cond, int32_t use_cond) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  static_assert(kRoundBins == 2 * kDecideThreads, "two bins per thread");
  __shared__ int32_t exps[kRoundBins], cands[kRoundBins];
  __shared__ unsigned long long rows[kRoundBins];
  __shared__ unsigned long long warp_sums[kDecideThreads / 32];
  __shared__ int32_t fresh[kMaxRoundItems];
  __shared__ uint32_t s_lo;
  __shared__ int32_t s_popped, s_top, s_tau, s_cut, s_room, s_rowcut, s_tiles;
  const DSlot& s = c.slots[blockIdx.z];
  const DRounds& r = s.r;
  RoundState* rs = r.st;
  const int tid = threadIdx.x;
  const int32_t L = c.p.num_leaves, need = L - 1;
  const RoundState st = *rs;
  const int32_t status = s.st->status;
  int32_t active = 0;
  if (!st.done) {
    const int32_t E = st.e0 + st.nb, N = 2 * E + 1;
    const int32_t new0 = st.root ? 0 : 2 * st.e0 + 1, nnew = N - new0;
    const int32_t total = st.ncand + nnew;  // the candidates: those kept, then the new nodes
    int32_t* ln = reinterpret_cast<int32_t*>(smem_raw);
    NodeFacts nd{r.gain, r.feat, r.exp, r.exp_node};
    if (N <= kDecideSmemNodes) {
      double* a = reinterpret_cast<double*>(smem_raw + ((size_t)L * sizeof(int32_t) + 15) / 16 * 16);
      int32_t* b = reinterpret_cast<int32_t*>(a + N);
      int32_t* d = b + N;
      int32_t* e = d + N;
      for (int32_t v = tid; v < N; v += kDecideThreads) {
        a[v] = r.gain[v];
        b[v] = r.feat[v];
        d[v] = r.exp[v];
      }
      for (int32_t i = tid; i < E; i += kDecideThreads) e[i] = r.exp_node[i];
      nd = NodeFacts{a, b, d, e};
    }
    for (int32_t l = tid; l <= st.popped; l += kDecideThreads) ln[l] = r.leaf_node[l];
    // this thread's first kOwn candidates and their rows stay in registers
    // (more only in trees of a thousand leaves); loaded while the replay runs
    constexpr int kOwn = 2;
    auto listed = [&](int32_t i) { return i < st.ncand ? r.cand[i] : new0 + i - st.ncand; };
    int32_t own_v[kOwn], own_n[kOwn], own_begin[kOwn], own_side[kOwn], own_buf[kOwn], own_inner[kOwn];
#pragma unroll
    for (int j = 0; j < kOwn; ++j) {
      const int32_t i = tid + j * kDecideThreads;
      own_v[j] = i < total ? listed(i) : -1;
    }
#pragma unroll
    for (int j = 0; j < kOwn; ++j) {
      const RNode& nv = r.node[max(own_v[j], 0)];
      own_n[j] = own_v[j] >= 0 ? nv.count : 0;
      own_begin[j] = nv.begin;
      own_side[j] = nv.side;
      own_buf[j] = nv.buf;
      own_inner[j] = r.best[max(own_v[j], 0)].inner;
    }
    // the buffers the round may take, from the end of the list
    for (int i = tid; i < min(r.bmax, st.nfree); i += kDecideThreads) fresh[i] = r.free[st.nfree - 1 - i];
    for (int b = tid; b < kRoundBins; b += kDecideThreads) {
      exps[b] = 0;
      cands[b] = 0;
      rows[b] = 0;
    }
    if (tid == 0) {
      s_lo = 0xffffffffu;
      s_tau = kRoundBins - 1;
      s_cut = kRoundBins - 1;
      s_room = r.bmax;
      s_rowcut = kRoundBins;
    }
    __syncthreads();
    if (tid < 32) {
      int32_t popped = st.popped;
      const int32_t top = L <= 32 * kReplaySlots ? replay<true>(r, nd, ln, need, popped)
                                                 : replay<false>(r, nd, ln, need, popped);
      if (tid == 0) {
        s_popped = popped;
        s_top = top;
      }
    }
    __syncthreads();
    const int32_t popped = s_popped, top = s_top;
    for (int32_t l = tid; l <= popped; l += kDecideThreads) r.leaf_node[l] = ln[l];
    // a partition whose look-back gave up ends the tree here: its row lists are
    // incomplete, and the rounds to come would each wait as long again
    bool done = top < 0 || status != kStatusOk;
    if (!done && st.rounds > need) {  // every round replays a split: never more rounds than splits
      if (tid == 0) s.st->status = kStatusTimeout;
      done = true;
    }
    if (!done) {
      const int32_t open = need - popped, spare = min(st.nfree, r.ecap - E);
      // only the node the replay waits for when one split is left to come
      const int32_t most = open == 1 ? 1 : max(1, min(min(r.bmax, spare - open + 1), max(r.least, (open + r.share - 1) / r.share)));
      // 0: the node cannot be split; positive for every positive gain
      auto key_of = [&](int32_t v) {
        float k = nd.gain[v] > 0.0 ? fmaxf((float)nd.gain[v], 1.4e-45f) : 0.0f;
        while (v > 0) {
          v = nd.exp_node[(v - 1) >> 1];
          if (nd.exp[v] & kReplayed) break;
          k = fminf(k, fmaxf((float)nd.gain[v], 1.4e-45f));
        }
        return __float_as_uint(k);
      };
      auto tiles_of = [](int32_t n) { return (n + kPartTileRows - 1) / kPartTileRows; };
      const uint32_t hi = key_of(top);  // no key is larger
      uint32_t own_k[kOwn];
      // visits this thread's candidates: fn(candidate), for every multiple of
      // kDecideThreads below `total` (node -1 past it)
      struct Cand {
        int32_t v, n, begin, side, buf, inner;
        uint32_t key;
      };
      auto each_cand = [&](auto fn) {
#pragma unroll
        for (int j = 0; j < kOwn; ++j)
          if (j * kDecideThreads < total)
            fn(Cand{own_v[j], own_n[j], own_begin[j], own_side[j], own_buf[j], own_inner[j], own_k[j]});
        for (int32_t i0 = kOwn * kDecideThreads; i0 < total; i0 += kDecideThreads) {
          const int32_t i = i0 + tid, v = i < total ? listed(i) : -1;
          const RNode& nv = r.node[max(v, 0)];
          fn(Cand{v, nv.count, nv.begin, nv.side, nv.buf, r.best[max(v, 0)].inner, v >= 0 ? key_of(v) : 0u});
        }
      };
      {
        uint32_t lo = 0xffffffffu;
#pragma unroll
        for (int j = 0; j < kOwn; ++j) own_k[j] = own_v[j] >= 0 ? key_of(own_v[j]) : 0u;
        each_cand([&](const Cand& x) {
          if (x.key > 0) lo = min(lo, x.key);
        });
        lo = __reduce_min_sync(0xffffffffu, lo);
        if ((tid & 31) == 0) atomicMin(&s_lo, lo);
      }
      __syncthreads();
      const int shift = max(0, 32 - __clz(hi - min(hi, s_lo)) - 10);
      static_assert(kRoundBins == 1 << 10, "the range of keys shifted to ten bits");
      auto bin_of = [&](uint32_t k) { return k ? min((int32_t)((hi - k) >> shift), kRoundBins - 1) : kRoundBins; };
      each_cand([&](const Cand& x) {
        const int32_t b = bin_of(x.key);
        if (b < kRoundBins) {
          if (x.n <= kRoundRows / 2 && x.v != top) atomicAdd(&rows[b], (unsigned long long)x.n);
          atomicAdd(&cands[b], 1);
        }
        if (x.v == top) s_tiles = tiles_of(x.n);
      });
      for (int32_t e = tid; e < E; e += kDecideThreads) {
        const int32_t v = nd.exp_node[e];
        if (!(nd.exp[v] & kReplayed)) atomicAdd(&exps[bin_of(key_of(v))], 1);
      }
      __syncthreads();
      {
        unsigned long long tot;
        const int32_t c0 = cands[2 * tid], c1 = cands[2 * tid + 1];
        const int32_t k0 = exps[2 * tid] + c0, k1 = exps[2 * tid + 1] + c1;
        const unsigned long long before = block_prefix<kDecideThreads>(
            ((unsigned long long)(uint32_t)(k0 + k1) << 32) | (uint32_t)(c0 + c1), warp_sums, tot);
        unsigned long long rb = block_prefix<kDecideThreads>(rows[2 * tid] + rows[2 * tid + 1], warp_sums, tot);
        int32_t kb = (int32_t)(before >> 32), cb = (int32_t)(uint32_t)before;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int b = 2 * tid + j, k = j ? k1 : k0, n = j ? c1 : c0;
          if (kb < open && kb + k >= open) s_tau = b;  // the last bin that can still be among the splits
          if (cb < most && cb + n >= most) {           // the last bin with room this round
            s_cut = b;
            s_room = most - cb - (b == 0 ? 1 : 0);  // the node the replay waits for is in bin 0
          }
          // the first bin that would take the round past kRoundRows rows ahead of need
          if (rb <= kRoundRows && rb + rows[b] > kRoundRows) s_rowcut = b;
          kb += k;
          cb += n;
          rb += rows[b];
        }
      }
      __syncthreads();
      const int32_t tau = s_tau, cut = s_cut, share = s_room, rowcut = s_rowcut;
      // one pass over the candidates in list order: the ones expanded (the
      // node the replay waits for is always the first), the ones kept, and the
      // buffers of the ones dropped
      int32_t took = 1, kept = 0, freed = 0, tiles = 0, at_cut0 = 0;
      auto place = [&](int32_t at, const Cand& x, int32_t tile0) {
        r.item[at] = RItem{x.v, x.begin, x.n, x.side, x.inner, tile0, fresh[at], 0};
        r.exp_node[E + at] = x.v;
        r.exp[x.v] = E + at;
        r.scan_cnt[2 * at] = 0;
        r.scan_cnt[2 * at + 1] = 0;
      };
      tiles = s_tiles;
      each_cand([&](const Cand& x) {
        bool pick = false, keep = false, drop = false, edge = false;
        if (x.v == top) place(0, x, 0);
        if (x.v >= 0 && x.v != top) {
          const int32_t b = bin_of(x.key);
          drop = b > tau;
          const bool fits = !drop && x.n <= kRoundRows / 2 && b < rowcut;
          pick = fits && b < cut;
          edge = fits && b == cut;
          keep = !drop;
        }
        unsigned long long tot;
        const int32_t edge0 = (int32_t)block_prefix<kDecideThreads>((unsigned long long)edge, warp_sums, tot);
        // the cut leaves room for `most` in all, the node the replay waits for among them
        pick = pick || (edge && at_cut0 + edge0 < share);
        at_cut0 += (int32_t)tot;
        keep = keep && !pick;
        // one sum of four counts: tiles (32 bits), picked, kept and dropped (10 bits each)
        const int32_t nt = tiles_of(x.n);
        const unsigned long long before = block_prefix<kDecideThreads>(
            (pick ? (1ull << 32) | (uint32_t)nt : 0ull) | (unsigned long long)keep << 42 | (unsigned long long)drop << 52,
            warp_sums, tot);
        static_assert(kDecideThreads < 1024, "ten bits a count");
        const int32_t at = took + (int32_t)(before >> 32 & 1023);
        if (pick && at < r.bmax && E + at < r.ecap) place(at, x, tiles + (int32_t)(uint32_t)before);
        // the list is compacted in place: an entry moves to a place at or
        // before its own, which this pass or an earlier one has read
        if (keep) r.cand[kept + (int32_t)(before >> 42 & 1023)] = x.v;
        if (drop) r.free_next[freed + (int32_t)(before >> 52)] = x.buf;
        took += (int32_t)(tot >> 32 & 1023);
        tiles += (int32_t)(uint32_t)tot;
        kept += (int32_t)(tot >> 42 & 1023);
        freed += (int32_t)(tot >> 52);
      });
      __syncthreads();
      // the round's buffers leave the list, the dropped candidates' join it
      for (int32_t i = tid; i < freed; i += kDecideThreads) r.free[st.nfree - took + i] = r.free_next[i];
      if (tid == 0) {
        rs->e0 = E;
        rs->nb = took;
        rs->ntiles = tiles;
        rs->ticket = 0;
        rs->epoch = st.epoch + 1;
        rs->rounds = st.rounds + 1;
        rs->ncand = kept;
        rs->nfree = st.nfree - took + freed;
      }
      active = 1;
    } else if (tid == 0) {
      rs->e0 = E;
      rs->nb = 0;
      rs->done = 1;
    }
    if (tid == 0) {
      rs->popped = popped;
      rs->root = 0;
    }
  }
  // whether any slot goes on: by the last slot's CTA
  if (tid == 0 && gridDim.z == 1) {
    ctrl[2] = active;
    if (use_cond) cudaGraphSetConditional(cond, (unsigned)active);
  } else if (tid == 0) {
    if (active) atomicAdd(&ctrl[1], 1);
    __threadfence();
    if (atomicAdd(&ctrl[0], 1) == (int)gridDim.z - 1) {
      __threadfence();
      const int32_t any = atomicExch(&ctrl[1], 0) > 0;
      ctrl[0] = 0;
      ctrl[2] = any;
      if (use_cond) cudaGraphSetConditional(cond, (unsigned)any);
    }
  }
}

// ---- the finished tree -----------------------------------------------------------------

// Grid (1, 1, slots), kDecideThreads threads: the replayed splits as the
// reference's tree arrays (Tree::split, tree.rs:254-297) and leaf ranges. A
// leaf that was expanded past its children has lost its own row list to its
// grandchildren's; its rows then lie in the ranges of the unexpanded nodes
// under it, which are listed leaf by leaf for k_round_restore and
// k_round_order.
__global__ void __launch_bounds__(kDecideThreads) k_round_emit(const __grid_constant__ DCtx c) {
  __shared__ unsigned long long warp_sums[kDecideThreads / 32];
  __shared__ int32_t s_bad, s_pieces;
  const DSlot& s = c.slots[blockIdx.z];
  const DRounds& r = s.r;
  RoundState* rs = r.st;
  DSlotState* st = s.st;
  const DTree& t = s.tree;
  const int tid = threadIdx.x;
  const int32_t P = rs->popped, N = 2 * (rs->e0 + rs->nb) + 1;
  for (int32_t v = tid; v < N; v += kDecideThreads) {
    r.pop_time[v] = -1;
    r.node_leaf[v] = -1;
  }
  for (int32_t l = tid; l <= P; l += kDecideThreads) r.piece_head[l] = -1;
  if (tid == 0) s_bad = s_pieces = 0;
  __syncthreads();
  for (int32_t i = tid; i < P; i += kDecideThreads) r.pop_time[r.pop_node[i]] = i;
  for (int32_t l = tid; l <= P; l += kDecideThreads) r.node_leaf[r.leaf_node[l]] = l;
  __syncthreads();
  // output of a node as its parent's split stored it
  auto output_of = [&](int32_t v) {
    if (v == 0) return rs->root_value;
    const DSplit& up = r.best[r.node[v].parent];
    const double o = (v & 1) ? up.left_output : up.right_output;
    return isnan(o) ? 0.0 : o;
  };
  auto child_of = [&](int32_t v) { return r.pop_time[v] >= 0 ? r.pop_time[v] : ~r.node_leaf[v]; };
  int32_t cats = 0;
  for (int32_t i0 = 0; i0 < P; i0 += kDecideThreads) {
    const int32_t i = i0 + tid;
    bool cat = false;
    int32_t x = 0;
    if (i < P) {
      x = r.pop_node[i];
      cat = c.feats[r.best[x].inner].bin_type != 0;
    }
    unsigned long long tot;
    const unsigned long long before = block_prefix<kDecideThreads>((unsigned long long)cat, warp_sums, tot);
    if (i < P) {
      const DSplit& info = r.best[x];
      const DFeature& m = c.feats[info.inner];
      const int32_t e = r.exp[x] & ~kReplayed, a = 2 * e + 1, b = 2 * e + 2;
      const bool numerical = m.bin_type == 0;
      t.split_feature_inner[i] = info.inner;
      t.split_feature[i] = info.feature;
      t.split_gain[i] = (float)(info.gain + c.p.min_gain_to_split);
      t.node_gain[i] = info.gain;
      t.left_child[i] = child_of(a);
      t.right_child[i] = child_of(b);
      t.internal_weight[i] = info.left_sum_hessian + info.right_sum_hessian;
      t.internal_value[i] = output_of(x);
      t.internal_count[i] = r.node[a].count + r.node[b].count;
      int8_t dt = 0;
      if (numerical && info.default_left != 0) dt |= 2;
      dt = (int8_t)((dt & 3) | (m.missing_type << 2));
      if (!numerical) dt |= 1;
      t.decision_type[i] = dt;
      t.threshold_in_bin[i] = numerical ? info.threshold : (uint32_t)(cats + (int32_t)before);
      for (int w = 0; w < kCatWords; ++w) t.cat_bits[i * kCatWords + w] = numerical ? 0u : info.cat_bits[w];
      if (min(r.node[a].count, r.node[b].count) <= 0) s_bad = 1;
    }
    cats += (int32_t)tot;
  }
  for (int32_t l = tid; l <= P; l += kDecideThreads) {
    const int32_t v = r.leaf_node[l];
    const RNode& nd = r.node[v];
    s.leaf_begin[l] = nd.begin;
    s.leaf_count[l] = nd.count;
    s.leaf_gcount[l] = nd.count;
    // past its children, a leaf's rows are gathered in its children's buffer
    const int32_t e = r.exp[v];
    const bool lost = e >= 0 && (r.exp[2 * e + 1] >= 0 || r.exp[2 * e + 2] >= 0);
    s.leaf_side[l] = lost ? 1 - nd.side : nd.side;
    if (P > 0) {
      const DSplit& up = r.best[nd.parent];
      t.leaf_parent[l] = r.pop_time[nd.parent];
      t.leaf_value[l] = output_of(v);
      t.leaf_weight[l] = (v & 1) ? up.left_sum_hessian : up.right_sum_hessian;
      t.leaf_count[l] = nd.count;
      t.leaf_depth[l] = nd.depth;
    }
  }
  // unexpanded nodes under a leaf that lost its list
  for (int32_t v = tid; v < N; v += kDecideThreads) {
    if (r.exp[v] >= 0 || r.node_leaf[v] >= 0) continue;
    int32_t up = r.node[v].parent;
    while (r.node_leaf[up] < 0) up = r.node[up].parent;
    const int32_t e = r.exp[up];
    const bool lost = r.exp[2 * e + 1] >= 0 || r.exp[2 * e + 2] >= 0;
    const RNode& nd = r.node[v];
    if (lost && nd.count > 0) {
      const int32_t l = r.node_leaf[up], at = atomicAdd(&s_pieces, 1);
      r.piece[at] = RPiece{nd.begin, nd.count, nd.side, nd.desc, l, atomicExch(&r.piece_head[l], at), r.node[up].desc, r.node[up].side};
    }
  }
  __syncthreads();
  if (tid == 0) {
    rs->npiece = s_pieces;
    rs->disorder = 0;
    st->num_leaves_cur = P + 1;
    st->num_cat = cats;
    if (s_bad && st->status == kStatusOk) st->status = kStatusEmptyChild;
    st->done = 1;
  }
}

// The listed row pieces that lie in the leaf's own buffer copied into the
// other one, at the same positions (every piece owns its positions in both).
// Grid (G, 1, slots).
__global__ void __launch_bounds__(256) k_round_restore(const __grid_constant__ DCtx c) {
  __shared__ int4 piece[256];  // begin, count, side and index of those that move
  __shared__ int32_t s_moves;
  const DSlot& s = c.slots[blockIdx.z];
  const int32_t n = s.r.st->npiece;
  for (int32_t i0 = 0; i0 < n; i0 += 256) {
    __syncthreads();
    if (threadIdx.x == 0) s_moves = 0;
    __syncthreads();
    if (i0 + (int)threadIdx.x < n) {
      const RPiece p = s.r.piece[i0 + threadIdx.x];
      if (p.side == p.own) piece[atomicAdd(&s_moves, 1)] = make_int4(p.begin, p.count, p.side, i0 + (int)threadIdx.x);
    }
    __syncthreads();
    const int32_t m = s_moves;
    for (int32_t i = 0; i < m; ++i) {
      const int4 p = piece[i];
      const uint32_t* from = s.idx[p.z] + p.x;
      uint32_t* to = s.idx[1 - p.z] + p.x;
      // small pieces start at different CTAs
      const uint32_t b = (blockIdx.x + (uint32_t)p.w * 37u) % gridDim.x;
      for (uint32_t k = b * 256u + threadIdx.x; k < (uint32_t)p.y; k += gridDim.x * 256u) to[k] = from[k];
    }
  }
}

// Whether every listed piece, in the children's buffer (k_round_restore), is
// ascending or descending as its node's list is: a bag in no order leaves
// none. Grid (G, 1, slots).
__global__ void __launch_bounds__(256) k_round_check(const __grid_constant__ DCtx c) {
  const DSlot& s = c.slots[blockIdx.z];
  const DRounds& r = s.r;
  const int32_t n = r.st->npiece;
  bool disorder = false;
  for (int32_t i = 0; i < n; ++i) {
    const RPiece p = r.piece[i];
    const uint32_t* x = s.idx[1 - p.own] + p.begin;
    for (uint32_t k = blockIdx.x * 256u + threadIdx.x; k + 1 < (uint32_t)p.count; k += gridDim.x * 256u)
      disorder |= (x[k + 1] < x[k]) != (p.desc != 0);
  }
  if (disorder) r.st->disorder = 1;
}

// Rows of the list x[0, n) below `row`.
__device__ __forceinline__ int32_t rows_below(const uint32_t* x, int32_t n, bool desc, uint32_t row) {
  int32_t lo = 0, hi = n;  // the first place on the other side of `row`
  while (lo < hi) {
    const int32_t mid = (lo + hi) >> 1;
    if ((x[mid] < row) != desc) lo = mid + 1;
    else hi = mid;
  }
  return desc ? n - lo : lo;
}

// The rows of the leaves that lost their lists in the lists' own order, that
// of growth split by split: a split keeps its left rows' order and reverses
// its right rows', so every list of the tree is ascending or descending and a
// row's place is its rank among the leaf's pieces, found by bisection. The
// pieces lie in the children's buffer (k_round_restore); the leaf's own takes
// the result. For the partition's readback alone; the lists' other readers
// take a leaf's rows in any order. Grid (G, 1, slots); a second run changes
// nothing.
__global__ void __launch_bounds__(256) k_round_order(const __grid_constant__ DCtx c) {
  // a chunk of the pieces and their leaves' lists, loaded side by side: one
  // piece at a time, each cost a chain of four loads (40 us of a 31-leaf tree)
  __shared__ RPiece piece[256];
  __shared__ int32_t begin[256], count[256], head[256];
  const DSlot& s = c.slots[blockIdx.z];
  const DRounds& r = s.r;
  const int32_t n = r.st->npiece;
  if (r.st->disorder) return;
  for (int32_t i0 = 0; i0 < n; i0 += 256) {
    const int32_t m = min(256, n - i0);
    __syncthreads();
    if ((int)threadIdx.x < m) {
      const RPiece p = r.piece[i0 + threadIdx.x];
      piece[threadIdx.x] = p;
      begin[threadIdx.x] = s.leaf_begin[p.leaf];
      count[threadIdx.x] = s.leaf_count[p.leaf];
      head[threadIdx.x] = r.piece_head[p.leaf];
    }
    __syncthreads();
    for (int32_t i = 0; i < m; ++i) {
      const RPiece p = piece[i];
      const uint32_t* from = s.idx[1 - p.own];
      uint32_t* to = s.idx[p.own] + begin[i];
      const uint32_t b = (blockIdx.x + (uint32_t)(i0 + i) * 37u) % gridDim.x;
      for (uint32_t k = b * 256u + threadIdx.x; k < (uint32_t)p.count; k += gridDim.x * 256u) {
        const uint32_t row = from[p.begin + k];
        int32_t rank = p.desc ? p.count - 1 - (int32_t)k : (int32_t)k;
        for (int32_t q = head[i]; q >= 0;) {
          const RPiece o = q >= i0 && q < i0 + m ? piece[q - i0] : r.piece[q];
          if (q != i0 + i) rank += rows_below(from + o.begin, o.count, o.desc != 0, row);
          q = o.next;
        }
        to[p.leaf_desc ? count[i] - 1 - rank : rank] = row;
      }
      if (p.next < 0 && b == 0 && threadIdx.x == 0) s.leaf_side[p.leaf] = p.own;  // the leaf's last piece
    }
  }
}
