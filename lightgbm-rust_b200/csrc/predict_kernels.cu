// Batched raw-score prediction: Gbdt::predict_matrix_early_stop with
// PredictKind::Raw (crates/lgbm-core/src/predict.rs:43-138, :231-339).
//
// The reference walks 16-row blocks level by level (predict.rs:43-138); here
// a thread walks its own row through two or four trees at once and a warp
// advances 32 rows together. What bounds a walk is the shared-memory pipe: a step is
// one 8-byte node load and one 4-byte value load.
//   - A CTA's rows are staged in shared memory by column (value of column c of
//     row r at c * R + r), so that the 32 lanes of a value load fall into 32
//     banks whatever features their nodes test.
//   - The trees are staged too, a few at a time, copied asynchronously while
//     the ones before are walked.
// With the rows staged by row, 16-byte nodes read through L1 and one tree at a
// time, 2,000,000 rows x 136 features under 300 trees of 255 leaves took
// 30.8 ms, bound by the latency of the dependent node loads (12 warps an SM).
//
// Few rows leave most SMs idle that way, so there a CTA takes 32 rows and its
// warps take different trees; one warp adds the leaf values in model order.
//
// Each row's sum, per class k, adds the leaf values of trees k, k + ntpi, ...
// in model order, which is the reference's summation order for that class
// (predict.rs:231-339), so the FP64 sums are the reference's. Any number of
// classes works: no per-class array is kept.
#include <algorithm>
#include <mutex>

#include "predict.h"

namespace lgbm_b200 {

constexpr int kRowThreads = 128;      // rows of a CTA of k_predict_rows
constexpr int kRowStageCols = 223;    // columns up to which it stages them: 128 x 224 floats are half an SM's memory
constexpr int kMaxPredictDevices = 64;
constexpr int kPredictSmem = 224 * 1024;

__device__ __forceinline__ bool find_in_bitset(const uint32_t* bits, int32_t n, int32_t pos) {  // tree.rs:46-52
  int32_t i1 = pos / 32;
  if (i1 >= n) return false;
  return ((bits[i1] >> (pos % 32)) & 1u) == 1u;
}

// The row is converted to f64 and |v| <= kZeroThreshold dropped
// (predict.rs:265-275).
__device__ __forceinline__ float drop_tiny(float x) {
  const double v = (double)x;
  return (!isnan(v) && fabs(v) <= kZeroThreshold) ? 0.0f : x;
}

// A categorical decision (step_any, predict.rs:77-90).
__device__ __noinline__ bool category_left(const DForest& f, int32_t ci, float v) {
  const int32_t b0 = f.cat_bnd[ci], b1 = f.cat_bnd[ci + 1];
  return !isnan(v) && (int32_t)v >= 0 && find_in_bitset(f.cat_words + b0, b1 - b0, (int32_t)v);
}

// One decision (FlatTree::step, predict.rs:95-111, or step_any) on a value
// free of tiny values: whether the walk goes to the node's first child.
// kSpecial: the node may be categorical, or have zero as its missing value and
// send it to the other side than the comparison would.
template <bool kSpecial>
__device__ __forceinline__ bool to_first(const DForest& f, const PNode& n, float v) {
  const float x = __uint_as_float(__float_as_uint(v) ^ (n.meta & kPNodeNegate));
  bool c = x <= n.threshold;
  if constexpr (kSpecial) {
    if (n.meta & kPNodeCat) c = category_left(f, __float_as_int(n.threshold), v);
    else if (v == 0.0f && (n.meta & kPNodeZeroFlip)) c = !c;
  }
  return c;
}

// R rows per CTA (a multiple of 32) and G = blockDim / R groups of R threads;
// a round of the loop walks G * kWalks trees of a class, kWalks a thread.
// kRows: the rows are staged; kTrees: so are the trees, in two buffers, else
// they are read from global memory; kSpecial: special nodes or features past
// the row. A round's leaf values are loaded while the next round walks, stored
// to shared memory after it, and added in model order by the first group in
// the round after that, so a round has one barrier.
template <int kWalks, bool kRows, bool kTrees, bool kSpecial>
__global__ void __launch_bounds__(1024) k_predict(const __grid_constant__ DForest f, const float* X, int64_t nrow,
                                                  int32_t ncol, double* out, int32_t R) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int T = blockDim.x, tid = threadIdx.x;
  const int row = tid % R, grp = tid / R, G = T / R;
  const int64_t r0 = (int64_t)blockIdx.x * R, r = r0 + row;
  const int per = G * kWalks;
  const int slot = f.max_nodes;
  // shared memory: two buffers of trees, two of leaf values, the rows, each staged tree's first node
  PNode* trees = reinterpret_cast<PNode*>(smem);
  double* vals = reinterpret_cast<double*>(smem + (kTrees ? (size_t)2 * per * slot * sizeof(PNode) : 0));
  int32_t* firsts = reinterpret_cast<int32_t*>(vals + (size_t)2 * per * R);
  float* xs = reinterpret_cast<float*>(firsts + 2 * per);
  const PNode* nodes = static_cast<const PNode*>(f.nodes);
  const int ntpi = f.ntpi;
  // copies the trees of round j of class k (nt trees) into buffer j & 1
  auto stage = [&](int k, int32_t j, int32_t nt) {
    const int m = min(per, nt - j * per), to = j & 1;
    for (int i = tid >> 5; i < m; i += T >> 5) {  // a warp per tree
      const int4 tt = __ldg(&f.tree[k + (j * per + i) * ntpi]);
      if ((tid & 31) == 0) firsts[to * per + i] = tt.x;
      if constexpr (kTrees) {
        const uint32_t dst = (uint32_t)__cvta_generic_to_shared(trees + ((size_t)to * per + i) * slot);
        const PNode* src = nodes + tt.x;
        for (int u = tid & 31; u < (tt.w >> 1); u += 32)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16u * (uint32_t)u), "l"(src + 2 * u) : "memory");
      }
    }
  };
  auto trees_of = [&](int k) { return f.num_trees > k ? (f.num_trees - k + ntpi - 1) / ntpi : 0; };
  stage(0, 0, trees_of(0));
  if constexpr (kRows) {
    // lanes take neighbouring rows, warps the columns: a row's sectors are
    // used up by the next columns' loads, and the stores fall into 32 banks
    const int warp = tid >> 5, lane = tid & 31, nw = T >> 5, rw = R >> 5;  // nw is a multiple of rw
    const bool vec = (ncol & 3) == 0 && (reinterpret_cast<uintptr_t>(X) & 15) == 0;
    const int ncv = vec ? ncol >> 2 : ncol;
    const int rl = (warp % rw) * 32 + lane;
    const bool live = r0 + rl < nrow;
    const float* src = X + (r0 + rl) * ncol;
#pragma unroll 4
    for (int c = warp / rw; c < ncv; c += nw / rw) {
      if (vec) {
        const float4 v = live ? __ldg(reinterpret_cast<const float4*>(src) + c) : make_float4(0.f, 0.f, 0.f, 0.f);
        float* d = xs + (size_t)4 * c * R + rl;
        d[0] = drop_tiny(v.x);
        d[R] = drop_tiny(v.y);
        d[2 * R] = drop_tiny(v.z);
        d[3 * R] = drop_tiny(v.w);
      } else {
        xs[(size_t)c * R + rl] = live ? drop_tiny(__ldg(src + c)) : 0.0f;
      }
    }
    for (int i = tid; i < R; i += T) xs[(size_t)ncol * R + i] = 0.0f;  // features past the row read 0.0
  }
  const float* xrow = kRows ? xs + row : X + min(r, nrow - 1) * ncol;
  auto value = [&](uint32_t meta) {
    const int32_t feat = (int32_t)(meta >> 16) & ((1 << kPNodeFeatureBits) - 1);
    if constexpr (kRows) return xrow[(uint32_t)((kSpecial ? min(feat, ncol) : feat) * R)];
    else return feat < ncol ? drop_tiny(__ldg(xrow + feat)) : 0.0f;
  };
  for (int k = 0; k < ntpi; ++k) {
    const int32_t nt = trees_of(k), rounds = (nt + per - 1) / per;
    if (k > 0) {
      __syncthreads();  // the class before is walked
      stage(k, 0, nt);
    }
    double acc = 0.0;
    double lv[kWalks];
    // round j walks the trees of round j; rounds and rounds + 1 only pass the last leaf values on
    for (int32_t j = 0; j < rounds + 2; ++j) {
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncthreads();
      if (j + 1 < rounds) stage(k, j + 1, nt);
      if (grp == 0 && j >= 2) {
        const int m = min(per, nt - (j - 2) * per);
        const double* v = vals + (size_t)(j & 1) * per * R + row;
#pragma unroll 4
        for (int b = 0; b < m; ++b) acc += v[(size_t)b * R];
      }
      uint32_t leaf[kWalks];
      if (j < rounds) {
        const int m = min(per, nt - j * per), buf = j & 1, b0 = grp * kWalks;
        uint32_t at[kWalks];
        const PNode* base[kWalks];
#pragma unroll
        for (int i = 0; i < kWalks; ++i) {
          const int b = min(b0 + i, m - 1);  // past the round's trees: walked, not used
          leaf[i] = (uint32_t)firsts[buf * per + b];
          if constexpr (kTrees) base[i] = trees + ((size_t)buf * per + b) * slot;
          else base[i] = nodes + leaf[i];
          at[i] = 0;
        }
        bool more = true;
        while (__any_sync(0xffffffffu, more)) {
          PNode n[kWalks];
#pragma unroll
          for (int i = 0; i < kWalks; ++i) n[i] = base[i][at[i]];
          float v[kWalks];
#pragma unroll
          for (int i = 0; i < kWalks; ++i) v[i] = value(n[i].meta);
          more = false;
#pragma unroll
          for (int i = 0; i < kWalks; ++i) {
            const uint32_t next = (n[i].meta & 0xffffu) + (to_first<kSpecial>(f, n[i], v[i]) ? 0u : 1u);
            more |= next != at[i];
            at[i] = next;
          }
        }
#pragma unroll
        for (int i = 0; i < kWalks; ++i) leaf[i] += at[i];
      }
      if (j >= 1 && j <= rounds) {
        double* v = vals + (size_t)((j - 1) & 1) * per * R + row;
#pragma unroll
        for (int i = 0; i < kWalks; ++i) v[(size_t)(grp * kWalks + i) * R] = lv[i];
      }
      if (j < rounds) {
#pragma unroll
        for (int i = 0; i < kWalks; ++i) lv[i] = __ldg(f.leaf_value + leaf[i]);
      }
    }
    if (grp == 0 && r < nrow) out[r * ntpi + k] = acc;
  }
}

// A thread per row that walks one tree after the other, nodes read through
// L1: the wide layout, and forests with too little work a row for the rounds'
// barriers and staged trees (launch_predict). kStage: the CTA's rows, one
// contiguous block of X, are staged in shared memory by row (`stride` floats
// apart, odd), so that the loads are coalesced.
template <bool kCompact, bool kStage>
__global__ void __launch_bounds__(kRowThreads) k_predict_rows(const __grid_constant__ DForest f, const float* X,
                                                              int64_t nrow, int32_t ncol, int32_t stride, double* out) {
  extern __shared__ __align__(16) unsigned char smem[];
  float* xs = reinterpret_cast<float*>(smem);
  const int64_t r0 = (int64_t)blockIdx.x * kRowThreads, r = r0 + threadIdx.x;
  if constexpr (kStage) {
    const int32_t total = (int32_t)min((int64_t)kRowThreads, nrow - r0) * ncol;
    const float* src = X + r0 * ncol;
    if ((ncol & 3) == 0 && (reinterpret_cast<uintptr_t>(src) & 15) == 0) {
      for (int32_t i = threadIdx.x; i < total >> 2; i += kRowThreads) {
        const float4 v = __ldg(reinterpret_cast<const float4*>(src) + i);
        const int32_t row = (i << 2) / ncol, col = (i << 2) - row * ncol;  // the 4 values lie in one row
        float* d = xs + row * stride + col;
        d[0] = drop_tiny(v.x);
        d[1] = drop_tiny(v.y);
        d[2] = drop_tiny(v.z);
        d[3] = drop_tiny(v.w);
      }
    } else {
      for (int32_t i = threadIdx.x; i < total; i += kRowThreads) {
        const int32_t row = i / ncol;
        xs[row * stride + i - row * ncol] = drop_tiny(__ldg(src + i));
      }
    }
    __syncthreads();
  }
  if (r >= nrow) return;
  const float* row = kStage ? xs + threadIdx.x * stride : X + r * ncol;
  auto value = [&](int32_t feat) {  // features past the row read 0.0
    if (feat >= ncol) return 0.0f;
    if constexpr (kStage) return row[feat];
    else return drop_tiny(__ldg(row + feat));
  };
  const int ntpi = f.ntpi;
  for (int k = 0; k < ntpi; ++k) {
    double acc = 0.0;
    for (int32_t t = k; t < f.num_trees; t += ntpi) {
      const int4 tt = __ldg(&f.tree[t]);
      int32_t leaf = 0;
      if constexpr (kCompact) {
        const PNode* nodes = static_cast<const PNode*>(f.nodes) + tt.x;
        uint32_t at = tt.z > 1 ? 0 : 1;  // a constant tree's leaf is at place 1
        while (tt.z > 1) {
          const uint2 u = __ldg(reinterpret_cast<const uint2*>(nodes + at));
          const PNode n{__uint_as_float(u.x), u.y};
          const uint32_t first = n.meta & 0xffffu;
          if (first < at) break;  // a leaf: a node's children lie behind it
          const float v = value((int32_t)(n.meta >> 16) & ((1 << kPNodeFeatureBits) - 1));
          at = first + (to_first<true>(f, n, v) ? 0u : 1u);
        }
        leaf = tt.x + (int32_t)at;
      } else {
        const DNodeWide* nodes = static_cast<const DNodeWide*>(f.nodes) + tt.x;
        int32_t node = tt.z > 1 ? 0 : ~0;
        while (node >= 0) {
          const DNodeWide n = nodes[node];
          const int8_t dt = (int8_t)(n.feat_dt >> kNodeFeatureBits);
          double v = (double)value(n.feat_dt & ((1 << kNodeFeatureBits) - 1));
          bool left;
          if (dt & 1) {
            left = category_left(f, (int32_t)__double_as_longlong(n.threshold), (float)v);
          } else {  // FlatTree::step (predict.rs:95-111)
            const int mt = (dt >> 2) & 3;
            const bool nan = isnan(v), nan_split = mt == 2;
            if (nan && !nan_split) v = 0.0;
            const bool zero = v >= -kZeroThreshold && v <= kZeroThreshold;
            const bool is_default = (mt == 1 && zero) || (nan_split && nan);
            left = is_default ? (dt & 2) != 0 : v <= n.threshold;
          }
          node = left ? n.left : n.right;
        }
        leaf = tt.y + ~node;
      }
      acc += __ldg(f.leaf_value + leaf);
    }
    out[r * ntpi + k] = acc;
  }
}

using PredictKernel = void (*)(DForest, const float*, int64_t, int32_t, double*, int32_t);
template <int kWalks>
static PredictKernel predict_kernel(bool rows, bool trees, bool special) {
  if (special)
    return rows ? (trees ? k_predict<kWalks, true, true, true> : k_predict<kWalks, true, false, true>)
                : (trees ? k_predict<kWalks, false, true, true> : k_predict<kWalks, false, false, true>);
  return rows ? (trees ? k_predict<kWalks, true, true, false> : k_predict<kWalks, true, false, false>)
              : (trees ? k_predict<kWalks, false, true, false> : k_predict<kWalks, false, false, false>);
}

static std::once_flag g_predict_once[kMaxPredictDevices];
static cudaError_t g_predict_err[kMaxPredictDevices];
static int g_predict_sms[kMaxPredictDevices];

// Opt the kernels in to more than 48 KiB of dynamic shared memory, once per
// device (the setting belongs to the device's context).
static cudaError_t predict_device(int* sms) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= kMaxPredictDevices) return cudaErrorInvalidDevice;
  std::call_once(g_predict_once[dev], [dev] {
    cudaError_t x = cudaDeviceGetAttribute(&g_predict_sms[dev], cudaDevAttrMultiProcessorCount, dev);
    auto opt = [&](const void* k) {
      if (x == cudaSuccess) x = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kPredictSmem);
    };
    for (int i = 0; i < 8; ++i) {
      opt((const void*)predict_kernel<2>(i & 1, i & 2, i & 4));
      opt((const void*)predict_kernel<4>(i & 1, i & 2, i & 4));
    }
    opt((const void*)k_predict_rows<true, true>);
    opt((const void*)k_predict_rows<false, true>);
    g_predict_err[dev] = x;
  });
  *sms = g_predict_sms[dev];
  return g_predict_err[dev];
}

cudaError_t launch_predict(const DForest& f, const float* X, int64_t nrow, int32_t ncol, double* out, cudaStream_t s) {
  if (nrow <= 0) return cudaSuccess;
  int sms = 148;
  cudaError_t e = predict_device(&sms);
  if (e != cudaSuccess) return e;
  const int32_t per_class = (f.num_trees + f.ntpi - 1) / f.ntpi;
  // A CTA's threads are R rows times G groups that walk different trees: the
  // rows take the most shared memory, and a walk is a chain of dependent
  // loads, so several warps share a row's staged values. 128 rows where that
  // fills the SMs, else fewer, and few rows spread over the SMs 32 at a time
  // with up to 32 groups.
  int R = nrow >= (int64_t)sms * 128 ? 128 : nrow >= (int64_t)sms * 64 ? 64 : 32;
  const size_t col = sizeof(float) * ((size_t)ncol + 1);
  while (R > 32 && R * col > 150 * 1024) R /= 2;
  const bool rows = R * col <= 150 * 1024;
  const size_t row_bytes = rows ? R * col : 0;
  const size_t tree = sizeof(PNode) * (size_t)f.max_nodes;
  // a round's trees in two buffers, two leaf values per row and tree and two
  // indices per tree, beside the rows
  const size_t left = kPredictSmem - row_bytes;
  auto bytes = [&](int per, bool staged) {
    return (size_t)per * ((staged ? 2 * tree : 0) + 2 * sizeof(double) * R + 2 * sizeof(int32_t));
  };
  // Four trees a thread where 16 trees leave room for a second CTA on the SM
  // (500,000 rows x 28 features, 100 trees of 31 leaves: 396 us against 493
  // with two), else two trees and twice the groups, whose shorter walks wait
  // less for the deepest of their rows (2,000,000 x 136, 300 trees of 255
  // leaves: 7.9 ms against 9.7 with four).
  const int walks = row_bytes + bytes(16, true) <= kPredictSmem / 2 ? 4 : 2;
  const int want = std::max(1, (per_class + walks - 1) / walks);  // groups that all have trees
  int G = std::min(want, R == 128 ? 16 / walks : R == 64 ? 32 / walks : 32);
  int Gs = G;
  while (Gs > 1 && bytes(Gs * walks, true) > left) --Gs;
  const bool staged = bytes(Gs * walks, true) <= left;
  if (staged) {
    G = Gs;
  } else {
    while (G > 1 && bytes(G * walks, false) > left) --G;
  }
  // no more groups than the rounds need: 20 trees are two rounds of 5 groups, not of 8
  const int rounds = std::max(1, (per_class + G * walks - 1) / (G * walks));
  G = std::max(1, (per_class + rounds * walks - 1) / (rounds * walks));
  // A thread a row where a row's walks are too short for the rounds' barriers
  // and staged trees. One tree a class: 1M rows x 28, 31 leaves, 47 us against
  // 83; ten classes 159 against 294 (few rows the same). Few levels in all, with
  // rows enough for a wave of CTAs' walks to hide another's loads: three trees of
  // 31 leaves 65 against 84, six 97 against 100, eight 118 against 102; 12 of 2
  // leaves 73 against 119; 100k rows, two of 31 leaves 23 against 25, six 31
  // against 27. Half as many where several classes share the rows' staging: two
  // trees a class, ten classes, 31 leaves 268 against 309, 255 leaves 372
  // against 351. Constant trees. Where the trees are too large to stage, both read
  // them through L1 and rows enough hide it: 1M rows, 20 trees of 30,000 leaves
  // 577 against 670, 100k rows 131 against 94.
  int levels = 0;
  while ((1 << levels) < f.max_nodes) ++levels;
  const bool by_row = !f.compact || per_class <= 1 || levels <= 1 ||
                      (nrow >= (int64_t)sms * 512 && per_class * levels * (f.ntpi > 1 ? 2 : 1) <= 24) ||
                      (nrow >= (int64_t)sms * 2048 && !staged && per_class <= 20);
  if (by_row) {
    const int64_t blocks = (nrow + kRowThreads - 1) / kRowThreads;
    if (blocks > 0x7fffffff) return cudaErrorInvalidValue;
    const bool stage = ncol <= kRowStageCols;
    const int32_t stride = ncol | 1;
    const size_t smem = stage ? sizeof(float) * kRowThreads * (size_t)stride : 0;
    auto kernel = f.compact ? (stage ? k_predict_rows<true, true> : k_predict_rows<true, false>)
                            : (stage ? k_predict_rows<false, true> : k_predict_rows<false, false>);
    kernel<<<(unsigned)blocks, kRowThreads, smem, s>>>(f, X, nrow, ncol, stride, out);
    return cudaGetLastError();
  }
  const size_t smem = bytes(G * walks, staged) + row_bytes;
  const int64_t blocks = (nrow + R - 1) / R;
  if (blocks > 0x7fffffff) return cudaErrorInvalidValue;
  const bool special = f.special || f.max_feature >= ncol;
  const PredictKernel kernel =
      walks == 4 ? predict_kernel<4>(rows, staged, special) : predict_kernel<2>(rows, staged, special);
  kernel<<<(unsigned)blocks, R * G, smem, s>>>(f, X, nrow, ncol, out, R);
  return cudaGetLastError();
}

}  // namespace lgbm_b200
