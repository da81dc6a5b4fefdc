// LambdarankNDCG gradients (crates/lgbm-core/src/objective/rank.rs:119-262,
// RankingBase::gradients :63-111) on the device, in one launch:
//   k_lambdarank   one CTA of 4 warps per query.
//     order   the stable descending order of the query's scores
//             (dcg.rs:167-179) by rank counting; the sorted scores, gains
//             and labels stay in shared memory (queries above kRankRows
//             rows: in global memory)
//     pairs   the reference's pair loop (outer position i below the
//             truncation level, inner j > i) as one sequence, in tiles of
//             kRankTile pairs: each pair's lambda and hessian are evaluated
//             once, by any thread, into shared memory
//     sums    the row at position p adds first the pairs (i, p), i < p, in
//             order of i, then, when p itself is an outer position, the
//             pairs (p, j) in order of j, one thread per row, so every f32
//             lambda and hessian is formed as on the CPU. The FP64 sum of
//             the lambdas (for the normalisation) is one sequential chain in
//             the sequence's order; it runs in one thread beside the rows'
//             sums (a pair that is skipped would add 0.0, which changes no
//             sum, and is left out of the chain).
// k_ndcg's order comes from k_rank_sort, the same rank counting on its own.
// The tables the reference builds in its constructor (label gains,
// discounts, inverse max DCG per query, the 2^20-entry sigmoid table) are
// built on the host by the same arithmetic and uploaded once.
#include "rank.h"

namespace lgbm_b200 {

constexpr double kMinScoreD = -INFINITY;  // consts.rs kMinScore
constexpr int kRankThreads = 128;
constexpr int kRankTile = 1024;  // pairs evaluated between two barriers
constexpr int kRankRows = 256;   // rows of a query whose sorted order stays in shared memory
constexpr int kRankHold = 4;     // rows ranked at once by a thread of a larger query
// Queries of so few rows are taken by 8 lanes each: a CTA's barriers and
// idle threads cost them more than their pairs (an iteration of 800k rows in
// queries of 2, trees of one split: 1160 us with a CTA each, 205 with these;
// of 5, 682 and 195; of 10, which keep their CTAs, 498).
constexpr int kRankSmall = 8;
constexpr int kRankSmallPerCta = kRankThreads / kRankSmall;

// Monotone map of a score onto uint64: larger score, larger key; -0 and +0
// are equal, and a NaN orders after every number.
__device__ __forceinline__ uint64_t rank_key(double s) {
  if (isnan(s)) return 0;
  const uint64_t b = (uint64_t)__double_as_longlong(s == 0.0 ? 0.0 : s);
  return (b & 0x8000000000000000ull) ? ~b : (b | 0x8000000000000000ull);
}

// Position i's place in the stable descending order of key[0, cnt). (No key
// is the largest uint64, so the key after it is one too.)
__device__ __forceinline__ int32_t rank_of(const uint64_t* key, int32_t cnt, int32_t i) {
  const uint64_t ki = key[i];
  int32_t rank = 0;
#pragma unroll 4
  for (int32_t j = 0; j < cnt; ++j) rank += key[j] >= (j < i ? ki : ki + 1) ? 1 : 0;
  return rank;
}

// The same for every row of a query too large for shared memory: a thread
// keeps the places of kRankHold of its rows while the keys pass through
// `key` (kRankTile of them at a time); place(i, rank) takes each result.
// All threads of the CTA call it.
template <class F>
__device__ __forceinline__ void rank_large(const double* score, int32_t cnt, uint64_t* key, F place) {
  for (int32_t i0 = 0; i0 < cnt; i0 += kRankHold * blockDim.x) {
    uint64_t mine[kRankHold];
    int32_t rank[kRankHold], row[kRankHold];
#pragma unroll
    for (int k = 0; k < kRankHold; ++k) {
      row[k] = i0 + k * (int32_t)blockDim.x + (int32_t)threadIdx.x;
      mine[k] = row[k] < cnt ? rank_key(score[row[k]]) : 0;
      rank[k] = 0;
    }
    for (int32_t j0 = 0; j0 < cnt; j0 += kRankTile) {
      const int32_t here = min(kRankTile, cnt - j0);
      __syncthreads();
      for (int32_t j = threadIdx.x; j < here; j += blockDim.x) key[j] = rank_key(score[j0 + j]);
      __syncthreads();
      for (int32_t j = 0; j < here; ++j) {
        const uint64_t kj = key[j];
#pragma unroll
        for (int k = 0; k < kRankHold; ++k) rank[k] += kj >= (j0 + j < row[k] ? mine[k] : mine[k] + 1) ? 1 : 0;
      }
    }
#pragma unroll
    for (int k = 0; k < kRankHold; ++k)
      if (row[k] < cnt) place(row[k], rank[k]);
  }
}

__global__ void __launch_bounds__(kRankThreads) k_rank_sort(DRank r, const double* score) {
  __shared__ uint64_t key[kRankTile];
  for (int32_t q = blockIdx.x; q < r.nq; q += gridDim.x) {
    const int32_t b0 = r.bnd[q], cnt = r.bnd[q + 1] - b0;
    rank_large(score + b0, cnt, key, [&](int32_t i, int32_t at) { r.sorted[b0 + at] = (uint32_t)i; });
  }
}

__device__ __forceinline__ double rank_sigmoid(const DRank& r, double score) {  // rank.rs:178-186
  if (!(score > r.min_in)) return r.sigmoid_table[0];  // a NaN too, as its cast to an index
  if (score >= r.max_in) return r.sigmoid_table[kRankSigmoidBins - 1];
  return r.sigmoid_table[(size_t)((score - r.min_in) * r.idx_factor)];
}

// One query's rows in sorted order and the values its pairs share.
struct QueryView {
  const double* score;
  const double* gain;  // of the label
  const float* label;
  double inverse_max_dcg;
  bool scale_by_score;  // norm and best_score != worst_score (rank.rs:231-233)
};

// The pair of two rows whose labels differ, neither score the minimum: its
// lambda and hessian by the reference's FP64 operations (rank.rs:217-252), from
// the higher-labelled row's score and label gain less the other's and the
// discounts of their places.
__device__ __forceinline__ void pair_value(const DRank& r, double delta_score, double dcg_gap, double discount_high,
                                           double discount_low, double inverse_max_dcg, bool scale_by_score,
                                           double& p_lambda, double& p_hessian) {
  const double paired_discount = fabs(discount_high - discount_low);
  double delta_pair_ndcg = dcg_gap * paired_discount * inverse_max_dcg;
  if (scale_by_score) delta_pair_ndcg /= (double)0.01f + fabs(delta_score);
  double pl = rank_sigmoid(r, delta_score);
  double ph = pl * (1.0 - pl);
  pl *= -r.sigmoid * delta_pair_ndcg;
  ph *= r.sigmoid * r.sigmoid * delta_pair_ndcg;
  p_lambda = pl;
  p_hessian = ph;
}

// The query of kRankSmall rows at most that the 8 lanes of this thread's group
// share, a row each (every thread of the warp calls it; cnt 0: no query). The
// same pairs and sums as k_lambdarank's, passed between the lanes: outer row i's
// pairs are evaluated side by side, their inner rows take them at once, and
// the outer row and the FP64 chain add them in order.
__device__ __forceinline__ void lambdarank_small(const DRank& r, int32_t b0, int32_t cnt, double inverse_max_dcg,
                                                 const double* score, const float* label, float* g, float* h,
                                                 float2* gh) {
  constexpr unsigned kAll = 0xffffffffu;
  constexpr int W = kRankSmall;
  const int l = threadIdx.x & (W - 1);
  const bool live = l < cnt;
  const int32_t most = __reduce_max_sync(kAll, cnt);  // of the warp's queries
  double sc = live ? score[b0 + l] : 0.0;
  float lab = live ? label[b0 + l] : 0.0f;
  int32_t at = l;  // the row's place in the stable descending order
  {
    const uint64_t key = live ? rank_key(sc) : 0;
    int32_t rank = 0;
    for (int j = 0; j < most; ++j) {
      const uint64_t kj = __shfl_sync(kAll, key, j, W);
      if (j < cnt) rank += kj >= (j < l ? key : key + 1) ? 1 : 0;
    }
    if (live) at = rank;
  }
  int32_t row = l;  // the row at this lane's place
  for (int j = 0; j < most; ++j)
    if (__shfl_sync(kAll, at, j, W) == l) row = j;
  sc = __shfl_sync(kAll, sc, row, W);
  lab = __shfl_sync(kAll, lab, row, W);
  const double gain = r.label_gain[(int32_t)lab], disc = r.discount[l];
  int32_t worst = max(cnt - 1, 0);
  const bool last_min = __shfl_sync(kAll, sc, worst, W) == kMinScoreD;
  if (worst > 0 && last_min) worst -= 1;
  const double best_score = __shfl_sync(kAll, sc, 0, W), worst_score = __shfl_sync(kAll, sc, worst, W);
  const bool scale = r.norm && best_score != worst_score;
  const int32_t outer = max(0, min(r.truncation_level, cnt - 1));
  const int32_t most_outer = __reduce_max_sync(kAll, outer);
  float acc_l = 0.0f, acc_h = 0.0f;
  double sum_lambdas = 0.0;
  for (int i = 0; i < most_outer; ++i) {
    const double si = __shfl_sync(kAll, sc, i, W), gi = __shfl_sync(kAll, gain, i, W), di = __shfl_sync(kAll, disc, i, W);
    const float li = __shfl_sync(kAll, lab, i, W);
    const bool pair = i < outer && l > i && live;
    const bool i_high = li > lab, counts = pair && li != lab && si != kMinScoreD && sc != kMinScoreD;
    double pl = 0.0, ph = 0.0;
    if (counts) {
      const double gap = i_high ? gi - gain : gain - gi;
      pair_value(r, i_high ? si - sc : sc - si, gap, i_high ? di : disc, i_high ? disc : di, inverse_max_dcg, scale, pl,
                 ph);
    }
    const float vl = i_high ? (float)pl : -(float)pl, vh = (float)ph;
    if (pair) {
      acc_l -= vl;
      acc_h += vh;
    }
    for (int j = i + 1; j < most; ++j) {
      const float ol = __shfl_sync(kAll, vl, j, W), oh = __shfl_sync(kAll, vh, j, W);
      const double oc = __shfl_sync(kAll, 2.0 * pl, j, W);  // 0 where the pair does not count
      if (i < outer && j < cnt) {
        sum_lambdas -= oc;
        if (l == i) {
          acc_l += ol;
          acc_h += oh;
        }
      }
    }
  }
  if (r.norm && sum_lambdas > 0.0) {
    const double norm_factor = log2(1.0 + sum_lambdas) / sum_lambdas;
    acc_l = (float)((double)acc_l * norm_factor);
    acc_h = (float)((double)acc_h * norm_factor);
  }
  if (!live) return;
  if (g) {
    g[b0 + row] = acc_l;
    h[b0 + row] = acc_h;
  } else {
    gh[b0 + row] = make_float2(acc_l, acc_h);
  }
}

// LambdarankNDCG::one_query (rank.rs:192-262), a CTA per query of more than
// kRankSmall rows, and CTAs that take kRankSmallPerCta of the others. Writes
// g/h (class-major float arrays) or the interleaved pairs.
//
// What bounds it: issue slots (2.2 instructions a cycle) and the barriers
// between the parts, since a pair costs an FP64 divide, index arithmetic and
// a load from the 8 MB sigmoid table, and one thread has the FP64 chain. A
// pair is evaluated once (each of its two rows and the chain read it from
// shared memory; a warp per query that evaluated it in all three places had
// no barriers and three times the work), and the whole CTA is on one query's
// pairs, so the largest query does not run on alone. Order and gradients,
// two launches -> this one, on B200 with 5 labels and truncation 30: 800k
// rows in queries of 40 rows (geometric) 1130 -> 455 us; of 400 rows 13.2
// -> 3.8 ms; 20k rows of 40 670 -> 160 us; one query of 10000 rows 81 -> 17
// ms. CTAs of 64, 96 and 256 threads take 1.25, 1.07 and 1.2 times as long
// at 40 rows a query (256 would win above 400).
__global__ void __launch_bounds__(kRankThreads, 9) k_lambdarank(DRank r, const double* score, const float* label,
                                                             float* g, float* h, float2* gh) {
  __shared__ __align__(16) double t_chain[kRankTile];  // 2 * lambda of the pairs that count, in order, by 32 slots
  __shared__ float t_lambda[kRankTile];  // what the pair adds to its outer row (its inner row takes the negative)
  __shared__ float t_hess[kRankTile];
  __shared__ double s_score[kRankRows], s_gain[kRankRows];
  __shared__ float s_label[kRankRows];
  __shared__ uint16_t s_row[kRankRows];
  __shared__ int32_t t_count[kRankTile / 32];
  __shared__ double s_sum;
  const int tid = threadIdx.x, lane = tid & 31;
  if ((int32_t)blockIdx.x >= r.num_large) {
    const int32_t x = ((int32_t)blockIdx.x - r.num_large) * kRankSmallPerCta + tid / kRankSmall;
    const int32_t q = x < r.num_small ? r.query[r.num_large + x] : -1;
    const int32_t b0 = q >= 0 ? r.bnd[q] : 0, cnt = q >= 0 ? r.bnd[q + 1] - b0 : 0;
    lambdarank_small(r, b0, cnt, q >= 0 ? r.inv_max_dcg[q] : 0.0, score, label, g, h, gh);
    return;
  }
  {
    const int32_t q = r.query[blockIdx.x];
    const int32_t b0 = r.bnd[q], cnt = r.bnd[q + 1] - b0;
    const bool small = cnt <= kRankRows;
    QueryView v;
    v.score = small ? s_score : r.sorted_score + b0;
    v.gain = small ? s_gain : r.sorted_gain + b0;
    v.label = small ? s_label : r.sorted_label + b0;
    v.inverse_max_dcg = r.inv_max_dcg[q];
    if (small) {
      uint64_t* key = reinterpret_cast<uint64_t*>(t_chain);
      for (int32_t i = tid; i < cnt; i += kRankThreads) key[i] = rank_key(score[b0 + i]);
      __syncthreads();
      for (int32_t i = tid; i < cnt; i += kRankThreads) {
        const int32_t at = rank_of(key, cnt, i);
        const float l = label[b0 + i];
        s_score[at] = score[b0 + i];
        s_gain[at] = r.label_gain[(int32_t)l];
        s_label[at] = l;
        s_row[at] = (uint16_t)i;
      }
    } else {
      rank_large(score + b0, cnt, reinterpret_cast<uint64_t*>(t_chain), [&](int32_t i, int32_t rank) {
        const int32_t at = b0 + rank;
        const float l = label[b0 + i];
        r.sorted_score[at] = score[b0 + i];
        r.sorted_gain[at] = r.label_gain[(int32_t)l];
        r.sorted_label[at] = l;
        r.sorted[at] = (uint32_t)i;
      });
    }
    __syncthreads();
    int32_t worst_idx = cnt - 1;
    if (worst_idx > 0 && v.score[worst_idx] == kMinScoreD) worst_idx -= 1;
    v.scale_by_score = r.norm && v.score[0] != v.score[worst_idx];
    // the sequence of pairs: rows i = 0 .. outer - 1, row i the pairs (i, i + 1 .. cnt - 1), from `start(i)` on
    const int32_t outer = max(0, min(r.truncation_level, cnt - 1));
    const int32_t pairs = outer * (cnt - 1) - (int32_t)((int64_t)outer * (outer - 1) / 2);
    auto start = [&](int32_t i) { return i * (cnt - 1) - (int32_t)((int64_t)i * (i - 1) / 2); };
    double sum_lambdas = 0.0;  // thread 0's chain
    int32_t i = 0, j = 1 + tid;                   // this thread's next pair
    int32_t first = 0;                            // the row that holds the tile's first pair
    for (int32_t base = 0; base == 0 || base < pairs; base += kRankTile) {
      const int32_t here = min(kRankTile, pairs - base);  // 0 for a query of one row
      for (int32_t t = tid; t < kRankTile; t += kRankThreads) {
        while (i < outer && j >= cnt) {
          ++i;
          j = j - cnt + i + 1;
        }
        double pl = 0.0, ph = 0.0;
        bool counts = false, i_high = false;
        if (i < outer) {
          const float li = v.label[i], lj = v.label[j];
          i_high = li > lj;
          counts = li != lj && v.score[i] != kMinScoreD && v.score[j] != kMinScoreD;
          if (counts) {
            const int32_t high = i_high ? i : j, low = i_high ? j : i;
            pair_value(r, v.score[high] - v.score[low], v.gain[high] - v.gain[low], r.discount[high], r.discount[low],
                       v.inverse_max_dcg, v.scale_by_score, pl, ph);
          }
        }
        t_lambda[t] = i_high ? (float)pl : -(float)pl;
        t_hess[t] = (float)ph;
        const uint32_t m = __ballot_sync(0xffffffffu, counts);
        const int32_t n = max(__popc(m), 1);  // one zero where no pair counts
        if (counts) t_chain[(t & ~31) + __popc(m & ((1u << lane) - 1))] = 2.0 * pl;
        if (lane >= __popc(m) && lane < ((n + 3) & ~3)) t_chain[(t & ~31) + lane] = 0.0;
        if (lane == 0) t_count[t >> 5] = n;
        j += kRankThreads;
        if (base + t - tid + kRankThreads >= pairs) break;  // uniform: no pair is left
      }
      __syncthreads();
      const int32_t last = base + here;  // pairs of the tile: [base, last)
      while (first + 1 < outer && start(first + 1) <= base) ++first;
      if (tid == 0 && r.norm) {
        double2 x = *reinterpret_cast<const double2*>(&t_chain[0]), y = *reinterpret_cast<const double2*>(&t_chain[2]);
        int32_t n = here > 0 ? t_count[0] : 0;
        for (int32_t w = 0; w * 32 < here; ++w) {
          const int32_t after = (w + 1) * 32 < here ? t_count[w + 1] : 0;
          for (int32_t k = 0; k < n; k += 4) {
            // the next four: of this group, or the first of the group after it
            const int32_t at = min(w * 32 + (k + 4 < n ? k + 4 : 32), kRankTile - 4);
            const double2 nx = *reinterpret_cast<const double2*>(&t_chain[at]);
            const double2 ny = *reinterpret_cast<const double2*>(&t_chain[at + 2]);
            sum_lambdas -= x.x;
            sum_lambdas -= x.y;
            sum_lambdas -= y.x;
            sum_lambdas -= y.y;
            x = nx;
            y = ny;
          }
          n = after;
        }
      }
      // the rows' sums; warp 0 keeps to the chain when there is one
      const int32_t skip = r.norm ? 32 : 0;
      for (int32_t p = (base == 0 ? 0 : first) + tid - skip; tid >= skip && p < cnt; p += kRankThreads - skip) {
        // as the inner position of rows first ..: pair (i, p) is slot start(i) + p - i - 1
        const int32_t inner = min(p, outer);
        int32_t o = first, slot = start(first) + p - first - 1 - base;
        if (slot < 0 && o < inner) slot += cnt - 2 - o++;  // row `first` began in the tile before
        const int32_t from = max(base, start(p)), to = min(last, start(p) + cnt - 1 - p);
        if (base > 0 && !(o < inner && slot < here) && !(p < outer && from < to)) continue;  // none of its pairs
        const uint32_t row = b0 + (small ? (uint32_t)s_row[p] : r.sorted[b0 + p]);
        float acc_l = 0.0f, acc_h = 0.0f;
        if (base > 0) {
          acc_l = g ? g[row] : gh[row].x;
          acc_h = g ? h[row] : gh[row].y;
        }
#pragma unroll 4
        for (; o < inner && slot < here; slot += cnt - 2 - o++) {
          acc_l -= t_lambda[slot];
          acc_h += t_hess[slot];
        }
        // as the outer position: its row's pairs inside the tile
        if (p < outer) {
#pragma unroll 8
          for (int32_t t = from; t < to; ++t) {
            acc_l += t_lambda[t - base];
            acc_h += t_hess[t - base];
          }
        }
        if (g) {
          g[row] = acc_l;
          h[row] = acc_h;
        } else {
          gh[row] = make_float2(acc_l, acc_h);
        }
      }
      __syncthreads();  // the sums are written, and the tile is free
    }
    if (!r.norm) return;
    if (tid == 0) s_sum = sum_lambdas;
    __syncthreads();
    sum_lambdas = s_sum;
    if (sum_lambdas > 0.0) {
      const double norm_factor = log2(1.0 + sum_lambdas) / sum_lambdas;
      for (int32_t x = tid; x < cnt; x += kRankThreads) {
        if (g) {
          g[b0 + x] = (float)((double)g[b0 + x] * norm_factor);
          h[b0 + x] = (float)((double)h[b0 + x] * norm_factor);
        } else {
          const float2 a = gh[b0 + x];
          gh[b0 + x] = make_float2((float)((double)a.x * norm_factor), (float)((double)a.y * norm_factor));
        }
      }
    }
  }
}

// NDCG@k of every query (metric.rs:546-598, no query weights), one thread
// per query, with the additions in the reference's order: out[q * nk + j]
// (1.0 for every k when the query's best DCG at ks[0] is 0). `r.sorted`
// holds the stable descending order of the query's scores (k_rank_sort).
__global__ void __launch_bounds__(128) k_ndcg(DRank r, const float* label, const int32_t* ks, int32_t nk,
                                              double* out) {
  for (int32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < r.nq; q += gridDim.x * blockDim.x) {
    const int32_t b0 = r.bnd[q], cnt = r.bnd[q + 1] - b0;
    const float* lb = label + b0;
    const uint32_t* sorted = r.sorted + b0;
    double* o = out + (size_t)q * nk;
    // dcg.rs max_dcg_at_k for each k, from the label counts
    bool first_ok = true;
    for (int32_t j = 0; j < nk; ++j) {
      int32_t counts[31];
      for (int v = 0; v < 31; ++v) counts[v] = 0;
      for (int32_t i = 0; i < cnt; ++i) counts[(int32_t)lb[i]] += 1;
      int32_t top = 30;
      double v = 0.0;
      const int32_t kk = min(ks[j], cnt);
      for (int32_t i = 0; i < kk; ++i) {
        while (top > 0 && counts[top] <= 0) top -= 1;
        v += r.discount[i] * r.label_gain[top];
        counts[top] -= 1;
      }
      o[j] = v > 0.0 ? 1.0 / v : -1.0;  // the inverse for now
      if (j == 0) first_ok = o[0] > 0.0;
    }
    if (!first_ok) {
      for (int32_t j = 0; j < nk; ++j) o[j] = 1.0;
      continue;
    }
    double cur = 0.0;
    int32_t left = 0;
    for (int32_t j = 0; j < nk; ++j) {
      const int32_t kk = min(ks[j], cnt);
      for (int32_t i = left; i < kk; ++i) cur += r.label_gain[(int32_t)lb[sorted[i]]] * r.discount[i];
      o[j] = cur * o[j];
      left = kk;
    }
  }
}

Status launch_ndcg(const DRank& r, const float* label, const double* score, const int32_t* ks, int32_t nk,
                   double* out, int sms, cudaStream_t s) {
  if (r.nq == 0) return Status();
  const int sort_grid = (int)std::min<int64_t>(r.nq, (int64_t)sms * 16);
  k_rank_sort<<<sort_grid, kRankThreads, 0, s>>>(r, score);
  CU_LAUNCH();
  const int grid = (int)std::max<int64_t>(1, std::min<int64_t>((r.nq + 127) / 128, (int64_t)sms * 16));
  k_ndcg<<<grid, 128, 0, s>>>(r, label, ks, nk, out);
  CU_LAUNCH();
  return Status();
}

Status RankTables::build(const float* label_h, const int32_t* bnd_h, int32_t nq_, double sigmoid, int32_t trunc,
                         bool norm) {
  nq = nq_;
  const int64_t n = bnd_h[nq];
  for (int32_t q = 0; q < nq; ++q)
    if (bnd_h[q + 1] < bnd_h[q]) return Status(LGBM_B200_ERR_INVALID_DATA, "query boundaries must not decrease");
  // dcg.rs: label gains 2^i - 1 and discounts 1 / log2(2 + i)
  std::vector<double> label_gain, discount;
  label_gain.push_back(0.0);
  for (int i = 1; i < 31; ++i) label_gain.push_back((double)((1 << i) - 1));
  for (int i = 0; i < kRankMaxQuery; ++i) discount.push_back(1.0 / std::log2(2.0 + (double)i));
  for (int64_t i = 0; i < n; ++i) {
    const float l = label_h[i];
    if (!(l >= 0.0f) || (int32_t)l >= (int32_t)label_gain.size())
      return Status(LGBM_B200_ERR_INVALID_DATA, "lambdarank labels must be integers in [0, 30]");
  }
  // inverse max DCG at the truncation level per query (rank.rs:140-156)
  std::vector<double> inv((size_t)nq);
  const size_t k = (size_t)std::max(trunc, 0);
  for (int32_t q = 0; q < nq; ++q) {
    const size_t cnt_q = (size_t)(bnd_h[q + 1] - bnd_h[q]);
    if (cnt_q > (size_t)kRankMaxQuery)
      return Status(LGBM_B200_ERR_UNSUPPORTED, "a query holds more than 10000 rows");
    std::vector<int32_t> cnt(label_gain.size(), 0);
    for (size_t i = 0; i < cnt_q; ++i) cnt[(int32_t)label_h[bnd_h[q] + i]] += 1;
    int32_t top = (int32_t)label_gain.size() - 1;
    double v = 0.0;
    for (size_t j = 0; j < std::min(k, cnt_q); ++j) {
      while (top > 0 && cnt[top] <= 0) top -= 1;
      if (top < 0) break;
      v += discount[j] * label_gain[top];
      cnt[top] -= 1;
    }
    inv[(size_t)q] = v > 0.0 ? 1.0 / v : v;
  }
  // the sigmoid table (rank.rs:162-176)
  double min_in = -50.0 / sigmoid / 2.0;
  double max_in = -min_in;
  double idx_factor = (double)kRankSigmoidBins / (max_in - min_in);
  std::vector<double> table((size_t)kRankSigmoidBins);
  for (size_t i = 0; i < (size_t)kRankSigmoidBins; ++i) {
    double score = (double)i / idx_factor + min_in;
    table[i] = 1.0 / (1.0 + std::exp(score * sigmoid));
  }
  // the queries with rows, those of more than kRankSmall first
  std::vector<int32_t> query;
  for (int large = 1; large >= 0; --large) {
    for (int32_t q = 0; q < nq; ++q) {
      const int32_t rows = bnd_h[q + 1] - bnd_h[q];
      if (rows > 0 && (rows > kRankSmall) == (large != 0)) query.push_back(q);
    }
    if (large) d.num_large = (int32_t)query.size();
  }
  d.num_small = (int32_t)query.size() - d.num_large;
  // one block, each array on a 256-byte boundary
  size_t bytes = 0;
  auto take = [&](size_t b) {
    const size_t o = bytes;
    bytes += (std::max<size_t>(b, 1) + 255) / 256 * 256;
    return o;
  };
  const size_t rows = (size_t)n;
  const size_t at_bnd = take(sizeof(int32_t) * ((size_t)nq + 1)), at_query = take(sizeof(int32_t) * query.size()),
               at_inv = take(sizeof(double) * (size_t)nq), at_table = take(sizeof(double) * table.size()),
               at_gain = take(sizeof(double) * label_gain.size()), at_disc = take(sizeof(double) * discount.size()),
               at_sorted = take(sizeof(uint32_t) * rows), at_score = take(sizeof(double) * rows),
               at_sgain = take(sizeof(double) * rows), at_label = take(sizeof(float) * rows);
  arena.free_all();
  unsigned char* block = nullptr;
  Status s = arena.alloc_n(&block, bytes);
  if (!s.ok()) return s;
  auto send = [&](size_t at, const void* src, size_t b) {
    return b ? cudaMemcpy(block + at, src, b, cudaMemcpyHostToDevice) : cudaSuccess;
  };
  CU(send(at_bnd, bnd_h, sizeof(int32_t) * ((size_t)nq + 1)));
  CU(send(at_query, query.data(), sizeof(int32_t) * query.size()));
  CU(send(at_inv, inv.data(), sizeof(double) * inv.size()));
  CU(send(at_table, table.data(), sizeof(double) * table.size()));
  CU(send(at_gain, label_gain.data(), sizeof(double) * label_gain.size()));
  CU(send(at_disc, discount.data(), sizeof(double) * discount.size()));
  d.bnd = reinterpret_cast<const int32_t*>(block + at_bnd);
  d.query = reinterpret_cast<const int32_t*>(block + at_query);
  d.nq = nq;
  d.inv_max_dcg = reinterpret_cast<const double*>(block + at_inv);
  d.sigmoid_table = reinterpret_cast<const double*>(block + at_table);
  d.label_gain = reinterpret_cast<const double*>(block + at_gain);
  d.discount = reinterpret_cast<const double*>(block + at_disc);
  d.sorted = reinterpret_cast<uint32_t*>(block + at_sorted);
  d.sorted_score = reinterpret_cast<double*>(block + at_score);
  d.sorted_gain = reinterpret_cast<double*>(block + at_sgain);
  d.sorted_label = reinterpret_cast<float*>(block + at_label);
  d.sigmoid = sigmoid;
  d.min_in = min_in;
  d.max_in = max_in;
  d.idx_factor = idx_factor;
  d.truncation_level = trunc;
  d.norm = norm ? 1 : 0;
  return Status();
}

Status launch_lambdarank(const DRank& r, const float* label, const double* score, float* g, float* h, float2* gh,
                         cudaStream_t s) {
  if (r.nq == 0) return Status();
  const int64_t grid = r.num_large + ((int64_t)r.num_small + kRankSmallPerCta - 1) / kRankSmallPerCta;
  if (grid == 0) return Status();
  k_lambdarank<<<(unsigned)grid, kRankThreads, 0, s>>>(r, score, label, g, h, gh);
  CU_LAUNCH();
  return Status();
}

}  // namespace lgbm_b200
