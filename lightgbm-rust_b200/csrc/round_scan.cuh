// The threshold scans of a growth round: both children of every expanded
// node, all features, in one launch (included by round_kernels.cuh).
//
// A round searches up to 256 nodes (43 of a 255-leaf tree) x 2 children x
// features at once, so unlike a single split step it is bound by throughput:
// what counts is work per warp instruction, not the latency of one scan.
//
//   quantized   one warp per scan: the views are loaded coalesced, and packed
//               integer sums are exact in any order (a warp prefix).
//   FP64        one warp per scan: the cumulative sums must be added in the
//               reference's order, serial chains of up to 255 adds, which four
//               lanes run side by side (gradients and hessians of both
//               directions); everything else is spread over the 32 lanes.
//
// Both evaluate the gain of every admissible threshold in FP32 first and in
// FP64 only where the FP32 value is within 1e-5 of the largest: the FP32
// value's relative error is below 1e-6 (four roundings and an approximate
// divide), so the FP64 maximum and its ties are always among those, and the
// result is the FP64 search's bit for bit. (Only the largest gain decides
// whether a feature is splittable.) The bound needs divisors well inside
// FP32's range and a largest gain above 1e-30: a square below FP32's normal
// numbers is off by up to 2^-150, and over a divisor of 1e-8 or more by 7e-38,
// which 1e-5 of such a gain covers; the approximate divide returns 0 from a
// divisor of 2^126 on. The least hessian sum of a leaf usually says so for a
// whole scan (a test of each estimate cost multiclass trees 2%); else the
// admissible thresholds are tested, and one outside has all evaluated in FP64.
// Parameters that change the gain's formula (L1, max_delta_step, path
// smoothing, monotone bounds) evaluate all in FP64.
#pragma once

// FP32 estimate of the plain gain of a threshold.
__device__ __forceinline__ float gain_estimate(float lg, float lh, float rg, float rh, float l2) {
  return __fdividef(lg * lg, lh + l2) + __fdividef(rg * rg, rh + l2);
}
// Whether the estimates hold for divisors lh + l2 and rh + l2.
__device__ __forceinline__ bool divisors_safe(float lh, float rh, float l2) {
  return fminf(lh, rh) + l2 >= 1e-8f && fmaxf(lh, rh) + l2 <= 1e37f;
}
// Whether they hold for every admissible threshold of a leaf whose hessians sum up to `total`.
__device__ __forceinline__ bool scan_safe(const DParams& p, double total) {
  return p.min_sum_hessian_in_leaf + p.lambda_l2 >= 2e-8 && total + p.lambda_l2 <= 1e36;
}
// The estimates from which a threshold is evaluated in FP64, given the
// largest: all of them when it is outside FP32's comfortable range.
__device__ __forceinline__ float estimate_floor(float most) {
  const float a = fabsf(most);
  return a > 1e-30f && a < 1e37f ? most - 1e-5f * a : -INFINITY;
}

// The job of leaf side `side` (0: the smaller child) of expansion e, item i
// of the round, up to its output; child: the node it fills.
__device__ __forceinline__ ScanJob round_job(const DCtx& c, const DSlot& s, bool root, int32_t e, int side,
                                             int32_t& child, int32_t& parent, int32_t& depth) {
  const DRounds& r = s.r;
  const int32_t a = root ? 0 : 2 * e + 1, b = root ? 0 : 2 * e + 2;
  const RNode &na = r.node[a], &nb = r.node[b];
  const bool left_smaller = na.ls.num_data < nb.ls.num_data;
  const RNode &sm = left_smaller ? na : nb, &lg = left_smaller ? nb : na;
  const RNode& me = side == 0 ? sm : lg;
  child = (side == 0) == left_smaller ? a : b;
  parent = na.parent;
  depth = na.depth;
  ScanJob j;
  j.sl = sm.ls;
  j.ls = me.ls;
  j.s_buf = sm.buf;
  j.l_buf = lg.buf;
  j.live = na.need != 0;
  j.root = root;
  j.cmin = me.cmin;
  j.cmax = me.cmax;
  j.gsc = s.st->grad_scale;
  j.hsc = s.st->hess_scale;
  j.out = nullptr;
  return j;
}

// The best split of a new node over its features (learner/mod.rs:842-849,
// :1066-1086), by one warp, once every feature's scan is stored.
__device__ void round_best(const DCtx& c, const DSlot& s, int slot, int32_t child, int32_t depth) {
  const DRounds& r = s.r;
  const int lane = threadIdx.x & 31;
  const int32_t nf = c.num_features;
  const DSplit* res = r.fres + (size_t)slot * nf;
  const double pen = c.p.use_monotone ? monotone_split_gain_penalty(depth, c.p.monotone_penalty) : 1.0;
  double bg = -INFINITY;
  int32_t bfeat = -1, bf = -1;
  for (int f = lane; f < nf; f += 32) {  // other CTAs' results: loaded through L2
    double g = __ldcg(&res[f].gain);
    const int32_t fe = __ldcg(&res[f].feature);
    if (__ldcg(&res[f].monotone_type) != 0) g *= pen;
    if (better_than(g, fe, bg, bfeat)) {
      bg = g;
      bfeat = fe;
      bf = f;
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    const double og = __shfl_xor_sync(0xffffffffu, bg, o);
    const int32_t ofe = __shfl_xor_sync(0xffffffffu, bfeat, o);
    const int32_t of = __shfl_xor_sync(0xffffffffu, bf, o);
    if (better_than(og, ofe, bg, bfeat)) {
      bg = og;
      bfeat = ofe;
      bf = of;
    }
  }
  if (bf < 0) return;  // the node keeps its gain of -inf
  const uint32_t* from = reinterpret_cast<const uint32_t*>(res + bf);
  uint32_t* to = reinterpret_cast<uint32_t*>(r.best + child);
  for (int i = lane; i < (int)(sizeof(DSplit) / 4); i += 32) to[i] = __ldcg(from + i);
  __syncwarp();
  if (lane == 0) {
    r.best[child].gain = bg;
    r.gain[child] = bg;
    r.feat[child] = bfeat;
  }
}

// `count` more scans of item side q are stored by this warp; the warp that
// stores the last one picks the node's best split.
__device__ __forceinline__ void scans_stored(const DCtx& c, const DSlot& s, int q, int count, int32_t child,
                                             int32_t depth) {
  int last = 0;
  __syncwarp();
  if ((threadIdx.x & 31) == 0) {
    // releases this warp's results, and acquires the others' for the last
    int32_t before;
    asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], %2;"
                 : "=r"(before)
                 : "l"(&s.r.scan_cnt[q]), "r"(count)
                 : "memory");
    last = before + count == c.num_features;
  }
  __syncwarp();
  last = __shfl_sync(0xffffffffu, last, 0);
  if (last) round_best(c, s, q, child, depth);
  __syncwarp();
}

// ---- quantized: one warp per (node, feature) ------------------------------------------

// A view in shared memory: bin t at element t + t / 8, so that lane l's bins
// 8l .. 8l + 7 and 32 consecutive bins both fall into different banks.
constexpr int kViewPad = kMaxBins + kMaxBins / kPer;
__device__ __forceinline__ int view_at(int t) { return t + (t >> 3); }

// Scratch of a categorical scan by one warp.
struct CatScratch {
  int64_t ig[kMaxBins];
  double key[kMaxBins];
  int32_t tpos[kMaxBins], sorted[kMaxBins];
};

// The accumulated hessian integers a threshold may have: [lo, hi], hi < lo
// when there are none. Where counts and hessian sums only grow in scan order,
// a threshold passes the reference's data and hessian minima on both sides
// exactly within a range, which depends on the leaf alone. They need not grow:
// the reference sums the root's packed values by position when it bags
// (quant.rs:452-477), so the most frequent bin, which takes what the other
// bins leave of that sum, can hold a negative hessian.
struct HessRange {
  uint32_t lo, hi;
};

// The first H in [0, last] for which pred holds (it then holds for every
// larger one), last + 1 if none; by one warp, which tests 32 values at once
// around `guess` and searches 32-fold when the guess is off.
template <class Pred>
__device__ __forceinline__ long long first_true(long long last, float guess, Pred pred) {
  const int lane = threadIdx.x & 31;
  long long g = (long long)guess - 15;
  g = g < 0 ? 0 : (g > last ? last : g);
  unsigned m = __ballot_sync(0xffffffffu, g + lane > last || pred((uint32_t)(g + lane)));
  if (m != 0 && (g == 0 || !(m & 1))) return g + __ffs(m) - 1;
  long long lo = 0, n = last + 1;  // the answer lies in [lo, lo + n]
  while (n > 0) {
    const long long step = (n + 31) / 32;
    const long long h = lo + step * (lane + 1) - 1;
    m = __ballot_sync(0xffffffffu, h >= lo + n || pred((uint32_t)h));
    const int k = m ? __ffs(m) - 1 : 32;  // [lo + step k, lo + step (k + 1)) holds it
    const long long end = min(lo + n, lo + step * (k + 1) - 1);
    lo = min(lo + n, lo + step * k);
    n = max(0LL, end - lo);
  }
  return lo;
}

__device__ __forceinline__ HessRange admissible_hess(const DParams& p, const LeafCtx& lc, double cnt_factor) {
  const uint32_t sum = int_hess(lc.int_sum);
  const double hs = lc.hs, min_hess = p.min_sum_hessian_in_leaf;
  const int32_t min_data = p.min_data_in_leaf, n = lc.num_data;
  const float cf = (float)cnt_factor, by_hess = __fdividef((float)min_hess, (float)hs);
  const long long lo =
      first_true(sum, fmaxf(__fdividef((float)min_data - 0.5f, cf), by_hess), [&](uint32_t h) {
        return round_int((double)h * cnt_factor) >= min_data && (double)h * hs >= min_hess;
      });
  const long long past =
      first_true(sum, fminf(__fdividef((float)(n - min_data) + 0.5f, cf), (float)sum - by_hess), [&](uint32_t h) {
        return n - round_int((double)h * cnt_factor) < min_data || (double)(sum - h) * hs < min_hess;
      });
  if (past == 0 || lo > (long long)sum) return HessRange{1, 0};
  return HessRange{(uint32_t)lo, (uint32_t)(past - 1)};
}

// The admissible thresholds of a view whose packed sums do not only grow, by
// the reference's tests one by one: too little on the accumulated side passes
// over a threshold, on the other side it ends the scan. Bit j of the result is
// bin 8 lane + j (t_lo .. t_hi except skip_t are visited), bit 8, on lane 0, the
// extra candidate before them (extra; its sum is base). One warp; out of line
// for its registers, and the sums formed again, since bagged trees alone come
// here.
__device__ __noinline__ uint32_t admissible_one_by_one(const int64_t* view, int32_t t_lo, int32_t t_hi, int32_t skip_t,
                                                       bool reverse, bool extra, uint64_t base, uint64_t sum, double hs,
                                                       int32_t num_data, double cnt_factor, int32_t min_data,
                                                       double min_hess) {
  const int lane = threadIdx.x & 31;
  auto visited = [&](int t) { return t >= t_lo && t <= t_hi && t != skip_t; };
  uint64_t pre = 0;
  for (int j = 0; j < kPer; ++j)
    if (visited(lane * kPer + j)) pre += (uint64_t)view[view_at(lane * kPer + j)];
  uint64_t run = pre;
  for (int o = 1; o < 32; o <<= 1) {
    const uint64_t other = __shfl_up_sync(0xffffffffu, run, o);
    if (lane >= o) run += other;
  }
  // the sum before this lane's bins in scan order
  run = reverse ? __shfl_sync(0xffffffffu, run, 31) - run : base + run - pre;
  uint32_t pend = 0;
  int32_t brk = reverse ? INT32_MIN : INT32_MAX;
  auto test = [&](uint64_t a, int32_t t) {
    const double h = (double)int_hess((int64_t)a);
    const int32_t ac = round_int(h * cnt_factor);
    if (ac < min_data || h * hs < min_hess) return false;
    const bool end = num_data - ac < min_data || (double)int_hess((int64_t)(sum - a)) * hs < min_hess;
    if (end) brk = reverse ? max(brk, t) : min(brk, t);
    return !end;
  };
  for (int i = 0; i < kPer; ++i) {
    const int j = reverse ? kPer - 1 - i : i, t = lane * kPer + j;
    if (!visited(t)) continue;
    run += (uint64_t)view[view_at(t)];
    if (test(run, t)) pend |= 1u << j;
  }
  if (extra && test(base, -1)) pend |= 1u << kPer;
  brk = reverse ? __reduce_max_sync(0xffffffffu, brk) : __reduce_min_sync(0xffffffffu, brk);
  for (int j = 0; j < kPer; ++j) {
    const int t = lane * kPer + j;
    if (reverse ? t <= brk : t >= brk) pend &= ~(1u << j);
  }
  return pend;
}

// One direction of the quantized scan (split.rs:995-1190) by one warp, over
// the view in shared memory (its most frequent bin fixed).
__device__ __forceinline__ bool scan_direction_packed(const int64_t* view, const DFeature& m, const DParams& p,
                                                      const LeafCtx& lc, const HessRange& range, double min_gain_shift,
                                                      double cnt_factor, bool reverse, bool skip_default,
                                                      bool na_as_missing, DSplit& out) {
  const int lane = threadIdx.x & 31;
  const int offset = m.offset;
  const int len = m.view_len;
  int32_t t_lo, t_hi;
  if (reverse) {
    t_hi = m.num_bin - 1 - offset - (int32_t)na_as_missing;
    t_lo = 1 - offset;
  } else {
    t_lo = 0;
    t_hi = m.num_bin - 2 - offset;
  }
  t_hi = min(t_hi, len - 1);
  const int32_t skip_t = skip_default ? m.default_bin - offset : INT32_MIN;
  const bool first_extra = !reverse && na_as_missing && offset == 1;
  const uint64_t sum = (uint64_t)lc.int_sum;
  const bool plain = plain_split(p, lc.mc);
  uint64_t x[kPer];
  uint32_t visited = 0;
  uint64_t pre = 0, all = 0;
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    const int t = lane * kPer + j;
    x[j] = (uint64_t)view[view_at(t)];
    if (first_extra && t < len) all += x[j];
    if (t >= t_lo && t <= t_hi && t != skip_t) {
      visited |= 1u << j;
      pre += x[j];
    } else {
      x[j] = 0;
    }
  }
  uint64_t incl = pre;  // inclusive over lanes of this lane's visited sum
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint64_t other = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += other;
  }
  uint64_t base = 0;
  if (first_extra) {  // split.rs:1097-1103: the leaf sum minus every stored bin
    for (int o = 16; o > 0; o >>= 1) all += __shfl_xor_sync(0xffffffffu, all, o);
    base = sum - all;
  }
  // the packed sum of the accumulated side at bin j is start + run
  // (ascending: the visited bins up to j; descending: the visited bins from
  // j up, the total minus those below)
  uint64_t q[kPer];
  {
    uint64_t run = incl - pre;
    if (reverse) {
      run = __shfl_sync(0xffffffffu, incl, 31) - run;
#pragma unroll
      for (int j = 0; j < kPer; ++j) {
        q[j] = run;
        run -= x[j];
      }
    } else {
      run += base;
#pragma unroll
      for (int j = 0; j < kPer; ++j) {
        run += x[j];
        q[j] = run;
      }
    }
  }
  const float gsf = (float)lc.gs, hsf = (float)lc.hs, l2f = (float)p.lambda_l2 + (float)kEpsilon;
  auto estimate = [&](uint64_t a) {
    const uint64_t rest = sum - a;
    return gain_estimate((float)int_grad((int64_t)a) * gsf, (float)int_hess((int64_t)a) * hsf,
                         (float)int_grad((int64_t)rest) * gsf, (float)int_hess((int64_t)rest) * hsf, l2f);
  };
  // which thresholds are admissible (extra: the candidate t = -1, lane 0's)
  uint32_t pend = 0;
  bool extra = first_extra && lane == 0;
  bool falls = (base >> 31 & 1) != 0;  // a negative hessian: the sums do not only grow
#pragma unroll
  for (int j = 0; j < kPer; ++j) falls |= (x[j] >> 31 & 1) != 0;
  if (!__any_sync(0xffffffffu, falls)) {
    auto admissible = [&](uint64_t a) {
      const uint32_t h = int_hess((int64_t)a);
      return h >= range.lo && h <= range.hi;
    };
#pragma unroll
    for (int j = 0; j < kPer; ++j)
      if ((visited >> j & 1) && admissible(q[j])) pend |= 1u << j;
    extra = extra && admissible(base);
  } else {
    pend = admissible_one_by_one(view, t_lo, t_hi, skip_t, reverse, extra, base, sum, lc.hs, lc.num_data, cnt_factor,
                                 p.min_data_in_leaf, p.min_sum_hessian_in_leaf);
    extra = pend >> kPer & 1;
    pend &= (1u << kPer) - 1;
  }
  // their estimates
  float est[kPer];
  float most = -INFINITY;
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    est[j] = estimate(q[j]);
    if (pend >> j & 1) most = fmaxf(most, est[j]);
  }
  if (extra) most = fmaxf(most, estimate(base));
  if (!__any_sync(0xffffffffu, pend != 0 || extra)) return false;
  if (!scan_safe(p, 4294967296.0 * lc.hs)) {  // a packed hessian is 32 bits, whatever the leaf's sum
    auto safe = [&](uint64_t a) {
      return divisors_safe((float)int_hess((int64_t)a) * hsf, (float)int_hess((int64_t)(sum - a)) * hsf, l2f);
    };
#pragma unroll
    for (int j = 0; j < kPer; ++j)
      if ((pend >> j & 1) && !safe(q[j])) most = INFINITY;  // no floor
    if (extra && !safe(base)) most = INFINITY;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, o));
  const float floor = plain ? estimate_floor(most) : -INFINITY;
#pragma unroll
  for (int j = 0; j < kPer; ++j)
    if (est[j] < floor) pend &= ~(1u << j);
  // FP64 gains
  double best_gain = -INFINITY;
  int32_t best_t = INT32_MIN;
  bool splittable = false;
  uint64_t wq = 0;  // this lane's best candidate's packed sum
  auto consider = [&](int t, uint64_t a) {
    const int64_t rest = (int64_t)(sum - a);
    const int32_t ac = round_int((double)int_hess((int64_t)a) * cnt_factor), rc = lc.num_data - ac;
    const double ga = (double)int_grad((int64_t)a) * lc.gs, gr = (double)int_grad(rest) * lc.gs;
    const double ha = (double)int_hess((int64_t)a) * lc.hs + kEpsilon, hr = (double)int_hess(rest) * lc.hs + kEpsilon;
    // the left child is the rest when scanning in reverse
    const double g1 = reverse ? gr : ga, h1 = reverse ? hr : ha, g2 = reverse ? ga : gr, h2 = reverse ? ha : hr;
    const int32_t c1 = reverse ? rc : ac, c2 = reverse ? ac : rc;
    const double gain = split_gain_hot(plain, g1, h1, g2, h2, p, c1, c2, lc.parent_output, lc.mc, lc.cmin, lc.cmax,
                                       m.monotone_type);
    if (gain <= min_gain_shift) return;
    splittable = true;
    if (gain > best_gain || (gain == best_gain && best_t != INT32_MIN && (reverse ? t > best_t : t < best_t))) {
      best_gain = gain;
      best_t = t;
      wq = a;
    }
  };
  // a lane's admissible thresholds one at a time, the lanes side by side
  // (bit 8: the extra candidate)
  if (extra) pend |= 1u << kPer;
  while (__any_sync(0xffffffffu, pend != 0)) {
    if (pend) {
      const int j = __ffs(pend) - 1;
      pend &= pend - 1;
      uint64_t a = base;
#pragma unroll
      for (int k = 0; k < kPer; ++k)
        if (k == j) a = q[k];
      consider(j == kPer ? -1 : lane * kPer + j, a);
    }
  }
  warp_pick(reverse, best_gain, best_t);
  const bool any = __any_sync(0xffffffffu, splittable) != 0;
  ScanBest r;
  r.splittable = any;
  r.gain = best_gain;
  r.t = best_t;
  r.acc_g = r.acc_h = 0.0;
  // the winner's packed sum, from the lane whose best it was (the extra
  // candidate t = -1 is lane 0's)
  wq = __shfl_sync(0xffffffffu, wq, best_t >= 0 ? best_t / kPer : 0);
  r.acc_q = best_t == INT32_MIN ? 0 : (int64_t)wq;
  r.acc_c = 0;  // the packed form takes its counts from the sums
  apply_direction<true>(r, m, p, lc.sum_g, lc.sum_h, lc.int_sum, lc.gs, lc.hs, lc.num_data, lc.parent_output, lc.mc,
                        lc.cmin, lc.cmax, min_gain_shift, cnt_factor, reverse, out);
  __syncwarp();
  return any;
}

// find_best_threshold (split.rs:246-271, :930-950) of the quantized form for
// one leaf and feature, by one warp.
__device__ __forceinline__ bool find_best_threshold_packed(const int64_t* view, CatScratch* cat, const DFeature& m,
                                                           const DParams& p, const DParams& p_cat, const LeafCtx& lc,
                                                           DSplit& out) {
  const int lane = threadIdx.x & 31;
  if (lane == 0) {
    out.default_left = 1;
    out.gain = -INFINITY;
    out.num_cat = 0;
    out.monotone_type = m.bin_type == 1 ? 0 : m.monotone_type;
  }
  __syncwarp();
  bool ok = false;
  if (m.bin_type == 1) {
    for (int t = lane; t < m.view_len; t += 32) cat->ig[t] = view[view_at(t)];
    __syncwarp();
    ok = scan_categorical<true>(*cat, m, p, p_cat, lc, out);
  } else {
    const double sg = (double)int_grad(lc.int_sum) * lc.gs;
    const double sh = (double)int_hess(lc.int_sum) * lc.hs;
    const double min_gain_shift =
        leaf_gain_hot(plain_split(p, lc.mc), sg, sh, p, lc.num_data, lc.parent_output) + p.min_gain_to_split;
    const double cnt_factor = (double)lc.num_data / (double)int_hess(lc.int_sum);
    const HessRange range = admissible_hess(p, lc, cnt_factor);
    // split.rs:426-439: the directions scanned and their missing-value rules
    const bool two = m.num_bin > 2 && m.missing_type != 0;
    const bool skip_default = two && m.missing_type == 1;
    const bool na_missing = two && m.missing_type == 2;
#pragma unroll 1
    for (int d = 0; d < (two ? 2 : 1); ++d)
      ok |= scan_direction_packed(view, m, p, lc, range, min_gain_shift, cnt_factor, d == 0, skip_default, na_missing,
                                  out);
    if (!two && lane == 0 && m.missing_type == 2) out.default_left = 0;
  }
  __syncwarp();
  if (lane == 0) out.gain *= m.penalty;
  __syncwarp();
  return ok;
}

constexpr size_t kScanWarpViews = (kScanThreads / 32) * (kViewPad * sizeof(int64_t));
constexpr size_t kScanWarpBase = kScanWarpViews + (kScanThreads / 32) * sizeof(DSplit);
size_t round_scan_int_smem(bool cat) { return kScanWarpBase + (cat ? (kScanThreads / 32) * sizeof(CatScratch) : 0); }

// One quantized scan by one warp: feature f, side (0 smaller, 1 larger) of job
// j, whose histogram views are fixed, subtracted and stored; view, cat and out
// are the warp's shared memory. The result goes to *dst when the feature is
// searched (left in `out`, too); returns whether it is splittable.
__device__ __forceinline__ bool scan_packed(const DCtx& c, const DSlot& s, const DFeature& m, int32_t f, int side,
                                            const ScanJob& j, bool search, int64_t* view, CatScratch* cat, DSplit& out,
                                            DSplit* dst) {
  const int lane = threadIdx.x & 31;
  const int len = m.view_len;
  long long* hs = reinterpret_cast<long long*>(s.hist) + (size_t)j.s_buf * c.total_bins + m.view_start;
  long long* hp = reinterpret_cast<long long*>(s.hist) + (size_t)j.l_buf * c.total_bins + m.view_start;
  uint64_t v[kPer], pv[kPer];
#pragma unroll
  for (int k = 0; k < kPer; ++k) {
    const int t = 32 * k + lane;
    // histogram cells are written by other CTAs' atomics: loaded through L2
    v[k] = t < len ? (uint64_t)__ldcg(hs + t) : 0ull;
    pv[k] = t < len && side == 1 ? (uint64_t)__ldcg(hp + t) : 0ull;
  }
  if (!search) return false;
  // the smaller leaf's most frequent bin (histogram.rs:42-56; exact in any order)
  if (m.most_freq_bin > 0) {
    uint64_t part = 0;
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      const int t = 32 * k + lane;
      if (t < m.num_bin && t != m.most_freq_bin) part += v[k];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
    const uint64_t fixed = (uint64_t)j.sl.int_sum - part;
#pragma unroll
    for (int k = 0; k < kPer; ++k)
      if (32 * k + lane == m.most_freq_bin) {
        v[k] = fixed;
        if (side == 0) hs[m.most_freq_bin] = (long long)fixed;
      }
  }
#pragma unroll
  for (int k = 0; k < kPer; ++k) {
    const int t = 32 * k + lane;
    if (side == 1) {  // larger = parent - smaller, in the parent's buffer (histogram.rs:59-63)
      v[k] = pv[k] - v[k];
      if (t < len) hp[t] = (long long)v[k];
    }
    view[view_at(t)] = (int64_t)v[k];
  }
  __syncwarp();
  const bool ok = find_best_threshold_packed(view, cat, m, c.p, c.p_cat, leaf_ctx(c, j), out);
  if (lane == 0) {
    out.feature = m.real_index;
    out.inner = f;
  }
  __syncwarp();
  const uint32_t* src = reinterpret_cast<const uint32_t*>(&out);
  for (int k = lane; k < (int)(sizeof(DSplit) / 4); k += 32) reinterpret_cast<uint32_t*>(dst)[k] = src[k];
  return ok;
}

// Grid (G, 1, slots), kScanThreads threads: each warp takes scans of its own;
// neighbouring scans go to different CTAs, so a round of few scans spreads
// over the SMs.
__global__ void __launch_bounds__(kScanThreads, kScanIntBlocks) k_round_scan_int(const __grid_constant__ DCtx c) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int kWarps = kScanThreads / 32;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int64_t* view = reinterpret_cast<int64_t*>(smem_raw) + (size_t)warp * kViewPad;
  DSplit& out = reinterpret_cast<DSplit*>(smem_raw + kScanWarpViews)[warp];
  CatScratch* cat = reinterpret_cast<CatScratch*>(smem_raw + kScanWarpBase) + warp;
  const DSlot& s = c.slots[blockIdx.z];
  const DRounds& r = s.r;
  const int32_t nf = c.num_features;
  const bool root = r.st->root != 0;
  const int32_t n = root ? nf : r.st->nb * 2 * nf, e0 = r.st->e0;
  for (int32_t w = warp * gridDim.x + blockIdx.x; w < n; w += kWarps * gridDim.x) {
    const int32_t item = w / nf, f = w - item * nf, side = item & 1;
    const DFeature m = c.feats[f];
    const uint8_t in_tree = s.bytree[f];
    int32_t child, parent, depth;
    const ScanJob j = round_job(c, s, root, e0 + (item >> 1), side, child, parent, depth);
    if (!j.live) continue;
    const uint8_t split_ok = parent < 0 ? 1 : r.splittable[(size_t)parent * nf + f];
    const bool search = in_tree && split_ok;
    DSplit* dst = r.fres + ((size_t)item * nf + f);
    const bool ok = scan_packed(c, s, m, f, side, j, search, view, cat, out, dst);
    if (!search && lane == 0) {
      dst->gain = -INFINITY;
      dst->feature = -1;
      dst->monotone_type = 0;
    }
    if (lane == 0) r.splittable[(size_t)child * nf + f] = ok;
    scans_stored(c, s, item, 1, child, depth);
  }
}

// The scans of a split step, a warp each, in the place of k_scan where those
// would run in waves (data-parallel growth of quantized trees on many
// features: a block scan's 256 threads and barriers per scan are for few of
// them). Grid (G, 1, slots), kScanThreads threads.
__global__ void __launch_bounds__(kScanThreads, kScanIntBlocks) k_scan_warp(const __grid_constant__ DCtx c) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int kWarps = kScanThreads / 32;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int64_t* view = reinterpret_cast<int64_t*>(smem_raw) + (size_t)warp * kViewPad;
  DSplit& out = reinterpret_cast<DSplit*>(smem_raw + kScanWarpViews)[warp];
  CatScratch* cat = reinterpret_cast<CatScratch*>(smem_raw + kScanWarpBase) + warp;
  const DSlot& s = c.slots[blockIdx.z];
  const int32_t nf = c.num_features;
  // the partition that follows claims its row tiles from this counter
  if (blockIdx.x == 0 && threadIdx.x == 0 && !s.st->done) {
    s.st->part_ticket = 0;
    s.st->part_done = 0;
  }
  for (int32_t w = warp * gridDim.x + blockIdx.x; w < 2 * nf; w += kWarps * gridDim.x) {
    const int32_t side = w / nf, f = w - side * nf;
    const DFeature m = c.feats[f];
    int32_t larger_leaf, L;
    const ScanJob j = step_job(c, s, f, side, larger_leaf, L);
    if (!j.live) continue;
    if (!s.bytree[f] || (larger_leaf >= 0 && !s.splittable[L * nf + f])) continue;
    const bool ok = scan_packed(c, s, m, f, side, j, true, view, cat, out, j.out);
    if (lane == 0) s.feat_ok[w] = ok ? 1 : 0;
    // the partition's goes-left table for this candidate, ready if it wins
    if (ok) build_partition_lut(m, out, s.lut_cand + (size_t)w * kMaxBins, lane, 32);
    __syncwarp();
  }
}

// ---- FP64: one warp per scan ------------------------------------------------------------

// A warp's shared memory: the view's gradients and hessians, and the
// cumulative sums of both directions (reverse g, h, forward g, h). Values
// move in 16-byte pairs. A pair of padding after every 16 values lets lanes
// on consecutive groups of 8 meet different banks and leaves a chain's
// addresses constant offsets (pairs permuted by their chunk took 15.5 cycles
// a value, this 9.9); one more after the last lets the four lanes that walk
// the four sums side by side meet different banks too.
constexpr int kF64Chunk = 16;  // values of a chain's step
constexpr int kF64Pad = kMaxBins + 2 * (kMaxBins / kF64Chunk) + 2;
static_assert(kF64Pad % 16 == 2, "the arrays start one 16-byte bank apart");
struct __align__(16) F64Scratch {
  double view[2][kF64Pad];
  double cum[4][kF64Pad];
};
__device__ __forceinline__ int f64_at(int t) { return t + 2 * (t >> 4); }
// Values 8 * seg .. 8 * seg + 7.
__device__ __forceinline__ void f64_load8(const double* x, int seg, double (&v)[kPer]) {
  static_assert(kPer == 8 && kF64Chunk == 16, "two groups a chunk");
  const double2* q = reinterpret_cast<const double2*>(x + f64_at(kPer * seg));
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const double2 two = q[i];
    v[2 * i] = two.x;
    v[2 * i + 1] = two.y;
  }
}
// A categorical scan's scratch, in the place of the cumulative sums.
struct CatScratchF64 {
  double g[kMaxBins], h[kMaxBins], key[kMaxBins];
  int32_t tpos[kMaxBins], sorted[kMaxBins];
};
static_assert(sizeof(CatScratchF64) <= sizeof(F64Scratch::cum), "the scratch overlays the sums");
constexpr int kF64Warps = kF64ScanThreads / 32;
size_t round_scan_f64_smem() { return kF64Warps * (sizeof(F64Scratch) + sizeof(DSplit)); }

// Thresholds a direction visits: t in [lo, hi] except skip.
struct ScanSpan {
  int32_t lo, hi, skip;
  __device__ __forceinline__ bool has(int t) const { return t >= lo && t <= hi && t != skip; }
};
__device__ __forceinline__ ScanSpan scan_span(const DFeature& m, bool reverse, bool skip_default, bool na_as_missing) {
  ScanSpan v;
  if (reverse) {
    v.hi = m.num_bin - 1 - m.offset - (int32_t)na_as_missing;
    v.lo = 1 - m.offset;
  } else {
    v.lo = 0;
    v.hi = m.num_bin - 2 - m.offset;
  }
  v.hi = min(v.hi, m.view_len - 1);
  v.skip = skip_default ? m.default_bin - m.offset : INT32_MIN;
  return v;
}

// Chunks of kF64Chunk values that hold a view.
__device__ __forceinline__ int f64_chunks(int len) { return (len + kF64Chunk - 1) / kF64Chunk; }

// A serial chain of adds (kMinus: subtractions) over `chunks` chunks of
// kF64Chunk values of x, in order, each replaced by its running value if
// kStore. Values that take no part are zeros (a running sum here is never
// -0.0, so adding zero changes nothing), which leaves an add and half a
// 16-byte load and store per value: with the visited tests in the loop a
// chain took 45 cycles a value. Half a chunk is loaded while the other half
// is added. Only the lanes with a chain of their own come here: a 16-byte
// access of 32 lanes is four wavefronts even when they name the same four
// addresses, and the shared-memory pipe is what a full round is bound by (60%
// of its peak with scalar accesses of arrays whose starts shared a bank). An
// FP64 add takes 8.2 cycles to its result, a value of the chain 9.5. Scans of
// an iteration of 1M x 100 with 255 leaves 1238 -> 710 us, the iteration 3.04
// -> 2.44 ms.
template <bool kMinus, bool kStore>
__device__ __noinline__ double f64_chain(double a, double* x, int chunks) {
  double2* q = reinterpret_cast<double2*>(x);
  double2 lo[4], hi[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) lo[i] = q[i];
  auto add = [&](double2& two) {
    two.x = a = kMinus ? a - two.x : a + two.x;
    two.y = a = kMinus ? a - two.y : a + two.y;
  };
  for (int k = 0; k < chunks; ++k, q += kF64Chunk / 2 + 1) {
#pragma unroll
    for (int i = 0; i < 4; ++i) hi[i] = q[4 + i];
#pragma unroll
    for (int i = 0; i < 4; ++i) add(lo[i]);
    if constexpr (kStore) {
#pragma unroll
      for (int i = 0; i < 4; ++i) q[i] = lo[i];
    }
    // past the last chunk: the array, the split records or the warp after, not used
#pragma unroll
    for (int i = 0; i < 4; ++i) lo[i] = q[kF64Chunk / 2 + 1 + i];
#pragma unroll
    for (int i = 0; i < 4; ++i) add(hi[i]);
    if constexpr (kStore) {
#pragma unroll
      for (int i = 0; i < 4; ++i) q[4 + i] = hi[i];
    }
  }
  return a;
}

// The cumulative sums of both directions in the reference's order
// (split.rs:676-891), four serial chains side by side: lane 0 adds the
// gradients in reverse, lane 1 the hessians, lanes 2 and 3 the same forward
// (two: both directions are scanned). The forward chain starts, for a feature
// with NaN missing and no stored bin 0, from the leaf's sums minus every
// stored bin (split.rs:787-800), which base_g / base_h return. Past its length
// the view holds zeros. The reverse sums of bin t lie at place
// kF64Chunk * chunks - 1 - t, so that all lanes run forward.
__device__ __forceinline__ void f64_chains(F64Scratch& sm, const LeafCtx& lc, const ScanSpan& rev, const ScanSpan& fwd,
                                           int len, bool two, bool first_extra, double& base_g, double& base_h) {
  const int lane = threadIdx.x & 31;
  const bool forward = (lane & 3) >= 2 && two, hess = lane & 1;
  const int chunks = f64_chunks(len), last = kF64Chunk * chunks - 1;
#pragma unroll
  for (int k = 0; k < kPer; ++k) {
    const int t = 32 * k + lane;
    if (t > last) continue;
    const double g = sm.view[0][f64_at(t)], h = sm.view[1][f64_at(t)];
    sm.cum[0][f64_at(last - t)] = rev.has(t) ? g : 0.0;
    sm.cum[1][f64_at(last - t)] = rev.has(t) ? h : 0.0;
    if (two) {
      sm.cum[2][f64_at(t)] = fwd.has(t) ? g : 0.0;
      sm.cum[3][f64_at(t)] = fwd.has(t) ? h : 0.0;
    }
  }
  double a = hess ? kEpsilon : 0.0;
  if (first_extra) {
    double b = 0.0;
    if (lane < 4) b = f64_chain<true, false>(hess ? lc.sum_h - kEpsilon : lc.sum_g, sm.view[hess], chunks);
    if (forward) a = b;
    base_g = __shfl_sync(0xffffffffu, b, 2);
    base_h = __shfl_sync(0xffffffffu, b, 3);
  }
  __syncwarp();
  if (lane < (two ? 4 : 2)) f64_chain<false, true>(a, sm.cum[(forward ? 2 : 0) + hess], chunks);
  __syncwarp();
}

// One direction of FindBestThresholdSequentially (split.rs:676-891) by one
// warp, lane l on bins 8l .. 8l + 7, over the cumulative sums in cg / ch
// (f64_chains).
__device__ __forceinline__ bool scan_direction_f64(const double* cg, const double* ch, const double* view_h,
                                                   const ScanSpan& span, const DFeature& m, const DParams& p,
                                                   const LeafCtx& lc, double min_gain_shift, double cnt_factor,
                                                   bool reverse, bool first_extra, double base_g, double base_h,
                                                   DSplit& out) {
  const int lane = threadIdx.x & 31;
  const int len = m.view_len;
  const int32_t min_data = p.min_data_in_leaf;
  const double min_hess = p.min_sum_hessian_in_leaf;
  const bool plain = plain_split(p, lc.mc);
  const float l2f = (float)p.lambda_l2;
  // count estimates: each bin's rounded on its own, their sums exact in any order
  int32_t n[kPer], pre = 0, all = 0;
  uint32_t visited = 0;
  double a[kPer], b[kPer];
  f64_load8(view_h, lane, b);
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    const int t = lane * kPer + j;
    const int32_t ce = t < len ? round_int(b[j] * cnt_factor) : 0;
    if (first_extra) all += ce;
    n[j] = 0;
    if (span.has(t)) {
      visited |= 1u << j;
      n[j] = ce;
      pre += ce;
    }
  }
  int32_t incl = pre;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int32_t other = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += other;
  }
  int32_t base_n = 0;
  if (first_extra) base_n = lc.num_data - __reduce_add_sync(0xffffffffu, all);
  {
    int32_t run = incl - pre;
    if (reverse) {
      run = __shfl_sync(0xffffffffu, incl, 31) - run;
#pragma unroll
      for (int j = 0; j < kPer; ++j) {
        const int32_t x = n[j];
        n[j] = run;
        run -= x;
      }
    } else {
      run += base_n;
#pragma unroll
      for (int j = 0; j < kPer; ++j) {
        run += n[j];
        n[j] = run;
      }
    }
  }
  // thresholds with enough on the accumulated side; the first in scan order
  // with too little on the other ends the scan
  auto low = [&](double b, int32_t c) { return c < min_data || b < min_hess; };
  auto ends = [&](double b, int32_t c) { return lc.num_data - c < min_data || lc.sum_h - b < min_hess; };
  auto estimate = [&](double a, double b) {
    return gain_estimate((float)a, (float)b, (float)(lc.sum_g - a), (float)(lc.sum_h - b), l2f);
  };
  {  // the reverse sums lie mirrored (f64_chains)
    const int segs = f64_chunks(len) * (kF64Chunk / kPer);
    const int seg = reverse ? max(0, segs - 1 - lane) : lane;
    f64_load8(cg, seg, a);
    f64_load8(ch, seg, b);
    if (reverse) {
#pragma unroll
      for (int j = 0; j < kPer / 2; ++j) {
        const double x = a[j], y = b[j];
        a[j] = a[kPer - 1 - j];
        b[j] = b[kPer - 1 - j];
        a[kPer - 1 - j] = x;
        b[kPer - 1 - j] = y;
      }
    }
  }
  float est[kPer];
  uint32_t pend = 0, stop = 0;
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    est[j] = estimate(a[j], b[j]);
    if ((visited >> j & 1) && !low(b[j], n[j])) (ends(b[j], n[j]) ? stop : pend) |= 1u << j;
  }
  bool extra = false;
  int32_t brk = reverse ? INT32_MIN : INT32_MAX;
  if (stop) brk = lane * kPer + (reverse ? 31 - __clz(stop) : __ffs(stop) - 1);
  if (first_extra && lane == 0 && !low(base_h, base_n)) {
    if (ends(base_h, base_n)) brk = -1;
    else extra = true;
  }
  brk = reverse ? __reduce_max_sync(0xffffffffu, brk) : __reduce_min_sync(0xffffffffu, brk);
  float most = -INFINITY;
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    const int t = lane * kPer + j;
    if (reverse ? t <= brk : t >= brk) pend &= ~(1u << j);
    if (pend >> j & 1) most = fmaxf(most, est[j]);
  }
  if (extra) most = fmaxf(most, estimate(base_g, base_h));
  if (!__any_sync(0xffffffffu, pend != 0 || extra)) return false;
  if (!scan_safe(p, lc.sum_h)) {
#pragma unroll
    for (int j = 0; j < kPer; ++j)
      if ((pend >> j & 1) && !divisors_safe((float)b[j], (float)(lc.sum_h - b[j]), l2f)) most = INFINITY;  // no floor
    if (extra && !divisors_safe((float)base_h, (float)(lc.sum_h - base_h), l2f)) most = INFINITY;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, o));
  const float floor = plain ? estimate_floor(most) : -INFINITY;
#pragma unroll
  for (int j = 0; j < kPer; ++j)
    if (est[j] < floor) pend &= ~(1u << j);
  double best_gain = -INFINITY, wg = 0.0, wh = 0.0;  // this lane's best candidate and its sums
  int32_t best_t = INT32_MIN, wc = 0;
  bool splittable = false;
  auto consider = [&](int t, double ag, double ah, int32_t ac) {
    const double gr = lc.sum_g - ag, hr = lc.sum_h - ah;
    const int32_t rc = lc.num_data - ac;
    // the left child is the rest when scanning in reverse
    const double g1 = reverse ? gr : ag, h1 = reverse ? hr : ah, g2 = reverse ? ag : gr, h2 = reverse ? ah : hr;
    const int32_t c1 = reverse ? rc : ac, c2 = reverse ? ac : rc;
    const double gain = split_gain_hot(plain, g1, h1, g2, h2, p, c1, c2, lc.parent_output, lc.mc, lc.cmin, lc.cmax,
                                       m.monotone_type);
    if (gain <= min_gain_shift) return;
    splittable = true;
    if (gain > best_gain || (gain == best_gain && best_t != INT32_MIN && (reverse ? t > best_t : t < best_t))) {
      best_gain = gain;
      best_t = t;
      wg = ag;
      wh = ah;
      wc = ac;
    }
  };
  // a lane's thresholds one at a time, the lanes side by side (bit 8: the extra candidate)
  if (extra) pend |= 1u << kPer;
  while (__any_sync(0xffffffffu, pend != 0)) {
    if (pend) {
      const int j = __ffs(pend) - 1;
      pend &= pend - 1;
      double ag = base_g, ah = base_h;
      int32_t ac = base_n;
#pragma unroll
      for (int k = 0; k < kPer; ++k)
        if (k == j) {
          ag = a[k];
          ah = b[k];
          ac = n[k];
        }
      consider(j == kPer ? -1 : lane * kPer + j, ag, ah, ac);
    }
  }
  warp_pick(reverse, best_gain, best_t);
  const bool any = __any_sync(0xffffffffu, splittable) != 0;
  // the winner's sums, from the lane whose best it was (the extra candidate t = -1 is lane 0's)
  const int src = best_t >= 0 ? best_t / kPer : 0;
  ScanBest r;
  r.splittable = any;
  r.gain = best_gain;
  r.t = best_t;
  r.acc_g = __shfl_sync(0xffffffffu, wg, src);
  r.acc_h = __shfl_sync(0xffffffffu, wh, src);
  r.acc_c = __shfl_sync(0xffffffffu, wc, src);
  r.acc_q = 0;
  apply_direction<false>(r, m, p, lc.sum_g, lc.sum_h, 0, lc.gs, lc.hs, lc.num_data, lc.parent_output, lc.mc, lc.cmin,
                         lc.cmax, min_gain_shift, cnt_factor, reverse, out);
  __syncwarp();
  return any;
}

// find_best_threshold (split.rs:246-271, :402-441) for one leaf and feature,
// by one warp; the view is in sm.view.
__device__ __forceinline__ bool find_best_threshold_f64(F64Scratch& sm, const DFeature& m, const DParams& p,
                                                        const DParams& p_cat, LeafCtx lc, DSplit& out) {
  const int lane = threadIdx.x & 31;
  if (lane == 0) {
    out.default_left = 1;
    out.gain = -INFINITY;
    out.num_cat = 0;
    out.monotone_type = m.bin_type == 1 ? 0 : m.monotone_type;
  }
  lc.sum_h = lc.sum_h + 2.0 * kEpsilon;
  __syncwarp();
  bool ok = false;
  if (m.bin_type == 1) {
    CatScratchF64& cat = *reinterpret_cast<CatScratchF64*>(sm.cum);
    for (int t = lane; t < m.view_len; t += 32) {
      cat.g[t] = sm.view[0][f64_at(t)];
      cat.h[t] = sm.view[1][f64_at(t)];
    }
    __syncwarp();
    ok = scan_categorical<false>(cat, m, p, p_cat, lc, out);
  } else {
    const double min_gain_shift =
        leaf_gain_hot(plain_split(p, lc.mc), lc.sum_g, lc.sum_h, p, lc.num_data, lc.parent_output) +
        p.min_gain_to_split;
    const double cnt_factor = (double)lc.num_data / lc.sum_h;
    // split.rs:426-439: the directions scanned and their missing-value rules
    const bool two = m.num_bin > 2 && m.missing_type != 0;
    const bool skip_default = two && m.missing_type == 1;
    const bool na_missing = two && m.missing_type == 2;
    const bool first_extra = na_missing && m.offset == 1;
    const ScanSpan rev = scan_span(m, true, skip_default, na_missing), fwd = scan_span(m, false, skip_default, na_missing);
    double base_g = 0.0, base_h = 0.0;
    f64_chains(sm, lc, rev, fwd, m.view_len, two, first_extra, base_g, base_h);
#pragma unroll 1
    for (int d = 0; d < (two ? 2 : 1); ++d)
      ok |= scan_direction_f64(sm.cum[2 * d], sm.cum[2 * d + 1], sm.view[1], d == 0 ? rev : fwd, m, p, lc,
                               min_gain_shift, cnt_factor, d == 0, d == 1 && first_extra, base_g, base_h, out);
    if (!two && lane == 0 && m.missing_type == 2) out.default_left = 0;
  }
  __syncwarp();
  if (lane == 0) out.gain *= m.penalty;
  __syncwarp();
  return ok;
}

// Grid (G, 1, slots), kF64ScanThreads threads: each warp takes scans of its own.
__global__ void __launch_bounds__(kF64ScanThreads, kScanF64Blocks) k_round_scan_f64(const __grid_constant__ DCtx c) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  F64Scratch& sm = reinterpret_cast<F64Scratch*>(smem_raw)[warp];
  DSplit& out = reinterpret_cast<DSplit*>(smem_raw + kF64Warps * sizeof(F64Scratch))[warp];
  const DSlot& s = c.slots[blockIdx.z];
  const DRounds& r = s.r;
  const int32_t nf = c.num_features;
  const bool root = r.st->root != 0;
  const int32_t n = root ? nf : r.st->nb * 2 * nf, e0 = r.st->e0;
  for (int32_t w = warp * gridDim.x + blockIdx.x; w < n; w += kF64Warps * gridDim.x) {
    const int32_t item = w / nf, f = w - item * nf, side = item & 1;
    const DFeature m = c.feats[f];
    const uint8_t in_tree = s.bytree[f];
    int32_t child, parent, depth;
    const ScanJob j = round_job(c, s, root, e0 + (item >> 1), side, child, parent, depth);
    if (!j.live) continue;
    const uint8_t split_ok = parent < 0 ? 1 : r.splittable[(size_t)parent * nf + f];
    const int len = m.view_len;
    double2* hs = reinterpret_cast<double2*>(s.hist) + (size_t)j.s_buf * c.total_bins + m.view_start;
    double2* hp = reinterpret_cast<double2*>(s.hist) + (size_t)j.l_buf * c.total_bins + m.view_start;
    double2 v[kPer], pv[kPer];
    const double2 zero = make_double2(0.0, 0.0);
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      const int t = 32 * k + lane;
      // histogram cells are written by other CTAs' atomics: loaded through L2
      v[k] = t < len ? __ldcg(hs + t) : zero;
      pv[k] = t < len && side == 1 ? __ldcg(hp + t) : zero;
    }
    DSplit* dst = r.fres + ((size_t)item * nf + f);
    bool ok = false;
    if (in_tree && split_ok) {
      // the smaller leaf's most frequent bin (histogram.rs:42-56): the leaf's
      // sums minus every other bin, in bin order (lane 0 the gradients, lane 1
      // the hessians)
      if (m.most_freq_bin > 0) {
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
          const bool own = 32 * k + lane != m.most_freq_bin;
          sm.view[0][f64_at(32 * k + lane)] = own ? v[k].x : 0.0;
          sm.view[1][f64_at(32 * k + lane)] = own ? v[k].y : 0.0;
        }
        __syncwarp();
        double a = 0.0;
        if (lane < 2)
          a = f64_chain<true, false>(lane ? j.sl.sum_hessians : j.sl.sum_gradients, sm.view[lane], f64_chunks(len));
        const double2 fixed = make_double2(__shfl_sync(0xffffffffu, a, 0), __shfl_sync(0xffffffffu, a, 1));
#pragma unroll
        for (int k = 0; k < kPer; ++k)
          if (32 * k + lane == m.most_freq_bin) {
            v[k] = fixed;
            if (side == 0) hs[m.most_freq_bin] = fixed;
          }
        __syncwarp();
      }
#pragma unroll
      for (int k = 0; k < kPer; ++k) {
        const int t = 32 * k + lane;
        if (side == 1) {  // larger = parent - smaller, in the parent's buffer (histogram.rs:59-63)
          v[k] = make_double2(pv[k].x - v[k].x, pv[k].y - v[k].y);
          if (t < len) hp[t] = v[k];
        }
        sm.view[0][f64_at(t)] = v[k].x;
        sm.view[1][f64_at(t)] = v[k].y;
      }
      __syncwarp();
      ok = find_best_threshold_f64(sm, m, c.p, c.p_cat, leaf_ctx(c, j), out);
      if (lane == 0) {
        out.feature = m.real_index;
        out.inner = f;
      }
      __syncwarp();
      const uint32_t* src = reinterpret_cast<const uint32_t*>(&out);
      for (int k = lane; k < (int)(sizeof(DSplit) / 4); k += 32) reinterpret_cast<uint32_t*>(dst)[k] = src[k];
    } else if (lane == 0) {
      dst->gain = -INFINITY;
      dst->feature = -1;
      dst->monotone_type = 0;
    }
    if (lane == 0) r.splittable[(size_t)child * nf + f] = ok;
    scans_stored(c, s, item, 1, child, depth);
  }
}
