// Evaluation metrics on the device (Metric::eval, metric.rs:520-770):
// AUC, binary logloss and error, L2 and RMSE, multiclass logloss and error,
// over labels and scores already in device memory (a booster's validation
// scores need not come back to the host every iteration).
//
// AUC (metric.rs:701-731) without weights accumulates only counts and sums
// of count x (count / 2 + count): every partial sum is a multiple of 1/2
// below 2^52, exact in FP64, so the order of the additions does not matter
// and the device result equals the reference's bit for bit. The scores are
// sorted in descending order with their classes (a radix sort written here,
// 8 passes of 8 bits, each row and its class moved once a pass), positives
// are counted by prefix, and every negative adds half the positives before
// its group of tied scores and half those up to the group's end.
//
// The losses are FP64 sums of per-row terms; their order differs from the
// reference's sequential loop (within a few ulps of the mean).
#include <algorithm>
#include <cstring>
#include <mutex>
#include <vector>

#include "host_copy.h"
#include "learner_impl.h"
#include "rank.h"

namespace lgbm_b200 {

constexpr double kMetricEpsilon = (double)1e-15f;  // consts.rs K_EPSILON
constexpr int kAucBlock = 1024;                    // slots of one CTA of the positives' prefix
// The radix sort's tile: kRadixThreads threads of kRadixItems rows each.
constexpr int kRadixThreads = 256;
constexpr int kRadixItems = 8;
constexpr int kRadixTile = kRadixThreads * kRadixItems;
constexpr int kRadixWarps = kRadixThreads / 32;
constexpr int kRadixDigits = 256;

// Monotone map of a double onto uint64 (larger score, larger key).
__device__ __forceinline__ uint64_t score_key(double s) {
  if (s == 0.0) s = 0.0;  // -0 and +0 are one score, as the reference compares them
  const uint64_t b = (uint64_t)__double_as_longlong(s);
  return (b & 0x8000000000000000ull) ? ~b : (b | 0x8000000000000000ull);
}

// The per-row terms of the loss metrics.
struct LossArgs {
  int32_t metric, num_class, top_k;
  double sigmoid, neg_log_eps;
};

__device__ double row_loss(const LossArgs& a, const float* label, const double* score, int64_t n, int64_t i) {
  const float l = label[i];
  switch (a.metric) {
    case LGBM_B200_METRIC_BINARY_LOGLOSS:
    case LGBM_B200_METRIC_BINARY_ERROR: {
      const double prob = 1.0 / (1.0 + exp(-a.sigmoid * score[i]));  // binary.rs:164-166
      if (a.metric == LGBM_B200_METRIC_BINARY_ERROR) return prob <= 0.5 ? (l > 0.0f ? 1.0 : 0.0) : (l <= 0.0f ? 1.0 : 0.0);
      if (l <= 0.0f) return 1.0 - prob > kMetricEpsilon ? -log(1.0 - prob) : a.neg_log_eps;
      return prob > kMetricEpsilon ? -log(prob) : a.neg_log_eps;
    }
    case LGBM_B200_METRIC_L2:
    case LGBM_B200_METRIC_RMSE: {
      const double d = score[i] - (double)l;
      return d * d;
    }
    default: {  // multiclass: softmax over the class-major scores (multiclass.rs:165)
      const int k = a.num_class;
      const int lk = (int)l;
      double wmax = score[i];
      for (int c = 1; c < k; ++c) wmax = fmax(wmax, score[(int64_t)c * n + i]);
      double wsum = 0.0;
      for (int c = 0; c < k; ++c) wsum += exp(score[(int64_t)c * n + i] - wmax);
      const double pl = exp(score[(int64_t)lk * n + i] - wmax) / wsum;
      if (a.metric == LGBM_B200_METRIC_MULTI_LOGLOSS) return pl > kMetricEpsilon ? -log(pl) : a.neg_log_eps;
      int larger = 0;  // metric.rs:252-265
      for (int c = 0; c < k; ++c) {
        const double pc = exp(score[(int64_t)c * n + i] - wmax) / wsum;
        if (pc >= pl && ++larger > a.top_k) return 1.0;
      }
      return 0.0;
    }
  }
}

// Per-CTA partial sums of the loss terms (added on the host in CTA order).
__global__ void __launch_bounds__(256) k_metric_sum(LossArgs a, const float* label, const double* score, int64_t n,
                                                    double* partial) {
  double s = 0.0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    s += row_loss(a, label, score, n, i);
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  __shared__ double ws[8];
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += ws[w];
    partial[blockIdx.x] = t;
  }
}

// AUC: keys and classes: 0 negative (label <= 0), 1 positive (label > 0), 3 a
// NaN label (neither, as in the reference's loop). The key is inverted, so
// the ascending radix sort leaves the scores in descending order.
__global__ void __launch_bounds__(256) k_auc_keys(const float* label, const double* score, int64_t n, uint64_t* key,
                                                  uint8_t* cls) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    key[i] = ~score_key(score[i]);
    const float l = label[i];
    cls[i] = l > 0.0f ? 1 : (l <= 0.0f ? 0 : 3);
  }
}

// Rows of each digit in every tile: count[digit * tiles + tile].
__global__ void __launch_bounds__(kRadixThreads) k_radix_count(const uint64_t* key, int64_t n, int shift,
                                                               uint32_t* count, int64_t tiles) {
  __shared__ uint32_t hist[kRadixWarps][kRadixDigits];
  const int warp = threadIdx.x >> 5;
  for (int d = threadIdx.x; d < kRadixWarps * kRadixDigits; d += kRadixThreads) (&hist[0][0])[d] = 0;
  __syncthreads();
  const int64_t base = (int64_t)blockIdx.x * kRadixTile + threadIdx.x;
#pragma unroll
  for (int k = 0; k < kRadixItems; ++k) {
    const int64_t i = base + k * kRadixThreads;
    if (i < n) atomicAdd(&hist[warp][(key[i] >> shift) & (kRadixDigits - 1)], 1u);
  }
  __syncthreads();
  uint32_t c = 0;
  for (int w = 0; w < kRadixWarps; ++w) c += hist[w][threadIdx.x];
  count[threadIdx.x * tiles + blockIdx.x] = c;
}

// The inclusive sum of v over the threads of a CTA of at most 1024 (`ws`:
// one slot a warp); all threads call it.
__device__ __forceinline__ uint32_t block_inclusive(uint32_t v, uint32_t* ws) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t u = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += u;
  }
  __syncthreads();  // an earlier call's reads of ws
  if (lane == 31) ws[warp] = v;
  __syncthreads();
  for (int w = 0; w < warp; ++w) v += ws[w];
  return v;
}

// One CTA per digit: its tiles' counts become exclusive sums over the tiles,
// their total goes to total[digit]. Also the positives' sums over blocks
// (grid 1). Sums stay below n <= 2^31.
__global__ void __launch_bounds__(1024) k_tile_prefix(uint32_t* count, int64_t tiles, uint32_t* total) {
  __shared__ uint32_t ws[32];
  __shared__ uint32_t carry;
  uint32_t* c = count + (int64_t)blockIdx.x * tiles;
  uint32_t before = 0;
  for (int64_t t0 = 0; t0 < tiles; t0 += blockDim.x) {
    const int64_t t = t0 + threadIdx.x;
    const uint32_t v = t < tiles ? c[t] : 0;
    const uint32_t incl = block_inclusive(v, ws);
    if (t < tiles) c[t] = before + incl - v;
    if (threadIdx.x == blockDim.x - 1) carry = before + incl;
    __syncthreads();
    before = carry;
  }
  if (threadIdx.x == 0) total[blockIdx.x] = before;
}

// What bounds the sort: latency, at the sizes of a validation set. A tile of
// 2048 rows gives a million rows 489 CTAs (scatter 31 us a pass with tiles of
// 4096, 19 with these), and a pass is 30 us in three launches; the bitonic
// network it took the place of had 66 launches and 780 us for a million rows
// against 300 here.
//
// One pass: every row to its place by the digit, rows of one digit in their
// order. A warp owns kRadixItems x 32 consecutive rows and counts each
// 32 rows' equal digits by ballots, so a row's place inside the tile needs
// no atomics; places of the warps and the tile follow from the sums. The
// rows pass through shared memory in the tile's new order: the stores of one
// digit (8 rows a tile on average) are consecutive.
__global__ void __launch_bounds__(kRadixThreads) k_radix_scatter(const uint64_t* key, const uint8_t* cls, int64_t n,
                                                                 int shift, const uint32_t* count, int64_t tiles,
                                                                 const uint32_t* total, uint64_t* key_out,
                                                                 uint8_t* cls_out) {
  __shared__ uint64_t s_key[kRadixTile];
  __shared__ uint8_t s_cls[kRadixTile];
  __shared__ uint16_t whist[kRadixWarps][kRadixDigits];  // a warp's rows of each digit, then their first place
  __shared__ uint32_t dest[kRadixDigits];  // where the tile's rows of a digit go, less their place in the tile
  __shared__ uint32_t ws[kRadixWarps];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int d = tid; d < kRadixWarps * kRadixDigits; d += kRadixThreads) (&whist[0][0])[d] = 0;
  __syncthreads();
  const int64_t tile0 = (int64_t)blockIdx.x * kRadixTile;
  const int64_t base = tile0 + warp * (kRadixItems * 32) + lane;
  uint64_t k[kRadixItems];
  uint8_t c[kRadixItems];
  uint16_t at[kRadixItems];
#pragma unroll
  for (int r = 0; r < kRadixItems; ++r) {
    const int64_t i = base + r * 32;
    k[r] = i < n ? key[i] : 0;
    c[r] = i < n ? cls[i] : 0;
  }
#pragma unroll
  for (int r = 0; r < kRadixItems; ++r) {
    const bool in = base + r * 32 < n;
    const uint32_t d = (uint32_t)(k[r] >> shift) & (kRadixDigits - 1);
    uint32_t same = __ballot_sync(0xffffffffu, in);
    if (!in) same = ~same;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      const uint32_t m = __ballot_sync(0xffffffffu, (d >> b) & 1);
      same &= (d >> b) & 1 ? m : ~m;
    }
    const uint32_t lower = same & ((1u << lane) - 1);
    const uint16_t have = in ? whist[warp][d] : 0;
    at[r] = (uint16_t)(have + __popc(lower));
    __syncwarp();
    if (in && lower == 0) whist[warp][d] = (uint16_t)(have + __popc(same));
    __syncwarp();
  }
  __syncthreads();
  {  // thread d: the first place of digit d in the tile, and of each warp's rows of it
    uint32_t mine = 0;
    for (int w = 0; w < kRadixWarps; ++w) mine += whist[w][tid];
    uint32_t first = block_inclusive(mine, ws) - mine;
    const uint32_t all = total[tid];
    const uint32_t below = block_inclusive(all, ws) - all;
    dest[tid] = below + count[tid * tiles + blockIdx.x] - first;
    for (int w = 0; w < kRadixWarps; ++w) {
      const uint32_t h = whist[w][tid];
      whist[w][tid] = (uint16_t)first;
      first += h;
    }
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kRadixItems; ++r) {
    if (base + r * 32 < n) {
      const uint32_t p = whist[warp][(k[r] >> shift) & (kRadixDigits - 1)] + at[r];
      s_key[p] = k[r];
      s_cls[p] = c[r];
    }
  }
  __syncthreads();
  const int here = (int)min((int64_t)kRadixTile, n - tile0);
  for (int p = tid; p < here; p += kRadixThreads) {
    const uint64_t kp = s_key[p];
    const uint32_t to = dest[(kp >> shift) & (kRadixDigits - 1)] + (uint32_t)p;
    key_out[to] = kp;
    cls_out[to] = s_cls[p];
  }
}

// Positives in each block of kAucBlock sorted rows.
__global__ void __launch_bounds__(kAucBlock) k_auc_block_pos(const uint8_t* cls, int64_t n, uint32_t* block_pos) {
  const int64_t i = (int64_t)blockIdx.x * kAucBlock + threadIdx.x;
  const int c = __syncthreads_count(i < n && cls[i] == 1);
  if (threadIdx.x == 0) block_pos[blockIdx.x] = (uint32_t)c;
}

// Positives before every sorted row (block_pos: before each block).
__global__ void __launch_bounds__(kAucBlock) k_auc_before(const uint8_t* cls, int64_t n, const uint32_t* block_pos,
                                                          uint32_t* before) {
  __shared__ uint32_t ws[32];
  const int64_t i = (int64_t)blockIdx.x * kAucBlock + threadIdx.x;
  const uint32_t p = i < n && cls[i] == 1 ? 1 : 0;
  const uint32_t incl = block_inclusive(p, ws);
  if (i < n) before[i] = block_pos[blockIdx.x] + incl - p;
}

// Every group of tied scores adds neg_g * (pos_g / 2 + positives before it)
// (metric.rs:713-723): each of its negatives adds half of the positives
// before the group and half of those up to its end. Rows of a tied group
// find its ends by bisection; a score that stands alone needs none. Large
// CTAs, because each ends in an FP64 atomic on one address (17 ns).
__global__ void __launch_bounds__(kAucBlock) k_auc_sum(const uint64_t* key, const uint8_t* cls, const uint32_t* before,
                                                 int64_t n, const uint32_t* positives, double* accum) {
  double sum = 0.0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const uint8_t c = cls[i];
    const uint64_t k0 = key[i];
    const bool tied_up = i > 0 && key[i - 1] == k0, tied_down = i + 1 < n && key[i + 1] == k0;
    uint32_t upto = i + 1 < n ? before[i + 1] : *positives, first = before[i];
    if (c != 0) continue;
    if (tied_up) {
      int64_t lo = 0, hi = i - 1;  // the first row with the key is in [lo, hi]
      while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        if (key[mid] == k0) hi = mid;
        else lo = mid + 1;
      }
      first = before[lo];
    }
    if (tied_down) {
      int64_t lo = i + 2, hi = n;  // the first row past the key is in [lo, hi]
      while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        if (key[mid] == k0) lo = mid + 1;
        else hi = mid;
      }
      upto = lo < n ? before[lo] : *positives;
    }
    sum += 0.5 * ((double)first + (double)upto);
  }
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  __shared__ double ws[kAucBlock / 32];
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = sum;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += ws[w];
    atomicAdd(accum, t);
  }
}

// The same sum for few rows, without a sort: row i of block x, when it is a
// negative, counts the positives with a larger score twice and those with
// the same score once, over the rows of slice y. Two compares a pair, all of
// them independent.
constexpr int kDirectThreads = 256, kDirectSlice = 1024;
// Up to here pairs are counted, above it the rows are sorted: the sort's 28
// launches cost 150 us for any few rows, the pairs grow with the square (a
// host call of 1000 rows 56 us against 178, 8000 120 against 263, 20000 134
// against 226; the two meet near 32000).
constexpr int64_t kDirectRows = 24576;
__global__ void __launch_bounds__(kDirectThreads) k_auc_direct(const float* label, const double* score, int32_t n,
                                                               uint32_t* positives, double* accum) {
  __shared__ uint64_t s_key[kDirectSlice];
  __shared__ int32_t s_have, ws[kDirectThreads / 32];
  if (threadIdx.x == 0) s_have = 0;
  __syncthreads();
  const int32_t i = blockIdx.x * kDirectThreads + threadIdx.x, j0 = blockIdx.y * kDirectSlice;
  for (int32_t j = j0 + threadIdx.x; j < min(n, j0 + kDirectSlice); j += kDirectThreads)
    if (label[j] > 0.0f) s_key[atomicAdd(&s_have, 1)] = score_key(score[j]);  // in any order
  __syncthreads();
  const bool negative = i < n && label[i] <= 0.0f;
  const uint64_t mine = i < n ? score_key(score[i]) : 0;
  int32_t twice = 0;
#pragma unroll 4
  for (int32_t k = 0; k < s_have; ++k) twice += (s_key[k] > mine ? 1 : 0) + (s_key[k] >= mine ? 1 : 0);
  twice = negative ? twice : 0;
  for (int o = 16; o > 0; o >>= 1) twice += __shfl_xor_sync(0xffffffffu, twice, o);
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = twice;
  __syncthreads();
  if (threadIdx.x == 0) {
    int32_t t = 0;  // at most 256 x 1024 x 2
    for (int w = 0; w < kDirectThreads / 32; ++w) t += ws[w];
    atomicAdd(accum, 0.5 * (double)t);
    if (blockIdx.x == 0) atomicAdd(positives, (uint32_t)s_have);
  }
}

namespace {

// Device memory of metric_eval, one set per device: allocated on first use
// and reallocated only when a call needs more (never shrunk), so a call
// allocates and frees nothing (cudaFree synchronises the whole device).
// Calls on one device are serialised by the mutex. The buffers live until
// the process ends.
enum WsSlot { kWsKey, kWsCls, kWsCount, kWsBlockPos, kWsAcc, kWsPartial, kWsLabel, kWsScore, kWsSlots };
constexpr int kMaxMetricDevices = 64;

struct MetricWorkspace {
  std::mutex mu;
  void* buf[kWsSlots] = {};
  size_t cap[kWsSlots] = {};
  void* pin[2] = {};  // page-locked pieces of host inputs, and when each is free again
  cudaEvent_t sent[2] = {};
  cudaError_t get(WsSlot slot, size_t bytes, void** p) {
    bytes = std::max<size_t>(bytes, 256);
    if (cap[slot] < bytes) {
      if (buf[slot]) {
        cudaError_t e = cudaFree(buf[slot]);
        buf[slot] = nullptr;
        cap[slot] = 0;
        if (e != cudaSuccess) return e;
      }
      cudaError_t e = cudaMalloc(&buf[slot], bytes);
      if (e != cudaSuccess) {
        buf[slot] = nullptr;
        return e;
      }
      cap[slot] = bytes;
    }
    *p = buf[slot];
    return cudaSuccess;
  }
};

constexpr size_t kUploadPiece = (size_t)4 << 20;

// Host memory to the device on the legacy default stream. Pageable memory
// longer than a few pieces' overhead goes through the two page-locked
// pieces: the host's threads fill one while the copy engine sends the other
// (the driver's own staging is one thread's memcpy: RMSE of a million rows,
// 12 MB, 690 us a call against 480). Page-locked memory is sent as it is. `src` is free on return.
cudaError_t upload(MetricWorkspace& ws, void* dst, const void* src, size_t bytes) {
  cudaPointerAttributes at{};
  const bool locked = cudaPointerGetAttributes(&at, src) == cudaSuccess && at.type != cudaMemoryTypeUnregistered;
  if (locked || bytes <= kUploadPiece / 8) return cudaMemcpy(dst, src, bytes, cudaMemcpyHostToDevice);
  cudaError_t e = cudaSuccess;
  for (int b = 0; b < 2 && e == cudaSuccess; ++b) {
    if (!ws.pin[b]) e = cudaHostAlloc(&ws.pin[b], kUploadPiece, cudaHostAllocDefault);
    if (e == cudaSuccess && !ws.sent[b]) e = cudaEventCreateWithFlags(&ws.sent[b], cudaEventDisableTiming);
  }
  int b = 0;
  for (size_t o = 0; o < bytes && e == cudaSuccess; o += kUploadPiece, b ^= 1) {
    const size_t m = std::min(kUploadPiece, bytes - o);
    if ((e = cudaEventSynchronize(ws.sent[b])) != cudaSuccess) break;
    parallel_copy(ws.pin[b], static_cast<const char*>(src) + o, m);
    e = cudaMemcpyAsync(static_cast<char*>(dst) + o, ws.pin[b], m, cudaMemcpyHostToDevice, 0);
    if (e == cudaSuccess) e = cudaEventRecord(ws.sent[b], 0);
  }
  return e;
}

MetricWorkspace& metric_workspace(int device) {
  static MetricWorkspace ws[kMaxMetricDevices];
  return ws[device];
}

// The sum and the positives by the sort.
Status auc_sorted(MetricWorkspace& ws, const float* label, const double* score, int64_t n, cudaStream_t s,
                  uint32_t* positives, double* acc) {
  cudaError_t e = cudaSuccess;
  const int64_t tiles = (n + kRadixTile - 1) / kRadixTile, nb = (n + kAucBlock - 1) / kAucBlock;
  const size_t n8 = (size_t)((n + 31) / 32 * 32);  // the second half of a pair of buffers stays aligned
  uint64_t* key = nullptr;
  uint8_t* cls = nullptr;
  uint32_t *count = nullptr, *block_pos = nullptr;
  if ((e = ws.get(kWsKey, 2 * sizeof(uint64_t) * n8, (void**)&key)) != cudaSuccess ||
      (e = ws.get(kWsCls, 2 * n8, (void**)&cls)) != cudaSuccess ||
      (e = ws.get(kWsCount, sizeof(uint32_t) * kRadixDigits * tiles, (void**)&count)) != cudaSuccess ||
      (e = ws.get(kWsBlockPos, sizeof(uint32_t) * nb, (void**)&block_pos)) != cudaSuccess)
    return Status(LGBM_B200_ERR_CUDA, std::string("metric: ") + cudaGetErrorString(e));
  uint32_t* total = reinterpret_cast<uint32_t*>(acc + 2);
  const int grid = (int)std::min<int64_t>((n + 255) / 256, current_device_sms() * 16);
  k_auc_keys<<<grid, 256, 0, s>>>(label, score, n, key, cls);
  uint64_t* key2 = key + n8;
  uint8_t* cls2 = cls + n8;
  for (int shift = 0; shift < 64; shift += 8) {  // 8 passes: the rows end where they began
    k_radix_count<<<(unsigned)tiles, kRadixThreads, 0, s>>>(key, n, shift, count, tiles);
    k_tile_prefix<<<kRadixDigits, 1024, 0, s>>>(count, tiles, total);
    k_radix_scatter<<<(unsigned)tiles, kRadixThreads, 0, s>>>(key, cls, n, shift, count, tiles, total, key2, cls2);
    std::swap(key, key2);
    std::swap(cls, cls2);
  }
  uint32_t* before = reinterpret_cast<uint32_t*>(key2);  // the other buffer is free now
  k_auc_block_pos<<<(unsigned)nb, kAucBlock, 0, s>>>(cls, n, block_pos);
  k_tile_prefix<<<1, 1024, 0, s>>>(block_pos, nb, positives);
  k_auc_before<<<(unsigned)nb, kAucBlock, 0, s>>>(cls, n, block_pos, before);
  k_auc_sum<<<(unsigned)std::min<int64_t>(nb, current_device_sms() * 4), kAucBlock, 0, s>>>(key, cls, before, n, positives, acc);
  return Status();
}

Status metric_device(MetricWorkspace& ws, const LgbmB200MetricConfig& cfg, const float* label, const double* score,
                     int64_t n, cudaStream_t s, double* out) {
  auto dalloc = [&](WsSlot slot, void** p, size_t bytes) { return ws.get(slot, bytes, p); };
  cudaError_t e = cudaSuccess;
  if (cfg.metric == LGBM_B200_METRIC_AUC) {
    double* acc = nullptr;  // the sum, then uint32: the positives, the digits' totals
    e = dalloc(kWsAcc, (void**)&acc, 2 * sizeof(double) + sizeof(uint32_t) * kRadixDigits);
    if (e == cudaSuccess) e = cudaMemsetAsync(acc, 0, 2 * sizeof(double), s);
    if (e != cudaSuccess) return Status(LGBM_B200_ERR_CUDA, std::string("metric: ") + cudaGetErrorString(e));
    uint32_t* positives = reinterpret_cast<uint32_t*>(acc + 1);
    if (n <= kDirectRows) {
      const dim3 grid((unsigned)((n + kDirectThreads - 1) / kDirectThreads), (unsigned)((n + kDirectSlice - 1) / kDirectSlice));
      k_auc_direct<<<grid, kDirectThreads, 0, s>>>(label, score, (int32_t)n, positives, acc);
    } else {
      Status st = auc_sorted(ws, label, score, n, s, positives, acc);
      if (!st.ok()) return st;
    }
    double result[2] = {};  // the sum and the positives
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(result, acc, sizeof(result), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return Status(LGBM_B200_ERR_CUDA, std::string("metric: ") + cudaGetErrorString(e));
    const double accum = result[0];
    uint32_t sum_pos;
    std::memcpy(&sum_pos, &result[1], sizeof(sum_pos));
    const double sp = (double)sum_pos, sw = (double)n;
    *out = (sp > 0.0 && sp != sw) ? accum / (sp * (sw - sp)) : 1.0;  // metric.rs:724-730
    return Status();
  }
  LossArgs a;
  a.metric = cfg.metric;
  a.num_class = std::max(1, cfg.num_class);
  a.top_k = cfg.multi_error_top_k;
  a.sigmoid = cfg.sigmoid;
  a.neg_log_eps = -(double)std::log(1e-15f);  // consts.rs neg_log_epsilon: the f32 log, promoted
  const int grid = (int)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, current_device_sms() * 8));
  double* partial = nullptr;
  if ((e = dalloc(kWsPartial, (void**)&partial, sizeof(double) * grid)) != cudaSuccess)
    return Status(LGBM_B200_ERR_CUDA, std::string("metric: ") + cudaGetErrorString(e));
  k_metric_sum<<<grid, 256, 0, s>>>(a, label, score, n, partial);
  std::vector<double> ph((size_t)grid);
  e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpyAsync(ph.data(), partial, sizeof(double) * grid, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return Status(LGBM_B200_ERR_CUDA, std::string("metric: ") + cudaGetErrorString(e));
  double sum = 0.0;
  for (double v : ph) sum += v;
  const double mean = sum / (double)n;  // unweighted: sum_weights = n
  *out = cfg.metric == LGBM_B200_METRIC_RMSE ? std::sqrt(mean) : mean;
  return Status();
}

}  // namespace

}  // namespace lgbm_b200

using namespace lgbm_b200;

extern "C" int lgbm_b200_metric_eval(const LgbmB200MetricConfig* cfg, const float* label, const double* score,
                                     int64_t n, int32_t location, int32_t device, double* out) {
  if (!cfg || !label || !score || !out || n <= 0 || n > ((int64_t)1 << 31))
    return fail(Status(LGBM_B200_ERR_INVALID_PARAMETER, "metric: bad argument"));
  if (cfg->metric < LGBM_B200_METRIC_AUC || cfg->metric > LGBM_B200_METRIC_MULTI_ERROR)
    return fail(Status(LGBM_B200_ERR_INVALID_PARAMETER, "metric: unknown metric"));
  const bool multi = cfg->metric == LGBM_B200_METRIC_MULTI_LOGLOSS || cfg->metric == LGBM_B200_METRIC_MULTI_ERROR;
  if (multi && cfg->num_class < 2) return fail(Status(LGBM_B200_ERR_INVALID_PARAMETER, "metric: num_class < 2"));
  if (device < 0 || device >= kMaxMetricDevices) return fail(Status(LGBM_B200_ERR_INVALID_PARAMETER, "metric: device"));
  if (cudaSetDevice(device) != cudaSuccess) return fail(Status(LGBM_B200_ERR_CUDA, "cudaSetDevice"));
  const int64_t ns = n * (multi ? cfg->num_class : 1);
  MetricWorkspace& ws = metric_workspace(device);
  std::lock_guard<std::mutex> lock(ws.mu);
  // the legacy default stream: device inputs written by work on it are ordered before the metric
  if (location == LGBM_B200_DEVICE) {
    Status st = metric_device(ws, *cfg, label, score, n, 0, out);
    return st.ok() ? LGBM_B200_OK : fail(st);
  }
  float* ld = nullptr;
  double* sd = nullptr;
  if (ws.get(kWsLabel, sizeof(float) * n, (void**)&ld) != cudaSuccess ||
      ws.get(kWsScore, sizeof(double) * ns, (void**)&sd) != cudaSuccess)
    return fail(Status(LGBM_B200_ERR_CUDA, "metric: cudaMalloc"));
  Status st;
  if (upload(ws, ld, label, sizeof(float) * n) != cudaSuccess ||
      upload(ws, sd, score, sizeof(double) * ns) != cudaSuccess)
    st = Status(LGBM_B200_ERR_CUDA, "metric: copy");
  else
    st = metric_device(ws, *cfg, ld, sd, n, 0, out);
  return st.ok() ? LGBM_B200_OK : fail(st);
}

extern "C" int lgbm_b200_metric_ndcg(const float* label, const double* score, const int32_t* query_boundaries,
                                     int32_t num_queries, const int32_t* eval_at, int32_t num_eval_at,
                                     int32_t location, int32_t device, double* out) {
  if (!label || !score || !query_boundaries || num_queries <= 0 || !eval_at || num_eval_at <= 0 || !out ||
      query_boundaries[0] != 0)
    return fail(Status(LGBM_B200_ERR_INVALID_PARAMETER, "ndcg: bad argument"));
  for (int32_t j = 0; j < num_eval_at; ++j)
    if (eval_at[j] <= 0) return fail(Status(LGBM_B200_ERR_INVALID_PARAMETER, "ndcg: eval_at must be positive"));
  if (cudaSetDevice(device) != cudaSuccess) return fail(Status(LGBM_B200_ERR_CUDA, "cudaSetDevice"));
  const int64_t n = query_boundaries[num_queries];
  // the label gains, discounts and query checks of the ranking objective's tables
  std::vector<float> lh;
  const float* lp = label;
  if (location == LGBM_B200_DEVICE) {
    lh.resize((size_t)n);
    if (cudaMemcpy(lh.data(), label, sizeof(float) * n, cudaMemcpyDeviceToHost) != cudaSuccess)
      return fail(Status(LGBM_B200_ERR_CUDA, "ndcg: label copy"));
    lp = lh.data();
  }
  RankTables rt;
  Status st = rt.build(lp, query_boundaries, num_queries, 1.0, 1, false);
  if (!st.ok()) return fail(st);
  float* ld = nullptr;
  double* sd = nullptr;
  int32_t* kd = nullptr;
  double* od = nullptr;
  const size_t nq = (size_t)num_queries, nk = (size_t)num_eval_at;
  cudaError_t e = cudaSuccess;
  if (location != LGBM_B200_DEVICE) {
    if ((e = cudaMalloc(&ld, sizeof(float) * n)) == cudaSuccess) e = cudaMalloc(&sd, sizeof(double) * n);
    if (e == cudaSuccess) e = cudaMemcpy(ld, label, sizeof(float) * n, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(sd, score, sizeof(double) * n, cudaMemcpyHostToDevice);
  }
  if (e == cudaSuccess) e = cudaMalloc(&kd, sizeof(int32_t) * nk);
  if (e == cudaSuccess) e = cudaMalloc(&od, sizeof(double) * nq * nk);
  if (e == cudaSuccess) e = cudaMemcpy(kd, eval_at, sizeof(int32_t) * nk, cudaMemcpyHostToDevice);
  std::vector<double> per(nq * nk);
  if (e == cudaSuccess) {
    const float* lbl = location == LGBM_B200_DEVICE ? label : ld;
    const double* sc = location == LGBM_B200_DEVICE ? score : sd;
    st = launch_ndcg(rt.d, lbl, sc, kd, num_eval_at, od, current_device_sms(), 0);
    if (st.ok()) e = cudaMemcpy(per.data(), od, sizeof(double) * nq * nk, cudaMemcpyDeviceToHost);
  }
  if (ld) cudaFree(ld);
  if (sd) cudaFree(sd);
  if (kd) cudaFree(kd);
  if (od) cudaFree(od);
  if (!st.ok()) return fail(st);
  if (e != cudaSuccess) return fail(Status(LGBM_B200_ERR_CUDA, std::string("ndcg: ") + cudaGetErrorString(e)));
  // the mean over queries, added in query order
  for (size_t j = 0; j < nk; ++j) {
    double acc = 0.0;
    for (size_t q = 0; q < nq; ++q) acc += per[q * nk + j];
    out[j] = acc / (double)num_queries;
  }
  return LGBM_B200_OK;
}
