// C-ABI layer: argument validation, variant dispatch, status codes.
// Entry points are declared (with the reference interfaces they replace) in
// include/hbsg.h.
#include <cuda_runtime.h>

#include <mutex>

#include "internal.h"

namespace hbsg {

static std::mutex g_dev_mu;
static int g_sms[kMaxDevices];
static int g_ok[kMaxDevices];  // 0 unknown, 1 sm_100, -1 other

int current_device_sms(int* device_out) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
    cudaGetLastError();
    return -1;
  }
  if (device_out) *device_out = dev;
  std::lock_guard<std::mutex> lk(g_dev_mu);
  if (g_ok[dev] == 0) {
    cudaDeviceProp prop;
    if (cudaGetDeviceProperties(&prop, dev) != cudaSuccess) {
      cudaGetLastError();
      return -1;
    }
    g_ok[dev] = (prop.major == 10 && prop.minor == 0) ? 1 : -1;
    g_sms[dev] = prop.multiProcessorCount;
  }
  return g_ok[dev] == 1 ? g_sms[dev] : -1;
}

bool set_smem_once(const void* func, int bytes, uint64_t* device_mask) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return false;
  const uint64_t bit = 1ull << dev;
  if (__atomic_load_n(device_mask, __ATOMIC_ACQUIRE) & bit) return true;
  if (cudaFuncSetAttribute(func, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess)
    return false;
  __atomic_fetch_or(device_mask, bit, __ATOMIC_ACQ_REL);
  return true;
}

static int status_from(cudaError_t e) {
  if (e == cudaSuccess) return HBSG_OK;
  cudaGetLastError();
  if (e == cudaErrorInvalidConfiguration || e == cudaErrorLaunchOutOfResources ||
      e == cudaErrorInvalidValue)
    return HBSG_ERR_LAUNCH;
  return HBSG_ERR_CUDA;
}

static bool variant_valid(int v) { return v >= HBSG_FFMA && v <= HBSG_BF16X6_SCALED; }

static size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

static int parts_of(int variant) {
  return (variant == HBSG_BF16X6 || variant == HBSG_BF16X6_SCALED) ? 3 : 2;
}
static bool scaled_of(int variant) {
  return variant == HBSG_BF16X3_SCALED || variant == HBSG_BF16X6_SCALED;
}

// Workspace layout of the split-BF16 path (one problem; batches reuse it).
struct SplitLayout {
  int Kp;
  size_t a_off, b_off, rowmax_off, colmax_off, total;
};
static SplitLayout split_layout(int M, int N, int K, int variant) {
  SplitLayout L{};
  const int P = parts_of(variant);
  L.Kp = (K + 31) / 32 * 32;
  if (L.Kp == 0) L.Kp = 32;
  L.a_off = 0;
  L.b_off = align256((size_t)P * M * L.Kp * 2);
  L.rowmax_off = L.b_off + align256((size_t)P * N * L.Kp * 2);
  L.colmax_off = L.rowmax_off + (scaled_of(variant) ? align256((size_t)M * 4) : 0);
  L.total = L.colmax_off + (scaled_of(variant) ? align256((size_t)N * 4) : 0);
  return L;
}

// Workspace layout of a fused-split schedule: the scaled forms' row and
// column maxima and, for the A-in-TMEM tiles, B's parts from the split pass
// (A's parts never reach HBM; the CTA-pair tiles split B in the kernel too);
// the K-slice partials follow.
static SplitLayout fused_layout(int M, int N, int K, int variant, bool ts) {
  SplitLayout L{};
  L.Kp = (K + 31) / 32 * 32;
  if (L.Kp == 0) L.Kp = 32;
  L.rowmax_off = 0;
  L.colmax_off = scaled_of(variant) ? align256((size_t)M * 4) : 0;
  L.b_off = L.colmax_off + (scaled_of(variant) ? align256((size_t)N * 4) : 0);
  L.total = L.b_off + (ts ? align256((size_t)parts_of(variant) * N * L.Kp * 2) : 0);
  L.a_off = L.total;
  return L;
}

// Global tile ids: 1..F are the FFMA family, F+1..F+T the split-BF16
// tensor-core family with a split pass, F+T+1..F+T+U the split-BF16 family
// with the split fused into the product kernel.
static int total_tiles() { return ffma_num_tiles() + tc_num_tiles() + fused_num_tiles(); }

struct TcChoice {
  bool fused;  // idx indexes the fused table (else the tensor-core table)
  int idx;
  int splits, kts;
  int whole = 0;   // > 0: only the tiles after the first `whole` are sliced
  long sliced = 0;  // floats of one slice's partials then
};

// Bytes of a schedule's K-slice partials.
static size_t partial_bytes(const TcChoice& c, int M, int N) {
  if (c.splits <= 1) return 0;
  const size_t floats = c.whole > 0 ? (size_t)c.sliced : (size_t)M * N;
  return (c.splits * floats * 4 + 255) / 256 * 256;
}

// ---- automatic split-BF16 schedule ----
// Estimated microseconds of a call on a tile with s K slices:
//   fixed                         launches, set-up, first loads, last stores
// + split  x operand bytes of the tile's split pass (read FP32, write the
//            parts) / 6 TB/s
// + wave   x rounds of the concurrent slots (an epilogue each)
// + ktile  x rounds x k-tiles per slice
// + s > 1: reduce x partial bytes written and read / 10 TB/s, + sliced
// The coefficients are a least-squares fit, tile by tile, to GPU times of 118
// shapes (M, N, K of 128-8192 and long-K and tall ones, every tile, 1-148
// slices; rms error 4-9 %). Taking the tile and slices of least estimate runs
// those shapes within 0.4 % of the best measured choice in the geometric mean
// (13 % at worst); the rule before it, which scored tiles by their last wave
// and sliced K only into slices of 16 k-tiles for outputs under half the SMs,
// within 20 % (6.4x at worst: 224 x 160 x 3136 in 6 products 44 against 17 us).
// `sliced` holds 3 us beyond the fit for the reduction's launch, which a
// host-bound caller pays in full.
struct TileCost {
  double fixed, split, wave, ktile, reduce, sliced;
};
static const TileCost kTcCost[] = {
    {5.6, 1.28, 5.13, 0.708, 1.38, 3.0},  // 6 products, 128 x 256
    {6.0, 1.09, 1.33, 0.507, 0.51, 4.5},  // 128 x 128
    {5.4, 1.01, 0.73, 0.452, 0.00, 4.9},  // 128 x 64
    {4.7, 1.20, 4.96, 0.413, 0.60, 4.1},  // 3 products, 128 x 256
    {5.2, 1.07, 1.49, 0.311, 0.29, 4.7},  // 128 x 128
    {4.9, 0.98, 0.77, 0.293, 0.00, 5.0},  // 128 x 64
    {6.1, 1.20, 2.39, 0.608, 0.97, 3.6},  // 6 products, 128 x 192
    {4.9, 1.11, 2.69, 0.352, 0.51, 4.4},  // 3 products, 128 x 192
    {5.3, 1.23, 4.79, 0.863, 0.57, 3.6},  // 6 products, pair 256 x 256
    {4.9, 1.20, 5.12, 0.417, 0.47, 4.2},  // 3 products, pair 256 x 256
};
static const TileCost kFusedCost[] = {
    {8.8, 0.00, 1.59, 1.394, 1.65, 3.0},  // 6 products, pair 256 x 256
    {8.7, 0.00, 1.34, 1.192, 1.34, 3.0},  // 3 products
    {7.3, 0.00, 0.00, 1.095, 1.06, 3.0},  // 6 products, pair 256 x 64
    {6.7, 0.00, 0.00, 0.992, 0.71, 3.0},  // 3 products
    {5.2, 1.10, 1.18, 0.364, 0.62, 5.1},  // 6 products, A in TMEM, 128 x 64
    {5.1, 1.12, 0.96, 0.257, 0.30, 5.1},  // 3 products
    {5.3, 1.07, 3.23, 0.557, 0.79, 5.1},  // 6 products, A in TMEM, 128 x 128
    {5.1, 1.09, 3.24, 0.352, 0.63, 5.2},  // 3 products
};
static_assert(sizeof(kTcCost) == kNumTcTiles * sizeof(TileCost) &&
                  sizeof(kFusedCost) == kNumFusedTiles * sizeof(TileCost),
              "a cost for each tile");

static double tile_us(const TileCost& c, double split_bytes, long tiles, int slots, int KT, int s,
                      double mn) {
  const int per = (KT + s - 1) / s;
  const int slices = (KT + per - 1) / per;
  const double waves = (double)((tiles * slices + slots - 1) / slots);
  double t = c.fixed + c.split * split_bytes / 6e6 + c.wave * waves + c.ktile * waves * per;
  if (slices > 1) t += c.reduce * slices * mn * 8.0 / 1e7 + c.sliced;
  return t;
}

// Slices of the last, unfilled round alone: a grid of 1 to 4 full rounds and
// some tiles more leaves most SMs idle for a whole tile's time at the end;
// those tiles in s slices each fill the SMs in rounds of 1/s. Only their
// partials are written and reduced. Best tile whole -> last round sliced, calls
// without the host interface's table in long alternating runs, us: 6 products
// 2048 x 2560 x 4096 277 -> 237, 1537 x 3333 x 4096 295 -> 262, 2100 x 2500 x 3000
// 207 -> 186, 4096^3 713 -> 688, 19072 x 250 x 1024 117 -> 109; 3 products, the
// first four, 163 -> 144, 179 -> 163, 123 -> 114, 408 -> 400. Past four rounds the
// round saved is under a fifth and the SM clock falls with the load (power cap),
// so it is not tried.
static double tail_us(const TileCost& c, double split_bytes, long tiles, int slots, int KT, int s,
                      double tile_elems) {
  const int per = (KT + s - 1) / s;
  const int slices = (KT + per - 1) / per;
  const long full = tiles / slots, rest = tiles - full * slots;
  const double tail = (double)((rest * slices + slots - 1) / slots);
  return c.fixed + c.split * split_bytes / 6e6 + c.wave * (full + tail) +
         c.ktile * (full * (double)KT + tail * per) +
         c.reduce * slices * rest * tile_elems * 8.0 / 1e7 + c.sliced + 3.0;
}


static void tc_pick_auto(int M, int N, int K, int variant, int sms, int req, bool fusable,
                         TcChoice* ch) {
  const int P = parts_of(variant);
  const int KT = K > 0 ? (K + 31) / 32 : 1;
  const double mk = (double)M * K, kn = (double)K * N, mn = (double)M * N;
  const double per_elem = 4.0 + 2.0 * P;
  const bool scaled = scaled_of(variant);
  double best = 0.0;
  int best_s = 1, whole = 0;
  bool have = false;
  // slice counts tried when the caller names none, up to one for every SM and
  // with the quarters of that: each at least 8 k-tiles, and no more than about
  // two rounds of the slots
  const int slice_counts[] = {1, 2, 3, 4, 6, 8, 12, 16, 24, sms / 4, 48, sms / 2, 3 * sms / 4, sms};
  auto consider = [&](bool fused, int idx, const TileCost& c, int bm, int bn, int slots,
                      double split_bytes) {
    const long tiles = (long)((M + bm - 1) / bm) * ((N + bn - 1) / bn);
    for (int s : slice_counts) {
      if (req > 0) s = req;
      if (req <= 0 && s > 1 && (KT / s < 8 || tiles * s * 5 > 11L * slots)) break;
      const double t = tile_us(c, split_bytes, tiles, slots, KT, s < KT ? s : KT, mn);
      if (!have || t < best) {
        have = true;
        best = t;
        best_s = s;
        ch->fused = fused;
        ch->idx = idx;
        whole = 0;
      }
      if (req > 0) break;
    }
    const long full = tiles / slots, rest = tiles - full * slots;
    if (fused || req > 0 || full < 1 || full > 4 || rest == 0) return;
    for (int s : {2, 3, 4, 6, 8}) {
      if (KT / s < 8) break;
      const double t = tail_us(c, split_bytes, tiles, slots, KT, s, (double)bm * bn);
      if (t < best) {
        best = t;
        best_s = s;
        ch->fused = false;
        ch->idx = idx;
        whole = (int)(full * slots);
        ch->sliced = rest * bm * bn;
      }
    }
  };
  for (int i = 0; i < tc_num_tiles(); ++i) {
    if (tc_tile_parts(i) != P) continue;
    const bool pair = tc_tile_pair(i) != 0;
    // scaled: the rows' maxima ride on their split, the columns are read again
    consider(false, i, kTcCost[i], pair ? 256 : 128, tc_tile_bn(i), pair ? sms / 2 : sms,
             (mk + kn) * per_elem + (scaled ? kn * 4.0 : 0.0));
  }
  if (fusable && K > 0) {
    for (int f = 0; f < fused_num_tiles(); ++f) {
      if (fused_tile_parts(f) != P) continue;
      const double bytes = (fused_tile_ts(f) ? kn * per_elem : 0.0) + (scaled ? (mk + kn) * 4.0 : 0.0);
      consider(true, f, kFusedCost[f], fused_tile_bm(f), fused_tile_bn(f),
               fused_tile_slots(f, sms), bytes);
    }
  }
  ch->whole = whole;
  ch->splits = ch->fused ? fused_pick_splits(ch->idx, M, N, K, best_s, sms, &ch->kts)
                         : tc_pick_splits(ch->idx, M, N, K, best_s, sms, &ch->kts);
}

// A schedule with fewer K slices, so usually less workspace: run where the
// automatic choice does not fit the caller's buffer, and with that one the
// measure of which problems the allocation-free entry point takes. Tiles by their score
// (split-pass tiles) or by waves of measured k-tile cycles (fused ones).
static void tc_pick_compact(int M, int N, int K, int variant, int sms, bool fusable, TcChoice* ch) {
  constexpr double kRate = 1.6e15;  // BF16 MMA flop/s of a well-fed tile
  constexpr double kHbm = 6.0e12;   // bytes/s of the split and product passes
  constexpr double kClock = 1.5e9;  // SM clock under load
  const int P = parts_of(variant);
  const double prods = P == 3 ? 6.0 : 3.0;
  const double flops = 2.0 * M * (double)N * K * prods;
  const double opnds = (double)M * K + (double)K * N;
  const double maxima = scaled_of(variant) ? opnds * 4.0 / kHbm : 0.0;
  double score = 0.0;
  ch->fused = false;
  ch->whole = 0;
  ch->idx = tc_pick_tile(M, N, K, P, sms, 0, &score);
  ch->splits = tc_pick_splits(ch->idx, M, N, K, 0, sms, &ch->kts);
  if (!fusable || K <= 0 || score <= 0.0) return;
  const double t_split = opnds * (4.0 + 2.0 * P) / (0.9 * kHbm) + 6e-6;
  const double t_unfused = t_split + flops / (kRate * score) + maxima;
  double best = 0.0;
  int best_idx = -1;
  for (int f = 0; f < fused_num_tiles(); ++f) {
    if (fused_tile_parts(f) != P) continue;
    const int bn = fused_tile_bn(f);
    const int bm = fused_tile_bm(f);
    const int slots = fused_tile_slots(f, sms);
    const long tiles = (long)((M + bm - 1) / bm) * ((N + bn - 1) / bn);
    int kts = 0;
    const int s = fused_pick_splits(f, M, N, K, 0, sms, &kts);
    const long waves = (tiles * s + slots - 1) / slots;
    const double t_conv = (double)waves * kts * fused_ktile_cycles(f) / kClock;
    const double t_mem = opnds * 4.0 / kHbm;
    const double t_reduce = s > 1 ? (double)s * M * N * 8.0 / kHbm : 0.0;
    // + ~3 us per wave to fill and drain the pipeline (first staging loads,
    // last MMAs, epilogue stores)
    // A-in-TMEM tiles split B in a pass of their own first
    const double t_split_b =
        fused_tile_ts(f) ? (double)K * N * (4.0 + 2.0 * P) / (0.9 * kHbm) + 4e-6 : 0.0;
    const double t = (t_conv > t_mem ? t_conv : t_mem) + 3e-6 * waves + t_reduce + maxima +
                     t_split_b;
    if (best_idx < 0 || t < best) {
      best = t;
      best_idx = f;
    }
  }
  if (best_idx >= 0 && best < 0.9 * t_unfused) {
    ch->fused = true;
    ch->idx = best_idx;
  }
  ch->splits = ch->fused ? fused_pick_splits(ch->idx, M, N, K, 0, sms, &ch->kts)
                         : tc_pick_splits(ch->idx, M, N, K, 0, sms, &ch->kts);
}

// Tensor-core tile and K-slice count for a split-BF16 problem (shared by the
// workspace query and the dispatcher so both agree). Returns false when an
// explicitly requested tile does not fit the variant or the operand layout
// (the fused kernels take row-major operands only).
static bool tc_schedule(int M, int N, int K, int variant, const hbsg_config* cfg, int sms,
                        bool transposed, bool fusable, TcChoice* ch) {
  const int P = parts_of(variant);
  const int tile = cfg && cfg->tile > 0 ? cfg->tile - 1 : -1;
  const int req = cfg ? cfg->split_k : 0;
  ch->fused = false;
  if (tile >= 0) {
    const int t = tile - ffma_num_tiles();
    if (t >= tc_num_tiles()) {
      ch->fused = true;
      ch->idx = t - tc_num_tiles();
      if (transposed || !fusable || ch->idx >= fused_num_tiles() ||
          fused_tile_parts(ch->idx) != P)
        return false;
    } else {
      ch->idx = t;
      if (t < 0 || tc_tile_parts(t) != P) return false;
    }
  } else {
    tc_pick_auto(M, N, K, variant, sms, req, !transposed && fusable, ch);
    return true;
  }
  ch->splits = ch->fused ? fused_pick_splits(ch->idx, M, N, K, req, sms, &ch->kts)
                         : tc_pick_splits(ch->idx, M, N, K, req, sms, &ch->kts);
  return true;
}

// fusable: 1 = the operands suit the fused-split tiles (16-byte aligned rows),
// 0 = they do not, -1 = unknown (the size covers either schedule).
static size_t workspace_needed(int M, int N, int K, int batch, int variant, const hbsg_config* cfg,
                               bool transposed = false, int fusable = -1) {
  if (variant == HBSG_FFMA) {
    const int splits = cfg && cfg->split_k > 1 ? cfg->split_k : 1;
    return ffma_workspace_bytes(M, N, batch, splits);
  }
  if (fusable < 0) {
    const size_t a = workspace_needed(M, N, K, batch, variant, cfg, transposed, 1);
    const size_t b = workspace_needed(M, N, K, batch, variant, cfg, transposed, 0);
    return a > b ? a : b;
  }
  // The schedule (and so the split-K partial buffer) depends on the SM count
  // of the device the product will run on: sizes are for the current device.
  const int sms = current_device_sms(nullptr);
  if (sms < 0) return 0;
  TcChoice ch;
  if (!tc_schedule(M, N, K, variant, cfg, sms, transposed, fusable == 1, &ch)) return 0;
  const size_t partial = partial_bytes(ch, M, N);
  return (ch.fused ? fused_layout(M, N, K, variant, fused_tile_ts(ch.idx))
                   : split_layout(M, N, K, variant)).total + partial;
}

// Whether gemm_dispatch may run these operands on a fused-split tile.
static bool operands_fusable(int K, const float* A, long lda, long strideA, const float* B,
                             long ldb, long strideB) {
  return K == 0 ||
         (fused_operands_ok(A, lda, B, ldb) && strideA % 4 == 0 && strideB % 4 == 0);
}

size_t gemm_workspace_exact(int trans_a, int trans_b, int m, int n, int k, const float* a,
                            long lda, const float* b, long ldb, int variant,
                            const hbsg_config* cfg) {
  if (m <= 0 || n <= 0 || k < 0 || !variant_valid(variant)) return 0;
  return workspace_needed(m, n, k, 1, variant, cfg, trans_a || trans_b,
                          operands_fusable(k, a, lda, 0, b, ldb, 0) ? 1 : 0);
}

size_t gemm_compact_workspace(int trans_a, int trans_b, int m, int n, int k, const float* a,
                              long lda, const float* b, long ldb, int variant) {
  const int sms = current_device_sms(nullptr);
  if (m <= 0 || n <= 0 || k < 0 || !variant_valid(variant) || sms < 0) return 0;
  const bool fusable = !(trans_a || trans_b) && operands_fusable(k, a, lda, 0, b, ldb, 0);
  TcChoice ch;
  tc_pick_compact(m, n, k, variant, sms, fusable, &ch);
  return (ch.fused ? fused_layout(m, n, k, variant, fused_tile_ts(ch.idx))
                   : split_layout(m, n, k, variant)).total +
         partial_bytes(ch, m, n);
}

// Core dispatcher for one (possibly batched) GEMM.
static int gemm_dispatch(int trans_a, int trans_b, int M, int N, int K, const float* A, long lda,
                         long strideA, const float* B, long ldb, long strideB, float* C, long ldc,
                         long strideC, int batch, int variant, const hbsg_config* cfg, void* ws,
                         size_t ws_bytes, cudaStream_t st) {
  if (M < 0 || N < 0 || K < 0 || batch < 0) return HBSG_ERR_INVALID_ARG;
  if (!variant_valid(variant)) return HBSG_ERR_UNSUPPORTED;
  if (M == 0 || N == 0 || batch == 0) return HBSG_OK;
  if (!C) return HBSG_ERR_INVALID_ARG;
  if (K > 0 && (!A || !B)) return HBSG_ERR_INVALID_ARG;
  // op(A) is M x K: stored M rows of K (row-major) or K rows of M (trans_a).
  const long a_row = trans_a ? M : K;
  const long b_row = trans_b ? K : N;
  if (K > 0 && (lda < (a_row > 0 ? a_row : 1) || ldb < (b_row > 0 ? b_row : 1)))
    return HBSG_ERR_INVALID_ARG;
  if (ldc < N) return HBSG_ERR_INVALID_ARG;
  int dev = 0;
  const int sms = current_device_sms(&dev);
  if (sms < 0) return HBSG_ERR_NO_DEVICE;

  int tile = cfg && cfg->tile > 0 ? cfg->tile - 1 : -1;
  if (tile >= total_tiles()) return HBSG_ERR_UNSUPPORTED;

  if (variant == HBSG_FFMA) {
    if (tile >= ffma_num_tiles()) return HBSG_ERR_UNSUPPORTED;
    if (tile < 0) tile = ffma_pick_tile(M, N, K, batch, sms, trans_a || trans_b);
    int splits = cfg && cfg->split_k > 1 ? cfg->split_k : 1;
    if (splits > 1 && K == 0) splits = 1;
    const size_t need = ffma_workspace_bytes(M, N, batch, splits);
    if (need > 0 && (!ws || ws_bytes < need || (reinterpret_cast<uintptr_t>(ws) & 255)))
      return HBSG_ERR_WORKSPACE;
    FfmaParams p{};
    p.A = A;
    p.B = B;
    p.C = C;
    p.partial = static_cast<float*>(ws);
    p.lda = lda;
    p.ldb = ldb;
    p.ldc = ldc;
    p.strideA = strideA;
    p.strideB = strideB;
    p.strideC = strideC;
    p.M = M;
    p.N = N;
    p.K = K;
    p.splits = splits;
    p.raster = cfg && cfg->raster_group > 0 ? cfg->raster_group : 8;
    return status_from(ffma_launch(tile, p, batch, st, trans_a ? 1 : 0, trans_b ? 1 : 0));
  }

  // ---- split-BF16 on the tensor cores ----
  const int P = parts_of(variant);
  const bool scaled = scaled_of(variant);
  TcChoice ch;
  // fused tiles read A and B through FP32 TMA maps (16-byte aligned rows;
  // with K = 0 nothing is read)
  const bool fusable = operands_fusable(K, A, lda, strideA, B, ldb, strideB);
  if (!tc_schedule(M, N, K, variant, cfg, sms, trans_a || trans_b, fusable, &ch))
    return HBSG_ERR_UNSUPPORTED;
  auto layout_of = [&](const TcChoice& c) {
    return c.fused ? fused_layout(M, N, K, variant, fused_tile_ts(c.idx))
                   : split_layout(M, N, K, variant);
  };
  auto fits = [&](const TcChoice& c) {
    const size_t need = layout_of(c).total + partial_bytes(c, M, N);
    return need == 0 || (ws && ws_bytes >= need && !(reinterpret_cast<uintptr_t>(ws) & 255));
  };
  if (!fits(ch)) {
    // an automatic schedule gives up K slices for a workspace that holds the
    // compact one (the allocation-free entry point's scratch, or a buffer
    // sized by the parts alone)
    if (tile >= 0 || (cfg && cfg->split_k > 0)) return HBSG_ERR_WORKSPACE;
    tc_pick_compact(M, N, K, variant, sms, !(trans_a || trans_b) && fusable, &ch);
    if (!fits(ch)) return HBSG_ERR_WORKSPACE;
  }
  const int tc = ch.idx, splits = ch.splits;
  const SplitLayout L = layout_of(ch);
  uint8_t* w = static_cast<uint8_t*>(ws);
  void* Ap = w + L.a_off;
  void* Bp = w + L.b_off;
  uint32_t* rowmax = scaled ? reinterpret_cast<uint32_t*>(w + L.rowmax_off) : nullptr;
  uint32_t* colmax = scaled ? reinterpret_cast<uint32_t*>(w + L.colmax_off) : nullptr;
  const int flags = cfg ? cfg->flags : 0;
  const int raster = cfg && cfg->raster_group > 0 ? cfg->raster_group : 0;
  const int chunk = cfg && cfg->chunk_k > 0 ? cfg->chunk_k : 0;
  if (ch.fused) {
    // The split of A (and, on the CTA-pair tiles, of B) runs inside the
    // product kernel; the workspace holds the scaled forms' maxima, the
    // A-in-TMEM tiles' B parts (PRESPLIT_A / _B: already current) and partials.
    const bool ts = fused_tile_ts(tc) != 0;
    for (int b = 0; b < batch; ++b) {
      const float* Ab = A + b * strideA;
      const float* Bb = B + b * strideB;
      // A's maxima, B's parts (A-in-TMEM tiles) and column maxima
      SplitOperand ops[2];
      int n_ops = 0;
      if (scaled && !(flags & HBSG_FLAG_PRESPLIT_A))
        ops[n_ops++] = {Ab, lda, M, K, L.Kp, false, nullptr, rowmax};
      if (!(flags & HBSG_FLAG_PRESPLIT_B))
        ops[n_ops++] = {Bb, ldb, N, K, L.Kp, true, ts ? Bp : nullptr, colmax};
      bool after_split = false;
      cudaError_t e = split_operands(ops, n_ops, P, scaled, st, &after_split);
      if (e != cudaSuccess) return status_from(e);
      if (flags & HBSG_FLAG_SPLIT_ONLY) continue;
      FusedParams fp{};
      fp.A = Ab;
      fp.B = Bb;
      fp.C = C + b * strideC;
      fp.lda = lda;
      fp.ldb = ldb;
      fp.ldc = ldc;
      fp.M = M;
      fp.N = N;
      fp.K = K;
      fp.splits = splits;
      fp.kt_per_split = ch.kts;
      fp.rowmax = rowmax;
      fp.colmax = colmax;
      fp.Bparts = ts ? Bp : nullptr;
      fp.Kp = L.Kp;
      e = fused_launch(tc, fp, raster, chunk, sms, 0, st,
                       reinterpret_cast<float*>(w + L.total), after_split);
      if (e != cudaSuccess) return status_from(e);
    }
    return HBSG_OK;
  }
  for (int b = 0; b < batch; ++b) {
    const float* Ab = A + b * strideA;
    const float* Bb = B + b * strideB;
    float* Cb = C + b * strideC;
    SplitOperand ops[2];
    int n_ops = 0;
    if (!(flags & HBSG_FLAG_PRESPLIT_A))
      ops[n_ops++] = {Ab, lda, M, K, L.Kp, trans_a != 0, Ap, rowmax};
    if (!(flags & HBSG_FLAG_PRESPLIT_B))
      ops[n_ops++] = {Bb, ldb, N, K, L.Kp, trans_b == 0, Bp, colmax};
    bool after_split = false;
    cudaError_t e = split_operands(ops, n_ops, P, scaled, st, &after_split);
    if (e != cudaSuccess) return status_from(e);
    if (flags & HBSG_FLAG_SPLIT_ONLY) continue;
    e = tc_launch(tc, Ap, Bp, M, N, K, L.Kp, Cb, ldc, rowmax, colmax, raster, chunk, sms, 0, 0, st,
                  splits, reinterpret_cast<float*>(w + L.total), after_split, ch.whole);
    if (e != cudaSuccess) return status_from(e);
  }
  return HBSG_OK;
}

}  // namespace hbsg

using namespace hbsg;

extern "C" {

int hbsg_sgemm(const float* mat1, const float* mat2, float* result, int n, int niter,
               hbsg_stream_t stream) {
  if (n < 0 || niter < 0) return HBSG_ERR_INVALID_ARG;
  if (n > 0 && niter > 0 && (!mat1 || !mat2 || !result)) return HBSG_ERR_INVALID_ARG;
  const long nn = (long)n * n;
  return gemm_dispatch(0, 0, n, n, n, mat1, n, nn, mat2, n, nn, result, n, nn, niter, HBSG_FFMA,
                       nullptr, nullptr, 0, reinterpret_cast<cudaStream_t>(stream));
}

int hbsg_sgemm_variant(const float* mat1, const float* mat2, float* result, int n, int niter,
                       int variant, void* workspace, size_t workspace_bytes,
                       hbsg_stream_t stream) {
  if (n < 0 || niter < 0) return HBSG_ERR_INVALID_ARG;
  if (n > 0 && niter > 0 && (!mat1 || !mat2 || !result)) return HBSG_ERR_INVALID_ARG;
  const long nn = (long)n * n;
  return gemm_dispatch(0, 0, n, n, n, mat1, n, nn, mat2, n, nn, result, n, nn, niter, variant,
                       nullptr, workspace, workspace_bytes,
                       reinterpret_cast<cudaStream_t>(stream));
}

size_t hbsg_sgemm_workspace_size(int n, int niter, int variant) {
  if (n <= 0 || niter <= 0 || !variant_valid(variant)) return 0;
  return workspace_needed(n, n, n, niter, variant, nullptr);
}

int hbsg_gemm(int trans_a, int trans_b, int m, int n, int k, const float* a, int64_t lda,
              const float* b, int64_t ldb, float* c, int64_t ldc, int variant, void* workspace,
              size_t workspace_bytes, hbsg_stream_t stream) {
  return gemm_dispatch(trans_a, trans_b, m, n, k, a, lda, 0, b, ldb, 0, c, ldc, 0, 1, variant,
                       nullptr, workspace, workspace_bytes,
                       reinterpret_cast<cudaStream_t>(stream));
}

int hbsg_gemm_ex(int trans_a, int trans_b, int m, int n, int k, const float* a, int64_t lda,
                 const float* b, int64_t ldb, float* c, int64_t ldc, int variant,
                 const hbsg_config* cfg, void* workspace, size_t workspace_bytes,
                 hbsg_stream_t stream) {
  return gemm_dispatch(trans_a, trans_b, m, n, k, a, lda, 0, b, ldb, 0, c, ldc, 0, 1, variant, cfg,
                       workspace, workspace_bytes, reinterpret_cast<cudaStream_t>(stream));
}

size_t hbsg_gemm_workspace_size(int m, int n, int k, int variant, const hbsg_config* cfg) {
  if (m <= 0 || n <= 0 || k < 0 || !variant_valid(variant)) return 0;
  return workspace_needed(m, n, k, 1, variant, cfg);
}

size_t hbsg_gemm_workspace_size_ex(int trans_a, int trans_b, int m, int n, int k, int variant,
                                   const hbsg_config* cfg) {
  if (m <= 0 || n <= 0 || k < 0 || !variant_valid(variant)) return 0;
  return workspace_needed(m, n, k, 1, variant, cfg, trans_a || trans_b);
}

size_t hbsg_gemm_workspace_size_for(int trans_a, int trans_b, int m, int n, int k, const float* a,
                                    int64_t lda, const float* b, int64_t ldb, int variant,
                                    const hbsg_config* cfg) {
  return gemm_workspace_exact(trans_a, trans_b, m, n, k, a, lda, b, ldb, variant, cfg);
}

int hbsg_get_split_layout(int m, int n, int k, int variant, hbsg_split_layout* out) {
  if (!out || m <= 0 || n <= 0 || k < 0) return HBSG_ERR_INVALID_ARG;
  if (!variant_valid(variant) || variant == HBSG_FFMA) return HBSG_ERR_UNSUPPORTED;
  const SplitLayout L = split_layout(m, n, k, variant);
  out->parts = parts_of(variant);
  out->kp = L.Kp;
  out->a_offset = L.a_off;
  out->b_offset = L.b_off;
  out->rowmax_offset = scaled_of(variant) ? L.rowmax_off : L.total;
  out->colmax_offset = scaled_of(variant) ? L.colmax_off : L.total;
  out->total_bytes = L.total;
  return HBSG_OK;
}

int hbsg_num_tiles(void) { return total_tiles(); }

int hbsg_tile_describe(int tile, hbsg_tile_info* out) {
  if (!out) return HBSG_ERR_INVALID_ARG;
  if (tile < 1 || tile > total_tiles()) return HBSG_ERR_INVALID_ARG;
  const int idx = tile - 1;
  const int F = ffma_num_tiles(), T = tc_num_tiles();
  const bool ok = idx < F       ? ffma_tile_info(idx, out)
                  : idx < F + T ? tc_tile_info(idx - F, out)
                                : fused_tile_info(idx - F - T, out);
  out->fused = idx >= F + T ? 1 : 0;
  return ok ? HBSG_OK : HBSG_ERR_INVALID_ARG;
}

const char* hbsg_strerror(int status) {
  switch (status) {
    case HBSG_OK: return "success";
    case HBSG_ERR_INVALID_ARG: return "invalid argument";
    case HBSG_ERR_UNSUPPORTED: return "unsupported variant, configuration or layout";
    case HBSG_ERR_WORKSPACE: return "workspace missing, misaligned or too small";
    case HBSG_ERR_LAUNCH: return "kernel launch failed";
    case HBSG_ERR_DEVICE_TIMEOUT: return "a bounded device-side wait expired";
    case HBSG_ERR_NO_DEVICE: return "no sm_100 device is current";
    case HBSG_ERR_CUDA: return "CUDA runtime error";
    default: return "unknown status";
  }
}

int hbsg_check_device(hbsg_stream_t stream) {
  if (current_device_sms(nullptr) < 0) return HBSG_ERR_NO_DEVICE;
  cudaError_t e = cudaStreamSynchronize(reinterpret_cast<cudaStream_t>(stream));
  if (e != cudaSuccess) return status_from(e);
  const int f1 = tc_read_and_clear_device_error();
  const int f2 = grouped_read_and_clear_device_error();
  const int f3 = fused_read_and_clear_device_error();
  const int f4 = jacobi_read_and_clear_device_error();
  return f1 != HBSG_OK ? f1 : f2 != HBSG_OK ? f2 : f3 != HBSG_OK ? f3 : f4;
}

int hbsg_debug_timeout_probe(void* workspace, size_t workspace_bytes, hbsg_stream_t stream) {
  if (!workspace || workspace_bytes < 65536 || (reinterpret_cast<uintptr_t>(workspace) & 255))
    return HBSG_ERR_WORKSPACE;
  const int sms = current_device_sms(nullptr);
  if (sms < 0) return HBSG_ERR_NO_DEVICE;
  // tiny problem: M = 128, N = 64, K = 32 on the 3-product, N = 64 tile
  int tc = -1;
  for (int i = 0; i < tc_num_tiles(); ++i) {
    hbsg_tile_info info;
    if (tc_tile_info(i, &info) && info.bn == 64 && tc_tile_parts(i) == 2) tc = i;
  }
  if (tc < 0) return HBSG_ERR_UNSUPPORTED;
  uint8_t* w = static_cast<uint8_t*>(workspace);
  cudaError_t e = tc_launch(tc, w, w + 16384, 128, 64, 32, 32, reinterpret_cast<float*>(w + 32768),
                            64, nullptr, nullptr, 1, 32, sms, 1, 200000000ull,
                            reinterpret_cast<cudaStream_t>(stream));
  return status_from(e);
}

int hbsg_version(void) { return 101; }

}  // extern "C"
