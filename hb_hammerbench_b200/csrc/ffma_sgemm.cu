// FP32 SIMT (FFMA) SGEMM for sm_100a.
//
// Replaces the HammerBench device kernel (apps/sgemm/kernel.cpp:279-333).
// The reference gives each tile of a 16x8 tile group 16x16 output blocks
// round-robin (kernel.cpp:300-302), streams 16x16 blocks of A and B from DRAM
// into scratchpad (load_block, kernel.cpp:36-109) and runs a 4x4
// register-blocked fmaf chain over k (compute_block, kernel.cpp:186-275).
// Here one CTA owns a BM x BN output tile: a producer warpgroup streams A and
// B tiles from HBM into a STAGES-deep shared-memory ring with cp.async
// (zero-filled past K), and each thread of the compute warps owns a TM x TN
// register block that it updates with one fused multiply-add per k in
// ascending k. The arithmetic per output element is therefore exactly the
// reference device kernel's:
// acc = 0.0f; for k = 0..K-1: acc = fmaf(a[m][k], b[k][n], acc).
//
// Layout in shared memory (per stage): BK rows of BM floats of A and BK rows
// of BN floats of B, m and n contiguous (an operand that is k-contiguous in
// memory is transposed on the way in, ffma_kernel.cuh).
// Thread layout inside a compute warp: lane = tn*8 + tm (tm < 8, tn < 4).
// Thread (tm, tn) owns rows {32i + 4tm + c} and columns {16j + 4tn + c}: the
// warp's fragment of one k is 128 contiguous bytes of A per i and 64 of B per
// j, read as 16-byte vectors without bank conflicts.
//
// What bounds it: the FMA pipe (a packed FMA holds it two cycles), once the
// loads are out of the FMA stream. 4096^3: 2.66 -> 2.23 ms (51.7 -> 61.5
// TFLOP/s, 0.87 of the measured packed-FMA roof) against the form whose
// compute warps issued the loads between two barriers per k-tile; two
// 512^3 products 24.6 -> 18.4 us; 1531 x 1009 x 2047 with A transposed and
// unaligned 239 -> 152 us.
#include "ffma_kernel.cuh"

namespace hbsg {

template <int BM, int BN, int BK, int WM, int WN, int STAGES, bool VEC, bool PAIR,
          bool TA = false, bool TB = false>
__global__ void __launch_bounds__(FfmaShape<BM, BN, BK, WM, WN, STAGES>::kThreads,
                                  FfmaShape<BM, BN, BK, WM, WN, STAGES>::kMinBlocks)
    ffma_sgemm_kernel(FfmaParams p) {
  extern __shared__ __align__(16) float smem[];
  // Rasterised tile order: groups of `raster` tile rows, column-major inside
  // a group, so CTAs resident at the same time share A and B strips in L2.
  const int t = blockIdx.x;
  const int group_span = p.raster * p.tiles_n;
  const int group = t / group_span;
  const int first_m = group * p.raster;
  const int gm = min(p.raster, p.tiles_m - first_m);
  const int in_group = t - group * group_span;
  const int m0 = (first_m + in_group % gm) * BM;
  const int n0 = (in_group / gm) * BN;
  const int batch = blockIdx.z;
  const int split = blockIdx.y;
  const int k_begin = split * p.k_per_split;
  const int k_end = min(p.K, k_begin + p.k_per_split);
  float* C;
  long ldc;
  bool vec_store;
  if (p.splits > 1) {  // split-K slices go to the partial buffer
    C = p.partial + ((long)batch * p.splits + split) * (long)p.M * p.N;
    ldc = p.N;
    vec_store = (p.N & 3) == 0;
  } else {
    C = p.C + batch * p.strideC;
    ldc = p.ldc;
    vec_store = p.vec_store;
  }
  using S = FfmaShape<BM, BN, BK, WM, WN, STAGES>;
  if (threadIdx.x >= S::kCompute) {
    ffma_regs_dec<S::kProducerRegs>();
    ffma_produce<S, BM, BN, BK, STAGES, VEC, TA, TB>(p.A + batch * p.strideA, p.lda,
                                                     p.B + batch * p.strideB, p.ldb, p.M, p.N,
                                                     k_begin, k_end, m0, n0, smem);
  } else {
    ffma_regs_inc<S::kComputeRegs>();
    ffma_compute<S, BM, BN, BK, WM, WN, STAGES, PAIR, TA, TB>(p.M, p.N, k_begin, k_end, m0, n0, C,
                                                              ldc, vec_store, smem);
  }
}

// Fixed-order reduction of split-K partial slices: C = ((p0 + p1) + p2) + ...,
// times 2^(row exponent + column exponent) in the scaled split-BF16 forms, whose
// slices are partial sums of the normalised operands.
// One thread per V consecutive outputs of a row (V = 4 when N and C's rows
// allow 16-byte access), the loads of 16 slices issued before their adds, so
// the serial chain is the adds alone: the partials come from L2 and one load
// at a time exposed its latency once per slice (148 slices of 256 x 256:
// 59 us, 24 us so, both from DRAM).
template <int V>
struct ReduceVec;
template <>
struct ReduceVec<4> {
  using T = float4;
  static __device__ __forceinline__ T add(T a, T b) {
    return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
  }
  using Bits = uint4;
  static __device__ __forceinline__ T scale(T a, uint32_t row, Bits c) {
    // a finite, normal maximum's exponent is E - 126: all but the ends of the
    // range take 2^(Er + Ec - 252) from the bits
    const uint32_t e = row >> 23, e0 = e + (c.x >> 23), e1 = e + (c.y >> 23), e2 = e + (c.z >> 23),
                   e3 = e + (c.w >> 23);
    if (min(e, min(min(c.x, c.y), min(c.z, c.w)) >> 23) >= 1 &&
        min(min(e0, e1), min(e2, e3)) > 125 && max(max(e0, e1), max(e2, e3)) <= 379 &&
        max(row, max(max(c.x, c.y), max(c.z, c.w))) < 0x7f800000u)
      return make_float4(a.x * __uint_as_float((e0 - 125) << 23),
                         a.y * __uint_as_float((e1 - 125) << 23),
                         a.z * __uint_as_float((e2 - 125) << 23),
                         a.w * __uint_as_float((e3 - 125) << 23));
    return scale_any(a, row, c);
  }
  static __device__ __noinline__ T scale_any(T a, uint32_t row, Bits c) {
    const int er = pow2_exp_of_bits(row);
    return make_float4(scale_pow2(a.x, er + pow2_exp_of_bits(c.x)),
                       scale_pow2(a.y, er + pow2_exp_of_bits(c.y)),
                       scale_pow2(a.z, er + pow2_exp_of_bits(c.z)),
                       scale_pow2(a.w, er + pow2_exp_of_bits(c.w)));
  }
};
template <>
struct ReduceVec<1> {
  using T = float;
  static __device__ __forceinline__ T add(T a, T b) { return a + b; }
  using Bits = uint32_t;
  static __device__ __forceinline__ T scale(T a, uint32_t row, Bits c) {
    return scale_pow2(a, pow2_exp_of_bits(row) + pow2_exp_of_bits(c));
  }
};

static constexpr int kReduceThreads = 128;
static constexpr int kReduceAhead = 16;

template <int V, bool SCALED>
__global__ void __launch_bounds__(kReduceThreads)
    splitk_reduce_kernel(const float* __restrict__ partial, float* __restrict__ C, int M, int N,
                         long ldc, long strideC, int splits, long total,
                         const uint32_t* __restrict__ rowmax,
                         const uint32_t* __restrict__ colmax) {
  using R = ReduceVec<V>;
  using T = typename R::T;
  const long idx = blockIdx.x * (long)kReduceThreads + threadIdx.x;
  if (idx >= total) return;
  const int nv = N / V;
  const long row = total <= 0xffffffffL ? (long)((unsigned)idx / (unsigned)nv) : idx / nv;
  const int col = (int)(idx - row * nv) * V;
  const int b = (int)(row / M);
  const int r = (int)(row - (long)b * M);
  const long MN = (long)M * N;
  const float* src = partial + (long)b * splits * MN + (long)r * N + col;
  T s = *reinterpret_cast<const T*>(src);
  int k = 1;
  for (; k + kReduceAhead <= splits; k += kReduceAhead) {
    T v[kReduceAhead];
#pragma unroll
    for (int u = 0; u < kReduceAhead; ++u)
      v[u] = __ldcs(reinterpret_cast<const T*>(src + (k + u) * MN));
#pragma unroll
    for (int u = 0; u < kReduceAhead; ++u) s = R::add(s, v[u]);
  }
  uint32_t rbits = 0;
  typename R::Bits cbits{};
  if constexpr (SCALED) {  // (beside the last slices' loads)
    rbits = __ldg(rowmax + r);
    cbits = __ldg(reinterpret_cast<const typename R::Bits*>(colmax + col));
  }
  for (; k < splits; ++k) s = R::add(s, __ldcs(reinterpret_cast<const T*>(src + k * MN)));
  if constexpr (SCALED) s = R::scale(s, rbits, cbits);
  *reinterpret_cast<T*>(C + b * strideC + r * ldc + col) = s;
}

// ---------------------------------------------------------------------------
// Tile table and launcher.

struct FfmaEntry {
  int bm, bn, bk, wm, wn, stages;
  int threads, smem;
  cudaError_t (*launch)(const FfmaParams&, dim3, cudaStream_t, bool vec);
};

template <int BM, int BN, int BK, int WM, int WN, int STAGES, bool PAIR>
static cudaError_t launch_ffma(const FfmaParams& p, dim3 grid, cudaStream_t st, bool vec) {
  using S = FfmaShape<BM, BN, BK, WM, WN, STAGES>;
  constexpr int smem = S::smem_bytes(false, false);
  auto kv = ffma_sgemm_kernel<BM, BN, BK, WM, WN, STAGES, true, PAIR>;
  auto ks = ffma_sgemm_kernel<BM, BN, BK, WM, WN, STAGES, false, PAIR>;
  auto k = vec ? kv : ks;
  static uint64_t mask_v = 0, mask_s = 0;
  static int regs_v = 0, regs_s = 0;
  if (!set_smem_once(reinterpret_cast<const void*>(k), smem, vec ? &mask_v : &mask_s))
    return cudaErrorInvalidValue;
  if (!ffma_regs_ok<S>(reinterpret_cast<const void*>(k), vec ? &regs_v : &regs_s))
    return cudaErrorInvalidConfiguration;
  k<<<grid, S::kThreads, smem, st>>>(p);
  return cudaGetLastError();
}

// Transposed-operand kernels for a tile shape.
template <int BM, int BN, int BK, int WM, int WN, int STAGES, bool VEC>
static cudaError_t launch_ffma_trans(const FfmaParams& p, dim3 grid, cudaStream_t st, int ta,
                                     int tb) {
  using S = FfmaShape<BM, BN, BK, WM, WN, STAGES>;
  auto k10 = ffma_sgemm_kernel<BM, BN, BK, WM, WN, STAGES, VEC, true, true, false>;
  auto k01 = ffma_sgemm_kernel<BM, BN, BK, WM, WN, STAGES, VEC, true, false, true>;
  auto k11 = ffma_sgemm_kernel<BM, BN, BK, WM, WN, STAGES, VEC, true, true, true>;
  auto k = ta && tb ? k11 : ta ? k10 : k01;
  static uint64_t masks[3] = {0, 0, 0};
  static int regs[3] = {0, 0, 0};
  const int slot = ta && tb ? 2 : ta ? 0 : 1;
  const int smem = S::smem_bytes(ta != 0, tb != 0);
  if (!set_smem_once(reinterpret_cast<const void*>(k), smem, &masks[slot]))
    return cudaErrorInvalidValue;
  if (!ffma_regs_ok<S>(reinterpret_cast<const void*>(k), &regs[slot]))
    return cudaErrorInvalidConfiguration;
  k<<<grid, S::kThreads, smem, st>>>(p);
  return cudaGetLastError();
}

#define HBSG_FFMA_ENTRY(BM, BN, BK, WM, WN, ST, PAIR)                                   \
  FfmaEntry {                                                                           \
    BM, BN, BK, WM, WN, ST, FfmaShape<BM, BN, BK, WM, WN, ST>::kThreads,                \
        FfmaShape<BM, BN, BK, WM, WN, ST>::smem_bytes(false, false),                    \
        &launch_ffma<BM, BN, BK, WM, WN, ST, PAIR>                                      \
  }

static const FfmaEntry kFfmaTiles[] = {
    HBSG_FFMA_ENTRY(128, 128, 16, 64, 64, 4, true),   // 1: 4 warps, 2 CTAs/SM, packed FMA
    HBSG_FFMA_ENTRY(128, 256, 16, 64, 64, 4, true),   // 2: 8 warps, packed FMA
    HBSG_FFMA_ENTRY(64, 64, 16, 32, 32, 6, true),     // 3: 4 warps, small problems
    HBSG_FFMA_ENTRY(128, 64, 16, 64, 32, 4, true),    // 4: 4 warps, narrow N
    HBSG_FFMA_ENTRY(128, 256, 32, 64, 64, 3, true),   // 5: 8 warps, deeper K tile
    HBSG_FFMA_ENTRY(256, 128, 16, 64, 64, 4, true),   // 6: 8 warps, tall
    HBSG_FFMA_ENTRY(128, 128, 32, 64, 64, 2, true),   // 7: 4 warps, deeper K tile
    HBSG_FFMA_ENTRY(128, 128, 16, 64, 64, 4, false),  // 8: as 1 with scalar FMA
    HBSG_FFMA_ENTRY(128, 128, 16, 64, 32, 4, true),   // 9: 8 warps, 8x8 per thread
};
static constexpr int kNumFfmaTiles = sizeof(kFfmaTiles) / sizeof(kFfmaTiles[0]);

int ffma_num_tiles() { return kNumFfmaTiles; }

bool ffma_tile_info(int idx, hbsg_tile_info* out) {
  if (idx < 0 || idx >= kNumFfmaTiles) return false;
  const FfmaEntry& e = kFfmaTiles[idx];
  out->variant_class = 0;
  out->bm = e.bm;
  out->bn = e.bn;
  out->bk = e.bk;
  out->threads = e.threads;
  out->smem_bytes = e.smem;
  out->parts = 0;
  return true;
}

// Tile for an M x N x K product (or a batch of them): the least estimated
// time of the SM that gets the most tiles. An SM's tiles run `res` at a time;
// the rates are those measured with 1 and with `res` tiles of a shape on every
// SM (TFLOP/s over 148 SMs, K = 4096, packed FMA), so a grid that leaves each
// SM one small tile, a ragged last round and the padding of edge tiles are
// all charged. 1536 x 1024 x 2048 takes 64 x 64 tiles (three per SM at most,
// 150 us) rather than 128 x 128 (one on 96 of the SMs, 177 us); 4096^3 takes
// 128 x 128 (2.24 ms). Transposed operands have kernels for two of the shapes.
// `res` is the row-major layout's: with only B transposed two 64 x 64 tiles fit
// an SM (88 KB, both staging rings), but charging it two at 46 TFLOP/s moves one
// ragged shape in twenty to 128 x 128, and of nine such one gained (1664 x 1836 x
// 3635 654 -> 624 us; 865 x 1398 x 352 33.1 -> 38.5, 2304 x 1386 x 1856 281 -> 309).
int ffma_pick_tile(int M, int N, int K, int batch, int num_sms, bool trans) {
  struct Rate {
    int idx, res;
    double one, full;
  };
  static const Rate kRates[] = {
      {0, 2, 57.0, 62.1},  // 128 x 128
      {1, 1, 62.4, 62.4},  // 128 x 256
      {3, 2, 51.0, 54.8},  // 128 x 64
      {2, 3, 41.8, 50.7},  // 64 x 64
  };
  constexpr double kTileUs = 1.5;  // first loads and the stores of a tile
  double best = 0.0;
  int best_idx = -1;
  for (const Rate& r : kRates) {
    if (trans && r.idx != 0 && r.idx != 2) continue;
    const FfmaEntry& e = kFfmaTiles[r.idx];
    const long tiles = (long)((M + e.bm - 1) / e.bm) * ((N + e.bn - 1) / e.bn) * batch;
    const long per_sm = (tiles + num_sms - 1) / num_sms;
    const long rounds = per_sm / r.res, rest = per_sm % r.res;
    const double us = 2.0 * e.bm * e.bn * (K > 0 ? K : 1) * 148.0 * 1e-6;  // x 1 / TFLOP/s
    const double rest_rate =
        r.res > 1 ? r.one + (r.full - r.one) * (rest - 1) / (r.res - 1) : r.full;
    double t = rounds * (r.res * us / r.full + kTileUs);
    if (rest > 0) t += rest * us / rest_rate + kTileUs;
    if (best_idx < 0 || t < best) {
      best = t;
      best_idx = r.idx;
    }
  }
  return best_idx;
}

size_t ffma_workspace_bytes(int M, int N, int batch, int splits) {
  return splits > 1 ? (size_t)M * N * batch * splits * sizeof(float) : 0;
}

cudaError_t ffma_launch(int tile_idx, FfmaParams p, int batch, cudaStream_t st, int ta, int tb) {
  // transposed operands: 128 x 128 or 64 x 64 tiles (the closest of the two)
  if (ta || tb) {
    const FfmaEntry& big = kFfmaTiles[0];
    const FfmaEntry& e0 = kFfmaTiles[tile_idx];
    tile_idx = (e0.bm * e0.bn >= big.bm * big.bn) ? 0 : 2;
  }
  const FfmaEntry& e = kFfmaTiles[tile_idx];
  p.tiles_m = (p.M + e.bm - 1) / e.bm;
  p.tiles_n = (p.N + e.bn - 1) / e.bn;
  if (p.raster <= 0) p.raster = 8;
  if (p.splits < 1) p.splits = 1;
  if (p.splits > 1) {
    // K slices are whole BK tiles.
    int per = (p.K + p.splits - 1) / p.splits;
    per = (per + e.bk - 1) / e.bk * e.bk;
    p.k_per_split = per;
    p.splits = (p.K + per - 1) / per;
  } else {
    p.k_per_split = p.K;
  }
  const bool vec = ((p.lda & 3) == 0) && ((p.ldb & 3) == 0) &&
                   ((reinterpret_cast<uintptr_t>(p.A) & 15) == 0) &&
                   ((reinterpret_cast<uintptr_t>(p.B) & 15) == 0) && ((p.strideA & 3) == 0) &&
                   ((p.strideB & 3) == 0);
  p.vec_store = ((p.ldc & 3) == 0) && ((reinterpret_cast<uintptr_t>(p.C) & 15) == 0) &&
                ((p.strideC & 3) == 0);
  dim3 grid((unsigned)(p.tiles_m * p.tiles_n), (unsigned)p.splits, (unsigned)batch);
  cudaError_t err;
  if (ta || tb) {
    if (tile_idx == 0)
      err = vec ? launch_ffma_trans<128, 128, 16, 64, 64, 4, true>(p, grid, st, ta, tb)
                : launch_ffma_trans<128, 128, 16, 64, 64, 4, false>(p, grid, st, ta, tb);
    else
      err = vec ? launch_ffma_trans<64, 64, 16, 32, 32, 6, true>(p, grid, st, ta, tb)
                : launch_ffma_trans<64, 64, 16, 32, 32, 6, false>(p, grid, st, ta, tb);
  } else {
    err = e.launch(p, grid, st, vec);
  }
  if (err != cudaSuccess || p.splits == 1) return err;
  return splitk_reduce(p.partial, p.C, p.M, p.N, p.ldc, p.strideC, p.splits, batch, st);
}

cudaError_t splitk_reduce(const float* partial, float* C, int M, int N, long ldc, long strideC,
                          int splits, int batches, cudaStream_t st, const uint32_t* rowmax,
                          const uint32_t* colmax) {
  const bool vec = (N & 3) == 0 && (ldc & 3) == 0 && (strideC & 3) == 0 &&
                   (reinterpret_cast<uintptr_t>(partial) & 15) == 0 &&
                   (reinterpret_cast<uintptr_t>(C) & 15) == 0;
  const long total = (long)batches * M * (vec ? N / 4 : N);
  const unsigned blocks = (unsigned)((total + kReduceThreads - 1) / kReduceThreads);
  auto kernel = rowmax ? (vec ? splitk_reduce_kernel<4, true> : splitk_reduce_kernel<1, true>)
                       : (vec ? splitk_reduce_kernel<4, false> : splitk_reduce_kernel<1, false>);
  kernel<<<blocks, kReduceThreads, 0, st>>>(partial, C, M, N, ldc, strideC, splits, total, rowmax,
                                            colmax);
  return cudaGetLastError();
}

}  // namespace hbsg
