// Split pre-pass for the split-BF16 tensor-core SGEMM (sm_100a).
//
// Every FP32 operand element x becomes BF16 parts (round to nearest even):
//   x' = x * 2^-e            (e = 0, or the row/column exponent when scaled)
//   hi  = bf16(x'),  r1 = x' - hi          (exact in FP32)
//   mid = bf16(r1),  r2 = r1 - mid         (exact in FP32)
//   lo  = bf16(r2)                          (3-part form only)
// With three parts hi + mid + lo == x' exactly for every normal FP32 value.
//
// Output layout (the K-major operand layout the tensor-core kernel's TMA reads):
//   Ap[p][m][k]  p < parts, m < M, k < Kp   (Kp = K rounded up to 32, zero-filled)
//   Bp[p][n][k]  B transposed: the K x N row-major input becomes N rows of Kp
// The scaled forms first reduce max|x| per row of A / per column of B into
// FP32 bit patterns (non-negative floats order like their bit patterns, so an
// integer atomicMax is an exact, order-independent max), then derive
// e = frexp exponent of that max: the row's largest |x'| lies in [0.5, 1).
//
// Bound by HBM (4 bytes read, 2 P written per element) once the operands are
// large, by launches and latency below that, so both operands share a launch:
// each is either row-major along k (A, transposed B: "rows") or k x n (B,
// transposed A: "columns", transposed through shared memory). Unscaled forms
// take one launch. Scaled forms take two: the first finishes rows (one CTA
// reads a row for its maximum and again, from the cache, for the split; many
// short rows see kShortRows) and reduces the column maxima, the second splits
// the columns. 3001 x 2503 x
// 3607 in the scaled 3-product form: 71 -> 48 us of split
// work, 4 launches and a memset before. At 8192^3 the passes run at 6.1 TB/s.
#include "internal.h"
#include "split_kernel.cuh"

namespace hbsg {

static constexpr int kSplitThreads = 256;
// Rows up to this long are finished by one CTA each (max and split); longer
// ones are cut into chunks of this many k for the maximum.
static constexpr int kRowChunk = 16384;
// Many short rows (kShortRows: K up to kShortK, kShortMany rows or more) go to
// groups of 4 to 64 lanes instead, which read a row once and keep up to
// kRowUnits units of 8 k a lane in registers between its maximum and its split.
// A CTA each left most of its threads, and most of the loads an SM can have in
// flight, unused: whole 3-product calls of 65536 x 64, transposed B, CTA -> group,
// K = 32 113 -> 18.5 us, 128 126 -> 31, 512 173 -> 90, 2048 336 -> 302 (6 products
// 155 -> 19, 178 -> 38, 228 -> 115, 443 -> 398). Longer rows give each thread of a
// CTA a unit or more: from K = 4096 on the groups lose 3-10 %, where only the
// maxima are wanted already at 2048 (10000 x 64 x 2048 67.6 -> 74.9 us; at 1500
// 65536 rows 265 -> 228), and fewer rows fit a few rounds of CTAs either way.
static constexpr int kRowUnits = 4;
static constexpr int kShortK = 2048;
static constexpr int kShortMaxK = 1536;  // the same for the maxima alone
static constexpr int kShortMany = 4096;
static constexpr int kColRows = 64;  // k rows per CTA of the column maxima

// One operand's share of a launch (blocks [first, first + blocks)).
enum SplitRole { kRowSplit, kRowMaxSplit, kRowMax, kColMax, kColSplit, kShortRows };
struct SplitJob {
  const float* X;  // rows: n x K with row stride ld; columns: K x n
  long ld;
  __nv_bfloat16* parts;  // [P][n][Kp], null: maxima only
  uint32_t* mx;          // n maxima (scaled forms)
  int n, K, Kp;
  int role;
  unsigned blocks;
};
struct SplitJobs {
  SplitJob job[2];
  unsigned first1;  // first block of job[1]
};

HBSG_DEV float finite_abs(float x) {
  const float a = fabsf(x);
  return isfinite(a) ? a : 0.0f;
}

HBSG_DEV float block_max(float mx, float* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
  __syncthreads();
  mx = red[threadIdx.x & (kSplitThreads / 32 - 1)];
#pragma unroll
  for (int o = kSplitThreads / 64; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  return mx;
}

// max|row[k]| over k in [k0, k1) by the whole CTA.
HBSG_DEV float row_max(const float* __restrict__ row, int k0, int k1, float* red) {
  float mx = 0.0f;
  if ((reinterpret_cast<uintptr_t>(row + k0) & 15) == 0) {
    const int k4 = k0 + (k1 - k0) / 4 * 4;
    for (int k = k0 + 4 * (int)threadIdx.x; k < k4; k += 4 * kSplitThreads) {
      const float4 v = *reinterpret_cast<const float4*>(row + k);
      mx = fmaxf(fmaxf(mx, fmaxf(finite_abs(v.x), finite_abs(v.y))),
                 fmaxf(finite_abs(v.z), finite_abs(v.w)));
    }
    k0 = k4;
  }
  for (int k = k0 + (int)threadIdx.x; k < k1; k += kSplitThreads) mx = fmaxf(mx, finite_abs(row[k]));
  return block_max(mx, red);
}

// Lanes of a short row's group: a unit each up to a warp, kRowUnits each beyond.
__host__ __device__ inline unsigned short_row_lanes(int Kp) {
  const int units = Kp / 8;
  unsigned g = 4;
  while ((int)g < units && (g < 32 || (int)g * kRowUnits < units)) g *= 2;
  return g;
}

// Short rows: their maximum and (with parts) their split, one group per row.
template <int P>
HBSG_DEV void split_short_rows(const SplitJob& j, unsigned block, float* red) {
  const unsigned g = short_row_lanes(j.Kp), l = threadIdx.x & (g - 1);
  const unsigned r = block * (kSplitThreads / g) + threadIdx.x / g;
  const bool live = r < (unsigned)j.n;
  const float* row = j.X + (long)(live ? r : 0) * j.ld;
  float v[kRowUnits][8];
  float mx = 0.0f;
#pragma unroll
  for (int u = 0; u < kRowUnits; ++u) {
    const int k0 = (int)(u * g + l) * 8;
    if (k0 < j.Kp) {  // (the padding past K loads as zeros)
      split_a_load(row + k0, k0, j.K, v[u]);
#pragma unroll
      for (int i = 0; i < 8; ++i) mx = fmaxf(mx, finite_abs(v[u][i]));
    }
  }
  for (unsigned o = (g < 32 ? g : 32) / 2; o > 0; o >>= 1)
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if (g > 32) {  // two warps a row
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
    __syncthreads();
    mx = fmaxf(mx, red[(threadIdx.x >> 5) ^ 1]);
  }
  if (!live) return;
  if (l == 0) j.mx[r] = __float_as_uint(mx);
  if (!j.parts) return;
  const SplitScale sc = split_scale(exp_from_maxbits(__float_as_uint(mx)));
  const long plane = (long)j.n * j.Kp;
#pragma unroll
  for (int u = 0; u < kRowUnits; ++u) {
    const int k0 = (int)(u * g + l) * 8;
    if (k0 < j.Kp) split_a_store<P, true>(v[u], sc, j.parts + (long)r * j.Kp + k0, plane);
  }
}

// SHORT: kernels that take kShortRows jobs (whose registers would cost the
// others a resident CTA).
template <int P, bool SCALED, bool SHORT>
HBSG_DEV void split_job(const SplitJob& j, unsigned block, float (*tile)[65]) {
  if (SHORT && j.role == kShortRows) {
    split_short_rows<P>(j, block, tile[0]);
    return;
  }
  switch (j.role) {
    case kRowSplit: {  // 8 consecutive k per thread, 4 units a block apart
      const unsigned upr = (unsigned)j.Kp / 8;
      const long total = (long)j.n * upr;
      const long plane = (long)j.n * j.Kp;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const long g = ((long)block * 4 + u) * kSplitThreads + threadIdx.x;
        if (g >= total) return;
        const long m = total <= 0xffffffffL ? (long)((unsigned)g / upr) : g / upr;
        const int k0 = (int)(g - m * upr) * 8;
        const SplitScale sc = split_scale(SCALED ? exp_from_maxbits(j.mx[m]) : 0);
        float v[8];
        split_a_load(j.X + m * j.ld + k0, k0, j.K, v);
        split_a_store<P, SCALED>(v, sc, j.parts + m * j.Kp + k0, plane);
      }
      break;
    }
    case kRowMaxSplit: {  // one row: its maximum, then its split
      const float* row = j.X + (long)block * j.ld;
      const float mx = row_max(row, 0, j.K, tile[0]);
      if (threadIdx.x == 0) j.mx[block] = __float_as_uint(mx);
      if (!j.parts) return;
      const SplitScale sc = split_scale(exp_from_maxbits(__float_as_uint(mx)));
      const long plane = (long)j.n * j.Kp;
      for (int k0 = 8 * (int)threadIdx.x; k0 < j.Kp; k0 += 8 * kSplitThreads) {
        float v[8];
        split_a_load(row + k0, k0, j.K, v);
        split_a_store<P, SCALED>(v, sc, j.parts + (long)block * j.Kp + k0, plane);
      }
      break;
    }
    case kRowMax: {  // one chunk of a long row into its (zeroed) maximum
      const int chunks = (j.K + kRowChunk - 1) / kRowChunk;
      const int r = (int)(block / (unsigned)chunks);
      const int k0 = (int)(block % (unsigned)chunks) * kRowChunk;
      const float mx = row_max(j.X + (long)r * j.ld, k0, min(j.K, k0 + kRowChunk), tile[0]);
      if (threadIdx.x == 0 && mx > 0.0f) atomicMax(j.mx + r, __float_as_uint(mx));
      break;
    }
    case kColMax: {  // 256 columns x kColRows k into the (zeroed) maxima
      const unsigned nb = ((unsigned)j.n + kSplitThreads - 1) / kSplitThreads;
      const int n = (int)(block % nb) * kSplitThreads + (int)threadIdx.x;
      const int k0 = (int)(block / nb) * kColRows;
      if (n >= j.n) return;
      const int k1 = min(j.K, k0 + kColRows);
      const float* p = j.X + (long)k0 * j.ld + n;
      float mx = 0.0f;
      int k = k0;
      for (; k + 8 <= k1; k += 8, p += 8 * j.ld) {
        float v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = p[i * j.ld];
#pragma unroll
        for (int i = 0; i < 8; ++i) mx = fmaxf(mx, finite_abs(v[i]));
      }
      for (; k < k1; ++k, p += j.ld) mx = fmaxf(mx, finite_abs(*p));
      if (mx > 0.0f) atomicMax(j.mx + n, __float_as_uint(mx));
      break;
    }
    default: {  // kColSplit: one 64 x 64 block, transposed
      const unsigned nb = ((unsigned)j.n + 63) / 64;
      const int n0 = (int)(block % nb) * 64, k0 = (int)(block / nb) * 64;
      float v[16];
      split_b_load(j.X, j.ld, j.K, j.n, k0, n0, v);
      split_b_to_tile(v, tile);
      __syncthreads();
      split_b_from_tile<P, SCALED>(j.n, j.Kp, j.parts, j.mx, k0, n0, tile);
    }
  }
}

template <int P, bool SCALED, bool SHORT>
__global__ void __launch_bounds__(kSplitThreads) split_kernel(const __grid_constant__ SplitJobs jobs) {
  __shared__ float tile[64][65];
  grid_dep_trigger();  // the next split launch or the product may set itself up
  grid_dep_wait();     // second launch: the first one's maxima
  if (blockIdx.x < jobs.first1) split_job<P, SCALED, SHORT>(jobs.job[0], blockIdx.x, tile);
  else split_job<P, SCALED, SHORT>(jobs.job[1], blockIdx.x - jobs.first1, tile);
}

static long blocks_of(const SplitJob& j) {
  auto cdiv = [](long a, long b) { return (a + b - 1) / b; };
  switch (j.role) {
    case kRowSplit: return cdiv((long)j.n * (j.Kp / 8), 4 * kSplitThreads);
    case kRowMaxSplit: return j.n;
    case kShortRows: return cdiv(j.n, kSplitThreads / short_row_lanes(j.Kp));
    case kRowMax: return (long)j.n * cdiv(j.K, kRowChunk);
    case kColMax: return cdiv(j.n, kSplitThreads) * cdiv(j.K, kColRows);
    default: return cdiv(j.n, 64) * cdiv(j.Kp, 64);
  }
}

static cudaError_t launch_jobs(SplitJob* job, int n, int parts, bool scaled, cudaStream_t st,
                               bool* launched) {
  // grids are one-dimensional: at most 2^31 - 1 blocks, each launch takes as
  // many jobs as fit (one operand alone always does: its elements are
  // addressable by 32-bit row and k)
  SplitJobs jobs{};
  long total = 0;
  int taken = 0;
  auto flush = [&]() -> cudaError_t {
    if (total == 0) return cudaSuccess;
    const unsigned grid = (unsigned)total;
    void (*k)(SplitJobs) =
        parts == 3 ? (scaled ? split_kernel<3, true, false> : split_kernel<3, false, false>)
                   : (scaled ? split_kernel<2, true, false> : split_kernel<2, false, false>);
    if (jobs.job[0].role == kShortRows || (taken > 1 && jobs.job[1].role == kShortRows))
      k = parts == 3 ? split_kernel<3, true, true> : split_kernel<2, true, true>;
    const cudaError_t e = launch_after(k, grid, kSplitThreads, 0, st, *launched, jobs);
    *launched = e == cudaSuccess;
    total = 0;
    taken = 0;
    return e;
  };
  for (int i = 0; i < n; ++i) {
    const long b = blocks_of(job[i]);
    if (b <= 0) continue;
    if (b > 0x7fffffffL) return cudaErrorInvalidConfiguration;
    if (total + b > 0x7fffffffL) {
      const cudaError_t e = flush();
      if (e != cudaSuccess) return e;
    }
    job[i].blocks = (unsigned)b;
    jobs.job[taken] = job[i];
    total += b;
    if (taken == 0) jobs.first1 = (unsigned)b;
    ++taken;
  }
  return flush();
}

cudaError_t split_operands(const SplitOperand* ops, int n, int parts, bool scaled,
                           cudaStream_t st, bool* launched) {
  *launched = false;
  SplitJob first[2], second[2];
  int n1 = 0, n2 = 0;
  for (int i = 0; i < n; ++i) {
    const SplitOperand& o = ops[i];
    if (o.n <= 0 || (!o.parts && !scaled)) continue;
    SplitJob j{o.X, o.ld, static_cast<__nv_bfloat16*>(o.parts), o.mx, o.n, o.K, o.Kp, 0, 0};
    if (!scaled) {
      j.role = o.columns ? kColSplit : kRowSplit;
      first[n1++] = j;
    } else if (!o.columns && o.K <= kRowChunk) {
      j.role = o.Kp <= (o.parts ? kShortK : kShortMaxK) && o.n >= kShortMany ? kShortRows
                                                                            : kRowMaxSplit;
      first[n1++] = j;
    } else {
      const cudaError_t e = cudaMemsetAsync(o.mx, 0, sizeof(uint32_t) * (size_t)o.n, st);
      if (e != cudaSuccess) return e;
      j.role = o.columns ? kColMax : kRowMax;
      if (o.K > 0) first[n1++] = j;
      j.role = o.columns ? kColSplit : kRowSplit;
      if (o.parts) second[n2++] = j;
    }
  }
  const cudaError_t e = launch_jobs(first, n1, parts, scaled, st, launched);
  return e != cudaSuccess ? e : launch_jobs(second, n2, parts, scaled, st, launched);
}

}  // namespace hbsg
