// Split helpers (FP32 -> BF16 parts) shared by the single and grouped split
// passes. The split itself is described in split_bf16.cu.
#pragma once

#include <cuda_bf16.h>

#include "common.cuh"

namespace hbsg {

HBSG_DEV int exp_from_maxbits(uint32_t bits) {
  const float mx = __uint_as_float(bits);
  if (!(mx > 0.0f) || !isfinite(mx)) return 0;
  int e;
  frexpf(mx, &e);
  return e;
}

// x * 2^-e as one multiply by a power of two (ldexpf's value: both round once),
// where 2^-e is a normal float; the few exponents beyond that (rows whose
// maximum is subnormal or above 2^126) take ldexpf out of line. ldexpf for
// every value made the scaled split passes issue-bound.
static __device__ __noinline__ float split_scale_slow(float x, int e) { return ldexpf(x, -e); }

struct SplitScale {
  int e;
  float f;  // 2^-e, or 0 when that is no normal float
};
HBSG_DEV SplitScale split_scale(int e) {
  return {e, e >= -127 && e <= 126 ? __uint_as_float((uint32_t)(127 - e) << 23) : 0.0f};
}
HBSG_DEV float apply_scale(float x, const SplitScale& s) {
  return s.f != 0.0f ? x * s.f : split_scale_slow(x, s.e);
}

template <int P, bool SCALED>
HBSG_DEV void split_value(float x, const SplitScale& sc, __nv_bfloat16* out) {
  if constexpr (SCALED) x = apply_scale(x, sc);
  const __nv_bfloat16 h = __float2bfloat16_rn(x);
  const float r1 = x - __bfloat162float(h);
  const __nv_bfloat16 m = __float2bfloat16_rn(r1);
  out[0] = h;
  out[1] = m;
  if constexpr (P == 3) {
    const float r2 = r1 - __bfloat162float(m);
    out[2] = __float2bfloat16_rn(r2);
  }
}

// One 64 (k) x 64 (n) block of B (K x N, row stride ldb) split into
// Bp[p][n][k0 .. k0+63], in three steps that callers may interleave with
// other blocks: split_b_load (16 values per thread into registers, coalesced
// along n), split_b_to_tile (into the shared tile), split_b_from_tile (split
// and store, 8 threads per 128-byte output row segment). 256 threads.
HBSG_DEV void split_b_load(const float* __restrict__ B, long ldb, int K, int N, int k0, int n0,
                           float* v) {
  const int tid = threadIdx.x;
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const int idx = tid + i * 256;
    const int k = k0 + (idx >> 6);
    const int n = n0 + (idx & 63);
    v[i] = (k < K && n < N) ? B[(long)k * ldb + n] : 0.0f;
  }
}

HBSG_DEV void split_b_to_tile(const float* v, float (*tile)[65]) {
  const int tid = threadIdx.x;
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const int idx = tid + i * 256;
    tile[idx >> 6][idx & 63] = v[i];
  }
}

template <int P, bool SCALED>
HBSG_DEV void split_b_from_tile(int N, int Kp, __nv_bfloat16* __restrict__ Bp,
                                const uint32_t* __restrict__ colmax, int k0, int n0,
                                const float (*tile)[65]) {
  const int tid = threadIdx.x;
  const long plane = (long)N * Kp;
#pragma unroll
  for (int pass = 0; pass < 2; ++pass) {
    const int j = pass * 32 + (tid >> 3);  // n offset
    const int kk = (tid & 7) * 8;          // k offset
    const int n = n0 + j;
    if (n >= N || k0 + kk >= Kp) continue;
    const SplitScale sc = split_scale(SCALED ? exp_from_maxbits(colmax[n]) : 0);
    __align__(16) __nv_bfloat16 parts[P][8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      __nv_bfloat16 o[3];
      split_value<P, SCALED>(tile[kk + i][j], sc, o);
#pragma unroll
      for (int p = 0; p < P; ++p) parts[p][i] = o[p];
    }
    __nv_bfloat16* dst = Bp + (long)n * Kp + k0 + kk;
#pragma unroll
    for (int p = 0; p < P; ++p)
      *reinterpret_cast<uint4*>(dst + p * plane) = *reinterpret_cast<const uint4*>(parts[p]);
  }
}

// 8 consecutive k of one row (or the part of them inside K), zero beyond it.
HBSG_DEV void split_a_load(const float* __restrict__ src, int k0, int K, float* v) {
  if (k0 + 8 <= K && ((reinterpret_cast<uintptr_t>(src) & 15) == 0)) {
    const float4 x0 = *reinterpret_cast<const float4*>(src);
    const float4 x1 = *reinterpret_cast<const float4*>(src + 4);
    v[0] = x0.x; v[1] = x0.y; v[2] = x0.z; v[3] = x0.w;
    v[4] = x1.x; v[5] = x1.y; v[6] = x1.z; v[7] = x1.w;
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = (k0 + i < K) ? src[i] : 0.0f;
  }
}

// Splits 8 values of a row into P parts of 16 bytes at dst + p * plane.
template <int P, bool SCALED>
HBSG_DEV void split_a_store(const float* v, const SplitScale& sc, __nv_bfloat16* dst, long plane) {
  __align__(16) __nv_bfloat16 parts[P][8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    __nv_bfloat16 o[3];
    split_value<P, SCALED>(v[i], sc, o);
#pragma unroll
    for (int p = 0; p < P; ++p) parts[p][i] = o[p];
  }
#pragma unroll
  for (int p = 0; p < P; ++p)
    *reinterpret_cast<uint4*>(dst + p * plane) = *reinterpret_cast<const uint4*>(parts[p]);
}

}  // namespace hbsg
