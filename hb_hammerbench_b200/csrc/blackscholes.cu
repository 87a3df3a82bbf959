// Black-Scholes European option pricing for sm_100a: the suite's
// apps/blackscholes benchmark on the same host interface as the SGEMM path.
//
// Reference: the device kernel `kernel(OptionData* data, int num_option,
// int pod_id)` (apps/blackscholes/kernel.cpp:27-113) prices each option
// record in place with BlkSchlsEqEuroNoDiv_kernel (bs_kernel.hpp:163-198);
// the testbench checks call and put against the host BlkSchlsEqEuroNoDiv
// (bs.hpp:60-125) by the sum of squared differences <= 0.01
// (main.cpp:119-141).
//
// Arithmetic: the device kernel's own approximations, each step the same IEEE
// operation, so results are bit-identical to that kernel:
//   - ln(s / strike) by its 5-term Taylor series around 1 in Horner form
//     (bs_kernel.hpp:33-49), 0 when s == strike;
//   - exp of a non-positive argument by whole steps of e^-1, one optional
//     e^-0.5 step and a 5-term Taylor polynomial of the remainder, 0 below -15
//     (bs_kernel.hpp:52-91);
//   - the cumulative normal by Hull's polynomial (bs_kernel.hpp:95-160);
// each `fmadd.s` / `fnmsub.s` of the reference is one fused multiply-add
// (__fmaf_rn); every other product, sum, quotient and square root is rounded
// on its own (the explicit __f*_rn intrinsics keep nvcc from contracting
// them); no library math function is called.
//
// B200 form: pricing reads 5 floats and writes 2 per option:
//   - records (the reference's OptionData, 8 floats = 32 bytes, call and put
//     updated in place): a record is loaded and stored back whole, one 32-byte
//     access each way (64 bytes per option). HBM-bound: 10M records 117 -> 96 us,
//     6.6 TB/s;
//   - separate arrays (s, strike, r, v, t in; call, put out): 28 bytes per
//     option. Bound by the issue rate: 10M options 66 -> 55-59 us by box.
// Each thread prices two options, with packed two-lane arithmetic.
#include <cuda_runtime.h>

#include "common.cuh"
#include "internal.h"

namespace hbsg {

static constexpr int kBsThreads = 256;

// Two options are priced at a time: every product, sum and fused multiply-add
// is a packed two-lane instruction (each lane the same IEEE operation), which
// halves the issue slots of the polynomials; the quotients, reciprocals and
// square roots, selections and table look-ups stay one per option.
HBSG_DEV float2 f2(float x) { return make_float2(x, x); }
HBSG_DEV float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
HBSG_DEV float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
HBSG_DEV float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
// a - b: b * -1 is exact, so the fused form rounds the difference once, as
// the subtraction does (signs of zero included)
HBSG_DEV float2 sub2(float2 a, float2 b) { return fma2(b, f2(-1.0f), a); }

// my_logf (bs_kernel.hpp:33-49)
HBSG_DEV float2 bs_logf(float2 x) {
  const float2 diff = add2(x, f2(-1.0f));
  float2 r = fma2(diff, f2(0.20000000f), f2(-0.25000000f));
  r = fma2(r, diff, f2(0.33333333f));
  r = fma2(r, diff, f2(-0.50000000f));
  r = fma2(r, diff, f2(1.00000000f));
  return mul2(r, diff);
}

// expf_0 (bs_kernel.hpp:52-65)
HBSG_DEV float2 bs_exp0(float2 x) {
  float2 r = fma2(x, f2(0.0083333338f), f2(0.04166667f));
  r = fma2(r, x, f2(0.16666666f));
  r = fma2(r, x, f2(0.5f));
  r = fma2(r, x, f2(1.0f));
  return fma2(r, x, f2(1.0f));
}

// fast_expf (bs_kernel.hpp:69-91), x <= 0, without its loop. The loop
// multiplies part1 by e^-1 and adds 1 to x while x <= -1. For -15 <= x <= -1
// every x + 1 is exact (1 is a multiple of x's ulp and |x + 1| < |x|), so the
// loop runs n = floor(-x) times, leaves x + n (exact, for the same reason) and
// part1 = the n-fold rounded product, which `pow_tab` (lane k of the warp
// holds the k-fold product, bs_pow_table) supplies by a shuffle: bit for bit
// the loop's result. n is read off 2^23 - x rounded down, whose low mantissa
// bits it is (0 for -1 < x <= 0; below -15 the result is 0 whatever n is).
// Every lane of the warp must call this together.
HBSG_DEV float2 bs_fast_expf(float2 x, float pow_tab) {
  const float2 t = make_float2(__fadd_rd(8388608.0f, -x.x), __fadd_rd(8388608.0f, -x.y));
  float2 part1 = make_float2(__shfl_sync(0xffffffffu, pow_tab, __float_as_int(t.x) & 15),
                             __shfl_sync(0xffffffffu, pow_tab, __float_as_int(t.y) & 15));
  const float2 y = add2(x, add2(t, f2(-8388608.0f)));
  // x <= -0.5: one e^-0.5 step (times 1 and plus 0 change nothing otherwise)
  const bool hx = y.x <= -0.5f, hy = y.y <= -0.5f;
  part1 = mul2(part1, make_float2(hx ? 0.60653066f : 1.0f, hy ? 0.60653066f : 1.0f));
  const float2 z = add2(y, make_float2(hx ? 0.5f : 0.0f, hy ? 0.5f : 0.0f));
  const float2 r = mul2(part1, bs_exp0(z));
  return make_float2(x.x < -15.0f ? 0.0f : r.x, x.y < -15.0f ? 0.0f : r.y);
}

// The k-fold product of e^-1 for k < 16, each product rounded, as fast_expf's
// loop forms it (IEEE float products, evaluated by the compiler).
struct BsPow {
  float v[16];
  constexpr BsPow() : v() {
    float p = 1.0f;
    for (int k = 0; k < 16; ++k) {
      v[k] = p;
      p = p * 0.36787945f;
    }
  }
};
static __device__ const BsPow g_bs_pow = BsPow();

// Lane k (< 16) of a warp holds the k-fold product.
HBSG_DEV float bs_pow_table() { return __ldg(&g_bs_pow.v[threadIdx.x & 15]); }

// one lane of dual_CNDF (bs_kernel.hpp:95-160); 1 / (1 + 0.2316419 |x|) as
// the correctly rounded reciprocal, the same value as the reference's divide
HBSG_DEV float2 bs_cndf(float2 x, float pow_tab) {
  const float2 xa = make_float2(fabsf(x.x), fabsf(x.y));
  // -(e^(-x^2/2) * 0.3989...): the sign of the product's constant, so that
  // fnmsub.s, -(f * e) + 1, is a fused multiply-add of f and -e
  const float2 ne = mul2(bs_fast_expf(mul2(mul2(f2(-0.5f), xa), xa), pow_tab),
                         f2(-0.39894228040143270286f));
  const float2 kd = fma2(f2(0.2316419f), xa, f2(1.0f));
  const float2 k = make_float2(__frcp_rn(kd.x), __frcp_rn(kd.y));
  float2 f = fma2(k, f2(1.330274429f), f2(-1.821255978f));
  f = fma2(f, k, f2(1.781477937f));
  f = fma2(f, k, f2(-0.356563782f));
  f = fma2(f, k, f2(0.319381530f));
  f = mul2(f, k);
  const float2 out = fma2(f, ne, f2(1.0f));
  const float2 flip = sub2(f2(1.0f), out);
  return make_float2(x.x < 0.0f ? flip.x : out.x, x.y < 0.0f ? flip.y : out.y);
}

// BlkSchlsEqEuroNoDiv_kernel (bs_kernel.hpp:163-198)
HBSG_DEV void bs_price(float2 s, float2 strike, float2 r, float2 v, float2 t, float2& call,
                       float2& put, float pow_tab) {
  const float2 sqrt_t = make_float2(__fsqrt_rn(t.x), __fsqrt_rn(t.y));
  const float2 lg = bs_logf(make_float2(__fdiv_rn(s.x, strike.x), __fdiv_rn(s.y, strike.y)));
  const float2 logv = make_float2(s.x == strike.x ? 0.0f : lg.x, s.y == strike.y ? 0.0f : lg.y);
  float2 d1 = fma2(mul2(v, v), f2(0.5f), r);
  d1 = fma2(d1, t, logv);
  const float2 den = mul2(v, sqrt_t);
  d1 = make_float2(__fdiv_rn(d1.x, den.x), __fdiv_rn(d1.y, den.y));
  const float2 d2 = sub2(d1, den);
  const float2 c1 = bs_cndf(d1, pow_tab);
  const float2 c2 = bs_cndf(d2, pow_tab);
  const float2 fv = mul2(strike, bs_exp0(mul2(mul2(r, f2(-1.0f)), t)));
  call = sub2(mul2(s, c1), mul2(fv, c2));
  put = sub2(mul2(fv, sub2(f2(1.0f), c2)), mul2(s, sub2(f2(1.0f), c1)));
}

// Every kernel below prices two options per thread, once: as many CTAs as the
// options need, so the hardware's scheduler evens out the SMs and a CTA's
// loads overlap its neighbours' arithmetic and stores. One wave of resident
// CTAs stepping through the options in a loop measured 107 against 96 us (10M
// records) and 60 against 58 us (10M in arrays). Lanes past the end price a
// dummy option and store nothing, because bs_fast_expf shuffles across the
// warp.

// A record as one 32-byte access: its whole DRAM sector in one instruction
// (as two 16-byte ones 119 instead of 107 us, 10M records). Streamed: nothing
// is reused.
struct BsRecord {
  float f[8];
};
template <bool V8>
HBSG_DEV BsRecord ld_record(const float* p) {
  BsRecord r;
  if constexpr (!V8) {  // 16-byte aligned records
    const float4 x = __ldcs(reinterpret_cast<const float4*>(p));
    const float4 y = __ldcs(reinterpret_cast<const float4*>(p) + 1);
    return {{x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w}};
  }
  asm volatile(
      "ld.global.L1::no_allocate.L2::evict_first.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n"
      : "=f"(r.f[0]), "=f"(r.f[1]), "=f"(r.f[2]), "=f"(r.f[3]), "=f"(r.f[4]), "=f"(r.f[5]),
        "=f"(r.f[6]), "=f"(r.f[7])
      : "l"(p));
  return r;
}
template <bool V8>
HBSG_DEV void st_record(float* p, const BsRecord& r) {
  if constexpr (!V8) {
    __stcs(reinterpret_cast<float4*>(p), make_float4(r.f[0], r.f[1], r.f[2], r.f[3]));
    __stcs(reinterpret_cast<float4*>(p) + 1, make_float4(r.f[4], r.f[5], r.f[6], r.f[7]));
    return;
  }
  asm volatile(
      "st.global.L1::no_allocate.L2::evict_first.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};\n" ::"l"(
          p),
      "f"(r.f[0]), "f"(r.f[1]), "f"(r.f[2]), "f"(r.f[3]), "f"(r.f[4]), "f"(r.f[5]), "f"(r.f[6]),
      "f"(r.f[7])
      : "memory");
}

// Records in place, 32-byte (V8) or 16-byte aligned; the whole record is stored back (its
// input fields unchanged), so its sector is written whole and never needs a
// fill from DRAM after the streaming load evicted it.
template <bool V8>
__global__ void __launch_bounds__(kBsThreads) bs_records_kernel(float* __restrict__ data,
                                                                long n) {
  const float pow_tab = bs_pow_table();
  const long i = (long)blockIdx.x * (2 * kBsThreads) + threadIdx.x, j = i + kBsThreads;
  BsRecord a = {{1.f, 1.f, 0.f, 1.f, 1.f, 0.f, 0.f, 0.f}}, b = a;
  if (i < n) a = ld_record<V8>(data + 8 * i);
  if (j < n) b = ld_record<V8>(data + 8 * j);
  float2 call, put;
  bs_price(make_float2(a.f[0], b.f[0]), make_float2(a.f[1], b.f[1]), make_float2(a.f[2], b.f[2]),
           make_float2(a.f[3], b.f[3]), make_float2(a.f[4], b.f[4]), call, put, pow_tab);
  a.f[5] = call.x;
  a.f[6] = put.x;
  b.f[5] = call.y;
  b.f[6] = put.y;
  if (i < n) st_record<V8>(data + 8 * i, a);
  if (j < n) st_record<V8>(data + 8 * j, b);
}

// Records at any 4-byte alignment: scalar loads, call and put stored alone.
__global__ void __launch_bounds__(kBsThreads) bs_records_scalar_kernel(float* __restrict__ data,
                                                                       long n) {
  const float pow_tab = bs_pow_table();
  const long i = (long)blockIdx.x * (2 * kBsThreads) + threadIdx.x, j = i + kBsThreads;
  const bool has0 = i < n, has1 = j < n;
  float* o = data + 8 * (has0 ? i : 0);
  float* p = data + 8 * (has1 ? j : 0);
  float2 call, put;
  bs_price(make_float2(has0 ? o[0] : 1.f, has1 ? p[0] : 1.f),
           make_float2(has0 ? o[1] : 1.f, has1 ? p[1] : 1.f),
           make_float2(has0 ? o[2] : 0.f, has1 ? p[2] : 0.f),
           make_float2(has0 ? o[3] : 1.f, has1 ? p[3] : 1.f),
           make_float2(has0 ? o[4] : 1.f, has1 ? p[4] : 1.f), call, put, pow_tab);
  if (has0) {
    o[5] = call.x;
    o[6] = put.x;
  }
  if (has1) {
    p[5] = call.y;
    p[6] = put.y;
  }
}

// Separate arrays. VEC (all seven 8-byte aligned): a thread's two options are
// consecutive, loaded and stored as 8-byte vectors (the last pair of an odd n
// holds one option); otherwise they are a CTA's width apart.
template <bool VEC>
__global__ void __launch_bounds__(kBsThreads)
    bs_arrays_kernel(const float* __restrict__ s, const float* __restrict__ strike,
                     const float* __restrict__ r, const float* __restrict__ v,
                     const float* __restrict__ t, float* __restrict__ call,
                     float* __restrict__ put, long n) {
  const float pow_tab = bs_pow_table();
  float2 C, P;
  if constexpr (VEC) {
    const long q = (long)blockIdx.x * kBsThreads + threadIdx.x;
    const bool both = q < n / 2, one = !both && 2 * q < n;
    float2 S = f2(1.f), K = f2(1.f), R = f2(0.f), V = f2(1.f), T = f2(1.f);
    if (both) {
      S = __ldcs(reinterpret_cast<const float2*>(s) + q);
      K = __ldcs(reinterpret_cast<const float2*>(strike) + q);
      R = __ldcs(reinterpret_cast<const float2*>(r) + q);
      V = __ldcs(reinterpret_cast<const float2*>(v) + q);
      T = __ldcs(reinterpret_cast<const float2*>(t) + q);
    } else if (one) {
      S.x = s[n - 1];
      K.x = strike[n - 1];
      R.x = r[n - 1];
      V.x = v[n - 1];
      T.x = t[n - 1];
    }
    bs_price(S, K, R, V, T, C, P, pow_tab);
    if (both) {
      __stcs(reinterpret_cast<float2*>(call) + q, C);
      __stcs(reinterpret_cast<float2*>(put) + q, P);
    } else if (one) {
      call[n - 1] = C.x;
      put[n - 1] = P.x;
    }
  } else {
    const long i = (long)blockIdx.x * (2 * kBsThreads) + threadIdx.x, j = i + kBsThreads;
    const bool has0 = i < n, has1 = j < n;
    const long ii = has0 ? i : n - 1, jj = has1 ? j : n - 1;  // past the end: the last option
    bs_price(make_float2(__ldcs(s + ii), __ldcs(s + jj)),
             make_float2(__ldcs(strike + ii), __ldcs(strike + jj)),
             make_float2(__ldcs(r + ii), __ldcs(r + jj)),
             make_float2(__ldcs(v + ii), __ldcs(v + jj)),
             make_float2(__ldcs(t + ii), __ldcs(t + jj)), C, P, pow_tab);
    if (has0) {
      __stcs(call + i, C.x);
      __stcs(put + i, P.x);
    }
    if (has1) {
      __stcs(call + j, C.y);
      __stcs(put + j, P.y);
    }
  }
}

static bool overlaps(const void* a, long abytes, const void* b, long bbytes) {
  const char* x = static_cast<const char*>(a);
  const char* y = static_cast<const char*>(b);
  return x < y + bbytes && y < x + abytes;
}

}  // namespace hbsg

using namespace hbsg;

extern "C" int hbsg_blackscholes(hbsg_option* options, int64_t num_option, hbsg_stream_t stream) {
  if (num_option < 0) return HBSG_ERR_INVALID_ARG;
  if (num_option == 0) return HBSG_OK;
  if (!options) return HBSG_ERR_INVALID_ARG;
  if (current_device_sms(nullptr) < 0) return HBSG_ERR_NO_DEVICE;
  float* data = reinterpret_cast<float*>(options);
  const cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const long blocks = (num_option + 2 * kBsThreads - 1) / (2 * kBsThreads);
  if (blocks > 0x7fffffffL) return HBSG_ERR_UNSUPPORTED;
  if ((reinterpret_cast<uintptr_t>(data) & 31) == 0)
    bs_records_kernel<true><<<(unsigned)blocks, kBsThreads, 0, st>>>(data, num_option);
  else if ((reinterpret_cast<uintptr_t>(data) & 15) == 0)
    bs_records_kernel<false><<<(unsigned)blocks, kBsThreads, 0, st>>>(data, num_option);
  else
    bs_records_scalar_kernel<<<(unsigned)blocks, kBsThreads, 0, st>>>(data, num_option);
  return cudaGetLastError() == cudaSuccess ? HBSG_OK : HBSG_ERR_LAUNCH;
}

extern "C" int hbsg_blackscholes_arrays(const float* s, const float* strike, const float* r,
                                        const float* v, const float* t, float* call, float* put,
                                        int64_t n, hbsg_stream_t stream) {
  if (n < 0) return HBSG_ERR_INVALID_ARG;
  if (n == 0) return HBSG_OK;
  if (!s || !strike || !r || !v || !t || !call || !put) return HBSG_ERR_INVALID_ARG;
  const long nb = (long)n * 4;
  const float* ins[5] = {s, strike, r, v, t};
  if (overlaps(call, nb, put, nb)) return HBSG_ERR_INVALID_ARG;
  for (const float* in : ins)
    if (overlaps(in, nb, call, nb) || overlaps(in, nb, put, nb)) return HBSG_ERR_INVALID_ARG;
  if (current_device_sms(nullptr) < 0) return HBSG_ERR_NO_DEVICE;
  uintptr_t bits = reinterpret_cast<uintptr_t>(call) | reinterpret_cast<uintptr_t>(put);
  for (const float* in : ins) bits |= reinterpret_cast<uintptr_t>(in);
  const cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const long blocks = (n + 2 * kBsThreads - 1) / (2 * kBsThreads);
  if (blocks > 0x7fffffffL) return HBSG_ERR_UNSUPPORTED;
  if ((bits & 7) == 0)
    bs_arrays_kernel<true>
        <<<(unsigned)blocks, kBsThreads, 0, st>>>(s, strike, r, v, t, call, put, n);
  else
    bs_arrays_kernel<false>
        <<<(unsigned)blocks, kBsThreads, 0, st>>>(s, strike, r, v, t, call, put, n);
  return cudaGetLastError() == cudaSuccess ? HBSG_OK : HBSG_ERR_LAUNCH;
}
