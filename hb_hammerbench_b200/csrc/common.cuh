// Shared device helpers for the sm_100a SGEMM kernels (cp.async, mbarrier,
// TMA, tcgen05). Inline PTX written from the PTX ISA; no library templates.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#define HBSG_DEV __device__ __forceinline__

namespace hbsg {

// ---- cp.async (global -> shared, bypassing registers) ---------------------
// src_bytes < cp-size zero-fills the rest of the destination; 0 reads nothing.
HBSG_DEV void cp_async16(void* smem, const void* gmem, int src_bytes) {
  unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(src_bytes)
               : "memory");
}
HBSG_DEV void cp_async4(void* smem, const void* gmem, int src_bytes) {
  unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(s), "l"(gmem), "r"(src_bytes)
               : "memory");
}
HBSG_DEV void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
HBSG_DEV void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// ---- programmatic dependent launch ------------------------------------------
// A kernel launched with launch_after(..., true) may start while the kernel
// before it in the stream still runs, once every CTA of that one has called
// grid_dep_trigger (or exited). grid_dep_wait returns when that kernel has
// completed and its writes are visible; nothing it writes may be touched
// before. Both do nothing in an ordinary launch.
HBSG_DEV void grid_dep_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
HBSG_DEV void grid_dep_trigger() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }

HBSG_DEV uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// ---- mbarrier ---------------------------------------------------------------
HBSG_DEV void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
HBSG_DEV void fence_barrier_init() {
  asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
}
HBSG_DEV void mbar_arrive(uint64_t* bar) {
  asm volatile(
      "{\n\t.reg .b64 st;\n\t"
      "mbarrier.arrive.shared::cta.b64 st, [%0];\n\t}\n" ::"r"(smem_u32(bar))
      : "memory");
}
HBSG_DEV void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile(
      "{\n\t.reg .b64 st;\n\t"
      "mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n\t}\n" ::"r"(smem_u32(bar)),
      "r"(bytes)
      : "memory");
}
// One probe of the phase with the given parity; returns true once it completed.
HBSG_DEV bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// ---- row and column scales of the scaled split-BF16 forms --------------------
// frexp exponent of max|x| from its FP32 bit pattern: the scale 2^-e the
// split applied to that row or column (0 for zero, non-finite or absent).
HBSG_DEV int pow2_exp_of_bits(uint32_t bits) {
  const int E = (int)((bits >> 23) & 0xffu);
  if (E == 0xff || bits == 0u) return 0;
  // a subnormal maximum is bits * 2^-149, its top bit 31 - clz
  return E != 0 ? E - 126 : -117 - __clz((int)bits);
}

// x * 2^s for scales that are no normal float, |s| < 1000: the product is exact
// in FP64, so the conversion back rounds once, as ldexpf does (and, unlike it,
// is no call, which would hold the epilogue's registers at every use).
HBSG_DEV float scale_pow2_wide(float x, int s) {
  return __double2float_rn((double)x * __hiloint2double((1023 + s) << 20, 0));
}

HBSG_DEV float scale_pow2(float x, int s) {
  return s >= -126 && s <= 127 ? x * __uint_as_float((uint32_t)(s + 127) << 23)
                               : scale_pow2_wide(x, s);
}

}  // namespace hbsg
