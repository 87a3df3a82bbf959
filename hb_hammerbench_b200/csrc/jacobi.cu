// 7-point Jacobi step on a 3-D grid for sm_100a: the suite's dense stencil
// benchmark (apps/jacobi) on the same host interface as the SGEMM path.
//
// Reference: the device kernel `kernel(c0, c1, A0, Anext, nx, ny, nz, pod_id)`
// (apps/jacobi/kernel.cpp:47-143) tiles x and y over the 16 x 8 tile group and
// streams z through scratchpad; its result must equal the host reference
// host_jacobi (apps/jacobi/main.cpp:19-48) exactly (main.cpp:141-150):
//   Anext[x,y,z] = c1 * (A[x-1] + A[x+1] + A[y-1] + A[y+1] + A[z-1] + A[z+1])
//                  - c0 * A[x,y,z]
// with neighbours outside the grid taken as 0.0f, the six-term sum taken left
// to right and the two products and the difference each rounded once (no
// fused multiply-add). Element (x, y, z) lies at ((y * nx) + x) * nz + z.
//
// B200 form: the step reads each element once and writes each once (8 bytes
// per point), so it is HBM-bound. A CTA of 32 (z) x 8 (x) threads marches
// along y over a slab of kYSlab planes: each thread keeps its column's y-1, y
// and y+1 values in registers, so only the new y+1 plane comes from DRAM,
// while the x and z neighbours come from the neighbouring threads' loads of
// the same plane (L1 hits). Loads go through the read-only path.
//
// Vector form (nz a multiple of 4, both grids 16-byte aligned): a thread owns
// 4 consecutive z of its column (one 16-byte load per plane and neighbour
// row, one 16-byte store), the z neighbours of its own 4 values are in its
// registers, those across lanes come by warp shuffle, and only the warp's
// two edge lanes load the z halo. That issues ~1/3 of the scalar form's
// instructions per point (the scalar form measured 66 % issue-active at 0.60
// of the HBM roof on 512^3).
//
// Ring form (the vector form's condition, grids that ring_wins): the vector form
// has one plane's loads in flight per warp and waits for each (5.3 TB/s at 53 %
// issue-active, DRAM traffic already the ideal 1.05 GB on 512^3). Here a
// producer warp streams whole (10 rows x 136 z) plane tiles, halos included,
// through TMA into a ring of kRing planes in shared memory; coordinates
// outside the grid arrive as zeros, which is the boundary condition. The
// compute warps march along y reading the ring: x neighbours from the plane's
// own tile, y neighbours kept in registers. 512^3: 201 -> 164 us (6.55 TB/s, the
// measured copy bandwidth), 207 -> 181 us repeated until the power cap holds
// the clock down; 256^3 33.6 -> 28.5 us. Rings of 4-12 planes and
// slabs of 12-128: 6 planes (33 KB, six CTAs per SM) and slabs of 12 were best
// (12 planes 171 us, slabs of 32 174 us, of 128 209 us).
#include <cuda.h>

#include "common.cuh"
#include "internal.h"

namespace hbsg {

static constexpr int kZT = 32;    // threads along z (one warp, coalesced)
static constexpr int kXT = 8;     // threads along x
static constexpr int kYSlab = 16;  // y planes per CTA

__global__ void __launch_bounds__(kZT * kXT) jacobi_kernel(float c0f, float c1f,
                                                           const float* __restrict__ A0,
                                                           float* __restrict__ An, int nx, int ny,
                                                           int nz) {
  const int z = blockIdx.x * kZT + threadIdx.x;
  const int x = blockIdx.y * kXT + threadIdx.y;
  const int y0 = blockIdx.z * kYSlab;
  if (z >= nz || x >= nx) return;
  const long sx = nz;
  const long sy = (long)nx * nz;
  const int y1 = min(ny, y0 + kYSlab);
  const long col = (long)x * sx + z;  // element (x, 0, z)
  float ym = y0 > 0 ? __ldg(A0 + col + (long)(y0 - 1) * sy) : 0.0f;
  float cur = __ldg(A0 + col + (long)y0 * sy);
  for (int y = y0; y < y1; ++y) {
    const long i = col + (long)y * sy;
    const float yp = y + 1 < ny ? __ldg(A0 + i + sy) : 0.0f;
    const float xm = x > 0 ? __ldg(A0 + i - sx) : 0.0f;
    const float xp = x < nx - 1 ? __ldg(A0 + i + sx) : 0.0f;
    const float zm = z > 0 ? __ldg(A0 + i - 1) : 0.0f;
    const float zp = z < nz - 1 ? __ldg(A0 + i + 1) : 0.0f;
    const float nb = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(xm, xp), ym), yp), zm), zp);
    An[i] = __fsub_rn(__fmul_rn(c1f, nb), __fmul_rn(c0f, cur));
    ym = cur;
    cur = yp;
  }
}

static constexpr int kZ4T = 32;  // threads along z in the vector form (128 z per warp)

__global__ void __launch_bounds__(kZ4T * kXT) jacobi_kernel4(float c0f, float c1f,
                                                             const float* __restrict__ A0,
                                                             float* __restrict__ An, int nx, int ny,
                                                             int nz) {
  const int lane = threadIdx.x;  // one warp per x row of the block
  const int zq = blockIdx.x * kZ4T + lane;
  const int x = blockIdx.y * kXT + threadIdx.y;
  const int y0 = blockIdx.z * kYSlab;
  if (x >= nx) return;  // whole warp (the warp shares x)
  const int nq = nz >> 2;
  const bool live = zq < nq;
  const int z0 = 4 * zq;
  const long sx = nz;
  const long sy = (long)nx * nz;
  const int y1 = min(ny, y0 + kYSlab);
  const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
  // element (x, y, z0) of the first plane; lanes past the end point at the
  // row's first quad and never load or store through it
  const long col = (long)x * sx + (live ? z0 : 0);
  const bool has_xm = x > 0, has_xp = x < nx - 1;
  const bool has_zm = live && z0 > 0, has_zp = live && z0 + 4 < nz;
  auto ld4 = [](const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); };
  float4 ym = (live && y0 > 0) ? ld4(A0 + col + (long)(y0 - 1) * sy) : zero4;
  float4 cur = live ? ld4(A0 + col + (long)y0 * sy) : zero4;
  for (int y = y0; y < y1; ++y) {
    const long i = col + (long)y * sy;
    const float4 yp = (live && y + 1 < ny) ? ld4(A0 + i + sy) : zero4;
    const float4 xm = (live && has_xm) ? ld4(A0 + i - sx) : zero4;
    const float4 xp = (live && has_xp) ? ld4(A0 + i + sx) : zero4;
    // z neighbours across the thread's quad: the lanes beside it, or the
    // global halo at the warp's edges; 0 outside the grid
    const float up = __shfl_up_sync(0xffffffffu, cur.w, 1);
    const float dn = __shfl_down_sync(0xffffffffu, cur.x, 1);
    float zm0 = 0.0f, zp3 = 0.0f;
    if (has_zm) zm0 = lane > 0 ? up : __ldg(A0 + i - 1);
    if (has_zp) zp3 = lane < kZ4T - 1 ? dn : __ldg(A0 + i + 4);
    const float xs[4] = {xm.x, xm.y, xm.z, xm.w}, xq[4] = {xp.x, xp.y, xp.z, xp.w};
    const float ys[4] = {ym.x, ym.y, ym.z, ym.w}, yq[4] = {yp.x, yp.y, yp.z, yp.w};
    const float c[4] = {cur.x, cur.y, cur.z, cur.w};
    const float zm[4] = {zm0, cur.x, cur.y, cur.z}, zp[4] = {cur.y, cur.z, cur.w, zp3};
    float o[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float nb =
          __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(xs[e], xq[e]), ys[e]), yq[e]), zm[e]),
                    zp[e]);
      o[e] = __fsub_rn(__fmul_rn(c1f, nb), __fmul_rn(c0f, c[e]));
    }
    if (live) *reinterpret_cast<float4*>(An + i) = make_float4(o[0], o[1], o[2], o[3]);
    ym = cur;
    cur = yp;
  }
}

// ---- ring form ----------------------------------------------------------------
static constexpr int kRing = 6;          // plane tiles in flight or in use
static constexpr int kRingSlab = 12;     // y planes per CTA
static constexpr int kRingZ = 4 * kZ4T;  // z per CTA
static constexpr int kTileZ = kRingZ + 8;  // + 4 on either side (16-byte aligned box)
static constexpr int kTileX = kXT + 2;
static constexpr int kTileBytes = kTileZ * kTileX * 4;
static constexpr int kTileStride = (kTileBytes + 127) / 128 * 128;
static constexpr int kRingThreads = kZ4T * kXT + 32;  // 8 compute warps, 1 producer
static constexpr int kRingSmem = 128 + kRing * kTileStride + 2 * kRing * 8 + 16;
static constexpr unsigned long long kRingWaitNs = 4000000000ull;  // bound of every wait

static __device__ int g_jacobi_error = 0;

HBSG_DEV unsigned long long ring_timer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

// Bounded wait on a barrier phase; false when it expired here or elsewhere in
// the CTA (every role then leaves its loop).
HBSG_DEV bool ring_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  if (mbar_try_wait(bar, parity)) return true;
  const unsigned long long t0 = ring_timer();
  for (uint32_t i = 0;; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((i & 63) == 0) {
      if (*abort_flag) return false;
      if (ring_timer() - t0 > kRingWaitNs) {
        *abort_flag = 1;
        atomicExch(&g_jacobi_error, (int)HBSG_ERR_DEVICE_TIMEOUT);
        return false;
      }
    }
  }
}

__global__ void __launch_bounds__(kRingThreads)
    jacobi_ring_kernel(const __grid_constant__ CUtensorMap map, float c0f, float c1f,
                       float* __restrict__ An, int nx, int ny, int nz) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((128u - (smem_u32(smem_raw) & 127u)) & 127u);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + kRing * kTileStride);
  uint64_t* empty = full + kRing;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(empty + kRing);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int zb = blockIdx.x * kRingZ, x0 = blockIdx.y * kXT, y0 = blockIdx.z * kRingSlab;
  const int y1 = min(ny, y0 + kRingSlab);
  const int planes = y1 - y0 + 2;  // y0 - 1 .. y1
  if (threadIdx.x == 0) {
    for (int i = 0; i < kRing; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], kXT);
    }
    *abort_flag = 0;
    fence_barrier_init();
  }
  __syncthreads();
  if (warp == kXT) {
    // ---- producer: plane p of the slab is y0 - 1 + p ----
    if (lane == 0) {
      for (int p = 0; p < planes; ++p) {
        const int s = p % kRing;
        if (!ring_wait(&empty[s], ((p / kRing) & 1) ^ 1, abort_flag)) break;
        mbar_arrive_expect_tx(&full[s], kTileBytes);
        asm volatile(
            "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes"
            " [%0], [%1, {%2, %3, %4}], [%5];\n" ::"r"(smem_u32(smem + s * kTileStride)),
            "l"(reinterpret_cast<uint64_t>(&map)), "r"(zb - 4), "r"(x0 - 1), "r"(y0 - 1 + p),
            "r"(smem_u32(&full[s]))
            : "memory");
      }
    }
  } else {
    // ---- compute: warp = x row, lane = 4 consecutive z ----
    const int x = x0 + warp;
    const int z0 = zb + 4 * lane;
    const bool live = x < nx && z0 < nz;
    const float* row = reinterpret_cast<const float*>(smem) + (warp + 1) * kTileZ + 4 + 4 * lane;
    constexpr int kTileFloats = kTileStride / 4;
    auto ld4 = [](const float* p) { return *reinterpret_cast<const float4*>(p); };
    float* out = An + ((long)y0 * nx + (live ? x : 0)) * nz + (live ? z0 : 0);
    const long sy = (long)nx * nz;
    float4 ym, cur;
    // a wait passes when it passed on every lane, so a warp leaves as one
    bool ok = __all_sync(0xffffffffu, ring_wait(&full[0], 0, abort_flag));
    if (ok) {
      ym = ld4(row);
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[0]);
      ok = __all_sync(0xffffffffu, ring_wait(&full[1], 0, abort_flag));
    }
    if (ok) cur = ld4(row + kTileFloats);
    for (int p = 1; ok && p + 1 < planes; ++p, out += sy) {
      const int s = p % kRing, sn = (p + 1) % kRing;
      const float* c_row = row + s * kTileFloats;
      const float4 xm = ld4(c_row - kTileZ), xp = ld4(c_row + kTileZ);
      const float up = __shfl_up_sync(0xffffffffu, cur.w, 1);
      const float dn = __shfl_down_sync(0xffffffffu, cur.x, 1);
      const float zm0 = lane > 0 ? up : c_row[-1];
      const float zp3 = lane < kZ4T - 1 ? dn : c_row[4];
      if (!__all_sync(0xffffffffu, ring_wait(&full[sn], ((p + 1) / kRing) & 1, abort_flag))) break;
      const float4 yp = ld4(row + sn * kTileFloats);
      const float xs[4] = {xm.x, xm.y, xm.z, xm.w}, xq[4] = {xp.x, xp.y, xp.z, xp.w};
      const float ys[4] = {ym.x, ym.y, ym.z, ym.w}, yq[4] = {yp.x, yp.y, yp.z, yp.w};
      const float c[4] = {cur.x, cur.y, cur.z, cur.w};
      const float zm[4] = {zm0, cur.x, cur.y, cur.z}, zp[4] = {cur.y, cur.z, cur.w, zp3};
      float o[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float nb = __fadd_rn(
            __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(xs[e], xq[e]), ys[e]), yq[e]), zm[e]), zp[e]);
        o[e] = __fsub_rn(__fmul_rn(c1f, nb), __fmul_rn(c0f, c[e]));
      }
      // plane p has been read (its values are in registers) by this warp
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[s]);
      if (live) __stcs(reinterpret_cast<float4*>(out), make_float4(o[0], o[1], o[2], o[3]));
      ym = cur;
      cur = yp;
    }
  }
  // after a bounded abort, copies still in flight get a moment to land
  if (*abort_flag) {
    const unsigned long long t0 = ring_timer();
    while (ring_timer() - t0 < 2000000ull) {
    }
  }
}

// Where the ring form is the faster, by GPU time of launches in a graph (vector
// against ring form, us). It needs a march to stream along, z that fills three
// quarters of its 128-wide tiles (512 x 512 x 32 39.3 against 41.7; 300 x 200 x
// 260 33.0 against 32.9-35.0), and:
//   - grids whose in- and output exceed what L2 holds of them (88 MB): 4 planes
//     or more (20000 x 4 x 512 65.5 / 62.2, 5000 x 5 x 512 21.3 / 18.1; but 10000 x
//     3 x 1024 51.5 / 54.8, 60000 x 1 x 256 34.3 / 45.0);
//   - smaller ones of several z tiles: a second slab, where the vector form waits
//     for 16 planes one by one (64 x 20 x 512 8.0 / 4.7, 300 x 14 x 256 7.0 / 5.1),
//     from 17 planes on or with a CTA for every SM (64 x 14 x 512 6.8 / 7.0); on one
//     slab each plane tile's halos cost more than the streaming saves (5000 x 1 x
//     512 5.3 / 7.3, 148 x 10 x 4096 9.4 / 10.2);
//   - smaller ones of a single z tile: from 17 planes on, where an SM takes no more
//     CTAs in turn than of the vector form, whose slabs are longer (64 x 64 x 128
//     5.5 / 4.9, 180 x 220 x 128 7.8 / 7.5; but 170 x 170 x 128, three CTAs an SM for
//     two, 6.8 / 7.7, 1200 x 40 x 128 8.6 / 10.4, 300 x 300 x 100 12.3 / 14.7).
static bool ring_wins(int nx, int ny, int nz, int sms) {
  const long zt = ((long)nz + kRingZ - 1) / kRingZ, xt = ((long)nx + kXT - 1) / kXT,
             yt = ((long)ny + kRingSlab - 1) / kRingSlab;
  if (4L * nz < 3 * zt * kRingZ || xt > 65535 || yt > 65535) return false;
  if ((long)nx * ny * nz > 11000000L) return ny >= 4;
  const long ctas = zt * xt * yt;
  if (zt == 1) {
    const long vector_ctas = xt * (((long)ny + kYSlab - 1) / kYSlab);
    return ny > kYSlab && (ctas + sms - 1) / sms <= (vector_ctas + sms - 1) / sms;
  }
  return ny > kYSlab || (ny > kRingSlab && ctas >= sms);
}

static bool ring_map(CUtensorMap* map, const float* A0, int nx, int ny, int nz) {
  return tc_make_f32_map_3d(map, A0, nz, nx, ny, kTileZ, kTileX, 1);
}

int jacobi_read_and_clear_device_error() {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_jacobi_error, sizeof(int)) != cudaSuccess) return HBSG_ERR_CUDA;
  if (v != 0) {
    const int zero = 0;
    cudaMemcpyToSymbol(g_jacobi_error, &zero, sizeof(int));
  }
  return v;
}

}  // namespace hbsg

using namespace hbsg;

extern "C" int hbsg_jacobi(int c0, int c1, const float* A0, float* Anext, int nx, int ny, int nz,
                           hbsg_stream_t stream) {
  if (nx < 0 || ny < 0 || nz < 0) return HBSG_ERR_INVALID_ARG;
  const long n = (long)nx * ny * nz;
  if (n == 0) return HBSG_OK;
  if (!A0 || !Anext) return HBSG_ERR_INVALID_ARG;
  // the step reads neighbours of every element: the output may not overlap the input
  const char* a = reinterpret_cast<const char*>(A0);
  const char* b = reinterpret_cast<const char*>(Anext);
  if (a < b + n * 4 && b < a + n * 4) return HBSG_ERR_INVALID_ARG;
  const int sms = current_device_sms(nullptr);
  if (sms < 0) return HBSG_ERR_NO_DEVICE;
  if ((nz + kZT - 1) / kZT > 0x7fffffff || (nx + kXT - 1) / kXT > 65535 ||
      (ny + kYSlab - 1) / kYSlab > 65535)
    return HBSG_ERR_UNSUPPORTED;
  const cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const bool vec = (nz & 3) == 0 && ((reinterpret_cast<uintptr_t>(A0) | reinterpret_cast<uintptr_t>(Anext)) & 15) == 0;
  const bool ring = vec && ring_wins(nx, ny, nz, sms);
  CUtensorMap map;
  if (ring && ring_map(&map, A0, nx, ny, nz)) {
    static uint64_t mask = 0;
    if (!set_smem_once(reinterpret_cast<const void*>(jacobi_ring_kernel), kRingSmem, &mask))
      return HBSG_ERR_LAUNCH;
    const dim3 grid((nz + kRingZ - 1) / kRingZ, (nx + kXT - 1) / kXT,
                    (ny + kRingSlab - 1) / kRingSlab);
    jacobi_ring_kernel<<<grid, kRingThreads, kRingSmem, st>>>(map, (float)c0, (float)c1, Anext, nx,
                                                              ny, nz);
  } else if (vec) {
    const dim3 grid((nz / 4 + kZ4T - 1) / kZ4T, (nx + kXT - 1) / kXT, (ny + kYSlab - 1) / kYSlab);
    jacobi_kernel4<<<grid, dim3(kZ4T, kXT), 0, st>>>((float)c0, (float)c1, A0, Anext, nx, ny, nz);
  } else {
    const dim3 grid((nz + kZT - 1) / kZT, (nx + kXT - 1) / kXT, (ny + kYSlab - 1) / kYSlab);
    jacobi_kernel<<<grid, dim3(kZT, kXT), 0, st>>>((float)c0, (float)c1, A0, Anext, nx, ny, nz);
  }
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? HBSG_OK : HBSG_ERR_LAUNCH;
}
