// FP32 SIMT (FFMA) SGEMM tile body for sm_100a, shared by the single and
// batched launch (ffma_sgemm.cu) and the grouped launch (grouped.cu). The
// design and the reference lines it follows are described in ffma_sgemm.cu.
#pragma once

#include "common.cuh"
#include "internal.h"

namespace hbsg {

static constexpr int kFfmaKU = 16;         // k steps the inner loop unrolls
static constexpr int kFfmaProducers = 128;  // producer threads (one warpgroup, the CTA's last)

template <int BM, int BN, int BK, int WM, int WN, int STAGES>
struct FfmaShape {
  static constexpr int kWarpsM = BM / WM;
  static constexpr int kWarpsN = BN / WN;
  static constexpr int kCompute = kWarpsM * kWarpsN * 32;  // compute threads
  static constexpr int kThreads = kCompute + kFfmaProducers;
  static constexpr int TM = WM / 8;
  static constexpr int TN = WN / 4;
  static constexpr int kAStage = BK * BM;
  static constexpr int kBStage = BK * BN;
  // Tiles whose copies are in flight before one is published to the compute
  // warps (see ffma_produce), and so the depth of the staging rings.
  static constexpr int kAhead = STAGES - 2;
  // the stage ring, then a staging ring per operand that is k-contiguous in
  // memory (row-major A, transposed B)
  static constexpr int smem_bytes(bool ta, bool tb) {
    return 4 * (STAGES * (kAStage + kBStage) +
                (kAhead + 1) * ((ta ? 0 : kAStage) + (tb ? kBStage : 0)));
  }
  // Resident CTAs per SM and the register split. All threads launch with
  // kLaunchRegs; setmaxnreg then moves registers from the producers to the
  // compute warps (0: no split).
  static constexpr int kMinBlocks = kCompute > 128 ? 1 : TM * TN <= 32 ? 3 : 2;
  static constexpr int kLaunchRegs = kThreads == 384 ? 168 : kMinBlocks == 3 ? 80 : 128;
  static constexpr int kComputeRegs =
      TM * TN == 128 ? (kCompute == 256 ? 216 : 208) : TM * TN == 32 ? 104 : 0;
  static constexpr int kProducerRegs =
      kComputeRegs == 0 ? 0 : (kLaunchRegs * kThreads - kComputeRegs * kCompute) / kFfmaProducers;
  static_assert(kComputeRegs == 0 ||
                    kProducerRegs * kFfmaProducers + kComputeRegs * kCompute <=
                        kLaunchRegs * kThreads,
                "setmaxnreg hands out no more than the launch's registers");
  static_assert(kProducerRegs % 8 == 0 && kComputeRegs % 8 == 0, "setmaxnreg granularity");
  static_assert(kThreads % 128 == 0 && kCompute % 128 == 0, "whole warpgroups");
  static_assert(STAGES >= 2, "ring");
  static_assert(2 * STAGES + 1 <= 16, "named barriers");
  static_assert(TM % 4 == 0 && TN % 4 == 0, "16-byte fragments");
  static_assert(BK % kFfmaKU == 0, "BK");
};

// Named barriers of the stage ring: full (the stage holds its tile), empty
// (every compute warp has read it). bar.sync / bar.arrive order the shared
// memory accesses on both sides; nothing spins. Barrier 0 is __syncthreads.
template <int COUNT>
HBSG_DEV void ffma_bar_sync(int id) {
  asm volatile("bar.sync %0, %1;\n" ::"r"(id), "n"(COUNT) : "memory");
}
template <int COUNT>
HBSG_DEV void ffma_bar_arrive(int id) {
  asm volatile("bar.arrive %0, %1;\n" ::"r"(id), "n"(COUNT) : "memory");
}
template <int N>
HBSG_DEV void ffma_regs_dec() {
  if constexpr (N > 0) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(N));
}
template <int N>
HBSG_DEV void ffma_regs_inc() {
  if constexpr (N > 0) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(N));
}

// setmaxnreg hands out registers of the block's launch allotment; a kernel
// built with another register count than the split assumes would wait forever
// in setmaxnreg.inc, so launchers check the count once per kernel (cache: 0
// unchecked, 1 ok, -1 wrong) and refuse to launch otherwise.
template <class S>
static inline bool ffma_regs_ok(const void* kernel, int* cache) {
  if (S::kComputeRegs == 0) return true;
  int st = __atomic_load_n(cache, __ATOMIC_ACQUIRE);
  if (st == 0) {
    cudaFuncAttributes fa;
    st = cudaFuncGetAttributes(&fa, kernel) == cudaSuccess && fa.numRegs == S::kLaunchRegs ? 1 : -1;
    __atomic_store_n(cache, st, __ATOMIC_RELEASE);
  }
  return st == 1;
}

// One operand's BK x BX tile (k rows of BX elements of the m or n axis, that
// axis contiguous) in shared memory, filled from global memory by the
// producer warps in one of two ways:
//   KC (k contiguous in memory: row-major A, transposed B): a warp copies
//     blocks of 8 rows x 16 k (cp.async) into staging slots of its own and,
//     once they have landed, each thread stores 4 consecutive k of a row
//     transposed, four 4-byte stores. No other warp reads the slots, so they
//     need no barrier, and the loads of several tiles are in flight without
//     holding registers. Element (k, x) lies at k * BX + (x ^ 8 * ((k / 4) %
//     4)): the xor spreads the 8 rows x 4 chunks a warp stores at once over
//     all 32 banks, and keeps 4 consecutive x together for the 16-byte
//     fragment loads.
//   else (x contiguous: transposed A, row-major B): cp.async straight into
//     the stage.
// Copies are of 16 bytes when VEC, of 4 otherwise; k past k_end is
// zero-filled. Rows or columns outside the matrix only reach outputs that are
// never stored, so their loads are moved to the last valid one (or copy no
// bytes) instead of being predicated: a full tile's loads are one pointer add
// and one instruction each, which matters because a producer warp shares its
// scheduler's issue slots with the compute warps (with a predicate, two
// selects and a 64-bit multiply per copy, one 64 x 64 tile per SM with
// unaligned operands ran at 20 TFLOP/s, 43 so).
template <int BX, int BK, int NT, bool KC, bool VEC>
struct FfmaLoader {
  static constexpr int kWarps = NT / 32;
  static constexpr int kElems = VEC ? 4 : 1;  // per copy
  // KC: units of 4 k per thread; a warp covers 8 rows x 4 units. Consecutive
  // lanes take one row's 64 bytes (4 lanes with 16-byte copies, 16 with
  // 4-byte ones): with the rows on consecutive lanes the L1 lookups of the
  // copies held up the compute warps' fragment loads (4736 x 4096 x 4096 at 55
  // instead of 62 TFLOP/s).
  static constexpr int kUnits = BX * BK / 4 / NT;
  static constexpr int kKQ = BK / 16;  // warps side by side along k
  static constexpr int kRowStep = 8 * kWarps / kKQ;
  // x contiguous: a thread copies the same kXReps x of every kCopyStep-th k
  static constexpr int kPerRow = BX / kElems < NT ? BX / kElems : NT;
  static constexpr int kXReps = BX / kElems / kPerRow;
  static constexpr int kCopies = BK * kPerRow / NT;
  static constexpr int kCopyStep = NT / kPerRow;
  static_assert(!KC || (kWarps % kKQ == 0 && (BX * BK / 4) % NT == 0), "KC unit split");
  static_assert(KC || (NT % kPerRow == 0 && kXReps * kCopies * kElems * NT == BX * BK),
                "copy split");

  const float* src[KC ? kUnits : kXReps];  // next tile's first element, per row / x
  long step;                               // floats between a thread's copies (unaligned KC: of
                                           // one unit)
  int rows[KC && !VEC ? kUnits : 1];       // unaligned KC: rows of the matrix from src[i]'s on
  int bytes[KC ? 1 : kXReps];              // x contiguous: valid bytes of a copy
  int k;                                   // this thread's first k of the next tile

  __device__ __forceinline__ void init(const float* p, long ld, int X, int x0, int k_begin,
                                       int tid) {
    if constexpr (KC) {
      const int w = tid >> 5, lane = tid & 31;
      const int x = x0 + (w / kKQ) * 8 + (VEC ? lane >> 2 : lane >> 4);
      k = k_begin + (w % kKQ) * 16 + (VEC ? (lane & 3) * 4 : lane & 15);
      step = 2 * ld;
#pragma unroll
      for (int i = 0; i < kUnits; ++i) {
        src[i] = p + (long)min(x + i * kRowStep, X - 1) * ld + k;
        if constexpr (!VEC) rows[i] = X - (x + i * kRowStep);
      }
    } else {
      k = k_begin + tid / kPerRow;
      step = (long)kCopyStep * ld;
#pragma unroll
      for (int e = 0; e < kXReps; ++e) {
        const int x = x0 + (tid % kPerRow + e * kPerRow) * kElems;
        bytes[e] = max(0, min(kElems, X - x)) * 4;
        src[e] = p + (long)k * ld + (bytes[e] > 0 ? x : 0);
      }
    }
  }

  // Starts the copies of the next tile: into `slot` (KC, the tile's part of
  // the staging ring) or straight into `tile`. FULL: the tile ends at or
  // before k_end; otherwise k past it is zero-filled by copies of no bytes,
  // which still get an address inside the matrix.
  template <bool FULL>
  __device__ __forceinline__ void copy(float* tile, float* slot, int k_end, int tid) {
    if constexpr (KC) {
#pragma unroll
      for (int i = 0; i < kUnits; ++i) {
        if constexpr (VEC) {
          const int left = FULL ? 4 : max(0, min(4, k_end - k));
          const float* s = left > 0 ? src[i] : src[i] - k;  // (k = 0 of the row)
          cp_async16(slot + 4 * tid + 4 * NT * i, s, 4 * left);
        } else {
          const bool in = FULL || k < k_end;
          const float* s0 = in ? src[i] : src[i] - k;
          float* d = slot + 4 * (tid & ~31) + (tid & 31) + 4 * NT * i;
#pragma unroll
          for (int c = 0; c < 4; ++c)
            cp_async4(d + 32 * c, 2 * c < rows[i] ? s0 + c * step : s0, in ? 4 : 0);
        }
        src[i] += BK;
      }
    } else {
      float* dst = tile + (tid / kPerRow) * BX + (tid % kPerRow) * kElems;
#pragma unroll
      for (int e = 0; e < kXReps; ++e) {
#pragma unroll
        for (int i = 0; i < kCopies; ++i) {
          const bool in = FULL || k + i * kCopyStep < k_end;
          const float* s = in ? src[e] : src[e] - (long)(k + i * kCopyStep) * (step / kCopyStep);
          float* d = dst + i * kCopyStep * BX + e * kPerRow * kElems;
          if constexpr (VEC) cp_async16(d, s, in ? bytes[e] : 0);
          else cp_async4(d, s, in ? bytes[e] : 0);
          src[e] += step;
        }
      }
    }
    k += BK;
  }

  // KC: the landed slot stored transposed into the stage.
  __device__ __forceinline__ void transpose(float* tile, const float* slot, int tid) const {
    if constexpr (KC) {
      if constexpr (!VEC) __syncwarp();  // other lanes copied parts of this thread's unit
      const int w = tid >> 5, lane = tid & 31;
      const int row = (w / kKQ) * 8 + (lane >> 2);
      const int q = lane & 3;
      float* dst = tile + ((w % kKQ) * 16 + q * 4) * BX;
#pragma unroll
      for (int i = 0; i < kUnits; ++i) {
        const float4 v = *reinterpret_cast<const float4*>(slot + 4 * tid + 4 * NT * i);
        // rows 32 apart share the xor (it only changes bits 3 and 4)
        float* d = kRowStep % 32 == 0 ? dst + (row ^ (8 * q)) + i * kRowStep
                                      : dst + ((row + i * kRowStep) ^ (8 * q));
        d[0 * BX] = v.x;
        d[1 * BX] = v.y;
        d[2 * BX] = v.z;
        d[3 * BX] = v.w;
      }
      if constexpr (!VEC) __syncwarp();  // the slot is read before a lane refills it
    }
  }
};

// The tile body runs on two roles. The producer warpgroup fills a STAGES-deep
// shared-memory ring with both operands' tiles; the compute warps only read
// fragments and issue FMAs. (With the loads issued by the compute warps
// themselves, between barriers, their address arithmetic and load latency sat
// in the FMA stream of the one or two warps a scheduler has: 52.8 TFLOP/s on
// 4736 x 4096 x 4096 against 66.9 for the same loop with its loads left out,
// and half the rate on one 64 x 64 tile per SM.)
//
// Producer: fills the ring for one BM x BN output tile over k in [k_begin,
// k_end). The copies of S::kAhead tiles are in flight when a tile is
// published. Progress: a compute warp waits for tile j + 1 before it releases
// tile j (its fragments are prefetched across tiles), so tile j + 1 must be
// published before the producer waits for tile j's release, i.e. before it
// starts tile j + STAGES: at most STAGES - 2 tiles may be started and not yet
// published when it waits.
template <class S, int BM, int BN, int BK, int STAGES, bool VEC, bool TA, bool TB>
__device__ __forceinline__ void ffma_produce(const float* __restrict__ A, long lda,
                                             const float* __restrict__ B, long ldb, int M, int N,
                                             int k_begin, int k_end, int m0, int n0,
                                             float* smem) {
  constexpr int NT = kFfmaProducers;
  constexpr int L = S::kAhead;
  float* As = smem;
  float* Bs = smem + STAGES * S::kAStage;
  float* Sa = Bs + STAGES * S::kBStage;                  // A's staging ring (row-major A)
  float* Sb = Sa + (TA ? 0 : (L + 1) * S::kAStage);      // B's (transposed B)
  const int KT = k_end > k_begin ? (k_end - k_begin + BK - 1) / BK : 0;
  const int FT = k_end > k_begin ? (k_end - k_begin) / BK : 0;  // full tiles
  if (KT == 0) return;
  const int tid = (int)threadIdx.x - S::kCompute;
  FfmaLoader<BM, BK, NT, !TA, VEC> la;
  FfmaLoader<BN, BK, NT, TB, VEC> lb;
  la.init(A, lda, M, m0, k_begin, tid);
  lb.init(B, ldb, N, n0, k_begin, tid);
  int s = 0, g = 0;    // stage and staging slot of tile i
  int sj = 0, gj = 0;  // of tile j = i - L
  for (int i = 0; i < KT + L; ++i) {
    if (i < KT) {
      if (i >= STAGES) ffma_bar_sync<S::kThreads>(1 + STAGES + s);
      if (i < FT) {
        la.template copy<true>(As + s * S::kAStage, Sa + g * S::kAStage, k_end, tid);
        lb.template copy<true>(Bs + s * S::kBStage, Sb + g * S::kBStage, k_end, tid);
      } else {
        la.template copy<false>(As + s * S::kAStage, Sa + g * S::kAStage, k_end, tid);
        lb.template copy<false>(Bs + s * S::kBStage, Sb + g * S::kBStage, k_end, tid);
      }
      s = s + 1 == STAGES ? 0 : s + 1;
      g = g == L ? 0 : g + 1;
    }
    cp_async_commit();
    if (i >= L) {
      cp_async_wait<L>();
      la.transpose(As + sj * S::kAStage, Sa + gj * S::kAStage, tid);
      lb.transpose(Bs + sj * S::kBStage, Sb + gj * S::kBStage, tid);
      ffma_bar_arrive<S::kThreads>(1 + sj);
      sj = sj + 1 == STAGES ? 0 : sj + 1;
      gj = gj == L ? 0 : gj + 1;
    }
  }
}

// Compute: C tile = A rows x B columns from the ring the producer fills,
// written to C (row stride ldc).
// PAIR selects the packed two-lane FMA (__ffma2_rn, sm_100): each instruction
// performs two independent IEEE fused multiply-adds, so the per-element
// arithmetic is unchanged while half as many FMA instructions are issued.
//
// Both operands lie in shared memory as k rows with m / n contiguous, so a
// thread's fragment of one k is TM + TN floats (16-byte loads) and two
// fragments fit in registers beside the accumulators: the loads of k + 1 are
// issued before the FMAs of k, across tile boundaries too. Measured as a bare
// inner loop on static operands (TFLOP/s, 8 x 16 accumulators, two CTAs of 4
// compute warps per SM): 66.2, against 60.5 with A kept k-contiguous (16-byte
// loads of 4 k per row, whose 32 registers leave no room for a second
// fragment) and 62.3 with scalar FMAs; 4 x 8 accumulators, one CTA per SM:
// 63.0 against 55.4.
template <class S, int BM, int BN, int BK, int WM, int WN, int STAGES, bool PAIR, bool TA, bool TB>
__device__ __forceinline__ void ffma_compute(int M, int N, int k_begin, int k_end, int m0, int n0,
                                             float* C, long ldc, bool vec_store,
                                             const float* smem) {
  constexpr int TM = S::TM;
  constexpr int TN = S::TN;
  constexpr bool kSwzA = !TA, kSwzB = TB;  // k-contiguous in memory: stored swizzled

  const int KT = k_end > k_begin ? (k_end - k_begin + BK - 1) / BK : 0;
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int wm = warp / S::kWarpsN;
  const int wn = warp % S::kWarpsN;
  const int tm = lane & 7;
  const int tn = lane >> 3;

  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.0f;

  if (KT > 0) {
    // fragment of one k: rows 32 i + 4 tm + c, columns 16 j + 4 tn + c
    float4 af[2][TM / 4], bf[2][TN / 4];
    const float* a_w = smem + wm * WM;
    const float* b_w = smem + STAGES * S::kAStage + wn * WN;
    auto ld_frag = [&](const float* a_s, const float* b_s, int k, int buf) {
      const int sw = 8 * ((k >> 2) & 3);  // k is a compile-time constant
#pragma unroll
      for (int i = 0; i < TM / 4; ++i)
        af[buf][i] = *reinterpret_cast<const float4*>(a_s + k * BM + 32 * i +
                                                      ((4 * tm) ^ (kSwzA ? sw : 0)));
#pragma unroll
      for (int j = 0; j < TN / 4; ++j)
        bf[buf][j] = *reinterpret_cast<const float4*>(
            b_s + k * BN +
            (kSwzB ? ((16 * j) ^ (sw & 16)) + ((4 * tn) ^ (sw & 8)) : 16 * j + 4 * tn));
    };
    ffma_bar_sync<S::kThreads>(1);
    ld_frag(a_w, b_w, 0, 0);

    int slot = 0;
    for (int kt = 0; kt < KT; ++kt) {
      const int next = slot + 1 == STAGES ? 0 : slot + 1;
      const float* a_s = a_w + slot * S::kAStage;
      const float* b_s = b_w + slot * S::kBStage;
      // runs of 16 k; those wholly past k_end are left out
      const int runs =
          BK == kFfmaKU
              ? 1
              : min(BK / kFfmaKU, (k_end - k_begin - kt * BK + kFfmaKU - 1) / kFfmaKU);
#pragma unroll 1
      for (int h = 0; h < runs; ++h) {
#pragma unroll
        for (int k = 0; k < kFfmaKU; ++k) {
          const int cur = k & 1;
          if (k + 1 < kFfmaKU) {
            ld_frag(a_s, b_s, k + 1, cur ^ 1);
          } else if (h + 1 < runs) {
            a_s += kFfmaKU * BM;
            b_s += kFfmaKU * BN;
            ld_frag(a_s, b_s, 0, cur ^ 1);
          } else if (kt + 1 < KT) {
            ffma_bar_sync<S::kThreads>(1 + next);
            ld_frag(a_w + next * S::kAStage, b_w + next * S::kBStage, 0, cur ^ 1);
          }
          const float4(&a)[TM / 4] = af[cur];
          const float4(&b)[TN / 4] = bf[cur];
#pragma unroll
          for (int i = 0; i < TM; ++i) {
            const float4 a4 = a[i / 4];
            const float av = i % 4 == 0 ? a4.x : i % 4 == 1 ? a4.y : i % 4 == 2 ? a4.z : a4.w;
            if constexpr (PAIR) {
              const float2 a2 = make_float2(av, av);
#pragma unroll
              for (int j = 0; j < TN / 4; ++j) {
                const float2 lo =
                    __ffma2_rn(a2, make_float2(b[j].x, b[j].y),
                               make_float2(acc[i][4 * j + 0], acc[i][4 * j + 1]));
                const float2 hi =
                    __ffma2_rn(a2, make_float2(b[j].z, b[j].w),
                               make_float2(acc[i][4 * j + 2], acc[i][4 * j + 3]));
                acc[i][4 * j + 0] = lo.x;
                acc[i][4 * j + 1] = lo.y;
                acc[i][4 * j + 2] = hi.x;
                acc[i][4 * j + 3] = hi.y;
              }
            } else {
#pragma unroll
              for (int j = 0; j < TN / 4; ++j) {
                acc[i][4 * j + 0] = __fmaf_rn(av, b[j].x, acc[i][4 * j + 0]);
                acc[i][4 * j + 1] = __fmaf_rn(av, b[j].y, acc[i][4 * j + 1]);
                acc[i][4 * j + 2] = __fmaf_rn(av, b[j].z, acc[i][4 * j + 2]);
                acc[i][4 * j + 3] = __fmaf_rn(av, b[j].w, acc[i][4 * j + 3]);
              }
            }
          }
        }
      }
      // the producer waits for this before it refills the stage (it fills
      // the last STAGES tiles' stages no more)
      if (kt + STAGES < KT) ffma_bar_arrive<S::kThreads>(1 + STAGES + slot);
      slot = next;
    }
  }

  // Epilogue: direct stores.
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int r = m0 + wm * WM + 32 * (i / 4) + 4 * tm + i % 4;
    if (r >= M) continue;
    float* crow = C + (long)r * ldc;
#pragma unroll
    for (int j = 0; j < TN / 4; ++j) {
      const int c = n0 + wn * WN + 16 * j + 4 * tn;
      if (vec_store && c + 3 < N) {
        *reinterpret_cast<float4*>(crow + c) =
            make_float4(acc[i][4 * j], acc[i][4 * j + 1], acc[i][4 * j + 2], acc[i][4 * j + 3]);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (c + e < N) crow[c + e] = acc[i][4 * j + e];
      }
    }
  }
}

}  // namespace hbsg
