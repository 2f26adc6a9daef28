// gemm_tf32.cu -- C = alpha A B + beta C on the fifth-generation tensor cores.
//
// One CTA computes a 128 x 128 (or 128 x 64) tile of C; wide products take a
// persistent kernel of 128 x 256 tiles (k_gemm_tf32_wide).  Warp 0 streams the K
// panels of A and B into a three-stage shared-memory ring with the tensor memory
// accelerator (cp.async.bulk.tensor, 128-byte swizzle, no multicast: every
// operand is this GPU's own memory); warp 1 owns the tile's 128 tensor-memory
// columns and issues tcgen05.mma kind::tf32 (M = 128, N = 128, K = 8) from
// one thread, four per 32-wide K panel, releasing each stage with
// tcgen05.commit; warps 2-5 read the FP32 accumulator back with tcgen05.ld
// (thread = row of the tile) and write alpha acc + beta C.  With 97 KB of
// shared memory and 128 tensor-memory columns, two CTAs share an SM, so one
// CTA's epilogue runs under the other's main loop.
//
// Out-of-range rows and columns of A and B (ragged M, N, K) are zero-filled
// by the copies; the epilogue writes only the rows and columns inside C.
//
// Every wait on a pipeline barrier is bounded.  A wait that gives up sets
// bit 0 of the error word and a shared abort flag; the other roles stop at
// their next wait, the copies already issued are waited for (bounded), the
// issued MMAs are waited for, and the CTA frees its tensor memory before it
// returns.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <map>
#include <mutex>

#include "gemm_tf32.h"
#include "pdl.cuh"

namespace {

constexpr int kBM = 128, kBK = 32;  // tile rows, K panel (32 floats = one 128-byte row)
constexpr int kThreads = 192;
constexpr int kABytes = kBM * kBK * 4;  // 16 KB per stage
constexpr long long kSpin = 1ll << 22;

// Tile shape of one variant: BN columns of C per CTA (the MMA's N and the
// tensor-memory columns), STAGES K panels in flight.  64 x 4 stages: 96 KB,
// two CTAs per SM; 128 x 3: 97 KB, two CTAs.  The 256-column variant is
// k_gemm_tf32_wide below.
template <int BN, int STAGES>
struct Tile {
  static constexpr int kBBytes = BN * kBK * 4;
  static constexpr int kOffB = STAGES * kABytes;
  static constexpr int kOffBar = kOffB + STAGES * kBBytes;  // full[STAGES], empty[STAGES], acc
  static constexpr int kOffMisc = kOffBar + 8 * (2 * STAGES + 1);
  static constexpr int kSmemBytes = kOffMisc + 16 + 1024;  // + alignment slack of the dynamic window
};

// instruction descriptor, kind::tf32: D f32 (bit 4), A and B tf32 (format 2
// at bits 7 and 10), both K-major, N >> 3 at bit 17, M >> 4 at bit 24
constexpr uint32_t idesc(int bn) {
  return (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(bn >> 3) << 17) | ((uint32_t)(kBM >> 4) << 24);
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// shared-memory descriptor of a K-major operand tile written by the copy
// engine with 128-byte swizzle: rows of 128 bytes, 8-row groups 1024 bytes
// apart (stride byte offset), version 1, layout SWIZZLE_128B
__device__ __forceinline__ uint64_t sdesc_sw128(uint32_t saddr) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) |
         (2ull << 61);
}

__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(done)
      : "r"(bar), "r"(parity)
      : "memory");
  return done != 0;
}

// bounded wait; false if it gave up or another role aborted the tile
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  for (long long it = 0; it < kSpin; ++it) {
    if (mbar_try(bar, parity)) return true;
    if ((it & 1023) == 1023 && *abort_flag) return false;
  }
  return false;
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
      "%15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
        "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
        "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
        "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(taddr));
}

__device__ __forceinline__ void tma_panel(const CUtensorMap* tm, uint32_t dst, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(tm)), "r"(x), "r"(y), "r"(bar)
      : "memory");
}

// the four K = 8 steps of one K panel (8 tf32 = 32 bytes along the swizzled
// row each); the first overwrites the accumulator when first is set
__device__ __forceinline__ void mma_panel(uint32_t tacc, uint64_t da, uint64_t db, uint32_t idesc, bool first) {
#pragma unroll
  for (int kk = 0; kk < kBK / 8; ++kk) {
    const uint32_t acc = !(first && kk == 0);
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tacc),
        "l"(da + (uint64_t)(2 * kk)), "l"(db + (uint64_t)(2 * kk)), "r"(idesc), "r"(acc));
  }
}

__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

template <int BN, int STAGES>
__global__ void __launch_bounds__(kThreads, 2)
    k_gemm_tf32(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, float* __restrict__ C,
                int ldc, int M, int N, int K, float alpha, float beta, int c_rowmajor, int* err) {
  using T = Tile<BN, STAGES>;
  constexpr int kBN = BN, kStages = STAGES, kBBytes = T::kBBytes, kOffB = T::kOffB, kOffBar = T::kOffBar,
                kOffMisc = T::kOffMisc;
  constexpr uint32_t kIdesc = idesc(BN);
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);  // 1024-aligned window
  const uint32_t sbase = smem_u32(smem);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kOffBar);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + kOffMisc);
  uint32_t* tslot = reinterpret_cast<uint32_t*>(smem + kOffMisc + 4);
  const uint32_t bar_full = smem_u32(&bars[0]), bar_empty = smem_u32(&bars[kStages]),
                 bar_acc = smem_u32(&bars[2 * kStages]);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m0 = blockIdx.x * kBM, n0 = blockIdx.y * kBN;
  const int nk = (K + kBK - 1) / kBK;

  if (tid == 0) {
    *abort_flag = 0;
    for (int s = 0; s < 2 * kStages + 1; ++s)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&bars[s])));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmA)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmB)) : "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tslot)), "r"(kBN));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = *reinterpret_cast<volatile uint32_t*>(tslot);
  pdl_wait();  // the operands and C are the predecessors' results
  pdl_next();

  if (warp == 0) {
    if (lane == 0) {  // producer
      int issued = 0;
      for (int kb = 0; kb < nk; ++kb) {
        const int s = kb % kStages;
        if (kb >= kStages && !mbar_wait(bar_empty + 8 * s, (uint32_t)((kb / kStages - 1) & 1), abort_flag)) {
          atomicOr(err, 1);
          *abort_flag = 1;
          break;
        }
        const uint32_t fb = bar_full + 8 * s;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(fb), "r"(kABytes + kBBytes)
                     : "memory");
        tma_panel(&tmA, sbase + s * kABytes, kb * kBK, m0, fb);
        tma_panel(&tmB, sbase + kOffB + s * kBBytes, kb * kBK, n0, fb);
        issued = kb + 1;
      }
      // the copies in flight land before the CTA leaves (bounded)
      for (int kb = issued > kStages ? issued - kStages : 0; kb < issued; ++kb) {
        const int s = kb % kStages;
        for (long long it = 0; it < kSpin && !mbar_try(bar_full + 8 * s, (uint32_t)((kb / kStages) & 1)); ++it) {
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {  // MMA issue
      for (int kb = 0; kb < nk; ++kb) {
        const int s = kb % kStages;
        if (!mbar_wait(bar_full + 8 * s, (uint32_t)((kb / kStages) & 1), abort_flag)) {
          atomicOr(err, 1);
          *abort_flag = 1;
          break;
        }
        tc_fence_after();
        mma_panel(tbase, sdesc_sw128(sbase + s * kABytes), sdesc_sw128(sbase + kOffB + s * kBBytes), kIdesc, kb == 0);
        tc_commit(bar_empty + 8 * s);
      }
      // completion of every MMA issued (also on abort, so that tensor memory is idle before it is freed)
      tc_commit(bar_acc);
      for (long long it = 0; it < kSpin && !mbar_try(bar_acc, 0); ++it) {
      }
    }
  } else {  // epilogue: warps 2-5, warp w reads tensor-memory lanes 32 (w % 4) ...
    const int q = warp & 3, row = m0 + 32 * q + lane;
    const bool live = row < M;
    // C of one 32-column chunk into registers, issued ahead of the previous
    // chunk's stores (the first chunk's under the main loop)
    constexpr int kCh = kBN < 32 ? kBN : 32;
    auto load_chunk = [&](int c0, float (&cv)[kCh]) {
#pragma unroll
      for (int j = 0; j < kCh; ++j) {
        const int col = n0 + c0 + j;
        cv[j] = (beta != 0.0f && live && col < N)
                    ? (c_rowmajor ? C[(size_t)row * ldc + col] : C[(size_t)col * ldc + row])
                    : 0.0f;
      }
    };
    float cn[kCh];
    load_chunk(0, cn);
    bool ok = mbar_wait(bar_acc, 0, abort_flag);
    if (!ok) {
      atomicOr(err, 1);
      *abort_flag = 1;
    }
    ok = __all_sync(0xffffffffu, ok && !*abort_flag);  // the tensor-memory loads below are warp-wide
    tc_fence_after();
    if (ok) {
      const uint32_t trow = tbase + ((uint32_t)(32 * q) << 16);
#pragma unroll 1
      for (int c0 = 0; c0 < kBN; c0 += kCh) {
        float cc[kCh];
#pragma unroll
        for (int j = 0; j < kCh; ++j) cc[j] = cn[j];
        if (c0 + kCh < kBN) load_chunk(c0 + kCh, cn);  // in flight while this chunk is written
        uint32_t v[32];
        tmem_ld32(trow + (uint32_t)c0, v);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (live) {
#pragma unroll
          for (int j = 0; j < kCh; ++j) {
            const int col = n0 + c0 + j;
            if (col < N) {
              float* dst = c_rowmajor ? C + (size_t)row * ldc + col : C + (size_t)col * ldc + row;
              *dst = fmaf(alpha, __uint_as_float(v[j]), beta * cc[j]);
            }
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tbase), "r"(kBN));
  }
}

// The wide variant: 128 x 256 tiles, a CTA per SM that takes tile after tile.
// Two accumulators of 256 tensor-memory columns let the main loop of a tile run
// under the epilogue of the one before, which the single-tile kernel gets from a
// second CTA per SM that 256 columns have no shared memory for; eight epilogue
// warps (two per tensor-memory quarter, 128 columns each) keep twice the reads
// of C in flight.  The wide tile reads its operands from L2 1.28 times less
// often than 128 x 128 ones, which bound the trailing updates.  Rank-512 updates
// against the fastest of the single-tile variants (128 x 256 tiles in single-tile
// form were slower than both, 4,329 us in the last case): 20.8 -> 16.8 us at
// 2,600 x 1,300, 194 -> 139 us (392 TFLOP/s) at 10,344 x 5,172, 3,166 -> 1,916 us
// (424 TFLOP/s) at 39,808 x 19,904, where C's read and write take 970 us at the
// copy bandwidth and the operands' 19 GB from L2 bound the rest.
constexpr int kWBN = 256, kWStages = 4, kWThreads = 320, kWEpi = 8;
struct Wide {
  static constexpr int kBBytes = kWBN * kBK * 4;
  static constexpr int kOffB = kWStages * kABytes;
  static constexpr int kOffBar = kOffB + kWStages * kBBytes;  // full, empty [stages], acc full, acc empty [2], done
  static constexpr int kBars = 2 * kWStages + 5;
  static constexpr int kOffMisc = kOffBar + 8 * kBars;
  static constexpr int kSmemBytes = kOffMisc + 16 + 1024;
};

__global__ void __launch_bounds__(kWThreads, 1)
    k_gemm_tf32_wide(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                     float* __restrict__ C, int ldc, int M, int N, int K, float alpha, float beta, int c_rowmajor,
                     int* err) {
  constexpr uint32_t kIdesc = idesc(kWBN);
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
  const uint32_t sbase = smem_u32(smem);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Wide::kOffBar);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + Wide::kOffMisc);
  uint32_t* tslot = reinterpret_cast<uint32_t*>(smem + Wide::kOffMisc + 4);
  const uint32_t bar_full = smem_u32(&bars[0]), bar_empty = smem_u32(&bars[kWStages]),
                 bar_acc = smem_u32(&bars[2 * kWStages]), bar_free = smem_u32(&bars[2 * kWStages + 2]),
                 bar_done = smem_u32(&bars[2 * kWStages + 4]);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nk = (K + kBK - 1) / kBK, mt = (M + kBM - 1) / kBM;
  const int tiles = mt * ((N + kWBN - 1) / kWBN);

  if (tid == 0) {
    *abort_flag = 0;
    for (int s = 0; s < Wide::kBars; ++s) {
      const int count = s == 2 * kWStages + 2 || s == 2 * kWStages + 3 ? kWEpi : 1;
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&bars[s])), "r"(count));
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmA)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmB)) : "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tslot)),
                 "r"(2 * kWBN));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = *reinterpret_cast<volatile uint32_t*>(tslot);
  pdl_wait();  // the operands and C are the predecessors' results
  pdl_next();
  auto give_up = [&] {
    atomicOr(err, 1);
    *abort_flag = 1;
  };

  if (warp == 0) {
    if (lane == 0) {  // producer: the K panels of all tiles, one after another
      int p = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x)
        for (int kb = 0; kb < nk; ++kb, ++p) {
          const int s = p % kWStages;
          if (p >= kWStages && !mbar_wait(bar_empty + 8 * s, (uint32_t)((p / kWStages - 1) & 1), abort_flag)) {
            give_up();
            ok = false;
            break;
          }
          const uint32_t fb = bar_full + 8 * s;
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(fb), "r"(kABytes + Wide::kBBytes)
                       : "memory");
          tma_panel(&tmA, sbase + s * kABytes, kb * kBK, t % mt * kBM, fb);
          tma_panel(&tmB, sbase + Wide::kOffB + s * Wide::kBBytes, kb * kBK, t / mt * kWBN, fb);
        }
      // the copies in flight land before the CTA leaves (bounded)
      for (int i = p > kWStages ? p - kWStages : 0; i < p; ++i) {
        const int s = i % kWStages;
        for (long long it = 0; it < kSpin && !mbar_try(bar_full + 8 * s, (uint32_t)((i / kWStages) & 1)); ++it) {
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {  // MMA issue
      int p = 0, u = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x, ++u) {
        const int b = u & 1;
        if (u >= 2) {  // the epilogue has read this accumulator's last tile
          if (!mbar_wait(bar_free + 8 * b, (uint32_t)((u / 2 - 1) & 1), abort_flag)) {
            give_up();
            break;
          }
          tc_fence_after();
        }
        for (int kb = 0; kb < nk; ++kb, ++p) {
          const int s = p % kWStages;
          if (!mbar_wait(bar_full + 8 * s, (uint32_t)((p / kWStages) & 1), abort_flag)) {
            give_up();
            ok = false;
            break;
          }
          tc_fence_after();
          mma_panel(tbase + (uint32_t)(b * kWBN), sdesc_sw128(sbase + s * kABytes),
                    sdesc_sw128(sbase + Wide::kOffB + s * Wide::kBBytes), kIdesc, kb == 0);
          tc_commit(bar_empty + 8 * s);
        }
        if (ok) tc_commit(bar_acc + 8 * b);
      }
      // completion of every MMA issued (also on abort, so that tensor memory is idle before it is freed)
      tc_commit(bar_done);
      for (long long it = 0; it < kSpin && !mbar_try(bar_done, 0); ++it) {
      }
    }
  } else {  // epilogue: warp w reads tensor-memory lanes 32 (w % 4) ..., columns 128 of one half
    const int q = warp & 3, half = (warp - 2) / 4 * (kWBN / 2);
    constexpr int kCh = 32;
    int u = 0;
    for (int t = blockIdx.x; t < tiles; t += gridDim.x, ++u) {
      const int b = u & 1, row = t % mt * kBM + 32 * q + lane, n0 = t / mt * kWBN + half;
      const bool live = row < M;
      auto load_chunk = [&](int c0, float (&cv)[kCh]) {
#pragma unroll
        for (int j = 0; j < kCh; ++j) {
          const int col = n0 + c0 + j;
          cv[j] = (beta != 0.0f && live && col < N)
                      ? (c_rowmajor ? C[(size_t)row * ldc + col] : C[(size_t)col * ldc + row])
                      : 0.0f;
        }
      };
      float cn[kCh];
      load_chunk(0, cn);
      bool ok = mbar_wait(bar_acc + 8 * b, (uint32_t)((u / 2) & 1), abort_flag);
      if (!ok) give_up();
      ok = __all_sync(0xffffffffu, ok && !*abort_flag);  // the tensor-memory loads below are warp-wide
      if (!ok) break;
      tc_fence_after();
      const uint32_t trow = tbase + (uint32_t)(b * kWBN + half) + ((uint32_t)(32 * q) << 16);
#pragma unroll 1
      for (int c0 = 0; c0 < kWBN / 2; c0 += kCh) {
        float cc[kCh];
#pragma unroll
        for (int j = 0; j < kCh; ++j) cc[j] = cn[j];
        if (c0 + kCh < kWBN / 2) load_chunk(c0 + kCh, cn);  // in flight while this chunk is written
        uint32_t v[32];
        tmem_ld32(trow + (uint32_t)c0, v);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (c0 + kCh == kWBN / 2) {  // the accumulator is free for the tile after next
          tc_fence_before();
          __syncwarp();
          if (lane == 0)
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar_free + 8 * b) : "memory");
        }
        if (live) {
#pragma unroll
          for (int j = 0; j < kCh; ++j) {
            const int col = n0 + c0 + j;
            if (col < N) {
              float* dst = c_rowmajor ? C + (size_t)row * ldc + col : C + (size_t)col * ldc + row;
              *dst = fmaf(alpha, __uint_as_float(v[j]), beta * cc[j]);
            }
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tbase), "r"(2 * kWBN));
  }
}

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  });
  return fn;
}

// 2-D map of a K-major operand: inner extent k floats, `rows` rows ld floats
// apart, box of 32 floats x box_rows rows, 128-byte swizzle, zero fill
bool make_map(CUtensorMap* tm, const float* base, int k, int rows, int ld, int box_rows) {
  auto fn = encode_fn();
  if (!fn) return false;
  cuuint64_t dims[2] = {(cuuint64_t)k, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)ld * 4};
  cuuint32_t box[2] = {(cuuint32_t)kBK, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  return fn(tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(base), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

namespace {

template <int BN, int STAGES>
int launch(cudaStream_t st, int dev, int m, int n, int k, float alpha, const float* A, int lda, const float* B, int ldb,
           float beta, float* C, int ldc, bool c_rowmajor, int* err) {
  using T = Tile<BN, STAGES>;
  // the shared-memory opt-in, once per device
  static std::mutex mu;
  static bool attr_set[64] = {};
  {
    std::lock_guard<std::mutex> lock(mu);
    if (!attr_set[dev]) {
      if (cudaFuncSetAttribute(k_gemm_tf32<BN, STAGES>, cudaFuncAttributeMaxDynamicSharedMemorySize, T::kSmemBytes) !=
          cudaSuccess)
        return 1;
      attr_set[dev] = true;
    }
  }
  CUtensorMap ta, tb;
  if (!make_map(&ta, A, k, m, lda, kBM) || !make_map(&tb, B, k, n, ldb, BN)) return 1;
  dim3 grid((unsigned)((m + kBM - 1) / kBM), (unsigned)((n + BN - 1) / BN));
  return pdl_launch(k_gemm_tf32<BN, STAGES>, grid, dim3(kThreads), T::kSmemBytes, st, ta, tb, C, ldc, m, n, k, alpha,
                    beta, c_rowmajor ? 1 : 0, err) == cudaSuccess
             ? 0
             : 1;
}

int launch_wide(cudaStream_t st, int dev, int m, int n, int k, float alpha, const float* A, int lda, const float* B,
                int ldb, float beta, float* C, int ldc, bool c_rowmajor, int* err) {
  // the shared-memory opt-in and the number of SMs, once per device
  static std::mutex mu;
  static int sms[64] = {};
  int ctas;
  {
    std::lock_guard<std::mutex> lock(mu);
    if (!sms[dev]) {
      int count = 0;
      if (cudaFuncSetAttribute(k_gemm_tf32_wide, cudaFuncAttributeMaxDynamicSharedMemorySize, Wide::kSmemBytes) !=
              cudaSuccess ||
          cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return 1;
      sms[dev] = count;
    }
    ctas = sms[dev];
  }
  CUtensorMap ta, tb;
  if (!make_map(&ta, A, k, m, lda, kBM) || !make_map(&tb, B, k, n, ldb, kWBN)) return 1;
  const long long tiles = (long long)((m + kBM - 1) / kBM) * ((n + kWBN - 1) / kWBN);
  if (tiles > 0x3fffffff) return 1;
  return pdl_launch(k_gemm_tf32_wide, dim3((unsigned)std::min<long long>(tiles, ctas)), dim3(kWThreads),
                    Wide::kSmemBytes, st, ta, tb, C, ldc, m, n, k, alpha, beta, c_rowmajor ? 1 : 0, err) == cudaSuccess
             ? 0
             : 1;
}

}  // namespace

int gemm_tf32_variant(cudaStream_t st, int variant, int m, int n, int k, float alpha, const float* A, int lda,
                      const float* B, int ldb, float beta, float* C, int ldc, bool c_rowmajor, int* err) {
  if (m <= 0 || n <= 0) return 0;
  if (k <= 0 || (reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(B) & 15) || (lda & 3) ||
      (ldb & 3) || lda < k || ldb < k)
    return 1;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 1;
  switch (variant) {
    case 0: return launch<64, 4>(st, dev, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, c_rowmajor, err);
    case 1: return launch<128, 3>(st, dev, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, c_rowmajor, err);
    case 2: return launch_wide(st, dev, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, c_rowmajor, err);
    default: return 1;
  }
}

// ---------------------------------------------------------------------------
// Autotuner: the tile variant of each shape class, measured on the device
// ---------------------------------------------------------------------------
namespace {

// shape class: M in 128-row tiles, N in 64-column tiles, both by powers of
// two, and K in 128-wide steps
struct Key {
  int dev, cm, cn, ck;
  bool operator<(const Key& o) const {
    return dev != o.dev ? dev < o.dev : cm != o.cm ? cm < o.cm : cn != o.cn ? cn < o.cn : ck < o.ck;
  }
};
int ceil_log2(long long x) {
  int c = 0;
  while ((1LL << c) < x) ++c;
  return c;
}
Key key_of(int dev, int m, int n, int k) {
  return Key{dev, ceil_log2((m + kBM - 1) / kBM), ceil_log2((n + 63) / 64), std::min((k + 127) / 128, 8)};
}
std::mutex g_tune_mu;
std::map<Key, int> g_tuned;

// the variant used before a class has been measured: the narrowest tile that
// still gives every SM work, else the widest
int heuristic(int m, int n) {
  const long long tiles128 = (long long)((m + kBM - 1) / kBM) * ((n + 127) / 128);
  if (n <= 64) return 0;
  if (tiles128 < 2 * 148) return n <= 128 ? 1 : 0;
  return tiles128 >= 8 * 148 ? 2 : 1;
}

}  // namespace

int gemm_tf32_pick(int m, int n, int k) {
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lock(g_tune_mu);
  auto it = g_tuned.find(key_of(dev, m, n, k));
  return it != g_tuned.end() ? it->second : heuristic(m, n);
}

int gemm_tf32_autotune(cudaStream_t st, int nshape, const int* shapes) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 1;
  std::lock_guard<std::mutex> lock(g_tune_mu);
  // the classes not measured yet, each with its largest shape
  std::map<Key, int3> todo;
  for (int s = 0; s < nshape; ++s) {
    const int m = shapes[3 * s], n = shapes[3 * s + 1], k = shapes[3 * s + 2];
    if (m <= 0 || n <= 0 || k <= 0) continue;
    const Key key = key_of(dev, m, n, k);
    if (g_tuned.count(key)) continue;
    int3& big = todo[key];
    if ((long long)m * n * k > (long long)big.x * big.y * big.z) big = make_int3(m, n, k);
  }
  if (todo.empty()) return 0;
  size_t na = 0, nb = 0, nc = 0;
  for (auto& t : todo) {
    const int ld = (t.second.z + 3) / 4 * 4;
    na = std::max(na, (size_t)t.second.x * ld);
    nb = std::max(nb, (size_t)t.second.y * ld);
    nc = std::max(nc, (size_t)t.second.x * t.second.y);
  }
  float *a = nullptr, *b = nullptr, *c = nullptr;
  int* err = nullptr;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  int rc = 0;
  if (cudaMalloc(&a, na * 4) != cudaSuccess || cudaMalloc(&b, nb * 4) != cudaSuccess ||
      cudaMalloc(&c, nc * 4) != cudaSuccess || cudaMalloc(&err, sizeof(int)) != cudaSuccess ||
      cudaEventCreate(&e0) != cudaSuccess || cudaEventCreate(&e1) != cudaSuccess)
    rc = 1;
  if (!rc && (cudaMemsetAsync(a, 0, na * 4, st) != cudaSuccess || cudaMemsetAsync(b, 0, nb * 4, st) != cudaSuccess ||
              cudaMemsetAsync(err, 0, sizeof(int), st) != cudaSuccess))
    rc = 1;
  for (auto it = todo.begin(); !rc && it != todo.end(); ++it) {
    const int m = it->second.x, n = it->second.y, k = it->second.z, ld = (k + 3) / 4 * 4;
    // the variants in turn, six rounds, each launch timed alone; the first
    // round warms up, the fastest of the other five counts (so that a clock
    // ramp or a passing neighbour does not decide the pick)
    float best_v[3] = {1e30f, 1e30f, 1e30f};
    for (int rep = 0; rep < 6 && !rc; ++rep)
      for (int v = 0; v < 3 && !rc; ++v) {
        float tv = 0.0f;
        if (cudaEventRecord(e0, st) != cudaSuccess ||
            gemm_tf32_variant(st, v, m, n, k, -1.0f, a, ld, b, ld, 1.0f, c, m, false, err) ||
            cudaEventRecord(e1, st) != cudaSuccess || cudaEventSynchronize(e1) != cudaSuccess ||
            cudaEventElapsedTime(&tv, e0, e1) != cudaSuccess)
          rc = 1;
        if (!rc && rep > 0) best_v[v] = std::min(best_v[v], tv);
      }
    int pick = heuristic(m, n);
    for (int v = 0; v < 3; ++v)
      if (best_v[v] < best_v[pick]) pick = v;
    if (!rc) g_tuned[it->first] = pick;
  }
  int werr = 0;
  if (err && cudaMemcpy(&werr, err, sizeof(int), cudaMemcpyDeviceToHost) == cudaSuccess && werr) rc = 1;
  if (e0) cudaEventDestroy(e0);
  if (e1) cudaEventDestroy(e1);
  cudaFree(a);
  cudaFree(b);
  cudaFree(c);
  cudaFree(err);
  return rc;
}

int gemm_tf32_tuned_count() {
  std::lock_guard<std::mutex> lock(g_tune_mu);
  return (int)g_tuned.size();
}

int gemm_tf32(cudaStream_t st, int m, int n, int k, float alpha, const float* A, int lda, const float* B, int ldb,
              float beta, float* C, int ldc, bool c_rowmajor, int* err) {
  return gemm_tf32_variant(st, gemm_tf32_pick(m, n, k), m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, c_rowmajor, err);
}
