// lu_fp64.cu -- complex128 LU with partial pivoting and the solve of its
// right-hand sides, for the plain form (ZGETRF/ZGETRS of RADIATION_SOLVER_MULTI
// / DIFFRACTION_SOLVER_MULTI, AssbMatxMulti.f90:112,279,346).
//
// Right-looking, in blocks of kZB = 64 columns made of four panels of kZW = 16:
//   k_zpanel   factors a panel in the registers of one cluster: a row per
//              thread, up to 16 blocks of 512 rows;
//   k_zapply   takes the panel's row exchanges to the other columns of the block
//              and solves for the panel's rows of U there;
//   k_zupdate  subtracts L U from the rest of the block's columns;
// then
//   k_zright   takes the block's row exchanges to all other columns and to the
//              right-hand sides, and solves for the block's rows of U (and of the
//              forward-substituted right-hand sides);
//   ZGEMM      the trailing matrix and the right-hand sides below, rank 64.
// The back substitution takes the blocks from the last: k_zback solves with the
// diagonal block, ZGEMM subtracts its columns above.
//
// The library's getrf spends 3.6 us per column on its panels (53 % of a
// 5,400-column factorisation, nearly all of an 800-column one) and its getrs two
// large triangular solves.  Factorisation and solve (58 right-hand sides at
// 5,400 panels) against it: 43.5 -> 31.0 ms at 5,400 panels, 14.9 -> 9.0 ms at
// 2,340 (two in flight), 4.9 -> 2.4 ms at 800 (eight in flight), 0.68 -> 0.66 ms
// at 234.  GMRES inverts its body blocks with it (identity right-hand sides,
// bodies of one size as one batch).  What bounds it: the panels' chains (1.9 us per column, 10.6 ms at 5,400
// panels), then ZGEMM (16 ms, 70 % of the FP64 tensor rate).
#include "lu_fp64.h"

#include <cstdint>

#include "pdl.cuh"

namespace {

constexpr int kZW = 16;             // panel columns
constexpr int kZB = 64;             // block columns
constexpr int kZP = kZB / kZW;      // panels per block
constexpr int kZThreads = 512;      // rows per block of the panel's cluster
constexpr int kZMoves = 2 * kZW;    // row moves of a panel at most
constexpr int kZList = 2 * kZMoves;  // workspace per panel of a block: (destination or -1, source) pairs

// Systems of one order factored together (blockIdx.z, or .y of the panels'
// clusters, the system): strides of A and X, the workspace after one another.
struct ZBatch {
  size_t a, x;
  __device__ __forceinline__ int* list(int* work, int sys) const { return work + (size_t)sys * kZP * kZList; }
};

__device__ __forceinline__ double2 zmul(double2 a, double2 b) {
  return make_double2(fma(-a.y, b.y, a.x * b.x), fma(a.y, b.x, a.x * b.y));
}
__device__ __forceinline__ void zsub(double2& s, double2 a, double2 b) {  // s -= a b
  s.x = fma(-a.x, b.x, fma(a.y, b.y, s.x));
  s.y = fma(-a.x, b.y, fma(-a.y, b.x, s.y));
}
// 1 / d by conj(d) / |d|^2, d first scaled by a power of two (exactly) so that
// the square neither overflows nor underflows; one reciprocal instead of the
// two divisions in a row of Smith's method.  Zero for d = 0.
__device__ __forceinline__ double2 zrcp(double2 d) {
  const int hi = __double2hiint(fmax(fabs(d.x), fabs(d.y))), e = min(max(hi >> 20, 1), 2045);
  const double s = __hiloint2double((2046 - e) << 20, 0);  // 2^(1023 - e)
  const double x = d.x * s, y = d.y * s, den = fma(x, x, y * y), r = den > 0.0 ? __drcp_rn(den) * s : 0.0;
  return make_double2(x * r, -y * r);
}

// One panel: columns c0 .. c0+w-1 of the rows from c0 on (w = kZW, or the last
// w rows and columns), a row per thread of the cluster, rows never moving
// between threads: the pivot of a column is the row of largest |re| + |im| (by
// the upper 32 bits: rows that agree in them are equally good) among those not
// taken.  Each warp offers its best row, each block its best warp's; the
// block's row goes to all blocks of the cluster, one cluster barrier, and every
// block picks the same one: 1.9 us per column, much the same with one block as
// with sixteen.  A row's current column is always entry 0: each
// update moves the entries down by one and the multiplier comes in at the end,
// so that one loop body serves all columns.  The pivot row of column j thus ends
// with U(j, c) at c - j and its multipliers after them, the others with theirs in
// order.  At the end the pivot rows are stored in their order,
// the rows they displace in the places they leave; moves lists both.
__global__ void __launch_bounds__(kZThreads, 1) k_zpanel(double2* __restrict__ A, int lda, int n, int c0, int w,
                                                        ZBatch zb, int* __restrict__ work, int panel, int* info) {
  __shared__ __align__(16) double2 offer[2][16][kZW];  // [column & 1][block]: each block's best row
  __shared__ uint32_t okey[2][16];
  __shared__ int orow[2][16];
  __shared__ double2 mine[kZW];
  __shared__ uint32_t wkey[kZThreads / 32];
  __shared__ int wtid[kZThreads / 32];
  __shared__ int piv[kZW];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  uint32_t rank, nct;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(nct));
  const int r = c0 + (int)rank * kZThreads + tid;
  const bool live = r < n;
  A += blockIdx.y * zb.a;
  int* moves = zb.list(work, blockIdx.y) + panel * kZList;
  pdl_wait();
  pdl_next();
  double2 a[kZW];
#pragma unroll
  for (int c = 0; c < kZW; ++c)
    a[c] = live && c < w ? A[(size_t)(c0 + c) * lda + r] : make_double2(0.0, 0.0);
  int step = -1;  // the column this row is the pivot of
  // every block of the cluster runs before another writes to its shared memory
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
#pragma unroll 1
  for (int j = 0; j < w; ++j) {
    const uint32_t key = live && step < 0 ? (uint32_t)__double2hiint(fabs(a[0].x) + fabs(a[0].y)) + 1u : 0u;
    const uint32_t wb = __reduce_max_sync(0xffffffffu, key);
    const int src = __ffs(__ballot_sync(0xffffffffu, key == wb)) - 1;
    if (lane == src) {
      wkey[warp] = wb;
      wtid[warp] = tid;
    }
    __syncthreads();
    const uint32_t k = lane < kZThreads / 32 ? wkey[lane] : 0u, cb = __reduce_max_sync(0xffffffffu, k);
    const int ws = __ffs(__ballot_sync(0xffffffffu, k == cb)) - 1;
    const int wt = wtid[ws];
    if (tid == wt) {  // its multipliers are no part of the update
#pragma unroll
      for (int c = 0; c < kZW; ++c) mine[c] = c < kZW - j ? a[c] : make_double2(0.0, 0.0);
    }
    __syncthreads();
    if (tid < (int)nct * kZW) {  // to block tid / kZW
      const int to = tid / kZW, c = tid % kZW;
      const uint32_t local = (uint32_t)__cvta_generic_to_shared(&offer[j & 1][rank][c]);
      uint32_t remote;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(to));
      const double2 v = mine[c];
      asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(remote), "d"(v.x), "d"(v.y) : "memory");
      if (c == 0) {
        const uint32_t lk = (uint32_t)__cvta_generic_to_shared(&okey[j & 1][rank]),
                       lr = (uint32_t)__cvta_generic_to_shared(&orow[j & 1][rank]);
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(lk), "r"(to));
        asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(remote), "r"(cb) : "memory");
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(lr), "r"(to));
        asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(remote), "r"(c0 + (int)rank * kZThreads + wt)
                     : "memory");
      }
    }
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    const uint32_t ck = lane < (int)nct ? okey[j & 1][lane] : 0u, best = __reduce_max_sync(0xffffffffu, ck);
    const int b = __ffs(__ballot_sync(0xffffffffu, ck == best)) - 1;
    const int p = orow[j & 1][b];
    const double2* u = offer[j & 1][b];
    const double2 d = u[0];
    if (tid == 0) {
      piv[j] = p;
      if (rank == 0 && d.x == 0.0 && d.y == 0.0) atomicCAS(info, 0, c0 + j + 1);
    }
    if (r == p) step = j;
    if (step < 0) {
      const double2 l = zmul(a[0], zrcp(d));
#pragma unroll
      for (int c = 1; c < kZW / 2; ++c) {
        a[c - 1] = a[c];
        zsub(a[c - 1], l, u[c]);
      }
      if (j < kZW / 2) {  // the upper half still holds columns of A
#pragma unroll
        for (int c = kZW / 2; c < kZW; ++c) {
          a[c - 1] = a[c];
          zsub(a[c - 1], l, u[c]);
        }
      } else {
#pragma unroll
        for (int c = kZW / 2; c < kZW; ++c) a[c - 1] = a[c];
      }
      a[kZW - 1] = l;
    }
  }
  __syncthreads();  // piv
  // rows of the panel's top that are no pivot, in order, take the places of the
  // pivots from below it, in the order of their columns
  auto chosen = [&](int q) {
    bool t = false;
    for (int j = 0; j < w; ++j) t |= piv[j] == q;
    return t;
  };
  auto vacated = [&](int k) {  // the k-th place left by a pivot from below the top, or -1
    for (int j = 0; j < w; ++j)
      if (piv[j] >= c0 + w && k-- == 0) return piv[j];
    return -1;
  };
  if (live) {
    int to = r;
    if (step >= 0) {
      to = c0 + step;
    } else if (r < c0 + w) {
      int before = 0;
      for (int q = c0; q < r; ++q) before += !chosen(q);
      to = vacated(before);
    }
    const int turn = step >= 0 ? step : 0;
#pragma unroll
    for (int c = 0; c < kZW; ++c) {
      const int cc = (c + turn) % kZW;
      if (cc < w) A[(size_t)(c0 + cc) * lda + to] = a[c];
    }
  }
  if (rank == 0 && tid < 2 * kZW) {
    int dst = -1, from = 0;
    if (tid < w && piv[tid] != c0 + tid) {
      dst = c0 + tid;
      from = piv[tid];
    } else if (tid >= kZW && tid - kZW < w) {
      dst = vacated(tid - kZW);
      int k = tid - kZW;  // the k-th top row that is no pivot
      for (int q = c0; dst >= 0 && q < c0 + w; ++q)
        if (!chosen(q) && k-- == 0) from = q;
    }
    moves[2 * tid] = dst;
    moves[2 * tid + 1] = from;
  }
}

// A panel's moves on the columns given by col(q), q < cols: all sources are
// read before any destination is written.  Called by a whole block; the columns
// belong to it alone.
template <class F>
__device__ __forceinline__ void move_rows(double2* buf, const int* __restrict__ moves, int cols, const F& col) {
#pragma unroll 2
  for (int e = threadIdx.x; e < kZMoves * cols; e += blockDim.x) {
    const int2 m = reinterpret_cast<const int2*>(moves)[e % kZMoves];
    if (m.x >= 0) buf[e] = col(e / kZMoves)[m.y];
  }
  __syncthreads();
#pragma unroll 2
  for (int e = threadIdx.x; e < kZMoves * cols; e += blockDim.x) {
    const int2 m = reinterpret_cast<const int2*>(moves)[e % kZMoves];
    if (m.x >= 0) col(e / kZMoves)[m.x] = buf[e];
  }
  __syncthreads();
}
// The kb x kb diagonal block at (k0, k0) into T[column][row], ld kZB + 1.
template <int NT>
__device__ __forceinline__ void load_diag(double2* T, const double2* __restrict__ A, int lda, int k0, int kb) {
#pragma unroll 8
  for (int e = threadIdx.x; e < kZB * kZB; e += NT) {
    const int i = e % kZB, k = e / kZB;
    if (i < kb && k < kb) T[k * (kZB + 1) + i] = A[(size_t)(k0 + k) * lda + k0 + i];
  }
}

// After panel p (columns c0 .. c0+w-1): its moves on the block's other columns
// k0 .. k1-1, and U = L_pp^-1 A on those right of it.  A block of 128 threads
// takes 8 columns: 16 threads each, one per panel row.
constexpr int kZApplyCols = 8;
__global__ void __launch_bounds__(128) k_zapply(double2* __restrict__ A, int lda, int k0, int k1, int c0, int w,
                                                ZBatch zb, int* work, int panel) {
  __shared__ double2 buf[kZMoves * kZApplyCols];
  __shared__ double2 L[kZW][kZW + 1];
  // the block's columns without the panel's
  const int left = c0 - k0, total = left + (k1 - c0 - w), q0 = blockIdx.x * kZApplyCols;
  const int cols = min(kZApplyCols, total - q0);
  A += blockIdx.z * zb.a;
  const int* moves = zb.list(work, blockIdx.z) + panel * kZList;
  pdl_wait();
  pdl_next();
  auto col = [&](int q) { return A + (size_t)(q0 + q < left ? k0 + q0 + q : c0 + w + (q0 + q - left)) * lda; };
  for (int e = threadIdx.x; e < w * w; e += blockDim.x) L[e % w][e / w] = A[(size_t)(c0 + e / w) * lda + c0 + e % w];
  move_rows(buf, moves, cols, col);
  const int q = threadIdx.x / kZW, i = threadIdx.x % kZW;
  const bool on = q < cols && i < w && q0 + q >= left;
  double2 x = on ? col(q)[c0 + i] : make_double2(0.0, 0.0);
  for (int k = 0; k + 1 < w; ++k) {  // the 16 threads of a column are half a warp
    const double2 xk = make_double2(__shfl_sync(0xffffffffu, x.x, k, kZW), __shfl_sync(0xffffffffu, x.y, k, kZW));
    if (i > k && i < w) zsub(x, L[i][k], xk);
  }
  if (on) col(q)[c0 + i] = x;
}

// A(r, c) -= sum_k L(r, k) U(k, c) for the rows from r0 = c0 + w on and the
// block's columns r0 .. k1-1, the panel's w columns k.  A block of 128 threads
// takes 128 rows and 8 columns, a row per thread.
constexpr int kZUpCols = 8;
__global__ void __launch_bounds__(128) k_zupdate(double2* __restrict__ A, int lda, int n, int k1, int c0, int w,
                                                 ZBatch zb) {
  __shared__ double2 U[kZW][kZUpCols];
  A += blockIdx.z * zb.a;
  pdl_wait();
  pdl_next();
  const int r0 = c0 + w, r = r0 + blockIdx.x * 128 + threadIdx.x, q0 = r0 + blockIdx.y * kZUpCols;
  const int cols = min(kZUpCols, k1 - q0);
  for (int e = threadIdx.x; e < kZW * kZUpCols; e += blockDim.x) {
    const int k = e % kZW, c = e / kZW;
    U[k][c] = k < w && c < cols ? A[(size_t)(q0 + c) * lda + c0 + k] : make_double2(0.0, 0.0);
  }
  const bool on = r < n;
  double2 s[kZUpCols], l[kZW];  // all in flight at once
#pragma unroll
  for (int k = 0; k < kZW; ++k) l[k] = on && k < w ? A[(size_t)(c0 + k) * lda + r] : make_double2(0.0, 0.0);
#pragma unroll
  for (int c = 0; c < kZUpCols; ++c) s[c] = on && c < cols ? A[(size_t)(q0 + c) * lda + r] : make_double2(0.0, 0.0);
  __syncthreads();
  if (!on) return;
#pragma unroll
  for (int k = 0; k < kZW; ++k)
#pragma unroll
    for (int c = 0; c < kZUpCols; ++c) zsub(s[c], l[k], U[k][c]);
#pragma unroll
  for (int c = 0; c < kZUpCols; ++c)
    if (c < cols) A[(size_t)(q0 + c) * lda + r] = s[c];
}

// The block's moves (its panels' lists in turn) on the columns outside it and
// on the right-hand sides, and U = L_bb^-1 A for the columns right of it and the
// right-hand sides.  A block of 256 threads takes 16 columns; their kb rows of
// the block go through shared memory, solved 16 rows at a time: the rows
// themselves in half-warps (a thread per row), then the rows below by all
// threads.
constexpr int kZRightCols = 16;
constexpr int kZRightSmem = (kZB * (kZB + 1) + kZB * (kZRightCols + 1)) * (int)sizeof(double2);
__global__ void __launch_bounds__(256) k_zright(double2* __restrict__ A, int lda, int n, int k0, int kb,
                                                double2* __restrict__ X, int nrhs, ZBatch zb, int* work) {
  extern __shared__ __align__(16) double2 zs[];
  double2* L = zs;                       // [column k][row i], ld kZB + 1
  double2* Y = zs + kZB * (kZB + 1);     // [row i][column q], ld kZRightCols + 1; the moves' buffer before
  constexpr int kLl = kZB + 1, kYl = kZRightCols + 1;
  const int right = n - k0 - kb, total = k0 + right + nrhs, q0 = blockIdx.x * kZRightCols;
  const int cols = min(kZRightCols, total - q0);
  A += blockIdx.z * zb.a;
  X += blockIdx.z * zb.x;
  const int* moves = zb.list(work, blockIdx.z);
  auto col = [&](int q) {
    const int c = q0 + q;
    return c < k0 ? A + (size_t)c * lda
                  : c < k0 + right ? A + (size_t)(c + kb) * lda : X + (size_t)(c - k0 - right) * n;
  };
  pdl_wait();
  pdl_next();
  const bool solve = q0 + cols > k0;  // else columns of L only
  if (solve) load_diag<256>(L, A, lda, k0, kb);
  for (int p = 0; p * kZW < kb; ++p) move_rows(Y, moves + p * kZList, cols, col);
  if (!solve) return;
#pragma unroll 4
  for (int e = threadIdx.x; e < kZB * kZRightCols; e += 256)
    if (e % kZB < kb && e / kZB < cols) Y[(e % kZB) * kYl + e / kZB] = col(e / kZB)[k0 + e % kZB];
  __syncthreads();
  const int q = threadIdx.x / kZW, i = threadIdx.x % kZW;
  for (int s0 = 0; s0 < kb; s0 += kZW) {
    const int sw = min(kZW, kb - s0);
    double2 x = q < cols && i < sw ? Y[(s0 + i) * kYl + q] : make_double2(0.0, 0.0);
    for (int k = 0; k + 1 < sw; ++k) {
      const double2 xk = make_double2(__shfl_sync(0xffffffffu, x.x, k, kZW), __shfl_sync(0xffffffffu, x.y, k, kZW));
      if (i > k && i < sw) zsub(x, L[(s0 + k) * kLl + s0 + i], xk);
    }
    if (q < cols && i < sw) Y[(s0 + i) * kYl + q] = x;
    __syncthreads();
    for (int e = threadIdx.x; e < (kb - s0 - sw) * kZRightCols; e += blockDim.x) {
      const int rr = s0 + sw + e / kZRightCols, c = e % kZRightCols;
      double2 y = Y[rr * kYl + c];
      if (c < cols) {
#pragma unroll 4
        for (int k = 0; k < sw; ++k) zsub(y, L[(s0 + k) * kLl + rr], Y[(s0 + k) * kYl + c]);
        Y[rr * kYl + c] = y;
      }
    }
    __syncthreads();
  }
#pragma unroll 4
  for (int e = threadIdx.x; e < kZB * kZRightCols; e += 256)
    if (e % kZB < kb && e / kZB < cols && q0 + e / kZB >= k0)
      col(e / kZB)[k0 + e % kZB] = Y[(e % kZB) * kYl + e / kZB];
}

// Rows k0 .. k0+kb-1 of X <- U_bb^-1 X: as k_zright from the last rows up.
constexpr int kZBackCols = 8;
constexpr int kZBackSmem = (kZB * (kZB + 1) + kZB * (kZBackCols + 1) + kZB) * (int)sizeof(double2);
__global__ void __launch_bounds__(128) k_zback(const double2* __restrict__ A, int lda, int n, int k0, int kb,
                                               double2* __restrict__ X, int nrhs, ZBatch zb) {
  extern __shared__ __align__(16) double2 zs[];
  double2* U = zs;
  double2* Y = zs + kZB * (kZB + 1);
  double2* R = Y + kZB * (kZBackCols + 1);  // reciprocals of the diagonal
  constexpr int kUl = kZB + 1, kYl = kZBackCols + 1;
  const int q0 = blockIdx.x * kZBackCols, cols = min(kZBackCols, nrhs - q0);
  A += blockIdx.z * zb.a;
  X += blockIdx.z * zb.x;
  pdl_wait();
  pdl_next();
  load_diag<128>(U, A, lda, k0, kb);
#pragma unroll
  for (int e = threadIdx.x; e < kZB * kZBackCols; e += 128)
    if (e % kZB < kb && e / kZB < cols)
      Y[(e % kZB) * kYl + e / kZB] = X[(size_t)(q0 + e / kZB) * n + k0 + e % kZB];
  __syncthreads();
  if (threadIdx.x < kb) R[threadIdx.x] = zrcp(U[threadIdx.x * kUl + threadIdx.x]);
  __syncthreads();
  const int q = threadIdx.x / kZW, i = threadIdx.x % kZW;
  for (int s0 = (kb - 1) / kZW * kZW; s0 >= 0; s0 -= kZW) {
    const int sw = min(kZW, kb - s0);
    double2 x = q < cols && i < sw ? Y[(s0 + i) * kYl + q] : make_double2(0.0, 0.0);
    for (int k = sw - 1; k >= 0; --k) {
      if (i == k) x = zmul(x, R[s0 + k]);
      const double2 xk = make_double2(__shfl_sync(0xffffffffu, x.x, k, kZW), __shfl_sync(0xffffffffu, x.y, k, kZW));
      if (i < k) zsub(x, U[(s0 + k) * kUl + s0 + i], xk);
    }
    if (q < cols && i < sw) Y[(s0 + i) * kYl + q] = x;
    __syncthreads();
    for (int e = threadIdx.x; e < s0 * kZBackCols; e += blockDim.x) {
      const int rr = e / kZBackCols, c = e % kZBackCols;
      if (c < cols) {
        double2 y = Y[rr * kYl + c];
#pragma unroll 4
        for (int k = 0; k < sw; ++k) zsub(y, U[(s0 + k) * kUl + rr], Y[(s0 + k) * kYl + c]);
        Y[rr * kYl + c] = y;
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int e = threadIdx.x; e < kZB * kZBackCols; e += 128)
    if (e % kZB < kb && e / kZB < cols)
      X[(size_t)(q0 + e / kZB) * n + k0 + e % kZB] = Y[(e % kZB) * kYl + e / kZB];
}

// Blocks of the cluster for a panel of `rows` rows: a power of two.
int cluster_of(int rows) {
  int c = 1;
  while (c * kZThreads < rows) c *= 2;
  return c;
}

cudaError_t launch_panel(cudaStream_t st, int batch, double2* A, int n, int c0, int w, ZBatch zb, int* work, int panel,
                         int* info) {
  const int cs = cluster_of(n - c0);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(cs, batch);
  cfg.blockDim = dim3(kZThreads);
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = cs;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, k_zpanel, A, n, n, c0, w, zb, work, panel, info);
}

}  // namespace

size_t zlu_work_ints(int batch) { return (size_t)batch * kZP * kZList; }

int zlu_supported(int n) {
  if (n < 1 || n > kZluMaxRows) return 1;
  if (cudaFuncSetAttribute(k_zpanel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
      cudaFuncSetAttribute(k_zright, cudaFuncAttributeMaxDynamicSharedMemorySize, kZRightSmem) != cudaSuccess ||
      cudaFuncSetAttribute(k_zback, cudaFuncAttributeMaxDynamicSharedMemorySize, kZBackSmem) != cudaSuccess) {
    cudaGetLastError();
    return 1;
  }
  const int cs = cluster_of(n);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(cs);
  cfg.blockDim = dim3(kZThreads);
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = cs;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  int clusters = 0;
  if (cudaOccupancyMaxActiveClusters(&clusters, k_zpanel, &cfg) != cudaSuccess || clusters < 1) {
    cudaGetLastError();
    return 1;
  }
  return 0;
}

int zlu_solve(cudaStream_t st, cublasHandle_t blas, int batch, int n, int nrhs, double2* A, size_t sa, double2* X,
              size_t sx, int* info, int* work, cudaEvent_t evf, long long* launches, long long* lib_calls) {
  const cuDoubleComplex one = make_cuDoubleComplex(1.0, 0.0), mone = make_cuDoubleComplex(-1.0, 0.0);
  if (cudaMemsetAsync(info, 0, sizeof(int), st) != cudaSuccess) return 1;
  const ZBatch zb{sa, sx};
  // c -= a b, a and c with their stride, b with sb
  auto gemm = [&](int m, int nn, int k, const double2* a, const double2* b, size_t sb, double2* c, size_t sc) {
    if (m <= 0 || nn <= 0) return 0;
    *lib_calls += 1;
    const cuDoubleComplex *pa = (const cuDoubleComplex*)a, *pb = (const cuDoubleComplex*)b;
    cuDoubleComplex* pc = (cuDoubleComplex*)c;
    const cublasStatus_t s =
        batch == 1 ? cublasZgemm(blas, CUBLAS_OP_N, CUBLAS_OP_N, m, nn, k, &mone, pa, n, pb, n, &one, pc, n)
                   : cublasZgemmStridedBatched(blas, CUBLAS_OP_N, CUBLAS_OP_N, m, nn, k, &mone, pa, n, (long long)sa, pb,
                                               n, (long long)sb, &one, pc, n, (long long)sc, batch);
    return s == CUBLAS_STATUS_SUCCESS ? 0 : 10 + (int)s;
  };
  auto blocks = [&](int count, int per) { return (unsigned)((count + per - 1) / per); };
  for (int k0 = 0; k0 < n; k0 += kZB) {
    const int k1 = k0 + kZB < n ? k0 + kZB : n, kb = k1 - k0, right = n - k1;
    for (int p = 0, c0 = k0; c0 < k1; ++p, c0 += kZW) {
      const int w = k1 - c0 < kZW ? k1 - c0 : kZW, others = kb - w;
      if (launch_panel(st, batch, A, n, c0, w, zb, work, p, info) != cudaSuccess) return 1;
      *launches += 1;
      if (others > 0) {
        pdl_launch(k_zapply, dim3(blocks(others, kZApplyCols), 1, batch), dim3(128), 0, st, A, n, k0, k1, c0, w, zb,
                   work, p);
        *launches += 1;
      }
      const int rest = k1 - c0 - w, below = n - c0 - w;
      if (rest > 0) {
        pdl_launch(k_zupdate, dim3(blocks(below, 128), blocks(rest, kZUpCols), batch), dim3(128), 0, st, A, n, n, k1,
                   c0, w, zb);
        *launches += 1;
      }
    }
    const int total = k0 + right + nrhs;
    if (total > 0) {
      pdl_launch(k_zright, dim3(blocks(total, kZRightCols), 1, batch), dim3(256), kZRightSmem, st, A, n, n, k0, kb, X,
                 nrhs, zb, work);
      *launches += 1;
    }
    if (cudaPeekAtLastError() != cudaSuccess) return 1;
    double2* Lk = A + (size_t)k0 * n + k1;
    int rc = gemm(right, right, kb, Lk, A + (size_t)k1 * n + k0, sa, A + (size_t)k1 * n + k1, sa);
    if (!rc) rc = gemm(right, nrhs, kb, Lk, X + k0, sx, X + k1, sx);
    if (rc) return rc;
  }
  if (evf && cudaEventRecord(evf, st) != cudaSuccess) return 1;
  if (nrhs <= 0) return 0;
  for (int k0 = (n - 1) / kZB * kZB; k0 >= 0; k0 -= kZB) {
    const int kb = k0 + kZB < n ? kZB : n - k0;
    pdl_launch(k_zback, dim3(blocks(nrhs, kZBackCols), 1, batch), dim3(128), kZBackSmem, st, A, n, n, k0, kb, X, nrhs,
               zb);
    *launches += 1;
    if (cudaPeekAtLastError() != cudaSuccess) return 1;
    const int rc = gemm(k0, nrhs, kb, A + (size_t)k0 * n, X + k0, sx, X, sx);
    if (rc) return rc;
  }
  return 0;
}
