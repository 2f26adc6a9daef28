/*
 * epsilon.h -- the Wynn epsilon extrapolation of Limes (FinGrnExtSubs.f90:
 * 370-470) taken row by row, for device and host.
 *
 * The reference fills its table one column at a time: column c of entry i
 * comes from columns c-1 and c-2, E(c,i) = E(c-2,i+1) + 1/(E(c-1,i+1) -
 * E(c-1,i)) (the first term alone where the two are equal); the even columns
 * hold the extrapolated values s, the odd ones the a = 1/differences.  It
 * returns the s beside the largest |a| met so far in column order, and stops
 * at the first such record whose s equals the entry it came from.
 *
 * Here the partial sums arrive in blocks of kEpsRows, and each block is taken
 * through all the columns it reaches: the block's rows of two neighbouring
 * columns stay in registers, and only the last row of the previous block is
 * kept per column (e).  Every entry has the same operands and the same
 * operations as in the column order, so it has the same bits; the kEpsRows
 * reciprocals of one column are independent, and memory holds one number per
 * column instead of two arrays that every column rewrites.  What depends on
 * the column order is restored from it:
 *   - the largest |a| wins; of equal ones the smallest column, then the first
 *     entry of that column (the entries of a column are met in order here too);
 *   - a record that stops the reference is one whose |a| exceeds every earlier
 *     entry's: those of the columns before it and of its own column.  m keeps
 *     the largest |a| of every column (its upper 32 bits), so that the test is
 *     exact for the rows met so far; a later row whose |a| in an earlier column
 *     is not below the stop's takes it back, and the caller repeats the table
 *     in column order (redo), as it does where the upper 32 bits do not decide
 *     or an entry is not finite.
 */
#ifndef HAMS_EPSILON_H
#define HAMS_EPSILON_H

#include <math.h>
#include <stdint.h>
#include <string.h>

#if defined(__CUDACC__)
#define EPS_FN __host__ __device__ __forceinline__
#else
#define EPS_FN static inline
#endif

namespace hams {

constexpr int kEpsRows = 8;  // rows of the table per block
constexpr uint32_t kEpsNoStop = 0xffffffffu;

EPS_FN uint32_t eps_hi(double x) {  // upper 32 bits of |x|
#if defined(__CUDA_ARCH__)
  return (uint32_t)__double2hiint(x) & 0x7fffffffu;
#else
  uint64_t b;
  memcpy(&b, &x, 8);
  return (uint32_t)(b >> 32) & 0x7fffffffu;
#endif
}

// The larger of the running |a|-like value m and |x|, |y|, by the upper 32
// bits read as a float: the order of the doubles below 2^1017; NaN, which
// stays, from there on.
EPS_FN float eps_top(float m, double x, double y) {
#if defined(__CUDA_ARCH__)
  float r;
  asm("max.NaN.abs.f32 %0, %1, %2, %3;"
      : "=f"(r)
      : "f"(m), "f"(__int_as_float(__double2hiint(x))), "f"(__int_as_float(__double2hiint(y))));
  return r;
#else
  const uint32_t h[3] = {0, eps_hi(x), eps_hi(y)};
  float f[3];
  memcpy(f, h, sizeof f);
  f[0] = m;
  float r = f[0];
  for (int q = 1; q < 3; ++q) r = r != r || f[q] != f[q] ? NAN : f[q] > r ? f[q] : r;
  return r;
#endif
}
EPS_FN uint32_t eps_bits(float m) {
#if defined(__CUDA_ARCH__)
  return __float_as_uint(m);
#else
  uint32_t u;
  memcpy(&u, &m, 4);
  return u;
#endif
}
// The largest of v[FROM..kEpsRows-1] in eps_top's sense; rows below from are left out.
template <int FROM>
EPS_FN float eps_top_of(const double (&v)[kEpsRows], int from) {
  float m = 0.0f;
#pragma unroll
  for (int j = FROM; j < kEpsRows; j += 2) {
    const double x = v[j], y = j + 1 < kEpsRows ? v[j + 1] : 0.0;
    m = eps_top(m, FROM > 0 && j < from ? 0.0 : x, FROM > 0 && j + 1 < from ? 0.0 : y);
  }
  return m;
}

// 1/d rounded to nearest for 2^-1021 < |d| < 2^1021; NaN for d = 0 and
// subnormal d (the callers look for it), tiny for larger d.  Free of branches,
// so that the eight reciprocals of a column overlap (with __drcp_rn EIGENE takes
// 19.3 instead of 13.6 ms and PIDCOCK 10.9 instead of 8.1 ms at 5,400 panels).
// From the hardware's seed y, with e = 1 - d y and so 1/d = y (1 + e + e^2 + ...):
//   - three terms of that series in Horner form leave e^3 < 2^-56: within one ulp;
//   - one more step, y + y e, rounds correctly from within one ulp, except where
//     d has a significand of all ones (P. Markstein, IBM J. Res. Dev. 34, 1990);
//   - there 1/d lies just above the middle of two numbers, and that step stays at
//     the lower one, a power of two, but ends at the upper one from the upper
//     one.  So the seed, whose lower word is zero, gets one of all ones (for the
//     price of the zero): e is then -2^-20, and the error of the three terms is
//     upwards.
// tests/test_epsilon_gpu.py compares the bits with __drcp_rn.
EPS_FN double eps_rcp(double d) {
#if defined(__CUDA_ARCH__)
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
  y = __hiloint2double(__double2hiint(y), -1);
  const double e = __fma_rn(-d, y, 1.0);
  y = __fma_rn(__fma_rn(y, e, y), e, y);
  return __fma_rn(y, __fma_rn(-d, y, 1.0), y);
#else
  return 1.0 / d;
#endif
}

// What a table pass carries from block to block.
struct EpsBest {
  double amax = 0.0, rl = 0.0;    // the largest |a| and the s beside it
  double stop = 0.0;              // the s of the stopping record
  uint32_t kbest = 0;             // column pair of amax
  uint32_t kstop = kEpsNoStop;    // column pair of the stopping record, and the upper bits of its |a|
  uint32_t stop_hi = 0xffffffffu;
  bool redo = false;
};

// r[j] = 1 / (x[j] - x[j-1]) for FROM <= j, zero where the two are equal;
// x[-1] is xb.  A reciprocal of 2^1017 or more, or none, in spite of that
// asks for redo.
template <int FROM>
EPS_FN void eps_recip(const double (&x)[kEpsRows], double xb, int from, double (&r)[kEpsRows], EpsBest& b) {
#pragma unroll
  for (int j = FROM; j < kEpsRows; ++j) r[j] = eps_rcp(x[j] - (j ? x[j - 1] : xb));
  const float top = eps_top_of<FROM>(r, from);
  if (__builtin_expect(top != top, 0)) {  // equal neighbours, rare
#pragma unroll
    for (int j = FROM; j < kEpsRows; ++j)
      if (x[j] == (j ? x[j - 1] : xb)) r[j] = 0.0;
    const float again = eps_top_of<FROM>(r, from);
    b.redo = b.redo || again != again;
  }
}

// One odd column c (= 2k-1) for the rows j >= FROM of the block (and j >= from
// in the first block): w holds column c-2 and becomes column c, x is column
// c-1; wb, xb are the previous block's last row of those columns.
template <int FROM>
EPS_FN void eps_odd(double (&w)[kEpsRows], double wb, const double (&x)[kEpsRows], double xb, int from, EpsBest& b) {
  double r[kEpsRows];
  eps_recip<FROM>(x, xb, from, r, b);
#pragma unroll
  for (int j = kEpsRows - 1; j >= FROM; --j) w[j] = (j ? w[j - 1] : wb) + r[j];
}

// One even column c = 2k: x holds column c-2 and becomes column c, w is
// column c-1 (the a), with the previous block's last rows xb, wb; mk is the
// largest |a| (upper bits) of column pair k so far, before that of the pairs
// below k.
template <int FROM>
EPS_FN void eps_even(double (&x)[kEpsRows], double xb, const double (&w)[kEpsRows], double wb, int from, uint32_t k,
                     uint32_t& mk, uint32_t& before, EpsBest& b) {
  double r[kEpsRows];
  eps_recip<FROM>(w, wb, from, r, b);
  // new entries, downwards (each needs the old entry below it), and which of
  // them equal that old entry
  uint32_t same = 0;
#pragma unroll
  for (int j = kEpsRows - 1; j >= FROM; --j) {
    const double old = j ? x[j - 1] : xb, y = old + r[j];
    if (y == old) same |= 1u << j;
    x[j] = y;
  }
  if (FROM > 0) same &= ~0u << from;
  // the largest |a| of the block's rows of this column (rows j-1), upper bits
  double av[kEpsRows];
#pragma unroll
  for (int j = FROM; j < kEpsRows; ++j) av[j] = j ? w[j - 1] : wb;
  const uint32_t th = eps_bits(eps_top_of<FROM>(av, from));
  if (__builtin_expect(same != 0, 0)) {  // a converged entry
    uint32_t prev = mk > before ? mk : before;
#pragma unroll
    for (int j = FROM; j < kEpsRows; ++j) {
      if (FROM > 0 && j < from) continue;
      const uint32_t h = eps_hi(av[j]);
      if ((same >> j & 1u) && k < b.kstop) {
        if (h > prev) {
          b.kstop = k;
          b.stop_hi = h;
          b.stop = x[j];
        } else if (h == prev) {
          b.redo = true;
        }
      }
      prev = h > prev ? h : prev;
    }
  }
  if (__builtin_expect(k < b.kstop && th >= b.stop_hi, 0)) b.redo = true;  // the stop was no record after all
  const uint32_t ah = eps_hi(b.amax);
  if (th >= ah) {
    // a new largest |a|, the first of equal ones; or one with the same upper
    // bits, which may equal the one so far and be of an earlier column
    const double top = b.amax;
    bool tie = th == ah && k < b.kbest;
#pragma unroll
    for (int j = FROM; j < kEpsRows; ++j) {
      if (FROM > 0 && j < from) continue;
      const double t = fabs(av[j]);
      if (t > b.amax || (tie && t == top)) {
        b.amax = t;
        b.rl = x[j];
        b.kbest = k;
        tie = false;
      }
    }
  }
  mk = th > mk ? th : mk;
  before = mk > before ? mk : before;
}

// The columns that only the rows from ODD0 on reach, c = q0 + T for rows
// j >= T; the odd column comes first.
template <int T>
EPS_FN void eps_tail(double (&x)[kEpsRows], double xb, double (&w)[kEpsRows], double wb, int pad, uint32_t c, double* e,
                     uint32_t* m, int ld, bool keep, uint32_t& before, EpsBest& b) {
  if constexpr (T < kEpsRows) {
    const int from = T + pad;
    eps_odd<T>(w, wb, x, xb, from, b);
    if (keep) e[(int)c * ld] = w[kEpsRows - 1];
    if constexpr (T + 1 < kEpsRows) {
      const uint32_t k = (c + 1) / 2;
      uint32_t mk = 0;  // a pair's first rows are met here
      eps_even<T + 1>(x, 0.0, w, 0.0, from + 1, k, mk, before, b);
      if (keep) {
        m[(int)k * ld] = mk;
        e[(int)(c + 1) * ld] = x[kEpsRows - 1];
      }
      eps_tail<T + 2>(x, 0.0, w, 0.0, pad, c + 2, e, m, ld, keep, before, b);
    }
  }
}

// Takes the block of partial sums x through the table.  The first block
// (q0 = 0) holds its rows at j >= pad; later ones are full (pad 0) and start at
// row q0; the last one of a sequence has keep false.  e[c ld] and m[k ld] belong
// to this sequence (eps_columns and eps_pairs of them).
EPS_FN void eps_block(double (&x)[kEpsRows], int q0, int pad, double* e, uint32_t* m, int ld, bool keep, EpsBest& b) {
  double w[kEpsRows];
#pragma unroll
  for (int j = 0; j < kEpsRows; ++j) w[j] = 0.0;
  double xb = 0.0, wb = 0.0;
  uint32_t before = 0;
  if (q0) xb = e[0];
  if (keep) e[0] = x[kEpsRows - 1];
  int c = 1;
  for (; c + 1 <= q0; c += 2) {
    const double wn = e[c * ld], xn = c + 1 < q0 ? e[(c + 1) * ld] : 0.0;
    const uint32_t k = (uint32_t)(c + 1) / 2;
    uint32_t mk = c + 1 < q0 ? m[(int)k * ld] : 0u;
    eps_odd<0>(w, wb, x, xb, 0, b);
    eps_even<0>(x, xb, w, wn, 0, k, mk, before, b);
    if (keep) {
      e[c * ld] = w[kEpsRows - 1];
      m[(int)k * ld] = mk;
      e[(c + 1) * ld] = x[kEpsRows - 1];
    }
    xb = xn;
    wb = wn;
  }
  if (q0 & 1) eps_tail<0>(x, xb, w, wb, 0, (uint32_t)c, e, m, ld, keep, before, b);
  else eps_tail<1>(x, 0.0, w, 0.0, pad, (uint32_t)c, e, m, ld, keep, before, b);
}

// Entries of e and of m that a sequence of n partial sums needs: the columns
// that the last block finds (its first row is at n - kEpsRows).
EPS_FN constexpr int eps_columns(int n) { return n > 2 * kEpsRows ? n - kEpsRows : kEpsRows; }
EPS_FN constexpr int eps_pairs(int n) { return eps_columns(n) / 2 + 1; }

// The result after the last block; last is the last partial sum.
EPS_FN double eps_result(const EpsBest& b, double last) {
  if (b.kstop != kEpsNoStop) return b.stop;
  return b.amax > 0.0 ? b.rl : last;
}

}  // namespace hams
#endif
