// green_series.cu -- the epsilon-accelerated finite-depth Green kernels.
//
// EIGENE and PIDCOCK (FinGreen3D.f90:413-660) sum up to 100 eigenfunction
// terms and extrapolate them with the Wynn epsilon algorithm (Limes), which
// divides by differences of nearly equal partial sums and stops on exact
// equalities.  This file is compiled with --fmad=false so that every product
// and sum of those series is rounded exactly as in the CPU oracle; the
// transcendental functions inside them come from detmath.h.  The remaining
// kernels (hams_gpu.cu) keep fused multiply-adds.
#include <atomic>

#include "kernels.cuh"
#include "epsilon.h"
#include "rankine.cuh"

// Horizontal distance of a pair, as fingreen3d of this file rounds it.
__device__ __forceinline__ double pair_distance(const DevGeom& g, uint32_t p) {
  const uint32_t tn = (uint32_t)g.tn;
  const int j = (int)(p / tn), i = (int)(p - (uint32_t)j * tn);
  const double xpq = g.xq[j] - g.fxyz[i], ypq = g.xq[j + g.n] - g.fxyz[i + g.tn];
  return sqrt(xpq * xpq + ypq * ypq);
}

__global__ void k_series_distance(DevGeom g, const uint32_t* __restrict__ pairs, long long count,
                                  double* __restrict__ r) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < count) r[t] = pair_distance(g, pairs[t]);
}

void launch_series_distance(cudaStream_t st, DevGeom g, const uint32_t* pairs, long long count, double* r) {
  k_series_distance<<<(unsigned)((count + 255) / 256), 256, 0, st>>>(g, pairs, count, r);
}

// Series length of a distance (FinGreen3D.f90:434, :592)
template <int BR>
__device__ __forceinline__ int series_terms(double r, double h) {
  const double rhp = fabs(r / h);
  return BR == hams::kPidcock ? (int)(HAMS_F4(-1010.10) * rhp + HAMS_F4(100.50))
                              : (int)(HAMS_F4(-88.89) * rhp + HAMS_F4(54.45));
}
template <int BR>
constexpr int series_max() {
  return BR == hams::kPidcock ? hams::kPidcockMax : hams::kEigenEMax;
}

// The radial table of a branch: one thread per (distance, mode), blockIdx.y
// the mode (0: the propagating mode's J and Y).  The threads of a warp hold
// neighbouring distances of one mode, so the loops of ik01a end together.
template <int BR>
__global__ void __launch_bounds__(128) k_rad_series(DevGeom g, WaveDev w, const double* __restrict__ wvn,
                                                    const double* __restrict__ ur, const uint32_t* __restrict__ pairs,
                                                    long long count, double* __restrict__ kt,
                                                    double4* __restrict__ jy) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= count) return;
  const double r = ur ? ur[t] : pair_distance(g, pairs[t]);
  if (blockIdx.y == 0) {
    double4 v;
    hams::jy01b(wvn[0] * r, v.x, v.y, v.z, v.w);
    jy[t] = v;
    return;
  }
  const int i = blockIdx.y + 1;
  if (i > min(series_terms<BR>(r, w.h), series_max<BR>())) return;
  double k0, k1;
  hams::ik01a(wvn[i - 1] * r, k0, k1);
  if (BR == hams::kPidcock) {
    const double umt = (i - 1) * 3.141592653589793 / w.h;
    double k0t, k1t;
    hams::ik01a(umt * r, k0t, k1t);
    reinterpret_cast<double2*>(kt)[(size_t)t * (rad_stride(BR) / 2) + 2 * (i - 2)] = make_double2(k0, k1);
    reinterpret_cast<double2*>(kt)[(size_t)t * (rad_stride(BR) / 2) + 2 * (i - 2) + 1] = make_double2(k0t, k1t);
  } else {
    reinterpret_cast<double2*>(kt)[(size_t)t * (rad_stride(BR) / 2) + (i - 2)] = make_double2(k0, k1);
  }
}

void launch_rad_series(int br, int ntmax, cudaStream_t st, DevGeom g, WaveDev w, const double* wvn, const double* ur,
                       const uint32_t* pairs, long long count, double* kt, double4* jy) {
  const dim3 grid((unsigned)((count + 127) / 128), ntmax);
  if (br == hams::kPidcock)
    k_rad_series<hams::kPidcock><<<grid, 128, 0, st>>>(
        g, w, wvn, ur, pairs, count, kt, jy);
  else
    k_rad_series<hams::kEigenE><<<grid, 128, 0, st>>>(
        g, w, wvn, ur, pairs, count, kt, jy);
}

// One term of table T (0: G, 1: dG/dR, 2: dG/dz) of mode i, FinGreen3D.f90:
// 446-470 (EIGENE) and :597-627 (PIDCOCK).
template <int BR>
struct SeriesTerm {
  const double* __restrict__ wvn;
  const double* __restrict__ pm;
  const double* __restrict__ ac;
  const double* __restrict__ kt;    // the pair's radial row, at K0 or K1
  const double* __restrict__ src;   // the source panel's sin or cos of mode 0, stride sn
  const double* __restrict__ srct;
  const double* __restrict__ fld;   // the field point's cos of mode 0, stride fn
  const double* __restrict__ fldt;
  size_t sn, fn;
  double h;
  int table;
  __device__ __forceinline__ double operator()(int i) const {
    if (BR == hams::kEigenE) {
      const double p = pm[i], c = table == 0 ? p : -p * wvn[i - 1];
      return c * kt[2 * (i - 2)] * src[i * sn] * fld[i * fn];
    }
    const double um = wvn[i - 1], umt = (i - 1) * 3.141592653589793 / h, a = ac[i];
    const double su = src[i * sn], sut = srct[i * sn], cup = fld[i * fn], cutp = fldt[i * fn];
    const double k = kt[4 * (i - 2)], kk = kt[4 * (i - 2) + 2];
    if (table == 2) {
      const double dam = -um * a * su * cup, damt = -umt * sut * cutp / h;
      return dam * k - damt * kk;
    }
    const double am = a * su * cup, amt = sut * cutp / h;
    return table == 0 ? am * k - amt * kk : -um * am * k + umt * amt * kk;
  }
};

// The same table in the reference's column order, for the rare sequences whose
// row-ordered pass asks for it (epsilon.h).
template <int BR>
__device__ __noinline__ double series_columns(const SeriesTerm<BR>& term, int nt) {
  double s[series_max<BR>()], a[series_max<BR>()];
  s[0] = 0.0;
  for (int i = 2; i <= nt; ++i) s[i - 1] = s[i - 2] + term(i);
  return hams::limes(nt - 1, s, a);
}

// Pidcock's image sum of one table (IMGS/DGSR/DGSZ), as pidcock_images.
__device__ __noinline__ double pidcock_image(int table, double r, double zf, double zp, double h) {
  const double t1 = r / h, t2 = (zf - zp) / h, t3 = (zf + zp + 2.0 * h) / h;
  double s = 0.0, q = 0.0;
  for (int l = -1; l <= 1; ++l) {
    const double a = t2 + 2.0 * l, b = t3 + 2.0 * l;
    const double ra = sqrt(t1 * t1 + a * a), rb = sqrt(t1 * t1 + b * b);
    if (table == 0) s += 1.0 / ra + 1.0 / rb;
    else if (table == 1) s += t1 / (ra * ra * ra) + t1 / (rb * rb * rb);
    else s += a / (ra * ra * ra) + b / (rb * rb * rb);
  }
  double p1[5], p23[5];
  for (int m = 0; m <= 4; ++m) {
    p1[m] = table == 1 ? pow(t1, 2.0 * m - 1.0) : pow(t1, 2.0 * m);
    p23[m] = table == 2 ? pow(t2, 2.0 * m - 1.0) + pow(t3, 2.0 * m - 1.0) : pow(t2, 2.0 * m) + pow(t3, 2.0 * m);
  }
  for (int m = 0; m <= 4; ++m)
    for (int n = 0; n <= 4; ++n) {
      const double amn = hams::c_amn[m + 5 * n];
      if (table == 0) q += amn * p1[m] * p23[n];
      else if (table == 1 && m >= 1) q += 2.0 * m * amn * p1[m] * p23[n];
      else if (table == 2 && n >= 1) q += 2.0 * n * amn * p1[m] * p23[n];
    }
  return table == 0 ? (s - 2.0 + q) / h : (-s + q) / (h * h);
}

// EIGENE and PIDCOCK pairs.  Three warps share 32 pairs, one per epsilon table
// (G, dG/dR, dG/dz): a table's chain of reciprocals is the pair's latency, and
// the three are independent.  The partial sums go through the epsilon table in
// blocks of 8 rows kept in registers (epsilon.h), so that 8 reciprocals are in
// flight per thread; the last row of each block (8 bytes per column) and the
// largest |a| per column pair (4 bytes) are in shared memory, sized for the
// launch's longest series (rows terms).
// Issue-bound: about 18 instructions per table entry, 8 of them FP64 (the FP64
// pipe is at half its rate).  Against one thread per pair with the Bessel
// functions in the loop and the tables column by column in local memory
// (5,400 panels, every pair): EIGENE 36.8 -> 13.9 ms for 11.2 M pairs, PIDCOCK
// 16.0 -> 7.9 ms for 0.63 M; an irregular mesh of 5,400 panels in 150 m, its pairs in
// the order of their distances, EIGENE 124.5 -> 92.9 ms for 26.8 M pairs and PIDCOCK
// 59.4 -> 48.9 ms for 2.29 M with their tables.  Blocks of 4 or 6 rows (more warps, more columns
// read and written per entry) measured the same within 3 %, one loop body for
// all columns (less code, idle rows computed) 6-20 % slower.
constexpr int kSerThreads = 96;
// What a launch evaluates: panel pairs, combined into A and S, or the points
// of hams_eval_green (a chunk of its list, point t of the chunk being source t
// and field point t of g), whose G and gradient go to out.
struct PairIO {
  static constexpr bool kPoints = false;
  const uint32_t* __restrict__ pairs;
  const double* __restrict__ rs;
  const double* __restrict__ rd;
  double2* __restrict__ A;
  double2* __restrict__ S;
};
struct PointIO {
  static constexpr bool kPoints = true;
  const uint32_t* __restrict__ list;
  const int* __restrict__ flag;
  double2* __restrict__ out;
  size_t npts;
};
template <int BR, class IO>
__global__ void __launch_bounds__(kSerThreads, 5) k_green_series(DevGeom g, WaveDev w, const double* __restrict__ wvn,
                                                                 hams::ModeTab mt, RadTab rt, IO io, long long count,
                                                                 int* ovf, int rows) {
  extern __shared__ double sm[];
  __shared__ double2 dz[32];
  const int table = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // the list is sorted by series length: the longest first
  const long long t0 = ((long long)gridDim.x - 1 - blockIdx.x) * 32 + lane;
  const bool live = t0 < count;
  const long long t = live ? t0 : count - 1;
  uint32_t p;
  int i, j, flag;
  if constexpr (IO::kPoints) {
    p = io.list[t];
    i = j = (int)t;
    flag = io.flag[p];
  } else {
    const uint32_t tn = (uint32_t)g.tn;
    p = io.pairs[t];
    j = (int)(p / tn);
    i = (int)(p - (uint32_t)j * tn);
    flag = near_flag(g, i, j);
  }
  const double xp = g.fxyz[i], yp = g.fxyz[i + g.tn], zp = g.fxyz[i + 2 * g.tn];
  const double xq = g.xq[j], yq = g.xq[j + g.n], zq = g.xq[j + 2 * g.n];
  if constexpr (!IO::kPoints) {
    if (w.limit) {
      if (table == 0 && live)
        store_pair(g, p, i, j, hams::green_limit(w.limit == 2, xq, xp, yq, yp, zq, zp, flag), io.rs, io.rd, io.A, io.S);
      return;
    }
  }
  const double xpq = xq - xp, ypq = yq - yp, zpq = zq + zp, h = w.h;
  const double rr = sqrt(xpq * xpq + ypq * ypq);
  const uint32_t row = rt.rid ? rt.rid[t] - rt.base : (uint32_t)t;

  // the extrapolated sum of this warp's table
  int nt = series_terms<BR>(rr, h);
  if (nt > rows) {  // outside the branch's range of R/h
    atomicOr(ovf, 1);
    nt = rows;
  }
  SeriesTerm<BR> term;
  term.wvn = wvn;
  term.pm = mt.pm;
  term.ac = mt.ac;
  term.kt = rt.kt + (size_t)row * rad_stride(BR) + (table == 1 ? 1 : 0);
  term.src = reinterpret_cast<const double*>(mt.src + j) + (table == 2 ? 0 : 1);
  term.srct = reinterpret_cast<const double*>(mt.srct + j) + (table == 2 ? 0 : 1);
  term.fld = mt.fld + i;
  term.fldt = mt.fldt + i;
  term.sn = 2 * (size_t)g.n;
  term.fn = (size_t)g.tn;
  term.h = h;
  term.table = table;
  double l;
  {
    double* e = sm + threadIdx.x;
    uint32_t* m = reinterpret_cast<uint32_t*>(sm + (size_t)hams::eps_columns(rows) * kSerThreads) + threadIdx.x;
    hams::EpsBest best;
    // the first block holds the rows that full blocks do not divide; a row's
    // sum s_q adds mode q + 1, and s_0 = 0
    const int r0 = (nt - 1) % hams::kEpsRows + 1, pad = hams::kEpsRows - r0;
    double x[hams::kEpsRows], s = 0.0;
#pragma unroll
    for (int k = 0; k < hams::kEpsRows; ++k) {
      if (k > pad) s += term(k - pad + 1);
      x[k] = s;
    }
    hams::eps_block(x, 0, pad, e, m, kSerThreads, r0 < nt, best);
    for (int q = r0; q < nt; q += hams::kEpsRows) {
#pragma unroll
      for (int k = 0; k < hams::kEpsRows; ++k) x[k] = term(q + k + 1);
#pragma unroll
      for (int k = 0; k < hams::kEpsRows; ++k) {
        s += x[k];
        x[k] = s;
      }
      hams::eps_block(x, q, 0, e, m, kSerThreads, q + hams::kEpsRows < nt, best);
    }
    l = best.redo ? series_columns<BR>(term, nt) : hams::eps_result(best, s);
  }

  // this table's component of G: the propagating mode, the series, minus the
  // Rankine terms, plus the point sources (FINGREEN3D)
  const double wk = wvn[0], czp = mt.fld[g.tn + i];
  const double2 szf = mt.src[g.n + j];  // sinh, cosh of k0 (zq + h)
  const double4 jy = rt.jy[row];
  const double p0 = mt.pm[1] * szf.y * czp;
  // the distances to the source and its image, with which FINGREEN3D both
  // removes and adds the point sources
  const double r = sqrt(rr * rr + (zq - zp) * (zq - zp)), r1 = sqrt(rr * rr + zpq * zpq);
  cplx v;
  if (BR == hams::kEigenE) {
    if (table == 0) v = hams::cmk(-p0 * jy.z, p0 * jy.x);
    else if (table == 1) v = hams::cmk(wk * p0 * jy.w, -wk * p0 * jy.y);
    else {
      const double dp0 = mt.pm[1] * szf.x * czp;
      v = hams::cmk(-wk * dp0 * jy.z, wk * dp0 * jy.x);
    }
    v.re += l;
  } else {
    if (table == 0) v = hams::cmk(-p0 * jy.z + 2.0 / h * (0.5772156649015328 + log(rr / 4.0 / h)), p0 * jy.x);
    else if (table == 1) v = hams::cmk(wk * p0 * jy.w + 2.0 / (rr * h), -wk * p0 * jy.y);
    else {
      const double dp0 = mt.ac[1] * szf.x * czp;
      v = hams::cmk(-dp0 * jy.z, dp0 * jy.x);
    }
    v.re = v.re + 4.0 * l + pidcock_image(table, rr, zq, zp, h);
  }
  const double ir1 = 1.0 / r1, ir13 = ir1 * ir1 * ir1, ir = 1.0 / r, ir3 = ir * ir * ir;
  if (table == 0) {
    v.re -= (ir + ir1);
    v.re += flag == 1 ? ir1 : ir1 + ir;
    if (live) {
      if constexpr (IO::kPoints) {
        io.out[p] = make_double2(v.re, v.im);
      } else {
        const double ds = g.ds[j];
        io.S[p] = make_double2(io.rs[p] + v.re * ds, v.im * ds);
      }
    }
  } else if (table == 2) {
    v.re += ((zq - zp) / r / (r * r) + zpq / r1 / (r1 * r1));
    v.re -= flag == 1 ? zpq * ir13 : zpq * ir13 + (zq - zp) * ir3;
    if constexpr (IO::kPoints) {
      if (live) io.out[p + 3 * io.npts] = make_double2(v.re, v.im);
    } else {
      dz[lane] = make_double2(v.re, v.im);
    }
  }
  __syncthreads();
  if (table == 1 && live) {
    v.re += (rr / r / (r * r) + rr / r1 / (r1 * r1));
    cplx gx = hams::cmk(0.0, 0.0), gy = hams::cmk(0.0, 0.0);
    if (rr > HAMS_F4(1.E-6)) {
      gx = v * (xpq / rr);
      gy = v * (ypq / rr);
    }
    gx.re -= flag == 1 ? xpq * ir13 : xpq * ir13 + xpq * ir3;
    gy.re -= flag == 1 ? ypq * ir13 : ypq * ir13 + ypq * ir3;
    if constexpr (IO::kPoints) {
      io.out[p + io.npts] = make_double2(gx.re, gx.im);
      io.out[p + 2 * io.npts] = make_double2(gy.re, gy.im);
      return;
    }
    const double2 gz = dz[lane];
    const double ds = g.ds[j], n1 = g.nrm[j], n2 = g.nrm[j + g.n], n3 = g.nrm[j + 2 * g.n];
    if constexpr (!IO::kPoints) {
      double are = io.rd[p] + ds * (gx.re * n1 + gy.re * n2 + gz.x * n3);
      const double aim = ds * (gx.im * n1 + gy.im * n2 + gz.y * n3);
      if (g.diag && i == j) are += 2.0 * 3.141592653589793;
      io.A[p] = make_double2(are, aim);
    }
  }
}

// Shared memory of a launch whose longest series has rows terms.
static size_t series_smem(int rows) {
  return ((size_t)hams::eps_columns(rows) * 8 + (size_t)hams::eps_pairs(rows) * 4) * kSerThreads;
}

// The shared-memory sizes of the series kernels, once per device.
int series_kernels_init() {
  static std::atomic<bool> done[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 1;
  if (dev < 64 && done[dev]) return 0;
  auto opt = [](const void* f, int rows) {
    return cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)series_smem(rows)) != cudaSuccess;
  };
  if (opt((const void*)k_green_series<hams::kPidcock, PairIO>, hams::kPidcockMax) ||
      opt((const void*)k_green_series<hams::kEigenE, PairIO>, hams::kEigenEMax) ||
      opt((const void*)k_green_series<hams::kPidcock, PointIO>, hams::kPidcockMax) ||
      opt((const void*)k_green_series<hams::kEigenE, PointIO>, hams::kEigenEMax))
    return 1;
  if (dev < 64) done[dev] = true;
  return 0;
}

template <class IO>
static void launch_series(int br, int ntmax, cudaStream_t st, const DevGeom& g, const WaveDev& w, const double* wvn,
                          const hams::ModeTab& mt, const RadTab& rt, const IO& io, long long count, int* ovf) {
  const unsigned blocks = (unsigned)((count + 31) / 32);
  const size_t sh = series_smem(ntmax);
  if (br == hams::kPidcock)
    k_green_series<hams::kPidcock, IO><<<blocks, kSerThreads, sh, st>>>(g, w, wvn, mt, rt, io, count, ovf, ntmax);
  else
    k_green_series<hams::kEigenE, IO><<<blocks, kSerThreads, sh, st>>>(g, w, wvn, mt, rt, io, count, ovf, ntmax);
}

void launch_green_series(int br, int ntmax, cudaStream_t st, DevGeom g, WaveDev w, const double* wvn,
                         const hams::ModeTab& mt, RadTab rt, const uint32_t* pairs, long long count, const double* rs,
                         const double* rd, double2* A, double2* S, int* ovf) {
  launch_series(br, ntmax, st, g, w, wvn, mt, rt, PairIO{pairs, rs, rd, A, S}, count, ovf);
}

// Per-frequency mode tables (ModeTab) for modes 2..nmode-1: one thread per
// (mode, panel) entry, the expressions of InlineModes (green.cuh), compiled
// here without fused multiply-adds like the series that read them.  Slot 1
// holds the propagating mode's factors: pm[1] = pi / NM0, ac[1] = k0 pi / NM0,
// src = (sinh, cosh) of k0 (zq + h), fld = cosh of k0 (zp + h).
__global__ void k_mode_tables(DevGeom g, WaveDev w, const double* __restrict__ wvn, int nmode, double* pm, double* ac,
                              double2* src, double2* srct, double* fld, double* fldt) {
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  int i = blockIdx.y + 1;  // mode number (1: propagating-mode factors)
  if (i >= nmode) return;
  const double h = w.h;
  if (i == 1) {
    const double wk = w.wk;
    if (k < g.n) {
      double zfh = g.xq[k + 2 * g.n] + h;
      src[g.n + k] = make_double2(sinh(wk * zfh), cosh(wk * zfh));
    }
    if (k < g.tn) fld[g.tn + k] = cosh(wk * (g.fxyz[k + 2 * g.tn] + h));
    if (k == 0) {
      const double nm0 = h / 2.0 * (1.0 + sinh(2.0 * wk * h) / (2.0 * wk * h));
      pm[1] = 3.141592653589793 / nm0;
      ac[1] = wk * 3.141592653589793 / nm0;
    }
    return;
  }
  if (k < g.n) {
    hams::InlineModes md{wvn, h, w.v, g.xq[k + 2 * g.n] + h, 0.0};
    double s, c;
    md.src(i, s, c);
    src[(size_t)i * g.n + k] = make_double2(s, c);
    md.srct(i, s, c);
    srct[(size_t)i * g.n + k] = make_double2(s, c);
  }
  if (k < g.tn) {
    hams::InlineModes md{wvn, h, w.v, 0.0, g.fxyz[k + 2 * g.tn] + h};
    fld[(size_t)i * g.tn + k] = md.fld(i);
    fldt[(size_t)i * g.tn + k] = md.fldt(i);
  }
  if (k == 0) {
    hams::InlineModes md{wvn, h, w.v, 0.0, 0.0};
    pm[i] = md.pm(i);
    ac[i] = md.ac(i);
  }
}

void launch_mode_tables(cudaStream_t st, DevGeom g, WaveDev w, const double* wvn, int nmode, double* pm, double* ac,
                        double2* src, double2* srct, double* fld, double* fldt) {
  dim3 grid((max(g.n, g.tn) + 127) / 128, nmode - 1);
  k_mode_tables<<<grid, 128, 0, st>>>(g, w, wvn, nmode, pm, ac, src, srct, fld, fldt);
}

// Batch Green evaluation: any branch, one pair per thread; list (count
// entries): the points to evaluate, or null for all.
__global__ void k_eval_green(int npts, const double* __restrict__ pts, const int* __restrict__ flag, WaveDev w,
                             const double* __restrict__ wvn, double2* __restrict__ out, int* ovf,
                             const uint32_t* __restrict__ list, int count) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= count) return;
  if (list) t = (int)list[t];
  double xq = pts[t], yq = pts[t + npts], zq = pts[t + 2 * (size_t)npts];
  double xp = pts[t + 3 * (size_t)npts], yp = pts[t + 4 * (size_t)npts], zp = pts[t + 5 * (size_t)npts];
  grn4 G;
  if (w.limit) {
    G = hams::green_limit(w.limit == 2, xq, xp, yq, yp, zq, zp, flag[t]);
  } else if (w.h < 0.0) {
    G = hams::infgreen3d(xq, xp, yq, yp, zq, zp, w.v, flag[t]);
  } else {
    int o = 0;
    double rr = sqrt((xq - xp) * (xq - xp) + (yq - yp) * (yq - yp));
    switch (hams::fin_branch(rr, w.h)) {
      case hams::kLinton: G = hams::fingreen3d<hams::kLinton>(xq, xp, yq, yp, zq, zp, w.v, wvn, w.h, flag[t], (void*)nullptr, &o); break;
      case hams::kPidcock: {
        hams::SeriesScratchN<hams::kPidcockMax> sc;
        G = hams::fingreen3d<hams::kPidcock>(xq, xp, yq, yp, zq, zp, w.v, wvn, w.h, flag[t], &sc, &o);
        break;
      }
      case hams::kEigenE: {
        hams::SeriesScratchN<hams::kEigenEMax> sc;
        G = hams::fingreen3d<hams::kEigenE>(xq, xp, yq, yp, zq, zp, w.v, wvn, w.h, flag[t], &sc, &o);
        break;
      }
      default: G = hams::fingreen3d<hams::kEigen>(xq, xp, yq, yp, zq, zp, w.v, wvn, w.h, flag[t], (void*)nullptr, &o); break;
    }
    if (o) atomicOr(ovf, 1);
  }
  for (int k = 0; k < 4; ++k) out[t + (size_t)k * npts] = make_double2(G.g[k].re, G.g[k].im);
}

// The points of hams_eval_green, sorted by branch and series length
// (kPointBins keys): a histogram, the offsets formed by the host, and the
// points filed into their bins (the order inside a bin is free: every point is
// computed by itself).
__global__ void __launch_bounds__(256) k_point_bins(int npts, const double* __restrict__ pts, double h,
                                                    unsigned short* __restrict__ key, uint32_t* __restrict__ hist) {
  __shared__ uint32_t sh[kPointBins];
  for (int b = threadIdx.x; b < kPointBins; b += blockDim.x) sh[b] = 0;
  __syncthreads();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < npts) {
    const double dx = pts[t] - pts[t + 3 * (size_t)npts], dy = pts[t + npts] - pts[t + 4 * (size_t)npts];
    const double rr = sqrt(dx * dx + dy * dy);
    const int k = hams::fin_branch(rr, h) * kPointTerms + min(max(hams::fin_terms(rr, h), 0), kPointTerms - 1);
    key[t] = (unsigned short)k;
    atomicAdd(&sh[k], 1u);
  }
  __syncthreads();
  for (int b = threadIdx.x; b < kPointBins; b += blockDim.x)
    if (sh[b]) atomicAdd(&hist[b], sh[b]);
}
__global__ void k_point_file(int npts, const unsigned short* __restrict__ key, uint32_t* __restrict__ next,
                             uint32_t* __restrict__ list) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < npts) list[atomicAdd(&next[key[t]], 1u)] = (uint32_t)t;
}
// A chunk of the list as sources xq and field points fx (m x 3 each) with
// their distances r.
__global__ void k_point_gather(int npts, const double* __restrict__ pts, const uint32_t* __restrict__ list, int m,
                               double* __restrict__ xq, double* __restrict__ fx, double* __restrict__ r) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= m) return;
  const size_t p = list[t];
  double q[6];
  for (int k = 0; k < 6; ++k) q[k] = pts[p + k * (size_t)npts];
  for (int k = 0; k < 3; ++k) {
    xq[t + k * m] = q[k];
    fx[t + k * m] = q[3 + k];
  }
  const double xpq = q[0] - q[3], ypq = q[1] - q[4];
  r[t] = sqrt(xpq * xpq + ypq * ypq);
}
// LINTON points, a warp each (hams::WarpQuad); lane 0 stores.
constexpr int kPointWarps = 4;
__global__ void __launch_bounds__(32 * kPointWarps) k_point_linton(int npts, const double* __restrict__ pts,
                                                                   const int* __restrict__ flag, WaveDev w,
                                                                   const double* __restrict__ wvn,
                                                                   const uint32_t* __restrict__ list, int count,
                                                                   double2* __restrict__ out, int* ovf) {
  __shared__ double stack[kPointWarps][2][hams::kQuadStack];
  const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5, k = blockIdx.x * kPointWarps + wl;
  if (k >= count) return;  // the whole warp
  const size_t t = list[k], n = npts;
  int o = 0;
  const hams::WarpQuad quad{stack[wl][0], stack[wl][1], lane};
  const grn4 G = hams::fingreen3d_linton(pts[t], pts[t + 3 * n], pts[t + n], pts[t + 4 * n], pts[t + 2 * n],
                                         pts[t + 5 * n], w.v, wvn, w.h, flag[t], &o, quad);
  if (lane != 0) return;
  if (o) atomicOr(ovf, 1);
  for (int q = 0; q < 4; ++q) out[t + q * n] = make_double2(G.g[q].re, G.g[q].im);
}

void launch_point_bins(cudaStream_t st, int npts, const double* pts, double h, unsigned short* key, uint32_t* hist) {
  k_point_bins<<<(npts + 255) / 256, 256, 0, st>>>(npts, pts, h, key, hist);
}
void launch_point_file(cudaStream_t st, int npts, const unsigned short* key, uint32_t* next, uint32_t* list) {
  k_point_file<<<(npts + 255) / 256, 256, 0, st>>>(npts, key, next, list);
}
void launch_point_linton(cudaStream_t st, int npts, const double* pts, const int* flag, WaveDev w, const double* wvn,
                         const uint32_t* list, int count, double2* out, int* ovf) {
  k_point_linton<<<(count + kPointWarps - 1) / kPointWarps, 32 * kPointWarps, 0, st>>>(npts, pts, flag, w, wvn, list,
                                                                                       count, out, ovf);
}
void launch_point_single(cudaStream_t st, int npts, const double* pts, const int* flag, WaveDev w, const double* wvn,
                        const uint32_t* list, int count, double2* out, int* ovf) {
  k_eval_green<<<(count + 127) / 128, 128, 0, st>>>(npts, pts, flag, w, wvn, out, ovf, list, count);
}
void launch_point_series(int br, int ntmax, cudaStream_t st, int npts, const double* pts, const int* flag, WaveDev w,
                         const double* wvn, const uint32_t* list, int m, const PointWork& pw, double2* out, int* ovf) {
  k_point_gather<<<(m + 127) / 128, 128, 0, st>>>(npts, pts, list, m, pw.xq, pw.fx, pw.r);
  DevGeom g{};
  g.n = g.tn = m;
  g.xq = pw.xq;
  g.fxyz = pw.fx;
  const int nmode = ntmax + 1;
  launch_mode_tables(st, g, w, wvn, nmode, pw.pm, pw.ac, pw.src, pw.srct, pw.fld, pw.fldt);
  const hams::ModeTab mt{m, m, nmode, pw.pm, pw.ac, pw.src, pw.srct, pw.fld, pw.fldt};
  launch_rad_series(br, ntmax, st, g, w, wvn, pw.r, nullptr, m, pw.kt, pw.jy);
  launch_series(br, ntmax, st, g, w, wvn, mt, RadTab{nullptr, 0, pw.kt, pw.jy}, PointIO{list, flag, out, (size_t)npts},
                m, ovf);
}

// Source (S) and normal-dipole (D) influence of every hull panel J at field
// point f without pair lists (sets of more than 2^32 - 1 pairs, or no memory
// for the lists), the terms CalPotentialMulti sums (PressureElevationMulti.f90:81-137):
// S = FLAG*SIJ + G ds, D = (FLAG*DIJ + grad G ds) . n_J, with the Rankine
// integrals at the field point (SGLINTBD_MULTI_QUAD2/TRI2,
// SingularIntgrMulti.f90:454-776) and FLAG = (distance <= 50 PNSZ_J).
__global__ void k_field_pairs(DevGeom g, WaveDev w, const double* __restrict__ wvn, int nfp,
                              const double* __restrict__ xfp, double2* __restrict__ Sf, double2* __restrict__ Df,
                              int* ovf) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y;
  if (f >= nfp) return;
  const double xp = xfp[f], yp = xfp[f + nfp], zp = xfp[f + 2 * (size_t)nfp];
  const double xq = g.xq[j], yq = g.xq[j + g.n], zq = g.xq[j + 2 * g.n];
  const double dist = sqrt((xp - xq) * (xp - xq) + (yp - yq) * (yp - yq) + (zp - zq) * (zp - zq));
  const int flag = dist <= 50.0 * g.pnsz[j] ? 1 : 0;
  const double xf[3] = {xp, yp, zp};
  hams::rk4 r;
  if (g.ncn[j] == 3) {
    double q[3][3];
    for (int v = 0; v < 3; ++v)
      for (int c = 0; c < 3; ++c) q[v][c] = g.vtx[(size_t)j * 12 + v * 3 + c];
    r = hams::sglint_tri(xf, q);
  } else {
    double q[4][3];
    for (int v = 0; v < 4; ++v)
      for (int c = 0; c < 3; ++c) q[v][c] = g.vtx[(size_t)j * 12 + v * 3 + c];
    r = hams::sglint_quad(xf, q);
  }
  grn4 G;
  if (w.limit) {
    G = hams::green_limit(w.limit == 2, xq, xp, yq, yp, zq, zp, flag);
  } else if (w.h < 0.0) {
    G = hams::infgreen3d(xq, xp, yq, yp, zq, zp, w.v, flag);
  } else {
    int o = 0;
    const double rr = sqrt((xq - xp) * (xq - xp) + (yq - yp) * (yq - yp));
    switch (hams::fin_branch(rr, w.h)) {
      case hams::kLinton: G = hams::fingreen3d<hams::kLinton>(xq, xp, yq, yp, zq, zp, w.v, wvn, w.h, flag, (void*)nullptr, &o); break;
      case hams::kPidcock: {
        hams::SeriesScratchN<hams::kPidcockMax> sc;
        G = hams::fingreen3d<hams::kPidcock>(xq, xp, yq, yp, zq, zp, w.v, wvn, w.h, flag, &sc, &o);
        break;
      }
      case hams::kEigenE: {
        hams::SeriesScratchN<hams::kEigenEMax> sc;
        G = hams::fingreen3d<hams::kEigenE>(xq, xp, yq, yp, zq, zp, w.v, wvn, w.h, flag, &sc, &o);
        break;
      }
      default: G = hams::fingreen3d<hams::kEigen>(xq, xp, yq, yp, zq, zp, w.v, wvn, w.h, flag, (void*)nullptr, &o); break;
    }
    if (o) atomicOr(ovf, 1);
  }
  const double ds = g.ds[j], n1 = g.nrm[j], n2 = g.nrm[j + g.n], n3 = g.nrm[j + 2 * g.n];
  double sre = G.g[0].re * ds, sim = G.g[0].im * ds;
  double dre = (G.g[1].re * n1 + G.g[2].re * n2 + G.g[3].re * n3) * ds;
  double dim = (G.g[1].im * n1 + G.g[2].im * n2 + G.g[3].im * n3) * ds;
  if (flag) {
    sre = r.s + G.g[0].re * ds;
    dre = (r.dx + G.g[1].re * ds) * n1 + (r.dy + G.g[2].re * ds) * n2 + (r.dz + G.g[3].re * ds) * n3;
  }
  Sf[f + (size_t)nfp * j] = make_double2(sre, sim);
  Df[f + (size_t)nfp * j] = make_double2(dre, dim);
}

void launch_field_pairs(cudaStream_t st, DevGeom g, WaveDev w, const double* wvn, int nfp, const double* xfp,
                        double2* Sf, double2* Df, int* ovf) {
  k_field_pairs<<<dim3((nfp + 127) / 128, g.n), 128, 0, st>>>(g, w, wvn, nfp, xfp, Sf, Df, ovf);
}

void launch_eval_green(unsigned blocks, cudaStream_t st, int npts, const double* pts, const int* flag, WaveDev w,
                       const double* wvn, double2* out, int* ovf) {
  k_eval_green<<<blocks, 128, 0, st>>>(npts, pts, flag, w, wvn, out, ovf, nullptr, npts);
}
