// hyc_fct2c.cu -- advem_fct2c (mod_tsadvc.F90:999-1368): FCT2 with the
// barotropic mass flux (btrmas), whose low-order part is a donor-cell scheme
// sub-cycled five times with a local time step per cell.
//
// FP64, one kernel per stage over whole slices, as the reference sweeps its
// arrays (the sub-cycling refreshes the halo of hloc and fldlo between
// iterations, mod_tsadvc.F90:1181-1182, which a fused tile would have to
// replace by an 8-cell halo).
// A launch covers up to 16 (field, layer) pairs; every pair has its own 11
// work slices (the reference's module arrays uloc, vloc, hloc, dtloc,
// ucumdt, vcumdt, flxcum, flycum, lcalc, fldlo, flx, fly, fax, fay, rp, rm,
// with fax/fay/rp/rm reusing the dead uloc/vloc/flx/fly).
//
// What bounds it: FP64 and integer issue, not memory, so products, divisions
// and comparisons run on the integer pipes (hyc_div.cuh, hyc_device.cuh),
// FP32 bounds settle limiter ratios of 1, and what has nothing left to do is
// not done: a cell whose four faces have used up the step (lcalc = 0, away
// from the coast all of them after the first iteration) needs no time step,
// and a face between two such cells no flux.  16 pairs of 900x700: 3.9 -> 1.9
// ms, of it start 0.20, the first iteration 0.41, the four others 0.16 each,
// fluxes, ratios and update 0.67; the FP64 pipe is 70-82 % busy in the first
// stages, 0-52 % in the others, whose issue slots are half to two thirds full.
//
// The stages keep
// the reference's margins and operation order and are built without FMA
// contraction, so results equal the oracle's bit for bit.
#include <cuda_runtime.h>

#include <cstdint>

#include "hyc_args.h"
#include "hyc_device.cuh"
#include "hyc_internal.h"
#include "hyc_pdl.cuh"

namespace hyc {

namespace {

constexpr double kEps = 1.e-10;  // epsil, mod_tsadvc.F90:1027
constexpr int kMb = 5;           // mbdy_advtyp(2)

enum { A_HLOC, A_FLDLO, A_DTLOC, A_UCUM, A_VCUM, A_ULOC, A_VLOC, A_FLX, A_FLY, A_FXC, A_FYC, A_N };
// after the sub-iterations: fax, fay, rp, rm live in uloc, vloc, flx, fly
enum { A_FAX = A_ULOC, A_FAY = A_VLOC, A_RP = A_FLX, A_RM = A_FLY };

__device__ __forceinline__ double *W(const Fct2cArgs &A, int arr, int p) {
  return A.work + ((long long)arr * A.npair + p) * A.slice;
}
__device__ __forceinline__ bool same_bits(double a, double b) { return __double_as_longlong(a) == __double_as_longlong(b); }

constexpr int kBX = 32, kBY = 8;  // the block of every stage

// cell (i,j) of the margin region [1-m, ii+m] x [1-m, jj+m] of this thread;
// false beyond the region
__device__ __forceinline__ bool cell_of(const Fct2cArgs &A, int m, long long &c, int &i, int &j) {
  const unsigned nbx = (unsigned)(A.ii + 2 * m + kBX - 1) / kBX, by = blockIdx.x / nbx;
  i = (int)((blockIdx.x - by * nbx) * kBX + threadIdx.x);
  j = (int)(by * kBY + threadIdx.y);
  c = (long long)(i + A.nb - m) + (long long)(j + A.nb - m) * A.ld1;
  return i < A.ii + 2 * m && j < A.jj + 2 * m;
}

__device__ __forceinline__ bool cell_of(const Fct2cArgs &A, int m, long long &c) {
  int i, j;
  return cell_of(A, m, c, i, j);
}

// Four cells of a column 8 rows apart for each thread (blocks of 32x32 cells):
// f(c) for those that want(c) says need work.  After the first iteration most
// cells need none, and what a stage costs is finding that out.
constexpr int kRows = 4;
template <class W, class F>
__device__ __forceinline__ void active_cells(const Fct2cArgs &A, int m, W &&want, F &&f) {
  const unsigned nbx = (unsigned)(A.ii + 2 * m + kBX - 1) / kBX, by = blockIdx.x / nbx;
  const int i = (int)((blockIdx.x - by * nbx) * kBX + threadIdx.x), j = (int)(by * (kBY * kRows) + threadIdx.y);
  if (i >= A.ii + 2 * m) return;
  const long long c = (long long)(i + A.nb - m) + (long long)(j + A.nb - m) * A.ld1;
  unsigned todo = 0;
#pragma unroll
  for (int r = 0; r < kRows; r++)
    if (j + kBY * r < A.jj + 2 * m && want(c + (long long)(kBY * r) * A.ld1)) todo |= 1u << r;
#pragma unroll 1
  for (int r = 0; r < kRows; r++)
    if (todo >> r & 1u) f(c + (long long)(kBY * r) * A.ld1);
}

__device__ __forceinline__ const double *U_(const Fct2cArgs &A, int p) {
  return A.mode == 0 ? A.uflx + (long long)A.k[p] * A.slice : A.uflx;
}
__device__ __forceinline__ const double *V_(const Fct2cArgs &A, int p) {
  return A.mode == 0 ? A.vflx + (long long)A.k[p] * A.slice : A.vflx;
}

// local time step of a sea cell of thickness h (:1086-1099)
__device__ __forceinline__ double local_dt(const Fct2cArgs &A, const double *u, const double *v, long long c, double h) {
  const double q = pos0(u[c + 1]) - neg0(u[c]) + pos0(v[c + A.ld1]) - neg0(v[c]);
  return gt0(q) ? kmin(A.dt2, div_rn(h, mul_rn(q, A.scali[c]))) : A.dt2;
}

// The whole arrays of hloc (mod_tsadvc.F90:1905-1942, with onetamas(m),
// :1804-1810) and fldlo, and the first local time step.  The other work
// arrays (:1068-1081) need no initial values: the first iteration writes them.
__global__ void __launch_bounds__(kBX * kBY) fct2c_start(Fct2cArgs A) {
  after_previous();
  const int p = blockIdx.y, nb = A.nb;
  long long t;
  int a, b;
  if (!cell_of(A, nb, t, a, b)) return;
  const long long sl = A.slice;
  const int ld1 = A.ld1;
  const double *u = U_(A, p), *v = V_(A, p);
  double fco;
  if (A.mode == 0) {
    const double d = A.dpn[(long long)A.k[p] * sl + t];
    const double o = A.oneta ? mul_rn(A.oneta[t], d) : d;
    double fdv = 0.0;
    if (a < ld1 - 1 && b < A.ld2 - 1)
      fdv = mul_rn(mul_rn((u[t + 1] - u[t]) + (v[t + ld1] - v[t]), A.dt2), A.scali[t]);
    fco = kmax(o + fdv, 0.0);
  } else {
    fco = A.fco[t];
  }
  W(A, A_HLOC, p)[t] = fco;
  W(A, A_FLDLO, p)[t] = A.fld[p][t];
  A.lcalc[p * sl + t] = 1;
  const bool in = a >= nb - kMb && a < nb + A.ii + kMb && b >= nb - kMb && b < nb + A.jj + kMb;
  if (in && (A.msk[t] & kIP)) W(A, A_DTLOC, p)[t] = local_dt(A, u, v, t, fco);
}

// Local time step per cell, later iterations.  A cell whose four faces have
// used up dt2 (lcalc = 0, most cells after the first iteration) gives its
// faces nothing more.
__global__ void __launch_bounds__(kBX * kBY) fct2c_dt(Fct2cArgs A) {
  after_previous();
  const int p = blockIdx.y;
  const uint8_t *lc = A.lcalc + (long long)p * A.slice;
  const double *u = U_(A, p), *v = V_(A, p), *h = W(A, A_HLOC, p);
  double *dt = W(A, A_DTLOC, p);
  active_cells(A, kMb, [&](long long c) { return (A.msk[c] & kIP) && lc[c]; },
               [&](long long c) { dt[c] = local_dt(A, u, v, c, h[c]); });
}

// One face (:1101-1149): its flux u from the cell at a (u >= 0) or at c for
// the rest of the step or the cell's local one.
template <bool FIRST>
__device__ __forceinline__ void face(const Fct2cArgs &A, bool open, long long c, long long a, const double *u,
                                     const double *dt, const double *lo, double *ucum, double *uloc, double *flx,
                                     double *fxc) {
  if (!open) {  // not between two sea cells: zero from the start
    if (FIRST) ucum[c] = uloc[c] = flx[c] = 0.0;
    return;
  }
  const double done = FIRST ? 0.0 : ucum[c];
  if (FIRST || !same_bits(done, A.dt2)) {
    const double uu = u[c];
    const long long up = ge0(uu) ? a : c;
    const double m = kmin(FIRST ? A.dt2 : A.dt2 - done, dt[up]), ul = mul_rn(m, uu), f = mul_rn(lo[up], ul);
    uloc[c] = ul;
    flx[c] = f;
    ucum[c] = FIRST ? m : done + m;
    fxc[c] = FIRST ? f : fxc[c] + f;
  } else {
    uloc[c] = 0.0;
    flx[c] = 0.0;
  }
}

// Partial-step donor fluxes and their sums.  A face between two cells with
// lcalc = 0 is not read any more.
__global__ void __launch_bounds__(kBX * kBY) fct2c_flux_first(Fct2cArgs A) {
  after_previous();
  const int p = blockIdx.y;
  long long c;
  if (!cell_of(A, kMb - 1, c)) return;
  const uint8_t m = A.msk[c];
  const double *dt = W(A, A_DTLOC, p), *lo = W(A, A_FLDLO, p);
  face<true>(A, m & kIU, c, c - 1, U_(A, p), dt, lo, W(A, A_UCUM, p), W(A, A_ULOC, p), W(A, A_FLX, p), W(A, A_FXC, p));
  face<true>(A, m & kIV, c, c - A.ld1, V_(A, p), dt, lo, W(A, A_VCUM, p), W(A, A_VLOC, p), W(A, A_FLY, p), W(A, A_FYC, p));
}
__global__ void __launch_bounds__(kBX * kBY) fct2c_flux(Fct2cArgs A) {
  after_previous();
  const int p = blockIdx.y, ld = A.ld1;
  const uint8_t *lc = A.lcalc + (long long)p * A.slice;
  const double *u = U_(A, p), *v = V_(A, p), *dt = W(A, A_DTLOC, p), *lo = W(A, A_FLDLO, p);
  active_cells(A, kMb - 1, [&](long long c) { return (A.msk[c] & (kIU | kIV)) && (lc[c] | lc[c - 1] | lc[c - ld]); },
               [&](long long c) {
                 const uint8_t m = A.msk[c];
                 face<false>(A, m & kIU, c, c - 1, u, dt, lo, W(A, A_UCUM, p), W(A, A_ULOC, p), W(A, A_FLX, p),
                             W(A, A_FXC, p));
                 face<false>(A, m & kIV, c, c - ld, v, dt, lo, W(A, A_VCUM, p), W(A, A_VLOC, p), W(A, A_FLY, p),
                             W(A, A_FYC, p));
               });
}

// low-order update of fldlo and hloc (:1153-1176)
__device__ __forceinline__ void low_order(const Fct2cArgs &A, int p, long long c, uint8_t *lc) {
  const int ld = A.ld1;
  const double dt2 = A.dt2;
  double *h = W(A, A_HLOC, p), *lo = W(A, A_FLDLO, p);
  const double *uloc = W(A, A_ULOC, p), *vloc = W(A, A_VLOC, p), *flx = W(A, A_FLX, p), *fly = W(A, A_FLY, p);
  const double *ucum = W(A, A_UCUM, p), *vcum = W(A, A_VCUM, p);
  const double u0 = uloc[c], u1 = uloc[c + 1], v0 = vloc[c], v1 = vloc[c + ld], x0 = flx[c], x1 = flx[c + 1], y0 = fly[c],
               y1 = fly[c + ld], hc = h[c], lc0 = lo[c], si = A.scali[c];
  const bool more = !same_bits(ucum[c + 1], dt2) || !same_bits(ucum[c], dt2) || !same_bits(vcum[c + ld], dt2) ||
                    !same_bits(vcum[c], dt2);
  const double qp = hc - mul_rn(u1 - u0 + v1 - v0, si);
  if (gt0(qp)) lo[c] = div_rn(mul_rn(kEps + hc, lc0) - mul_rn(x1 - x0 + y1 - y0, si), kEps + qp);
  h[c] = qp;
  lc[c] = more;
}
__global__ void __launch_bounds__(kBX * kBY) fct2c_cell_first(Fct2cArgs A) {
  after_previous();
  const int p = blockIdx.y;
  long long c;
  if (cell_of(A, kMb - 2, c) && (A.msk[c] & kIP)) low_order(A, p, c, A.lcalc + (long long)p * A.slice);
}
__global__ void __launch_bounds__(kBX * kBY) fct2c_cell(Fct2cArgs A) {
  after_previous();
  const int p = blockIdx.y;
  uint8_t *lc = A.lcalc + (long long)p * A.slice;
  active_cells(A, kMb - 2, [&](long long c) { return (A.msk[c] & kIP) && lc[c]; },
               [&](long long c) { low_order(A, p, c, lc); });
}

// antidiffusive fluxes (:1199-1215); faces that are not between two sea
// cells carry none (the section-edge zeroing :1223-1243 covers every such
// face a sea cell reads)
__global__ void __launch_bounds__(kBX * kBY) fct2c_anti(Fct2cArgs A) {
  after_previous();
  const int p = blockIdx.y;
  long long c;
  if (!cell_of(A, kMb - 2, c)) return;
  const uint8_t m = A.msk[c];
  const double *fc = A.fldc[p];
  const int ld = A.ld1;
  const uint32_t R = recip_of(A.dt2);
  double fax = 0.0, fay = 0.0;
  if (m & kIU) fax = mul_rn(half_of(U_(A, p)[c]), fc[c] + fc[c - 1]) - div_by(W(A, A_FXC, p)[c], A.dt2, R);
  if (m & kIV) fay = mul_rn(half_of(V_(A, p)[c]), fc[c] + fc[c - ld]) - div_by(W(A, A_FYC, p)[c], A.dt2, R);
  W(A, A_FAX, p)[c] = fax;
  W(A, A_FAY, p)[c] = fay;
}

// Zalesak ratios (:1257-1303), true i+1/j+1 neighbours.  FP32 bounds (below
// qp, above famax, and famax surely above kEps) show most to be 1.
__global__ void __launch_bounds__(kBX * kBY) fct2c_ratio(Fct2cArgs A) {
  after_previous();
  const int p = blockIdx.y;
  long long c;
  if (!cell_of(A, kMb - 3, c) || !(A.msk[c] & kIP)) return;
  const int ld = A.ld1;
  const double *lo = W(A, A_FLDLO, p), *fax = W(A, A_FAX, p), *fay = W(A, A_FAY, p);
  const long long ca = (A.msk[c - 1] & kIP) ? c - 1 : c, cb = (A.msk[c + 1] & kIP) ? c + 1 : c;
  const long long cja = (A.msk[c - ld] & kIP) ? c - ld : c, cjb = (A.msk[c + ld] & kIP) ? c + ld : c;
  const double l0 = lo[c], h = W(A, A_HLOC, p)[c], scal = A.scal[c];
  const double fx0 = fax[c], fx1 = fax[c + 1], fy0 = fay[c], fy1 = fay[c + ld];
  const long long k0 = dkey(l0), ka = dkey(lo[ca]), kb = dkey(lo[cb]), kja = dkey(lo[cja]), kjb = dkey(lo[cjb]);
  const double dmx = from_dkey(max(max(max(max(k0, ka), kb), kja), kjb)) - l0;
  const double dmn = l0 - from_dkey(min(min(min(min(k0, ka), kb), kja), kjb));
  const float a0 = f32_away(fx0), a1 = f32_away(fx1), b0 = f32_away(fy0), b1 = f32_away(fy1);
  const float hs = f32_below(h) * f32_below(scal), qf0 = hs * f32_below(A.qdt2);
  const float qf = hs > 1e-30f && hs < 1e30f && qf0 > 1e-30f && qf0 < 1e30f ? qf0 : 0.0f;
  const float amax = (fmaxf(a0, 0.0f) - fminf(a1, 0.0f)) + (fmaxf(b0, 0.0f) - fminf(b1, 0.0f));
  const float amin = (fmaxf(a1, 0.0f) - fminf(a0, 0.0f)) + (fmaxf(b1, 0.0f) - fminf(b0, 0.0f));
  const float eps = 1.0001e-10f;
  double rp = 1.0, rm = 1.0;
  if (!(amax > eps && f32_below(dmx) * qf > amax * 1.000004f)) {
    const double famax = pos0(fx0) - neg0(fx1) + pos0(fy0) - neg0(fy1);
    const double qp = mul_rn(mul_rn(mul_rn(dmx, h), scal), A.qdt2);
    rp = !klt(kEps, famax) ? 0.0 : klt(qp, famax) ? div_rn(qp, famax) : 1.0;
  }
  if (!(amin > eps && f32_below(dmn) * qf > amin * 1.000004f)) {
    const double famin = pos0(fx1) - neg0(fx0) + pos0(fy1) - neg0(fy0);
    const double qm = mul_rn(mul_rn(mul_rn(dmn, h), scal), A.qdt2);
    rm = !klt(kEps, famin) ? 0.0 : klt(qm, famin) ? div_rn(qm, famin) : 1.0;
  }
  W(A, A_RP, p)[c] = rp;
  W(A, A_RM, p)[c] = rm;
}

// Limited antidiffusive fluxes of a cell's four faces (:1308-1332) and the
// corrected update of the interior sea cells (:1340-1359).  A face is limited
// by both its cells: that is a product where the factor is not 1, against a
// pass that writes and reads both flux arrays.
__global__ void __launch_bounds__(kBX * kBY) fct2c_update(Fct2cArgs A) {
  after_previous();
  const int p = blockIdx.y;
  long long c;
  if (!cell_of(A, 0, c)) return;
  const uint8_t m = A.msk[c];
  if (!(m & kIP)) return;
  const int ld = A.ld1;
  const double *fax = W(A, A_FAX, p), *fay = W(A, A_FAY, p), *rp = W(A, A_RP, p), *rm = W(A, A_RM, p);
  const double l0 = W(A, A_FLDLO, p)[c], h = W(A, A_HLOC, p)[c], rp0 = rp[c], rm0 = rm[c];
  // f between the cells a (west, south) and b; 0 at a closed face
  auto limit = [](bool open, double f, double rpa, double rma, double rpb, double rmb) {
    if (!open) return f;
    const double fact = lt0(f) ? kmin(rpa, rmb) : kmin(rpb, rma);
    return __double_as_longlong(fact) == kOneBits ? f : mul_rn(fact, f);
  };
  const double x0 = limit(m & kIU, fax[c], rp[c - 1], rm[c - 1], rp0, rm0);
  const double x1 = limit(A.msk[c + 1] & kIU, fax[c + 1], rp0, rm0, rp[c + 1], rm[c + 1]);
  const double y0 = limit(m & kIV, fay[c], rp[c - ld], rm[c - ld], rp0, rm0);
  const double y1 = limit(A.msk[c + ld] & kIV, fay[c + ld], rp0, rm0, rp[c + ld], rm[c + ld]);
  double *f = A.fld[p];
  if (gt0(h)) {
    const double flxdiv = mul_rn(mul_rn((x1 - x0) + (y1 - y0), A.dt2), A.scali[c]);
    const double eh = kEps + h;
    f[c] = div_rn(mul_rn(eh, l0) - flxdiv, eh);
  } else {
    f[c] = l0;
  }
}

template <class K>
cudaError_t go(K kern, const Fct2cArgs &A, int margin, cudaStream_t s, int rows = 1) {
  const unsigned nbx = (unsigned)(A.ii + 2 * margin + kBX - 1) / kBX,
                 nby = (unsigned)(A.jj + 2 * margin + kBY * rows - 1) / (kBY * rows);
  const dim3 grid(nbx * nby, A.npair);
  return launch_after(kern, grid, dim3(kBX, kBY), s, A);
}

}  // namespace

size_t fct2c_work_doubles(long long slice) { return (size_t)slice * A_N; }
size_t fct2c_work_bytes(long long slice) { return (size_t)slice * (A_N * sizeof(double) + 1); }

cudaError_t launch_fct2c(const Fct2cArgs &A, int nreg, int *launches, cudaStream_t s) {
  cudaError_t e;
  int nl = 0;
  if ((e = go(fct2c_start, A, A.nb, s)) != cudaSuccess) return e;
  for (int it = 0; it < 5; it++) {  // :1083-1192
    if (it == 0) {
      if ((e = go(fct2c_flux_first, A, kMb - 1, s)) != cudaSuccess) return e;
      if ((e = go(fct2c_cell_first, A, kMb - 2, s)) != cudaSuccess) return e;
    } else {
      if ((e = go(fct2c_dt, A, kMb, s, kRows)) != cudaSuccess) return e;
      if ((e = go(fct2c_flux, A, kMb - 1, s, kRows)) != cudaSuccess) return e;
      if ((e = go(fct2c_cell, A, kMb - 2, s, kRows)) != cudaSuccess) return e;
    }
    // xctilr(hloc), xctilr(fldlo), :1181-1182
    if ((e = launch_xctilr(A.work + (long long)A_HLOC * A.npair * A.slice, A.slice, A.npair, A.ii, A.jj, A.nb, A.ld1,
                           kMb, kMb, nreg, s)) != cudaSuccess)
      return e;
    if ((e = launch_xctilr(A.work + (long long)A_FLDLO * A.npair * A.slice, A.slice, A.npair, A.ii, A.jj, A.nb,
                           A.ld1, kMb, kMb, nreg, s)) != cudaSuccess)
      return e;
    nl += 5;  // the start kernel counts with the first iteration, which has no time step of its own
  }
  if ((e = go(fct2c_anti, A, kMb - 2, s)) != cudaSuccess) return e;
  if ((e = go(fct2c_ratio, A, kMb - 3, s)) != cudaSuccess) return e;
  if ((e = go(fct2c_update, A, 0, s)) != cudaSuccess) return e;
  nl += 3;
  if (launches) *launches += nl;
  return cudaSuccess;
}

}  // namespace hyc
