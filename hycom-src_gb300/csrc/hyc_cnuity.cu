// hyc_cnuity.cu -- the continuity equation (cnuity.F90:14-1419): flux-
// corrected transport of the layer thicknesses, the barotropic restoration
// and bottom-pressure restoring (not btrmas), biharmonic or Laplacian
// interface-depth diffusion, the cumulative fluxes, the btrmas restoring and
// the Robert-Asselin filter of dp.
//
// The reference is a sequence of sweeps over the slice whose margins shrink
// from 6 to 0 within a layer, with a vertical recurrence (util3 = depth of
// the layer's top, p = interface pressures) from one layer to the next.  Here
// one kernel does a sweep over the same margin for a batch of layers: util3 is
// a running sum of the thicknesses as they came, p one of the results, and
// neither is read by another layer's sweeps in between, so both are formed by
// kernels of their own.  Every value the reference computes (halo cells
// included) is computed, in the same operation order, FP64 without FMA
// contraction: the results equal the oracle's bit for bit.
//
// What bounds them: at the start the FP64 pipe (71-82 % busy in every sweep);
// with products and divisions on the integer pipes (hyc_div.cuh) the pipe, the
// integer pipes and the memory system are each half to two thirds busy, so the
// operands of a sweep are loaded before the first is used.  1500x1100, one
// layer, before / after: cn_flux 45 / 41 us, cn_low 27 / 24, cn_ratio 55 / 32,
// cn_clip 40 / 26, cn_update 27 / 25, cn_btflux 37 / 28, cn_thk_util 34 / 27,
// cn_thk_flux 112 / 82, cn_thk_p 21 / 19.  The sweeps move about 55 slices per
// cell and layer against 11 for a fused form.
//
// Work slices (CnuityArgs::w): utotn, vtotn, util3 below the batch, pold, the
// reciprocal of p(kk+1), oneta_u, oneta_v, onetamas(:,:,1:2); then for each layer
// of a batch uflux, vflux, uflux2, vflux2, util1, util2, util3.
#include <cuda_runtime.h>

#include <climits>
#include <cstdint>

#include "hyc_args.h"
#include "hyc_device.cuh"
#include "hyc_internal.h"
#include "hyc_pdl.cuh"

namespace hyc {

namespace {

// one slice each, then A.nbatch slices each (layer k0 + l of a batch in slice l)
enum { W_UTN, W_VTN, W_U3T, W_POLD, W_RPB, W_OU, W_OV, W_OM, W_FIX = W_OM + 2 };
enum { B_UF, B_VF, B_UF2, B_VF2, B_U1, B_U2, B_U3, B_N };

constexpr double kOnem = 9.806 / (1.0 / 1000.0);  // onem = g/svref, mod_cb_arrays.F90:843-846
constexpr double kOnecm = kOnem * 0.01;
constexpr double kEpsilCb = 1.0e-11;   // epsil, mod_cb_arrays.F90:853
constexpr double kEpsilCn = 1.e-14;    // epsil_cnuity, cnuity.F90:52

struct Cell {
  int i, j;
  long long c;
};

// thread -> cell of the box i in [1-M, ii+M], j in [1-M, jj+M]; false when outside
__device__ __forceinline__ bool cell_of(const CnuityArgs &A, int M, Cell &x) {
  const int bi = blockIdx.x * blockDim.x + threadIdx.x, bj = blockIdx.y * blockDim.y + threadIdx.y;
  if (bi >= A.ii + 2 * M || bj >= A.jj + 2 * M) return false;
  x.i = 1 - M + bi;
  x.j = 1 - M + bj;
  x.c = (long long)(x.i + A.nb - 1) + (long long)(x.j + A.nb - 1) * A.ld1;
  return true;
}

__device__ __forceinline__ double *W(const CnuityArgs &A, int s) { return A.w + (long long)s * A.slice; }
__device__ __forceinline__ double *WB(const CnuityArgs &A, int s, int l) {
  return A.w + ((long long)W_FIX + (long long)s * A.nbatch + l) * A.slice;
}

// the reference's max/min of two reals (ordered as written; signs of zero
// never reach a result of this path)
__device__ __forceinline__ double mx(double a, double b) { return kmax(a, b); }
__device__ __forceinline__ double mn(double a, double b) { return kmin(a, b); }

__device__ __forceinline__ bool is0(double x) { return (unsigned long long)__double_as_longlong(x) << 1 == 0; }
// q*x, q finite: x = 0 (thin layers) does not go to the FP64 pipe
__device__ __forceinline__ double scaled(double q, double x) { return is0(x) ? 0.0 : mul_rn(q, x); }
// -x without the FP64 pipe
__device__ __forceinline__ double minus(double x) {
  return __longlong_as_double(__double_as_longlong(x) ^ (long long)0x8000000000000000ULL);
}
__device__ __forceinline__ bool finite(double x) { return (__double2hiint(x) & 0x7FF00000) != 0x7FF00000; }

// :112-157 at margin 6
__global__ void cn_init(const CnuityArgs A) {
  after_previous();
  Cell x;
  if (!cell_of(A, 6, x)) return;
  const long long c = x.c, sl = A.slice;
  const int mm = A.m - 1, nn = A.n - 1;
  const uint8_t mk = A.msk[c];
  double *om = W(A, W_OM);
  // the outermost halo column/row has no west/south neighbour; its u/v
  // factors are never read
  const bool w = x.i > 1 - A.nb, s = x.j > 1 - A.nb;
  if (A.btrmas) {
    om[c] = A.oneta[c];
    om[c + sl] = A.oneta[c + sl];
    if ((mk & kIU) && w) {
      const double a = A.oneta[c + mm * sl], b = A.oneta[c - 1 + mm * sl];
      W(A, W_OU)[c] = A.pbot[c] == A.pbot[c - 1] ? 0.5 * (a + b) : (A.pbot[c] == A.depthu[c] ? a : b);
    }
    if ((mk & kIV) && s) {
      const double a = A.oneta[c + mm * sl], b = A.oneta[c - A.ld1 + mm * sl];
      W(A, W_OV)[c] = A.pbot[c] == A.pbot[c - A.ld1] ? 0.5 * (a + b) : (A.pbot[c] == A.depthv[c] ? a : b);
    }
  } else {
    om[c] = 1.0;
    om[c + sl] = 1.0;
    W(A, W_OU)[c] = 1.0;
    W(A, W_OV)[c] = 1.0;
  }
  W(A, W_UTN)[c] = 0.0;
  W(A, W_VTN)[c] = 0.0;
  W(A, W_U3T)[c] = 0.0;
  for (int k = 0; k < A.kdm; k++) {
    const long long o = ((long long)k + (long long)nn * A.kdm) * sl + c;
    A.dpo[o] = A.dp[o];
  }
}

// util3, the depth of each layer's top, of the batch's layers: the running sum
// of dp(:,:,k,n) before the layers' own updates (:300-306), at the sea cells of
// margin 4, where the reference forms it layer after layer; 0 elsewhere
__global__ void cn_top(const CnuityArgs A, int nl) {
  after_previous();
  Cell x;
  if (!cell_of(A, 4, x)) return;
  const long long c = x.c, sl = A.slice;
  if (!(A.msk[c] & kIP)) return;
  const double *dk = A.dp + ((long long)A.k0 + (long long)(A.n - 1) * A.kdm) * sl + c;
  double t = W(A, W_U3T)[c];
  int l = 0;
  for (; l + 4 <= nl; l += 4) {
    double d[4];
#pragma unroll
    for (int r = 0; r < 4; r++) d[r] = dk[(long long)(l + r) * sl];
#pragma unroll
    for (int r = 0; r < 4; r++) {
      WB(A, B_U3, l + r)[c] = t;
      t = t + d[r];
    }
  }
  for (; l < nl; l++) {
    WB(A, B_U3, l)[c] = t;
    t = t + dk[(long long)l * sl];
  }
  W(A, W_U3T)[c] = t;
}

// loop 76, :240-285 at margin 5: low-order and antidiffusive fluxes of layer k.
// BT = btrmas.  Without it onetamas and the face factors oneta_u/v are 1.0
// (:142-145), and x*1.0 == x exactly, so those products (and their loads)
// are skipped; the FP64 pipe bounds this kernel.
template <bool BT>
__global__ void cn_flux(const CnuityArgs A) {
  after_previous();
  const int l = blockIdx.z, k = A.k0 + l;
  Cell x;
  if (!cell_of(A, 5, x)) return;
  const long long c = x.c, sl = A.slice, ld = A.ld1;
  const int mm = A.m - 1, nn = A.n - 1;
  const uint8_t mk = A.msk[c];
  const double *dk = A.dp + ((long long)k + (long long)nn * A.kdm) * sl;
  const double *u3 = WB(A, B_U3, l), *omn = W(A, W_OM) + nn * sl;
  const long long lm = ((long long)k + (long long)mm * A.kdm) * sl;
  if (!(mk & (kIU | kIV))) return;
  // every operand is loaded before the first is used: the upwind cell is
  // known only after the velocity is
  const double d0 = dk[c], dw = dk[c - 1], ds = dk[c - ld], t0 = u3[c], tw = u3[c - 1], ts = u3[c - ld];
  const double uu = A.u[lm + c], ub = A.ubavg[mm * sl + c], su = A.scuy[c], du = A.depthu[c], hu = A.dpu[lm + c];
  const double vv = A.v[lm + c], vb = A.vbavg[mm * sl + c], sv = A.scvx[c], dv = A.depthv[c], hv = A.dpv[lm + c];
  if (mk & kIU) {
    const double utotm = mul_rn(uu + ub, su);
    const bool up = ge0(utotm);
    const double q0 = mn(up ? dw : d0, mx(0., du - (up ? tw : t0)));
    const double uf = mul_rn(utotm, BT ? mul_rn(q0, omn[up ? c - 1 : c]) : q0);
    WB(A, B_UF, l)[c] = uf;
    const double ud = mul_rn(utotm, hu);
    WB(A, B_UF2, l)[c] = (BT ? mul_rn(ud, W(A, W_OU)[c]) : ud) - uf;
    A.uflx[(long long)k * sl + c] = uf;
  }
  if (mk & kIV) {
    const double vtotm = mul_rn(vv + vb, sv);
    const bool up = ge0(vtotm);
    const double q0 = mn(up ? ds : d0, mx(0., dv - (up ? ts : t0)));
    const double vf = mul_rn(vtotm, BT ? mul_rn(q0, omn[up ? c - ld : c]) : q0);
    WB(A, B_VF, l)[c] = vf;
    const double vd = mul_rn(vtotm, hv);
    WB(A, B_VF2, l)[c] = (BT ? mul_rn(vd, W(A, W_OV)[c]) : vd) - vf;
    A.vflx[(long long)k * sl + c] = vf;
  }
}

// per-warp minimum of a key, one atomic per warp (dpkmin rows j = 1..jj)
__device__ __forceinline__ void row_min(const CnuityArgs &A, const Cell &x, bool in, double v, int slot) {
  long long k = (in && x.j >= 1 && x.j <= A.jj) ? dkey(v) : LLONG_MAX;
  for (int o = 16; o > 0; o >>= 1) {
    const long long t = __shfl_xor_sync(0xffffffffu, k, o);
    k = t < k ? t : k;
  }
  if ((threadIdx.x & 31) == 0 && k != LLONG_MAX) atomicMin(&A.keys[slot], k);
}

// loop 19, :294-315 at margin 4: low-order update of dp(k,n) (BT as cn_flux)
template <bool BT>
__global__ void cn_low(const CnuityArgs A) {
  after_previous();
  const int l = blockIdx.z, k = A.k0 + l;
  Cell x;
  const bool in = cell_of(A, 4, x);
  bool sea = false;
  double d = 0.0;
  if (in && (A.msk[x.c] & kIP)) {
    const long long c = x.c, sl = A.slice, ld = A.ld1;
    const int mm = A.m - 1, nn = A.n - 1;
    double *dk = A.dp + ((long long)k + (long long)nn * A.kdm) * sl;
    const double *uf = WB(A, B_UF, l), *vf = WB(A, B_VF, l);
    d = (BT ? mul_rn(dk[c], W(A, W_OM)[nn * sl + c]) : dk[c]) -
        mul_rn(mul_rn((uf[c + 1] - uf[c]) + (vf[c + ld] - vf[c]), A.delt1), A.scp2i[c]);
    dk[c] = d;
    A.dpo[((long long)k + (long long)mm * A.kdm) * sl + c] = d;
    sea = true;
  }
  if (A.keys) row_min(A, x, in && sea, d, k);
}

// :400-430 at margin 4: the limiter's ratios
__global__ void cn_ratio(const CnuityArgs A) {
  after_previous();
  const int l = blockIdx.z, k = A.k0 + l;
  Cell x;
  if (!cell_of(A, 4, x)) return;
  const long long c = x.c, sl = A.slice, ld = A.ld1;
  if (!(A.msk[c] & kIP)) return;
  const int nn = A.n - 1;
  const double *dk = A.dp + ((long long)k + (long long)nn * A.kdm) * sl;
  // ipim1 etc. (bigrid.F90:316-340): the neighbour if sea, else the point itself
  const uint8_t *ms = A.msk;
  const long long ca = (ms[c - 1] & kIP) ? c - 1 : c, cb = (ms[c + 1] & kIP) ? c + 1 : c,
                  cja = (ms[c - ld] & kIP) ? c - ld : c, cjb = (ms[c + ld] & kIP) ? c + ld : c;
  const double d = dk[c];
  const double u1 = mx(mx(mx(mx(d, dk[ca]), dk[cb]), dk[cja]), dk[cjb]);
  const double u2 = mx(0., mn(mn(mn(mn(d, dk[ca]), dk[cb]), dk[cja]), dk[cjb]));
  const double *f2u = WB(A, B_UF2, l), *f2v = WB(A, B_VF2, l);
  const double fu0 = f2u[c], fu1 = f2u[c + 1], fv0 = f2v[c], fv1 = f2v[c + ld];
  // The ratios are used as min(1, ratio) only.  FP32 bounds (below the
  // numerator, above the denominator) show most of them to be at least 1, and
  // a numerator of 0 gives 0; the rest take the division.
  const float a0 = f32_away(fu0), a1 = f32_away(fu1), b0 = f32_away(fv0), b1 = f32_away(fv1);
  const float ds = f32_away(A.delt1) * f32_away(A.scp2i[c]);
  const float in = ((fmaxf(a0, 0.0f) - fminf(a1, 0.0f)) + (fmaxf(b0, 0.0f) - fminf(b1, 0.0f))) + 1.0001e-11f;
  const float out = ((fmaxf(a1, 0.0f) - fminf(a0, 0.0f)) + (fmaxf(b1, 0.0f) - fminf(b0, 0.0f))) + 1.0001e-11f;
  const float din = in * ds * 1.000004f, dout = out * ds * 1.000004f;
  const bool fine = ds > 1e-30f && din > 1e-30f && dout > 1e-30f && din < 1e37f && dout < 1e37f;
  const double n1 = u1 - d, n2 = d - u2;  // the second ratio with both signs turned
  double r1 = 1.0, r2 = 1.0;
  if (!(fine && f32_below(n1) > din)) {
    r1 = 0.0;
    if (!(fine && is0(n1)))
      r1 = div_rn(n1, mul_rn(mul_rn(((pos0(fu0) - neg0(fu1)) + (pos0(fv0) - neg0(fv1))) + kEpsilCb, A.delt1), A.scp2i[c]));
  }
  if (!(fine && f32_below(n2) > dout)) {
    r2 = 0.0;
    if (!(fine && is0(n2)))
      r2 = div_rn(n2, mul_rn(mul_rn(((pos0(fu1) - neg0(fu0)) + (pos0(fv1) - neg0(fv0))) + kEpsilCb, A.delt1), A.scp2i[c]));
  }
  WB(A, B_U1, l)[c] = r1;
  WB(A, B_U2, l)[c] = r2;
}

// f2*clip; the part clipped off is added to rest (nothing where clip = 1)
__device__ __forceinline__ double clipped(double f2, double clip, double *rest) {
  if (__double_as_longlong(clip) == kOneBits && finite(f2)) return f2;
  *rest = *rest + mul_rn(f2, 1. - clip);
  return mul_rn(f2, clip);
}

// :442-472 at margin 3: clip the antidiffusive fluxes of the batch's layers.
// A thread takes its faces through the layers, since utotn adds up in their order.
__global__ void cn_clip(const CnuityArgs A, int nl) {
  after_previous();
  Cell x;
  if (!cell_of(A, 3, x)) return;
  const long long c = x.c, sl = A.slice, ld = A.ld1;
  const uint8_t mk = A.msk[c];
  if (!(mk & (kIU | kIV))) return;
  double *ul = A.uflx + (long long)A.k0 * sl + c, *vl = A.vflx + (long long)A.k0 * sl + c;
  for (int l = 0; l < nl; l++, ul += sl, vl += sl) {
    const double *u1 = WB(A, B_U1, l), *u2 = WB(A, B_U2, l);
    const double a1 = u1[c], a2 = u2[c], w1 = u1[c - 1], w2 = u2[c - 1], s1 = u1[c - ld], s2 = u2[c - ld];
    const double f2 = WB(A, B_UF2, l)[c], g2 = WB(A, B_VF2, l)[c], ul0 = *ul, vl0 = *vl;
    if (mk & kIU) {
      const bool up = ge0(f2);
      const double clip = mn(mn(1., up ? a1 : a2), up ? w2 : w1);
      const double uf = clipped(f2, clip, W(A, W_UTN) + c);
      WB(A, B_UF, l)[c] = uf;
      *ul = ul0 + uf;
    }
    if (mk & kIV) {
      const bool up = ge0(g2);
      const double clip = mn(mn(1., up ? a1 : a2), up ? s2 : s1);
      const double vf = clipped(g2, clip, W(A, W_VTN) + c);
      WB(A, B_VF, l)[c] = vf;
      *vl = vl0 + vf;
    }
  }
}

// loop 15 (:480-498, margin 2) and loop 14 (:650-665, margin 0): flux update
// of dp(k,n); slot: dpkmin slot of layer 1, -1: none
__global__ void cn_update(const CnuityArgs A, int M, int slot) {
  after_previous();
  const int l = blockIdx.z, k = A.k0 + l;
  Cell x;
  const bool in = cell_of(A, M, x);
  bool sea = false;
  double d = 0.0;
  if (in && (A.msk[x.c] & kIP)) {
    const long long c = x.c, sl = A.slice, ld = A.ld1;
    const int nn = A.n - 1;
    double *dk = A.dp + ((long long)k + (long long)nn * A.kdm) * sl;
    const double *uf = WB(A, B_UF, l), *vf = WB(A, B_VF, l);
    d = dk[c] - mul_rn(mul_rn((uf[c + 1] - uf[c]) + (vf[c + ld] - vf[c]), A.delt1), A.scp2i[c]);
    dk[c] = d;
    sea = true;
  }
  if (A.keys && slot >= 0) row_min(A, x, in && sea, d, slot + k);
}

// p(k+1) = p(k) + dp(k,n) of every layer at margin M (:494-496, :661-663).  The
// layers' updates do not read it but for p(kk+1), which loop 77 takes as it was.
__global__ void cn_p(const CnuityArgs A, int M) {
  after_previous();
  Cell x;
  if (!cell_of(A, M, x)) return;
  const long long c = x.c, sl = A.slice;
  if (!(A.msk[c] & kIP)) return;
  const double *dk = A.dp + (long long)(A.n - 1) * A.kdm * sl + c;
  double *p = A.p + c, t = *p;
  int k = 0;
  for (; k + 4 <= A.kdm; k += 4) {
    double d[4];
#pragma unroll
    for (int r = 0; r < 4; r++) d[r] = dk[(long long)(k + r) * sl];
#pragma unroll
    for (int r = 0; r < 4; r++) {
      t = t + d[r];
      p[(long long)(k + r + 1) * sl] = t;
    }
  }
  for (; k < A.kdm; k++) {
    t = t + dk[(long long)k * sl];
    p[(long long)(k + 1) * sl] = t;
  }
}

// loop 77: the 32-bit reciprocal (recip_of) of p(kk+1) of every sea cell at
// margin 2.  p(kk+1) does not change during loop 77 before its last layer's
// fluxes are formed, so one reciprocal per cell serves every layer's division
// dp/p(kk+1).
__global__ void cn_rpb(const CnuityArgs A) {
  after_previous();
  Cell x;
  if (!cell_of(A, 2, x)) return;
  const long long c = x.c;
  if (!(A.msk[c] & kIP)) return;
  W(A, W_RPB)[c] = __longlong_as_double(recip_of(A.p[(long long)A.kdm * A.slice + c]));
}

// loop 77, :595-645 at margin 1: the barotropic correction fluxes of layer k.
// q = dp/p(kk+1) by div_by with the cell's reciprocal.  A face that clipped
// nothing (most) has no correction flux: uf = 0*q = 0 for its finite q.
__global__ void cn_btflux(const CnuityArgs A) {
  after_previous();
  const int l = blockIdx.z, k = A.k0 + l;
  Cell x;
  if (!cell_of(A, 1, x)) return;
  const long long c = x.c, sl = A.slice, ld = A.ld1;
  const uint8_t mk = A.msk[c];
  const int nn = A.n - 1;
  const double *dk = A.dp + ((long long)k + (long long)nn * A.kdm) * sl, *pb = A.p + (long long)A.kdm * sl;
  const double *rpb = W(A, W_RPB);
  if (!(mk & (kIU | kIV))) return;
  double *ul = A.uflx + (long long)k * sl + c, *vl = A.vflx + (long long)k * sl + c;
  const double ut = W(A, W_UTN)[c], vt = W(A, W_VTN)[c], d0 = dk[c], dw = dk[c - 1], ds = dk[c - ld], p0 = pb[c],
               pw = pb[c - 1], ps = pb[c - ld], r0 = rpb[c], rw = rpb[c - 1], rs = rpb[c - ld], ul0 = *ul, vl0 = *vl;
  // the correction flux of a face with transport t from a cell of thickness
  // d and total depth p, added onto *fl
  auto flux = [](double t, double d, double p, double r, double l0, double *fl) {
    const uint32_t R = (uint32_t)__double_as_longlong(r);
    if (is0(t) && R != 0 && finite(d)) return 0.0;
    const double f = mul_rn(t, div_by(d, p, R));
    *fl = l0 + f;
    return f;
  };
  if (mk & kIU) {
    const bool up = ge0(ut);
    WB(A, B_UF, l)[c] = flux(ut, up ? dw : d0, up ? pw : p0, up ? rw : r0, ul0, ul);
  }
  if (mk & kIV) {
    const bool up = ge0(vt);
    WB(A, B_VF, l)[c] = flux(vt, up ? ds : d0, up ? ps : p0, up ? rs : r0, vl0, vl);
  }
}

// :709-735 at margin 0: bottom-pressure restoring (not btrmas)
__global__ void cn_bottom(const CnuityArgs A) {
  after_previous();
  Cell x;
  if (!cell_of(A, 0, x)) return;
  const long long c = x.c, sl = A.slice;
  if (!(A.msk[c] & kIP)) return;
  const int nn = A.n - 1;
  const double q = div_rn(A.pbot[c], A.p[(long long)A.kdm * sl + c]);
  for (int k = 0; k < A.kdm; k++) {
    double *d = A.dp + ((long long)k + (long long)nn * A.kdm) * sl + c;
    *d = mul_rn(*d, q);
    A.p[(long long)(k + 1) * sl + c] = A.p[(long long)k * sl + c] + *d;
  }
}

// :770-785 / :993-1010 at margin 6: start of the interface diffusion
__global__ void cn_thk_init(const CnuityArgs A, int bih, int iflip) {
  after_previous();
  Cell x;
  if (!cell_of(A, 6, x)) return;
  const long long c = x.c;
  const uint8_t mk = A.msk[c];
  if (mk & kIU) WB(A, B_UF, 0)[c] = 0.;
  if (mk & kIV) WB(A, B_VF, 0)[c] = 0.;
  if (mk & kIP) {
    if (!bih) WB(A, B_VF, 0)[c] = 0.;
    W(A, W_POLD)[c] = iflip == 1 ? A.p[(long long)A.kdm * A.slice + c] : 0.;
  }
}

// ipim1x etc. (bigrid.F90:343-368): W (E, S, N) if sea, else the opposite
// neighbour if sea, else the point itself
__device__ __forceinline__ long long nbx(const CnuityArgs &A, long long c, long long d) {
  if (A.msk[c + d] & kIP) return c + d;
  if (A.msk[c - d] & kIP) return c - d;
  return c;
}

// loop 13, :790-830 at margin 5: biharmonic smoothing operands at the
// interfaces k = kf, kf + dir, .. (1-based) of a batch; they read only their own
// interface, which moves after them
__global__ void cn_thk_util(const CnuityArgs A, int kf, int dir) {
  after_previous();
  const int l = blockIdx.z, k = kf + dir * l;
  Cell x;
  if (!cell_of(A, 5, x)) return;
  const long long c = x.c, sl = A.slice, ld = A.ld1;
  if (!(A.msk[c] & kIP)) return;
  const int nn = A.n - 1;
  const double *dk = A.dp + ((long long)(k - 1) + (long long)nn * A.kdm) * sl,
               *dkm = A.dp + ((long long)(k - 2) + (long long)nn * A.kdm) * sl, *pk = A.p + (long long)(k - 1) * sl;
  double u1, u2;
  if (klt(mn(dk[c], dkm[c]), kOnecm)) {
    u1 = 0.0;
    u2 = 0.0;
  } else {
    const long long ca = nbx(A, c, -1), cb = nbx(A, c, 1), cja = nbx(A, c, -ld), cjb = nbx(A, c, ld);
    u1 = pk[c] - half_of(pk[ca] + pk[cb]);
    u2 = pk[c] - half_of(pk[cja] + pk[cjb]);
    if (gt0(u1)) {
      if (klt(mn(dk[ca], dk[cb]), kOnecm)) u1 = 0.0;
    } else {
      if (klt(mn(dkm[ca], dkm[cb]), kOnecm)) u1 = 0.0;
    }
    if (gt0(u2)) {
      if (klt(mn(dk[cja], dk[cjb]), kOnecm)) u2 = 0.0;
    } else {
      if (klt(mn(dkm[cja], dkm[cjb]), kOnecm)) u2 = 0.0;
    }
  }
  WB(A, B_U1, l)[c] = u1;
  WB(A, B_U2, l)[c] = u2;
}

// :838-900 (biharmonic) / :1030-1060 (Laplacian) at margin 4: limited
// interface fluxes at interface k (1-based).  The per-cell terms of the
// face bounds, G = .25*(p(kk+1)-p(k))*scp2 and (biharmonic) H =
// .25*(p(k)-pold)*scp2 (iflip 0) or .25*(pold-p(k))*scp2 (iflip 1), are
// formed once per cell in shared memory, each by the reference's own
// operations, and every face takes them from there (each is used by up to
// four faces): flxhi = G(i), flxlo = -G(i-1) (negation is exact), and the
// biharmonic bounds uflux + H, uflux - H of the cells the reference names.
constexpr int kTX = 32, kTY = 8;  // the block of every cnuity launch
// BIH, IFLIP: compile-time, so that no branch of the other form is predicated in.
// Six blocks an SM leave 40 registers, and the biharmonic forms spill 56 bytes a
// thread; without the bound it is 60 registers, no spill and fewer warps to hide
// the loads: a whole call on 1500x1100x41 14.46 against 14.49 ms (five blocks
// 14.48), with the Laplacian form 12.75 against 12.83.
template <bool BIH, bool IFLIP>
__global__ void __launch_bounds__(kTX * kTY, 6) cn_thk_flux(const CnuityArgs A, int k, int l) {
  after_previous();
  __shared__ double sG[kTY + 1][kTX + 1], sH[kTY + 1][kTX + 1];
  Cell x;
  const bool in = cell_of(A, 4, x);
  const int tx = threadIdx.x + 1, ty = threadIdx.y + 1;
  const long long sl = A.slice, ld = A.ld1;
  const double *pk = A.p + (long long)(k - 1) * sl, *ptop = A.p + (long long)A.kdm * sl;
  const double *pold = W(A, W_POLD), *scp2 = A.scp2;
  auto terms = [&](long long c, int sy, int sx) {
    sG[sy][sx] = mul_rn(half_of(half_of(ptop[c] - pk[c])), scp2[c]);
    if (BIH) sH[sy][sx] = mul_rn(half_of(half_of(IFLIP ? pold[c] - pk[c] : pk[c] - pold[c])), scp2[c]);
  };
  // every other operand is under way before the terms are exchanged
  const long long c = x.c;
  const uint8_t mk = in ? A.msk[c] : 0;
  double *uk1 = A.uflx + (long long)(k - 2) * sl, *uk = A.uflx + (long long)(k - 1) * sl;
  double *vk1 = A.vflx + (long long)(k - 2) * sl, *vk = A.vflx + (long long)(k - 1) * sl;
  double *uf = WB(A, B_UF, 0), *vf = WB(A, B_VF, 0);
  const double *pu = BIH ? WB(A, B_U1, l) : pk, *pv = BIH ? WB(A, B_U2, l) : pk;
  double tu = 0, uw = 0, uc = 0, uf0 = 0, ul1 = 0, ul0 = 0, tv = 0, vs = 0, vc = 0, vf0 = 0, vl1 = 0, vl0 = 0;
  if (mk & kIU) {
    tu = A.thkdfu[c], uw = pu[c - 1], uc = pu[c], ul1 = uk1[c], ul0 = uk[c];
    if (BIH) uf0 = uf[c];
  }
  if (mk & kIV) {
    tv = A.thkdfv[c], vs = pv[c - ld], vc = pv[c], vl1 = vk1[c], vl0 = vk[c];
    if (BIH) vf0 = vf[c];
  }
  // the box starts at margin 4, so the west and south neighbours of its
  // first column and row (margin 5) lie inside the array; one warp takes the
  // block's west column, one its south row
  if (in) terms(c, ty, tx);
  const long long c0 = (long long)((int)blockIdx.x * kTX - 3 + A.nb - 1) + (long long)((int)blockIdx.y * kTY - 3 + A.nb - 1) * ld;
  if (ty == 1 && tx <= kTY && (int)blockIdx.y * kTY + tx - 1 < A.jj + 8) terms(c0 - 1 + (tx - 1) * ld, tx, 0);
  if (ty == 2 && (int)blockIdx.x * kTX + tx - 1 < A.ii + 8) terms(c0 - ld + tx - 1, 0, tx);
  __syncthreads();
  if (!in) return;
  const double dtinv = A.dtinv;
  const double g = sG[ty][tx];
  if (mk & kIU) {
    double flxhi = g, flxlo = minus(sG[ty][tx - 1]);
    if (BIH) {
      const double hw = sH[ty][tx - 1], h = sH[ty][tx];
      flxhi = mn(flxhi, uf0 + (IFLIP ? h : hw));
      flxlo = mx(flxlo, uf0 - (IFLIP ? hw : h));
    }
    const double f = mn(flxhi, mx(flxlo, scaled(mul_rn(A.delt1, tu), uw - uc)));
    uf[c] = f;
    if (!is0(f)) {
      const double ft = mul_rn(f, dtinv);
      uk1[c] = ul1 + ft;
      uk[c] = ul0 - ft;
    }
  }
  if (mk & kIV) {
    double flxhi = g, flxlo = minus(sG[ty - 1][tx]);
    if (BIH) {
      const double hs = sH[ty - 1][tx], h = sH[ty][tx];
      flxhi = mn(flxhi, vf0 + (IFLIP ? h : hs));
      flxlo = mx(flxlo, vf0 - (IFLIP ? hs : h));
    }
    const double f = mn(flxhi, mx(flxlo, scaled(mul_rn(A.delt1, tv), vs - vc)));
    vf[c] = f;
    if (!is0(f)) {
      const double ft = mul_rn(f, dtinv);
      vk1[c] = vl1 + ft;
      vk[c] = vl0 - ft;
    }
  }
}

// :905-920 at margin 4: move interface k (1-based)
__global__ void cn_thk_p(const CnuityArgs A, int k) {
  after_previous();
  Cell x;
  if (!cell_of(A, 4, x)) return;
  const long long c = x.c, ld = A.ld1;
  if (!(A.msk[c] & kIP)) return;
  double *pk = A.p + (long long)(k - 1) * A.slice;
  const double *uf = WB(A, B_UF, 0), *vf = WB(A, B_VF, 0);
  W(A, W_POLD)[c] = pk[c];
  pk[c] = pk[c] - mul_rn((uf[c + 1] - uf[c]) + (vf[c + ld] - vf[c]), A.scp2i[c]);
}

// :925-950 at margin 4: interfaces kept ordered, dp(n) from p
__global__ void cn_thk_final(const CnuityArgs A) {
  after_previous();
  Cell x;
  if (!cell_of(A, 4, x)) return;
  const long long c = x.c, sl = A.slice;
  if (!(A.msk[c] & kIP)) return;
  const int nn = A.n - 1;
  for (int k = 0; k < A.kdm; k++) {
    double *p1 = A.p + (long long)(k + 1) * sl + c;
    const double p0 = A.p[(long long)k * sl + c];
    if (klt(*p1, p0)) *p1 = p0;
    A.dp[((long long)k + (long long)nn * A.kdm) * sl + c] = *p1 - p0;
  }
}

// :1326-1348 at margin 0: cumulative fluxes
__global__ void cn_cumul(const CnuityArgs A) {
  after_previous();
  Cell x;
  if (!cell_of(A, 0, x)) return;
  const long long c = x.c, sl = A.slice;
  const uint8_t mk = A.msk[c];
  const int nn = A.n - 1;
  for (int k = 0; k < A.kdm; k++) {
    const long long ck = (long long)k * sl + c;
    if (mk & kIU) A.uflxav[ck] = A.uflxav[ck] + A.uflx[ck];
    if (mk & kIV) A.vflxav[ck] = A.vflxav[ck] + A.vflx[ck];
    if (mk & kIP) A.dpav[ck] = A.dpav[ck] + A.dp[((long long)k + (long long)nn * A.kdm) * sl + c];
  }
}

// :1350-1385 at margin 1: btrmas restoring (dp back to dp')
__global__ void cn_btrmas(const CnuityArgs A) {
  after_previous();
  Cell x;
  if (!cell_of(A, 1, x)) return;
  const long long c = x.c, sl = A.slice;
  if (!(A.msk[c] & kIP)) return;
  const int nn = A.n - 1;
  const double cnt = div_rn(A.p[(long long)A.kdm * sl + c], A.pbot[c]);
  A.onetacnt[c] = cnt;
  double *dn = A.dp + (long long)nn * A.kdm * sl + c;
  if (cnt > kEpsilCn) {
    const double q = rcp_rn(cnt);
    for (int k = 0; k < A.kdm; k++) {
      dn[(long long)k * sl] = dn[(long long)k * sl] * q;
      A.p[(long long)(k + 1) * sl + c] = A.p[(long long)k * sl + c] + dn[(long long)k * sl];
    }
  } else {
    dn[0] = A.pbot[c];
    A.p[sl + c] = A.p[c] + dn[0];
    for (int k = 1; k < A.kdm; k++) {
      dn[(long long)k * sl] = 0.0;
      A.p[(long long)(k + 1) * sl + c] = A.p[(long long)k * sl + c] + dn[(long long)k * sl];
    }
  }
}

// :1387-1410 at margin 6: Robert-Asselin filter of dp
__global__ void cn_ra(const CnuityArgs A) {
  after_previous();
  Cell x;
  if (!cell_of(A, 6, x)) return;
  const long long c = x.c, sl = A.slice;
  if (!(A.msk[c] & kIP)) return;
  const int mm = A.m - 1, nn = A.n - 1;
  const double hra = 0.5 * A.ra2fac;
  for (int k = 0; k < A.kdm; k++) {
    const long long om = ((long long)k + (long long)mm * A.kdm) * sl + c, on = ((long long)k + (long long)nn * A.kdm) * sl + c;
    const double dpold = A.dpo[on], dpmid = A.dp[om], dpnew = A.dp[on];
    const double q = mul_rn(hra, dpold + dpnew - twice_of(dpmid));
    A.dpo[om] = dpmid;
    A.dp[om] = dpmid + q;
  }
}

dim3 grid_for(const CnuityArgs &a, int M, int layers = 1) {
  return dim3((unsigned)((a.ii + 2 * M + kTX - 1) / kTX), (unsigned)((a.jj + 2 * M + kTY - 1) / kTY), (unsigned)layers);
}

}  // namespace

size_t cnuity_work_slices(int nbatch) { return W_FIX + (size_t)B_N * nbatch; }

// Layers per launch of loops 76 and 77 (their layers are independent but for
// util3 and p, which are running sums) and interfaces per launch of the
// interface diffusion's operands: as many as 1 GiB of work slices holds.  One
// layer a launch and as many as 8 GiB holds: 257x193x22 1361 / 696 us (1 GiB:
// 696), 600x450x41 3737 / 2784 (2786), 1500x1100x41 16.9 / 14.9 ms (14.9),
// 3000x2200x10 15.1 / 14.2 (14.5).
int cnuity_batch(long long slice, int kdm) {
  const long long n = (1LL << 30) / (B_N * 8 * slice), most = kdm < 65535 ? kdm : 65535;  // the grid's limit
  return (int)(n < 1 ? 1 : n > most ? most : n);
}

cudaError_t launch_cnuity_layers(const CnuityArgs &a0, int *launches, cudaStream_t s) {
  const dim3 b(kTX, kTY);
  CnuityArgs a = a0;
  int nl = 0;
  launch_after(cn_init, grid_for(a, 6), b, s, a);
  nl++;
  for (a.k0 = 0; a.k0 < a.kdm; a.k0 += a.nbatch) {  // loop 76
    const int n = a.kdm - a.k0 < a.nbatch ? a.kdm - a.k0 : a.nbatch;
    launch_after(cn_top, grid_for(a, 4), b, s, a, n);
    if (a.btrmas) {
      launch_after(cn_flux<true>, grid_for(a, 5, n), b, s, a);
      launch_after(cn_low<true>, grid_for(a, 4, n), b, s, a);
    } else {
      launch_after(cn_flux<false>, grid_for(a, 5, n), b, s, a);
      launch_after(cn_low<false>, grid_for(a, 4, n), b, s, a);
    }
    launch_after(cn_ratio, grid_for(a, 4, n), b, s, a);
    launch_after(cn_clip, grid_for(a, 3), b, s, a, n);
    launch_after(cn_update, grid_for(a, 2, n), b, s, a, 2, a.kdm);
    nl += 6;
  }
  launch_after(cn_p, grid_for(a, 2), b, s, a, 2);
  nl++;
  *launches += nl;
  return cudaGetLastError();
}

cudaError_t launch_cnuity_rest(const CnuityArgs &a0, int *launches, cudaStream_t s) {
  const dim3 b(kTX, kTY);
  CnuityArgs a = a0;
  int nl = 0;
  if (!a.btrmas) {
    launch_after(cn_rpb, grid_for(a, 2), b, s, a);
    nl++;
    for (a.k0 = 0; a.k0 < a.kdm; a.k0 += a.nbatch) {  // loop 77
      const int n = a.kdm - a.k0 < a.nbatch ? a.kdm - a.k0 : a.nbatch;
      launch_after(cn_btflux, grid_for(a, 1, n), b, s, a);
      launch_after(cn_update, grid_for(a, 0, n), b, s, a, 0, -1);
      nl += 2;
    }
    launch_after(cn_p, grid_for(a, 0), b, s, a, 0);
    launch_after(cn_bottom, grid_for(a, 0), b, s, a);
    nl += 2;
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  if (a.thk == 4 || a.thk == 2) {
    const int bih = a.thk == 4, iflip = a.nstep % 2;
    const int nb = a.nb;
    e = launch_xctilr(a.dp + (long long)(a.n - 1) * a.kdm * a.slice, a.slice, a.kdm, a.ii, a.jj, nb, a.ld1, 6, 6,
                      a.nreg, s);
    if (e == cudaSuccess) e = launch_xctilr(a.p + a.slice, a.slice, a.kdm, a.ii, a.jj, nb, a.ld1, 6, 6, a.nreg, s);
    if (e != cudaSuccess) return e;
    nl += 2;
    launch_after(cn_thk_init, grid_for(a, 6), b, s, a, bih, iflip);
    nl++;
    const int k0 = bih ? (iflip ? a.kdm : 2) : 2, k1 = bih ? (iflip ? 2 : a.kdm) : a.kdm, dk = k1 >= k0 ? 1 : -1;
    const int ni = a.kdm < 2 ? 0 : (k1 - k0) * dk + 1;  // interior interfaces
    for (int q = 0; q < ni; q++) {
      const int k = k0 + dk * q, l = q % a.nbatch;
      if (bih && l == 0) {
        launch_after(cn_thk_util, grid_for(a, 5, ni - q < a.nbatch ? ni - q : a.nbatch), b, s, a, k, dk);
        nl++;
      }
      if (!bih) launch_after(cn_thk_flux<false, false>, grid_for(a, 4), b, s, a, k, l);
      else if (iflip) launch_after(cn_thk_flux<true, true>, grid_for(a, 4), b, s, a, k, l);
      else launch_after(cn_thk_flux<true, false>, grid_for(a, 4), b, s, a, k, l);
      launch_after(cn_thk_p, grid_for(a, 4), b, s, a, k);
      nl += 2;
    }
    launch_after(cn_thk_final, grid_for(a, 4), b, s, a);
    nl++;
  }
  if (a.uflxav && a.vflxav && a.dpav) {
    launch_after(cn_cumul, grid_for(a, 0), b, s, a);
    nl++;
  }
  if (a.btrmas) {
    launch_after(cn_btrmas, grid_for(a, 1), b, s, a);
    nl++;
  }
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  e = launch_xctilr(a.dp + (long long)(a.n - 1) * a.kdm * a.slice, a.slice, a.kdm, a.ii, a.jj, a.nb, a.ld1, 6, 6,
                    a.nreg, s);
  if (e != cudaSuccess) return e;
  launch_after(cn_ra, grid_for(a, 6), b, s, a);
  nl += 2;
  *launches += nl;
  return cudaGetLastError();
}

}  // namespace hyc
