// hyc_fct.cuh -- FP64 FCT2/FCT4 tile kernel tuned for GB300's FP64 pipe.
//
// Same stages and arithmetic as the generic tile kernel (hyc_tile.cuh; map to
// mod_tsadvc.F90:645-997 for FCT2 and :1370-1706 for FCT4), reorganised so
// that two CTAs fit on an SM (the FP64 pipe needs more resident warps to
// hide its latency than one 256-thread CTA gives):
//   * 12 shared arrays of doubles instead of 19: fmxlo/fmnlo overwrite
//     fld/fldc in place once fld and fldc are dead, fcn and scal are staged
//     where the limiter ratios go later, and fqmax/fqmin live in registers of
//     the thread that updates the same output cell;
//   * divisions and the products of the flux divergence run on the integer
//     pipes (hyc_div.cuh), and FP32 bounds settle most limiter ratios: FCT2,
//     T and S, 1500x1100x10 3.80 -> 3.27 ms (FP64 pipe 72 -> 59 % busy);
//   * fco+onemu is formed once per cell (the reference forms it per field);
//   * the stage loops have compile-time bounds and are unrolled, so a
//     thread's cells interleave (more independent FP64 work in flight).
// The region is staged by TMA (cp.async.bulk.tensor, one box per array and
// one mbarrier, every wait bounded) when the launch carries tensor maps,
// else by plain loads.  Only sea cells of the interior are written to the
// output slice.
// It serves launches too small for the strip kernel (hyc_march.cuh).
#pragma once
#include <cuda.h>

#include "hyc_args.h"
#include "hyc_device.cuh"
#include "hyc_pdl.cuh"
#include "hyc_tma.cuh"

namespace hyc {

// The region is RW x RY cells (the TX x TY output cells and a 3-cell ring).
// Its rows are stored RX = TX + 8 doubles apart, an even count, so that a
// TMA box row is a multiple of 16 bytes and the box can start on the even
// padded column at or before the region's first one (x coordinates of a
// box must be even for 8-byte elements); the region then sits at offset
// off = 0 or 1 in each array's slot.
template <int TX, int TY>
struct FctGeom {
  static constexpr int RW = TX + 6, RX = TX + 8, RY = TY + 6;
  static constexpr int NR = RX * RY;                     // cells of a staged box
  static constexpr int N = (NR + 1 + 15) / 16 * 16;      // one array's slot (128-byte multiple)
  // doubles U V HO HN SCI | FLD FLDC FX FY FLO RP RM, 4-byte RC QF FXF FYF, bytes MSK NBR
  static constexpr int NARR = 12;
  static constexpr unsigned BOX = NR * 8;                // bytes of one TMA box
  static constexpr size_t smem_bytes = 128 + (size_t)N * (NARR * 8 + 4 * 4 + 2);
};

// Compile-time rectangle [A0,A1) x [B0,B1) of a region of width RX, spread
// over 256 threads; f(a, b, e, it) with e = b*RX + a and it the iteration.
template <int RX, int A0, int A1, int B0, int B1, class F>
__device__ __forceinline__ void rect(F &&f) {
  constexpr int W = A1 - A0;
  constexpr int NN = W * (B1 - B0);
  constexpr int IT = (NN + 255) / 256;
#pragma unroll
  for (int it = 0; it < IT; it++) {
    const int t = threadIdx.x + it * 256;
    if (NN % 256 == 0 || t < NN) {
      const int bb = t / W;
      const int aa = t - bb * W;
      f(A0 + aa, B0 + bb, (B0 + bb) * RX + A0 + aa, it);
    }
  }
}

// One tile (tile index, 0-based layer k) of one basin; sm is the CTA's
// dynamic shared memory (FctGeom<TX,TY>::smem_bytes), bar its mbarrier and
// ph the count of the mbarrier's completed phases (uniform over the CTA).
// False when a TMA wait gave up (A.err is set; the CTA stops).
template <int SCHEME, int TX, int TY>
__device__ __forceinline__ bool fct_tile_body(const TileArgs &A, const int tile, const int k, double *sm,
                                              uint64_t *bar, uint32_t &ph) {
  using G = FctGeom<TX, TY>;
  constexpr int RX = G::RX, RW = G::RW, RY = G::RY, N = G::N, NR = G::NR;
  constexpr int NOUT_IT = (TX * TY + 255) / 256;
  const int tyi = tile / A.ntx, txi = tile - tyi * A.ntx;
  const int ib0 = 1 + txi * TX - 3, jb0 = 1 + tyi * TY - 3;  // region origin (Fortran index)
  const int nb = A.nbdy, ld1 = A.ld1, ii = A.ii, jj = A.jj;
  const int x0 = ib0 + nb - 1, y0 = jb0 + nb - 1;  // padded column / row of the region origin
  const int off = x0 & 1;                           // TMA boxes start at the even column x0 - off
  double *sal = reinterpret_cast<double *>((reinterpret_cast<uintptr_t>(sm) + 127) & ~uintptr_t(127));
  double *U = sal + off, *V = U + N, *HO = V + N, *HN = HO + N, *SCI = HN + N;
  double *FLD = SCI + N, *FLDC = FLD + N, *FX = FLDC + N, *FY = FX + N, *FLO = FY + N, *RP = FLO + N,
         *RM = RP + N;
  double *FCN = RP, *SCL = RM;  // staged there: dead before the first field's ratios
  uint32_t *RC = reinterpret_cast<uint32_t *>(sal + G::NARR * N);
  float *QF = reinterpret_cast<float *>(RC + N), *FXF = QF + N, *FYF = FXF + N;
  uint8_t *MSK = reinterpret_cast<uint8_t *>(FYF + N), *NBR = MSK + N;
  // fmxlo/fmnlo, as keys, in FLD/FLDC once those are dead
  auto kmx_at = [&](int e) { return __double_as_longlong(FLD[e]); };
  auto kmn_at = [&](int e) { return __double_as_longlong(FLDC[e]); };
  const CUtensorMap *tm = reinterpret_cast<const CUtensorMap *>(A.tmaps);
  const long long sl = A.slice;
  const double dt2 = A.dt2;
  // all threads wait for the mbarrier's next phase; if any gave up, let the
  // copies in flight land (bounded) and report failure
  auto landed = [&]() -> bool {
    const bool ok = tma::wait(bar, ph & 1u, A.err);
    ph++;
    if (__syncthreads_or(!ok)) {
      if (threadIdx.x == 0) tma::wait(bar, (ph - 1) & 1u, nullptr);
      return false;
    }
    return true;
  };

  // ---- per-layer inputs ------------------------------------------------------
  if (tm) {
    __syncthreads();  // the previous item's readers of these slots are done
    if (threadIdx.x == 0) {
      tma::fence_proxy_async();
      const int zk = A.mode == 0 ? k : 0;
      tma::expect_tx(bar, (A.tm_has3 ? 6u : 5u) * G::BOX);
      tma::load3(U - off, tm + 0, bar, x0 - off, y0, zk);
      tma::load3(V - off, tm + 1, bar, x0 - off, y0, zk);
      tma::load3(FCN - off, tm + 2, bar, x0 - off, y0, zk);
      if (A.tm_has3) tma::load3(HO - off, tm + 3, bar, x0 - off, y0, 0);
      tma::load3(SCL - off, tm + 4, bar, x0 - off, y0, 0);
      tma::load3(SCI - off, tm + 5, bar, x0 - off, y0, 0);
    }
    for (int t = threadIdx.x; t < NR; t += 256) {  // masks (bytes) by plain loads meanwhile
      const int bb = t / RX, aa = t - bb * RX;
      const int i = ib0 + aa, j = jb0 + bb;
      const bool in = (i >= 1 - nb) && (i <= ii + nb) && (j >= 1 - nb) && (j <= jj + nb);
      MSK[t] = in ? A.msk[(long long)(i + nb - 1) + (long long)(j + nb - 1) * ld1] : 0;
      if (!A.tm_has3) HO[t] = 1.0;  // tsadvc without btrmas: onetamas = 1
    }
    if (!landed()) return false;
  } else {
    const double *uk = A.mode == 0 ? A.uflx + k * sl : A.uflx;
    const double *vk = A.mode == 0 ? A.vflx + k * sl : A.vflx;
    for (int t = threadIdx.x; t < NR; t += 256) {
      const int bb = t / RX, aa = t - bb * RX;
      const int i = ib0 + aa, j = jb0 + bb;
      const bool in = (i >= 1 - nb) && (i <= ii + nb) && (j >= 1 - nb) && (j <= jj + nb);
      const long long o = in ? (long long)(i + nb - 1) + (long long)(j + nb - 1) * ld1 : 0;
      MSK[t] = in ? A.msk[o] : 0;
      U[t] = in ? uk[o] : 0.0;
      V[t] = in ? vk[o] : 0.0;
      SCL[t] = in ? A.scal[o] : 1.0;
      SCI[t] = in ? A.scali[o] : 1.0;
      if (A.mode == 0) {
        FCN[t] = in ? A.dpn[k * sl + o] : 0.0;            // dp(:,:,k,n)
        HO[t] = (in && A.oneta_n) ? A.oneta_n[o] : 1.0;   // onetamas(:,:,m)
      } else {
        HO[t] = in ? A.fco[o] : 0.0;
        FCN[t] = in ? A.fcn[o] : 0.0;
      }
    }
  }
  __syncthreads();
  const float qdt2f = f32_below(A.qdt2);
  for (int t = threadIdx.x; t < NR; t += 256) {
    const int bb = t / RX, aa = t - bb * RX;
    double fco, fcn;
    FX[t] = 0.0;  // faces that are not between two sea cells keep these zeros
    FY[t] = 0.0;
    FXF[t] = 0.0f;
    FYF[t] = 0.0f;
    if (aa > 0 && aa < RX - 1 && bb > 0 && bb < RY - 1)
      NBR[t] = (MSK[t - 1] & kIP) | (MSK[t + 1] & kIP) << 1 | (MSK[t - RX] & kIP) << 2 | (MSK[t + RX] & kIP) << 3;
    if (A.mode == 0) {  // mod_tsadvc.F90:1931-1938
      const double o = A.oneta_n ? HO[t] * FCN[t] : FCN[t];  // 1.0*x == x
      double fdv = 0.0;
      if (aa < RX - 1 && bb < RY - 1) {
        if (A.ufco) {
          // isopycnic layer 1: the divergence of the smoothed fluxes, read as
          // the staged ones would be (0 outside the array)
          const int i = ib0 + aa, j = jb0 + bb;
          auto at = [&](const double *f, int ic, int jc) -> double {
            const bool in = (ic >= 1 - nb) && (ic <= ii + nb) && (jc >= 1 - nb) && (jc <= jj + nb);
            return in ? f[(long long)(ic + nb - 1) + (long long)(jc + nb - 1) * ld1] : 0.0;
          };
          fdv = ((at(A.ufco, i + 1, j) - at(A.ufco, i, j)) + (at(A.vfco, i, j + 1) - at(A.vfco, i, j))) * dt2 *
                SCI[t];
        } else {
          fdv = ((U[t + 1] - U[t]) + (V[t + RX] - V[t])) * dt2 * SCI[t];
        }
      }
      fco = kmax(o + fdv, 0.0);
      fcn = kmax(o, 0.0);
    } else {
      fco = HO[t];
      fcn = FCN[t];
    }
    const double hn = fcn + kOnemu;
    HO[t] = fco + kOnemu;
    HN[t] = hn;
    RC[t] = recip_of(hn);
    // fcn*scal/dt2 from below, 0 where FP32 could lose it
    const float fs = f32_below(fcn) * f32_below(SCL[t]), qf = fs * qdt2f;
    QF[t] = fs > 1e-30f && fs < 1e30f && qf > 1e-30f && qf < 1e30f ? qf : 0.0f;
  }
  __syncthreads();

  const double qdt2 = A.qdt2;  // mod_tsadvc.F90:865
  // fcn and scal of a region cell again, for the few ratios that need them
  auto cell = [&](int a, int b) { return (long long)(x0 + a) + (long long)(y0 + b) * ld1; };
  auto fcn_of = [&](int a, int b) {
    const long long o = cell(a, b);
    if (A.mode != 0) return A.fcn[o];
    const double d = A.dpn[k * sl + o];
    return kmax(A.oneta_n ? A.oneta_n[o] * d : d, 0.0);
  };
  auto scl_of = [&](int a, int b) { return A.scal[cell(a, b)]; };
  for (int fi = 0; fi < A.nfld; fi++) {
    const FieldDesc fd = A.f[fi];
    if (k + 1 > fd.kmax || k + 1 < fd.kmin) continue;
    const double *fn = fd.nbase + (long long)(k + fd.k_off) * sl;
    const double *fm = fd.mbase + (long long)(k + fd.k_off) * sl;
    double *out = A.out + ((long long)fi * A.kdm + k) * sl;
    if (tm) {  // the previous field's readers passed the barrier that ends its loop
      if (threadIdx.x == 0) {
        tma::fence_proxy_async();
        tma::expect_tx(bar, 2u * G::BOX);
        tma::load3(FLD - off, tm + 6 + 2 * fi, bar, x0 - off, y0, k + fd.k_off);
        tma::load3(FLDC - off, tm + 7 + 2 * fi, bar, x0 - off, y0, k + fd.k_off);
      }
      if (!landed()) return false;
    } else {
      for (int t = threadIdx.x; t < NR; t += 256) {
        const int bb = t / RX, aa = t - bb * RX;
        const int i = ib0 + aa, j = jb0 + bb;
        const bool in = (i >= 1 - nb) && (i <= ii + nb) && (j >= 1 - nb) && (j <= jj + nb);
        const long long o = in ? (long long)(i + nb - 1) + (long long)(j + nb - 1) * ld1 : 0;
        FLD[t] = in ? fn[o] : 0.0;
        FLDC[t] = in ? fm[o] : 0.0;
      }
      __syncthreads();
    }

    // S1: upwind fluxes, :686-720 (zero on faces that are not sea-sea)
    rect<RX, 1, RW, 1, RY - 1>([&](int a, int b, int e, int) {
      if (MSK[e] & kIU) {
        const double uu = U[e];
        FX[e] = uu * (ge0(uu) ? FLD[e - 1] : FLD[e]);
      }
    });
    rect<RX, 1, RW - 1, 1, RY>([&](int a, int b, int e, int) {
      if (MSK[e] & kIV) {
        const double vv = V[e];
        FY[e] = vv * (ge0(vv) ? FLD[e - RX] : FLD[e]);
      }
    });
    __syncthreads();

    // S2: low-order solution on [1,RX-1)^2, :778-791
    rect<RX, 1, RW - 1, 1, RY - 1>([&](int a, int b, int e, int) {
      if (!(MSK[e] & kIP)) return;
      const int nbr = NBR[e];
      const double c = FLD[e];
      const long long kc = dkey(c), kw = dkey(FLD[nbr & 1 ? e - 1 : e]), ke = dkey(FLD[nbr & 2 ? e + 1 : e]),
                      ks = dkey(FLD[nbr & 4 ? e - RX : e]), kn = dkey(FLD[nbr & 8 ? e + RX : e]);
      const long long fmx = max(max(max(max(kc, kw), ke), ks), kn);
      const long long fmn = min(min(min(min(kc, kw), ke), ks), kn);
      const double fdv = mul_rn(mul_rn((FX[e + 1] - FX[e]) + (FY[e + RX] - FY[e]), dt2), SCI[e]);
      const double q = mul_rn(c, HO[e]) - fdv;
      FLO[e] = from_dkey(max(fmn, min(fmx, dkey(div_by(q, HN[e], RC[e])))));
    });
    __syncthreads();

    // S3: antidiffusive fluxes, :817-855 (FCT4: :1528-1580)
    rect<RX, 2, RW - 1, 2, RY - 2>([&](int a, int b, int e, int) {
      if (!(MSK[e] & kIU)) return;
      const double uu = U[e];
      double fhx;
      if (SCHEME == kFCT4 && (MSK[e - 1] & kIU) && (MSK[e + 1] & kIU)) {
        const double ft14 = 7.0 / 12.0, ft24 = -1.0 / 12.0;
        fhx = uu * (ft14 * (FLDC[e] + FLDC[e - 1]) + ft24 * (FLDC[e + 1] + FLDC[e - 2]));
      } else {
        fhx = uu * 0.5 * (FLDC[e] + FLDC[e - 1]);
      }
      const double fa = fhx - FX[e];
      FX[e] = fa;
      FXF[e] = f32_away(fa);
    });
    rect<RX, 2, RW - 2, 2, RY - 1>([&](int a, int b, int e, int) {
      if (!(MSK[e] & kIV)) return;
      const double vv = V[e];
      double fhy;
      if (SCHEME == kFCT4 && (MSK[e - RX] & kIV) && (MSK[e + RX] & kIV)) {
        const double ft14 = 7.0 / 12.0, ft24 = -1.0 / 12.0;
        fhy = vv * (ft14 * (FLDC[e] + FLDC[e - RX]) + ft24 * (FLDC[e + RX] + FLDC[e - 2 * RX]));
      } else {
        fhy = vv * 0.5 * (FLDC[e] + FLDC[e - RX]);
      }
      const double fa = fhy - FY[e];
      FY[e] = fa;
      FYF[e] = f32_away(fa);
    });
    __syncthreads();

    // fmxlo/fmnlo (:792-793) in place over fld/fldc, now dead
    rect<RX, 1, RW - 1, 1, RY - 1>([&](int a, int b, int e, int) {
      if (!(MSK[e] & kIP)) return;
      const long long c = dkey(FLD[e]), cc = dkey(FLDC[e]), lo = dkey(FLO[e]);
      FLD[e] = __longlong_as_double(max(max(c, cc), lo));
      FLDC[e] = __longlong_as_double(min(min(c, cc), lo));
    });
    __syncthreads();

    // S4: Zalesak bounds and ratios, :863-909.  Output cells keep
    // fqmax/fqmin (as keys) in registers for S6 (same thread-to-cell map).
    // A ratio is 1 unless qp < famax, mostly on one side of a cell (the side
    // t and t-1 do not differ towards): FP32 bounds of the two sides (below qp,
    // above famax, 2^-18 apart where the roundings of either are below
    // 2^-20) settle the others without the eight FP64 operations of each
    // side.  famax = 0: every flux the ratio multiplies is 0.
    long long qx[NOUT_IT], qn[NOUT_IT];
    auto zalesak = [&](int a, int b, int e, long long &kqx, long long &kqn) {
      const int nbr = NBR[e];
      const int ew = nbr & 1 ? e - 1 : e, ee = nbr & 2 ? e + 1 : e, es = nbr & 4 ? e - RX : e, en = nbr & 8 ? e + RX : e;
      kqx = max(max(max(max(kmx_at(e), kmx_at(ew)), kmx_at(ee)), kmx_at(es)), kmx_at(en));
      kqn = min(min(min(min(kmn_at(e), kmn_at(ew)), kmn_at(ee)), kmn_at(es)), kmn_at(en));
      const double lo = FLO[e];
      const double dmx = from_dkey(kqx) - lo, dmn = lo - from_dkey(kqn);
      // ib=ipip1, jb=ipjp1 (:873-875): land to the E/N -> own face twice
      const float xa = FXF[e], xb = FXF[ee], ya = FYF[e], yb = FYF[en], qf = QF[e];
      const float amax = (fmaxf(xa, 0.0f) - fminf(xb, 0.0f)) + (fmaxf(ya, 0.0f) - fminf(yb, 0.0f));
      const float amin = (fmaxf(xb, 0.0f) - fminf(xa, 0.0f)) + (fmaxf(yb, 0.0f) - fminf(ya, 0.0f));
      double rp = 1.0, rm = 1.0;
      if (!(f32_below(dmx) * qf > amax * 1.000004f || amax == 0.0f)) {
        const double famax = pos0(FX[e]) - neg0(FX[ee]) + pos0(FY[e]) - neg0(FY[en]);
        const double qp = dmx * fcn_of(a, b) * scl_of(a, b) * qdt2;
        rp = !gt0(famax) ? 0.0 : klt(qp, famax) ? div_rn(qp, famax) : 1.0;
      }
      if (!(f32_below(dmn) * qf > amin * 1.000004f || amin == 0.0f)) {
        const double famin = pos0(FX[ee]) - neg0(FX[e]) + pos0(FY[en]) - neg0(FY[e]);
        const double qm = dmn * fcn_of(a, b) * scl_of(a, b) * qdt2;
        rm = !gt0(famin) ? 0.0 : klt(qm, famin) ? div_rn(qm, famin) : 1.0;
      }
      RP[e] = rp;
      RM[e] = rm;
    };
    rect<RX, 3, RW - 3, 3, RY - 3>([&](int a, int b, int e, int it) {
      if (MSK[e] & kIP) zalesak(a, b, e, qx[it], qn[it]);
    });
    {  // the ring [2,RW-2) x [2,RY-2) minus the output cells: ratios only
      constexpr int NRING = 2 * (RW - 4) + 2 * (RY - 6);
      static_assert(NRING <= 256, "ring larger than the CTA");
      const int t = threadIdx.x;
      if (t < NRING) {
        int a, b;
        if (t < RW - 4) { a = 2 + t; b = 2; }
        else if (t < 2 * (RW - 4)) { a = 2 + t - (RW - 4); b = RY - 3; }
        else if (t < 2 * (RW - 4) + (RY - 6)) { a = 2; b = 3 + t - 2 * (RW - 4); }
        else { a = RW - 3; b = 3 + t - 2 * (RW - 4) - (RY - 6); }
        const int e = b * RX + a;
        long long dx, dn;
        if (MSK[e] & kIP) zalesak(a, b, e, dx, dn);
      }
    }
    __syncthreads();

    // S5: limit, :922-946
    rect<RX, 3, RW - 2, 3, RY - 3>([&](int a, int b, int e, int) {
      if (!(MSK[e] & kIU)) return;
      const double f = FX[e];
      const int ep = lt0(f) ? e - 1 : e, em = e + e - 1 - ep;
      const double fact = kmin(RP[ep], RM[em]);
      if (__double_as_longlong(fact) != kOneBits) FX[e] = fact * f;
    });
    rect<RX, 3, RW - 3, 3, RY - 2>([&](int a, int b, int e, int) {
      if (!(MSK[e] & kIV)) return;
      const double f = FY[e];
      const int ep = lt0(f) ? e - RX : e, em = e + e - RX - ep;
      const double fact = kmin(RP[ep], RM[em]);
      if (__double_as_longlong(fact) != kOneBits) FY[e] = fact * f;
    });
    __syncthreads();

    // S6: corrected update of the output cells, :962-982
    rect<RX, 3, RW - 3, 3, RY - 3>([&](int a, int b, int e, int it) {
      const int i = ib0 + a, j = jb0 + b;
      if (i > ii || j > jj || !(MSK[e] & kIP)) return;
      const double fdv = mul_rn(mul_rn((FX[e + 1] - FX[e]) + (FY[e + RX] - FY[e]), dt2), SCI[e]);
      const double res = from_dkey(max(qn[it], min(qx[it], dkey(FLO[e] - div_by(fdv, HN[e], RC[e])))));
      out[(long long)(i + nb - 1) + (long long)(j + nb - 1) * ld1] = res;
    });
    __syncthreads();
  }
  return true;
}

template <int SCHEME, int TX, int TY>
__global__ void __launch_bounds__(256, 2) fct_tile_kernel(const TileArgs A) {
  after_previous();
  extern __shared__ __align__(16) double sm[];
  __shared__ uint64_t bar;
  if (threadIdx.x == 0) {
    tma::bar_init(&bar, 1);
    tma::fence_bar_init();
  }
  __syncthreads();
  uint32_t ph = 0;
  fct_tile_body<SCHEME, TX, TY>(A, blockIdx.x, blockIdx.y, sm, &bar, ph);
}

}  // namespace hyc
