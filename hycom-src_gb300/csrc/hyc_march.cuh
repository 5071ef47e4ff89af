// hyc_march.cuh -- FP64 strip kernels (FCT2/FCT4, and below them MPDATA and
// donor cell): a CTA marches up the rows of a strip of columns, one barrier
// per row.
//
// Thread t owns column i0 - 3 + t of the strip (NT columns, the middle NT - 6
// are updated) for one field; the NG groups of NT threads of a CTA carry NG
// fields of the layer and share its thickness factors, which they form in
// turn, one group a row.  At row J a thread runs every stage of the scheme,
// each on an earlier row (map to mod_tsadvc.F90:645-997 for FCT2 and
// :1370-1706 for FCT4):
//   P  row J    fco+onemu, fcn+onemu, its reciprocal, fcn*scal/dt2  :1905-1942
//   A  row J    upwind and antidiffusive fluxes                :686-720, :817-855
//   B  row J-1  extrema, low-order fldlo, fmxlo/fmnlo               :778-797
//   D  row J-2  Zalesak bounds and ratios                           :863-909
//   E  row J-3  limited x-flux (y: row J-2)                         :922-946
//   F  row J-4  corrected update, clip                              :962-982
// North and south neighbours are the thread's own earlier rows, in registers;
// a west or east neighbour's value was written to a ring of rows in shared
// memory at an earlier row step, so one barrier a row orders everything.
//
// What bounds it: the FP64 pipe (a warp instruction per 16 clocks and SM; 72 %
// busy, about 85 % is reached in practice) and latency at 16 warps per SM
// (registers and shared memory both stop there); issue slots are 43 % used.
// FCT2, T and S, 1500x1100x10: 2.40 ms; the 32x16 tile kernel 3.80 ms with
// every operation on the FP64 pipe, 3.27 ms with the same integer operations
// as here.  A strip recomputes 6 of NT columns and 7 rows of a segment, where
// a tile recomputes 20-60 % of a stage, and the stages of one row step do not
// depend on one another but for B -> D -> E, so both pipes have work at any
// time.  NT = 64: four CTAs of four warps wait less at their barriers than
// two of eight (NT = 128: 2.54 ms), though 10 % of the columns are recomputed.
// Divisions and the products of P and B run on the integer pipes: with all of
// them on the FP64 pipe 2.53 ms, with A's too on the integer pipes 2.56 ms.
#pragma once
#include <cstddef>

#include "hyc_args.h"
#include "hyc_device.cuh"
#include "hyc_pdl.cuh"

namespace hyc {

template <int NT, int NG>
struct MarchGeom {
  static constexpr int OUT = NT - 6;   // columns a strip updates
  static constexpr int P = NT + 3;     // a row: two columns of padding to the west, one to the east
  static constexpr int ROW = P * 8;    // bytes of a row of doubles
  // rows shared by the fields, then rows of each field (ring length in [])
  enum { U = 0, V = U + 4, DP = V + 4, SCL = DP + 4, SCI = SCL + 8, HN = SCI + 8, RQ = HN + 8, FCN = RQ + 8, HO = FCN + 4,
         SHARED = HO + 2 };
  enum { F = 0, C = F + 4, FX = C + 4, FA = FX + 2, KX = FA + 4, KN = KX + 2, RP = KN + 2, RM = RP + 2, FXL = RM + 2,
         FAF = FXL + 2, FIELD = FAF + 2 };  // FAF: four rows of floats
  static constexpr int MSK = (SHARED + NG * FIELD) * ROW;  // four rows of bytes
  static constexpr size_t smem_bytes = MSK + 4 * P;
};

// |x| without the FP64 pipe
__device__ __forceinline__ double fabs_of(double x) { return __longlong_as_double(__double_as_longlong(x) & 0x7FFFFFFFFFFFFFFFLL); }

// 8 bytes from global to shared memory, or zeros
__device__ __forceinline__ void copy8(void *dst, const double *src, bool in) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  const int n = in ? 8 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}

// Rows [j0, j0 + nrow) of one strip of layer k (0-based), fields f0 .. f0+NG-1
// of the launch (those past nfld or outside their layers idle), described in
// fds (A.f is not read).
template <int SCHEME, int NT, int NG>
__device__ __forceinline__ void march_body(const TileArgs &A, const FieldDesc *fds, const int strip, const int j0,
                                           const int nrow, const int k, const int f0, char *sm) {
  using G = MarchGeom<NT, NG>;
  constexpr int ROW = G::ROW;
  constexpr uint8_t kW = 8, kE = 16, kS = 32, kN = 64;  // sea to the west, east, south, north
  const int t = NG == 1 ? threadIdx.x : threadIdx.x % NT, g = NG == 1 ? 0 : threadIdx.x / NT;
  const int i = 1 + strip * G::OUT - 3 + t;
  const int nb = A.nbdy, ld1 = A.ld1, ii = A.ii, jj = A.jj;
  const long long sl = A.slice;
  const double dt2 = A.dt2;
  char *sh = sm + (t + 2) * 8, *sf = sh + (G::SHARED + g * G::FIELD) * ROW;
  uint8_t *sk = reinterpret_cast<uint8_t *>(sm) + G::MSK + t + 2;
  auto S = [&](int arr, int slot, int dx = 0) -> double & {  // own column + dx of a shared row
    return *reinterpret_cast<double *>(sh + arr * ROW + slot * ROW + dx * 8);
  };
  auto Q = [&](int arr, int slot, int dx = 0) -> double & {  // of a row of this group's field
    return *reinterpret_cast<double *>(sf + arr * ROW + slot * ROW + dx * 8);
  };
  auto FAF = [&](int slot, int dx = 0) -> float & {
    return *reinterpret_cast<float *>(sf - (t + 2) * 4 + G::FAF * ROW + slot * (ROW / 2) + dx * 4);
  };
  const int fi = f0 + g;
  const FieldDesc &fd = fds[fi < A.nfld ? fi : 0];
  const bool on = fi < A.nfld && k + 1 <= fd.kmax && k + 1 >= fd.kmin;
  const bool incol = i >= 1 - nb && i <= ii + nb;
  const int xc = incol ? i + nb - 1 : 0;
  const double *fn = fd.nbase + (long long)(k + fd.k_off) * sl + xc;
  const double *fm = fd.mbase + (long long)(k + fd.k_off) * sl + xc;
  double *out = A.out + ((long long)fi * A.kdm + k) * sl + xc;
  const long long lk = A.mode == 0 ? k * sl : 0;
  const double *x3 = A.mode == 0 ? A.oneta_n : A.fco;  // onetamas(:,:,m) (null: 1) or fco
  const double *dpk = (A.mode == 0 ? A.dpn : A.fcn) + lk;
  const uint8_t *msk = A.msk;

  // row r of every array into its ring slots (zeros outside the arrays)
  auto fetch = [&](int r) -> uint8_t {
    const bool in = incol && r >= 1 - nb && r <= jj + nb;
    const long long o = in ? (long long)(r + nb - 1) * ld1 : 0;
    const int s4 = r & 3;
    if (on) {
      copy8(&Q(G::F, s4), fn + o, in);
      copy8(&Q(G::C, s4), fm + o, in);
    }
    if (g == 0) {
      copy8(&S(G::U, s4), A.uflx + lk + xc + o, in);
      copy8(&S(G::V, s4), A.vflx + lk + xc + o, in);
      copy8(&S(G::DP, s4), dpk + xc + o, in);
    }
    uint8_t m = 0;
    if (g == NG - 1) {
      copy8(&S(G::SCI, r & 7), A.scali + xc + o, in);
      copy8(&S(G::SCL, r & 7), A.scal + xc + o, in);
      if (in) m = msk[xc + o];
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    return m;
  };
  auto arrive = [&](int r, uint8_t m) {  // the row fetched last is there for every thread
    if (g == NG - 1) sk[(r & 3) * G::P] = m;
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
  };

  __syncthreads();  // the previous item's readers are done
  if (t < 2) {      // the padding columns
    for (int r = g; r < G::SHARED + NG * G::FIELD; r += NG) {
      *reinterpret_cast<double *>(sm + r * ROW + t * 8) = 0.0;
      if (t == 0) *reinterpret_cast<double *>(sm + r * ROW + (NT + 2) * 8) = 0.0;
    }
    for (int r = 0; r < 4; r++) {
      sk[r * G::P - 2] = 0;
      if (t == 0) sk[r * G::P + NT] = 0;
    }
  }
  const int jfirst = j0 - 3, jlast = j0 + nrow + 3;
  {
    const uint8_t m = fetch(jfirst);
    arrive(jfirst, m);
    const uint8_t m2 = fetch(jfirst + 1);
    arrive(jfirst + 1, m2);
  }
  const float qdt2f = f32_below(A.qdt2);
  // earlier rows of this column
  uint32_t fl = 0;                      // flags of rows J-1 (lowest byte) .. J-4
  uint8_t m1 = 0, m2 = 0;               // masks of rows J-1, J-2
  double f1 = 0, f2 = 0, c1 = 0, c2 = 0;  // old and centre level of rows J-1, J-2
  double fy1 = 0;                       // upwind y-flux of face J-1
  double ay1 = 0, ay2 = 0;              // antidiffusive y-fluxes of faces J-1, J-2
  float af1 = 0, af2 = 0;               // their FP32 bounds
  long long kx3 = 0, kn3 = 0;           // fmxlo/fmnlo of row J-3
  double lo2 = 0, lo3 = 0, lo4 = 0;     // fldlo of rows J-2 .. J-4
  long long qx3 = 0, qn3 = 0, qx4 = 0, qn4 = 0;  // fqmax/fqmin of rows J-3, J-4
  double yl3 = 0, yl4 = 0;              // limited y-fluxes of faces J-3, J-4

#pragma unroll 1
  for (int J = jfirst; J <= jlast; J++) {
    const uint8_t mnext = fetch(J + 2);
    const int s0 = J & 3, s1 = (J - 1) & 3, p0 = J & 1, p1 = p0 ^ 1;
    const uint8_t m0 = sk[s0 * G::P];

    // P: thickness factors of row J
    if ((NG == 1 || (J & (NG - 1)) == g) && __any_sync(0xffffffffu, m0 & kIP)) {
      const double d = S(G::DP, s0);
      double t3 = 0.0;  // onetamas(:,:,m) or fco
      if (x3 && (m0 & kIP)) t3 = x3[xc + (long long)(J + nb - 1) * ld1];
      double fco, fcn;
      if (A.mode == 0) {  // :1931-1938
        double o = d;
        if (x3) o = mul_rn(t3, d);
        const double fdv =
            mul_rn(mul_rn((S(G::U, s0, 1) - S(G::U, s0)) + (S(G::V, (J + 1) & 3) - S(G::V, s0)), dt2), S(G::SCI, J & 7));
        fco = kmax(o + fdv, 0.0);
        fcn = kmax(o, 0.0);
      } else {
        fco = t3;
        fcn = d;
      }
      const double hn = fcn + kOnemu;
      S(G::HO, p0) = fco + kOnemu;
      S(G::HN, J & 7) = hn;
      S(G::FCN, s0) = fcn;
      // fcn*scal/dt2 from below, 0 where FP32 could lose it
      const float fs = f32_below(fcn) * f32_below(S(G::SCL, J & 7)), qf = fs * qdt2f;
      *reinterpret_cast<uint2 *>(&S(G::RQ, J & 7)) =
          make_uint2(recip_of(hn), __float_as_uint(fs > 1e-30f && fs < 1e30f && qf > 1e-30f && qf < 1e30f ? qf : 0.0f));
    }

    if (on) {
      // A: fluxes through the west and south faces of row J (0 on faces that
      // are not between two sea cells)
      const double fc = Q(G::F, s0), cc = Q(G::C, s0);
      double fx = 0.0, ax = 0.0, fy = 0.0, ay = 0.0;
      long long kx1 = 0, kn1 = 0, kx2 = 0, kn2 = 0, qx = 0, qn = 0;
      double lo1 = 0.0, yl = 0.0;
      float af = 0.0f;
      const double ft14 = 7.0 / 12.0, ft24 = -1.0 / 12.0;
      fl <<= 8;
      // a warp whose columns are land on every row in flight only keeps its
      // faces' zeros
      if (!__any_sync(0xffffffffu, (fl | m0 | m1) != 0)) {
        Q(G::FX, p0) = 0.0;
        Q(G::FA, s0) = 0.0;
        FAF(s0) = 0.0f;
        Q(G::FXL, p1) = 0.0;
      } else {
      if (m0 & kIU) {
        const double u = S(G::U, s0), fw = Q(G::F, s0, -1), cw = Q(G::C, s0, -1);
        fx = u * (ge0(u) ? fw : fc);
        double c = cc + cw, uh = u;
        if (SCHEME == kFCT4 && (sk[s0 * G::P - 1] & sk[s0 * G::P + 1] & kIU))
          c = ft14 * c + ft24 * (Q(G::C, s0, 1) + Q(G::C, s0, -2));
        else
          uh = half_of(u);
        ax = uh * c - fx;
      }
      Q(G::FX, p0) = fx;
      Q(G::FA, s0) = ax;
      FAF(s0) = f32_away(ax);
      if (m0 & kIV) {
        const double v = S(G::V, s0);
        fy = v * (ge0(v) ? f1 : fc);
        double c = cc + c1, vh = v;
        if (SCHEME == kFCT4 && (m1 & sk[((J + 1) & 3) * G::P] & kIV))
          c = ft14 * c + ft24 * (Q(G::C, (J + 1) & 3) + c2);
        else
          vh = half_of(v);
        ay = vh * c - fy;
      }
      af = f32_away(ay);

      // B: low-order solution of row J-1
      fl |= m1 | (sk[s1 * G::P - 1] & kIP ? kW : 0) | (sk[s1 * G::P + 1] & kIP ? kE : 0) |
           (m2 & kIP ? kS : 0) | (m0 & kIP ? kN : 0);
      if (m1 & kIP) {
        const long long kc = dkey(f1), kw = dkey(Q(G::F, s1, fl & kW ? -1 : 0)), ke = dkey(Q(G::F, s1, fl & kE ? 1 : 0)),
                        ks = fl & kS ? dkey(f2) : kc, kn = fl & kN ? dkey(fc) : kc;
        const long long fmx = max(max(max(max(kc, kw), ke), ks), kn);
        const long long fmn = min(min(min(min(kc, kw), ke), ks), kn);
        const double fdv =
            mul_rn(mul_rn((Q(G::FX, p1, 1) - Q(G::FX, p1)) + (fy - fy1), dt2), S(G::SCI, (J - 1) & 7));
        const double q = mul_rn(f1, S(G::HO, p1)) - fdv;
        const uint32_t R = reinterpret_cast<const uint2 *>(&S(G::RQ, (J - 1) & 7))->x;
        const long long klo = max(fmn, min(fmx, dkey(div_by(q, S(G::HN, (J - 1) & 7), R))));
        lo1 = from_dkey(klo);
        const long long kcc = dkey(c1);
        kx1 = max(max(kc, kcc), klo);  // :792-793
        kn1 = min(min(kc, kcc), klo);
      }
      Q(G::KX, p1) = __longlong_as_double(kx1);
      Q(G::KN, p1) = __longlong_as_double(kn1);

      // D: Zalesak bounds (keys) and ratios of row J-2.  A ratio is 1 unless
      // qp < famax, mostly on one side of a cell (the side t and t-1 do not
      // differ towards): FP32 bounds of the two sides (below qp, above famax, 2^-18
      // apart where the roundings of either are below 2^-20) settle the others
      // without the eight FP64 operations of each side.  famax = 0: every flux
      // the ratio multiplies is 0.
      const uint32_t w2 = fl >> 8;
      kx2 = __double_as_longlong(Q(G::KX, p0)), kn2 = __double_as_longlong(Q(G::KN, p0));
      double rp = 1.0, rm = 1.0;
      if (w2 & kIP) {
        const int dw = w2 & kW ? -1 : 0, de = w2 & kE ? 1 : 0;
        qx = max(max(kx2, __double_as_longlong(Q(G::KX, p0, dw))), __double_as_longlong(Q(G::KX, p0, de)));
        qn = min(min(kn2, __double_as_longlong(Q(G::KN, p0, dw))), __double_as_longlong(Q(G::KN, p0, de)));
        if (w2 & kS) qx = max(qx, kx3), qn = min(qn, kn3);
        if (w2 & kN) qx = max(qx, kx1), qn = min(qn, kn1);
        const double dmx = from_dkey(qx) - lo2, dmn = lo2 - from_dkey(qn);
        // ib=ipip1, jb=ipjp1 (:873-875): land to the E/N -> own face twice
        const int s2 = (J - 2) & 3;
        const float xa = FAF(s2), xb = FAF(s2, de), ya = af2, yb = w2 & kN ? af1 : af2;
        const float qf = __uint_as_float(reinterpret_cast<const uint2 *>(&S(G::RQ, (J - 2) & 7))->y);
        const float amax = (fmaxf(xa, 0.0f) - fminf(xb, 0.0f)) + (fmaxf(ya, 0.0f) - fminf(yb, 0.0f));
        const float amin = (fmaxf(xb, 0.0f) - fminf(xa, 0.0f)) + (fmaxf(yb, 0.0f) - fminf(ya, 0.0f));
        bool ex = !(f32_below(dmx) * qf > amax * 1.000004f || amax == 0.0f);
        bool en = !(f32_below(dmn) * qf > amin * 1.000004f || amin == 0.0f);
        // at an extremum the distance is 0, and so is the ratio
        const float inf = __int_as_float(0x7F800000);
        if (ex && __double_as_longlong(dmx) == 0 && qf > 0.0f && amax < inf) ex = false, rp = 0.0;
        if (en && __double_as_longlong(dmn) == 0 && qf > 0.0f && amin < inf) en = false, rm = 0.0;
        if (ex || en) {
          const double fcn = S(G::FCN, s2), scl = S(G::SCL, (J - 2) & 7);
          const double fxa = Q(G::FA, s2), fxb = Q(G::FA, s2, de), fya = ay2, fyb = w2 & kN ? ay1 : ay2;
          if (ex) {
            const double famax = pos0(fxa) - neg0(fxb) + pos0(fya) - neg0(fyb);
            const double qp = dmx * fcn * scl * A.qdt2;
            rp = !gt0(famax) ? 0.0 : klt(qp, famax) ? div_rn(qp, famax) : 1.0;
          }
          if (en) {
            const double famin = pos0(fxb) - neg0(fxa) + pos0(fyb) - neg0(fya);
            const double qm = dmn * fcn * scl * A.qdt2;
            rm = !gt0(famin) ? 0.0 : klt(qm, famin) ? div_rn(qm, famin) : 1.0;
          }
        }
      }
      Q(G::RP, p0) = rp;
      Q(G::RM, p0) = rm;

      // E: limited fluxes, x of row J-3 and y of face J-2
      const double rp3 = Q(G::RP, p1), rm3 = Q(G::RM, p1);
      double xl = 0.0;
      if (fl >> 16 & kIU) {
        const double f = Q(G::FA, (J - 3) & 3);
        const bool neg = lt0(f);
        const double fact = kmin(neg ? Q(G::RP, p1, -1) : rp3, neg ? rm3 : Q(G::RM, p1, -1));
        xl = __double_as_longlong(fact) == kOneBits ? f : fact * f;
      }
      Q(G::FXL, p1) = xl;
      if (w2 & kIV) {
        const double f = ay2;
        const bool neg = lt0(f);
        const double fact = kmin(neg ? rp3 : rp, neg ? rm : rm3);
        yl = __double_as_longlong(fact) == kOneBits ? f : fact * f;
      }

      // F: corrected update of row J-4
      const int j = J - 4;
      if ((fl >> 24 & kIP) && j >= j0 && j <= jj && t >= 3 && t < NT - 3 && i <= ii) {
        const double fdv =
            ((Q(G::FXL, p0, 1) - Q(G::FXL, p0)) + (yl3 - yl4)) * dt2 * S(G::SCI, j & 7);
        const uint32_t R = reinterpret_cast<const uint2 *>(&S(G::RQ, j & 7))->x;
        const double res = from_dkey(max(qn4, min(qx4, dkey(lo4 - div_by(fdv, S(G::HN, j & 7), R)))));
        const long long o = (long long)(j + nb - 1) * ld1;
        out[o] = res;
        if (A.images) {  // periodic in x: the xctilr copy (mod_xc_sm.h:1415-1421) written here
          if (i <= A.images) out[o + ii] = res;
          if (i > ii - A.images) out[o - ii] = res;
        }
      }
      }

      f2 = f1, f1 = fc;
      if (SCHEME == kFCT4) c2 = c1;
      c1 = cc;
      fy1 = fy;
      ay2 = ay1, ay1 = ay, af2 = af1, af1 = af;
      kx3 = kx2, kn3 = kn2;
      lo4 = lo3, lo3 = lo2, lo2 = lo1;
      qx4 = qx3, qn4 = qn3, qx3 = qx, qn3 = qn;
      yl4 = yl3, yl3 = yl;
    }
    m2 = m1, m1 = m0;
    arrive(J + 2, mnext);
  }
}

// ---------------------------------------------------------------------------
// MPDATA (mod_tsadvc.F90:207-493) and donor cell (:495-643) in the same manner.
// At row J:
//   P  row J    thickness factors (one group); the other group the sums of
//               thicknesses around the faces of row J-1 that divide the
//               antidiffusive velocities (:377-387), shared by the fields
//   A  row J    upwind fluxes, tx1/ty1                          :248-270
//   B  row J-1  extrema, flux divergence, low-order fldlo       :277-352
//   C  row J-2  antidiffusive fluxes                            :377-387
//   D  row J-3  limiter ratios (used as min(1, ratio))          :411-419
//   E  row J-4  limited x-flux (y: face J-3)                    :440-441
//   F  row J-5  corrected update, clip                          :465-486
// The donor-cell scheme ends with B.  MPDATA, 1500x1100x10, T and S: 3.72 ms
// against 7.43 ms of the generic 32x16 tile kernel (one CTA an SM).  The FP64
// pipe bounds it (77 % busy, of the 80-85 % reached in practice): the sums
// stay there, with the products of A on it too 3.89 ms, with all products on
// the integer pipes 3.95 ms (they overflow the instruction cache).
// ---------------------------------------------------------------------------
template <int NT, int NG>
struct MarchGeom1 {
  static constexpr int OUT = NT - 6, P = NT + 3, ROW = P * 8;
  enum { U = 0, V = U + 8, DP = V + 4, SCL = DP + 4, SCI = SCL + 8, HN = SCI + 8, RQ = HN + 8, FCN = RQ + 8, FCO = FCN + 4,
         HO = FCO + 4, DX = HO + 2, DY = DX + 2, RD = DY + 2, SHARED = RD + 2 };
  enum { F = 0, FX = F + 4, FD = FX + 2, AX = FD + 2, RP = AX + 4, RM = RP + 2, XL = RM + 2, FAF = XL + 2, FIELD = FAF + 2 };
  static constexpr int MSK = (SHARED + NG * FIELD) * ROW;
  static constexpr size_t smem_bytes = MSK + 4 * P;
};

template <int SCHEME, int NT, int NG>
__device__ __forceinline__ void march1_body(const TileArgs &A, const FieldDesc *fds, const int strip, const int j0,
                                            const int nrow, const int k, const int f0, char *sm) {
  using G = MarchGeom1<NT, NG>;
  constexpr int ROW = G::ROW;
  constexpr bool MP = SCHEME == kMPDATA;
  constexpr int LAG = MP ? 5 : 1;
  constexpr uint8_t kW = 8, kE = 16, kS = 32, kN = 64;  // sea to the west, east, south, north
  const int t = NG == 1 ? threadIdx.x : threadIdx.x % NT, g = NG == 1 ? 0 : threadIdx.x / NT;
  const int i = 1 + strip * G::OUT - 3 + t;
  const int nb = A.nbdy, ld1 = A.ld1, ii = A.ii, jj = A.jj;
  const long long sl = A.slice;
  const double dt2 = A.dt2;
  char *sh = sm + (t + 2) * 8, *sf = sh + (G::SHARED + g * G::FIELD) * ROW;
  uint8_t *sk = reinterpret_cast<uint8_t *>(sm) + G::MSK + t + 2;
  auto S = [&](int arr, int slot, int dx = 0) -> double & {
    return *reinterpret_cast<double *>(sh + arr * ROW + slot * ROW + dx * 8);
  };
  auto Q = [&](int arr, int slot, int dx = 0) -> double & {
    return *reinterpret_cast<double *>(sf + arr * ROW + slot * ROW + dx * 8);
  };
  auto U2 = [&](int arr, int slot) -> uint2 & { return *reinterpret_cast<uint2 *>(&S(arr, slot)); };
  auto FAF = [&](int slot, int dx = 0) -> float & {
    return *reinterpret_cast<float *>(sf - (t + 2) * 4 + G::FAF * ROW + slot * (ROW / 2) + dx * 4);
  };
  const int fi = f0 + g;
  const FieldDesc &fd = fds[fi < A.nfld ? fi : 0];
  const bool on = fi < A.nfld && k + 1 <= fd.kmax && k + 1 >= fd.kmin;
  const double posdef = MP ? fd.posdef : 0.0;
  const bool shifted = MP && posdef != 0.0;
  const bool incol = i >= 1 - nb && i <= ii + nb;
  const int xc = incol ? i + nb - 1 : 0;
  const double *fn = fd.nbase + (long long)(k + fd.k_off) * sl + xc;
  double *out = A.out + ((long long)fi * A.kdm + k) * sl + xc;
  const long long lk = A.mode == 0 ? k * sl : 0;
  const double *x3 = A.mode == 0 ? A.oneta_n : A.fco;  // onetamas(:,:,m) (null: 1) or fco
  const double *dpk = (A.mode == 0 ? A.dpn : A.fcn) + lk;

  auto fetch = [&](int r) -> uint8_t {  // row r of every array into its ring slots (zeros outside the arrays)
    const bool in = incol && r >= 1 - nb && r <= jj + nb;
    const long long o = in ? (long long)(r + nb - 1) * ld1 : 0;
    if (on) copy8(&Q(G::F, r & 3), fn + o, in);
    if (g == 0) {
      copy8(&S(G::U, r & 7), A.uflx + lk + xc + o, in);
      copy8(&S(G::V, r & 3), A.vflx + lk + xc + o, in);
      copy8(&S(G::DP, r & 3), dpk + xc + o, in);
    }
    uint8_t m = 0;
    if (g == NG - 1) {
      copy8(&S(G::SCI, r & 7), A.scali + xc + o, in);
      copy8(&S(G::SCL, r & 7), A.scal + xc + o, in);
      if (in) m = A.msk[xc + o];
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    return m;
  };
  auto arrive = [&](int r, uint8_t m) {
    if (g == NG - 1) sk[(r & 3) * G::P] = m;
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
  };
  // the limited flux of a face: factor of the side it flows from
  auto limited = [](double f, double fact) { return __double_as_longlong(fact) == kOneBits ? f : fact * f; };

  __syncthreads();  // the previous item's readers are done
  if (t < 2) {      // the padding columns
    for (int r = g; r < G::SHARED + NG * G::FIELD; r += NG) {
      *reinterpret_cast<double *>(sm + r * ROW + t * 8) = 0.0;
      if (t == 0) *reinterpret_cast<double *>(sm + r * ROW + (NT + 2) * 8) = 0.0;
    }
    for (int r = 0; r < 4; r++) {
      sk[r * G::P - 2] = 0;
      if (t == 0) sk[r * G::P + NT] = 0;
    }
  }
  const int jfirst = j0 - 3, jlast = j0 + nrow - 1 + LAG;
  {
    const uint8_t m = fetch(jfirst);
    arrive(jfirst, m);
    const uint8_t m2 = fetch(jfirst + 1);
    arrive(jfirst + 1, m2);
  }
  const float qdt2f = f32_below(A.qdt2);
  uint32_t fl = 0, fl5 = 0;  // flags of rows J-1 (lowest byte) .. J-4, and J-5
  uint8_t m1 = 0, m2 = 0;    // masks of rows J-1, J-2
  double f1 = 0, f2 = 0;     // old level of rows J-1, J-2
  double fy1 = 0;            // upwind y-flux of face J-1
  double tx1 = 0, tx2 = 0, ty1 = 0, ty2 = 0;  // tx1/ty1 of rows J-1, J-2
  double v1 = 0, v2 = 0;     // vflx of rows J-1, J-2
  double fd3 = 0;            // flux divergence of row J-3
  double ay3 = 0;            // antidiffusive y-flux of face J-3
  float af3 = 0;
  double lo2 = 0, lo3 = 0, lo4 = 0, lo5 = 0;
  long long kx2 = 0, kx3 = 0, kx4 = 0, kx5 = 0, kn2 = 0, kn3 = 0, kn4 = 0, kn5 = 0;  // extrema (keys)
  double yl4 = 0, yl5 = 0;   // limited y-fluxes of faces J-4, J-5

#pragma unroll 1
  for (int J = jfirst; J <= jlast; J++) {
    const uint8_t mnext = fetch(J + 2);
    const int s0 = J & 3, s1 = (J - 1) & 3, p0 = J & 1, p1 = p0 ^ 1;
    const uint8_t m0 = sk[s0 * G::P];

    if ((NG == 1 || p0 == g) && __any_sync(0xffffffffu, m0 & kIP)) {  // P: thickness factors of row J
      const double d = S(G::DP, s0);
      double t3 = 0.0;
      if (x3 && (m0 & kIP)) t3 = x3[xc + (long long)(J + nb - 1) * ld1];
      double fco, fcn;
      if (A.mode == 0) {  // :1931-1938
        double o = d;
        if (x3) o = mul_rn(t3, d);
        const double fdv = mul_rn(
            mul_rn((S(G::U, J & 7, 1) - S(G::U, J & 7)) + (S(G::V, (J + 1) & 3) - S(G::V, s0)), dt2), S(G::SCI, J & 7));
        fco = kmax(o + fdv, 0.0);
        fcn = kmax(o, 0.0);
      } else {
        fco = t3;
        fcn = d;
      }
      const double hn = fcn + kOnemu;
      S(G::HO, p0) = fco + kOnemu;
      S(G::HN, J & 7) = hn;
      S(G::FCN, s0) = fcn;
      S(G::FCO, s0) = fco;
      // fcn*scal/dt2 from below, 0 where FP32 could lose it
      const float fs = f32_below(fcn) * f32_below(S(G::SCL, J & 7)), qf = fs * qdt2f;
      U2(G::RQ, J & 7) =
          make_uint2(recip_of(hn), __float_as_uint(fs > 1e-30f && fs < 1e30f && qf > 1e-30f && qf < 1e30f ? qf : 0.0f));
    }
    if (MP && (NG == 1 || p1 == g) && __any_sync(0xffffffffu, m1 & (kIU | kIV))) {  // the faces of row J-1
      const double fo = S(G::FCO, s1), fc = S(G::FCN, s1);
      const double dx = ((fo + S(G::FCO, s1, -1)) + (fc + S(G::FCN, s1, -1))) + kOnemu;
      const double dy = ((fo + S(G::FCO, (J - 2) & 3)) + (fc + S(G::FCN, (J - 2) & 3))) + kOnemu;
      S(G::DX, p1) = dx;
      S(G::DY, p1) = dy;
      U2(G::RD, p1) = make_uint2(recip_of(dx), recip_of(dy));
    }

    if (on) {
      const double fc = Q(G::F, s0), vv = S(G::V, s0);
      double fx = 0.0, fy = 0.0, tx = 0.0, ty = 0.0, fdv = 0.0, lo1 = 0.0, ax = 0.0, ay = 0.0, yl = 0.0;
      float af = 0.0f;
      long long kx1 = 0, kn1 = 0;
      fl5 = fl >> 24;
      fl = fl << 8 | m1 | (sk[s1 * G::P - 1] & kIP ? kW : 0) | (sk[s1 * G::P + 1] & kIP ? kE : 0) |
           (m2 & kIP ? kS : 0) | (m0 & kIP ? kN : 0);
      const int j = J - LAG;
      const bool stored = j >= j0 && j <= jj && t >= 3 && t < NT - 3 && i <= ii;
      if (!__any_sync(0xffffffffu, (fl | fl5 | m0) != 0)) {  // land on every row in flight: its faces' zeros
        Q(G::FX, p0) = 0.0;
        if (MP) {
          Q(G::AX, (J - 2) & 3) = 0.0;
          FAF((J - 2) & 3) = 0.0f;
          Q(G::XL, p0) = 0.0;
        }
      } else {
        // A: fluxes through the west and south faces of row J (0 on faces
        // that are not between two sea cells)
        if (m0 & kIU) {
          const double u = S(G::U, J & 7), fw = Q(G::F, s0, -1);
          if (MP) tx = mul_rn(half_of(fabs_of(u)), fc - fw);
          double q = ge0(u) ? fw : fc;
          if (shifted) q = q + posdef;
          fx = mul_rn(u, q);
        }
        if (m0 & kIV) {
          if (MP) ty = mul_rn(half_of(fabs_of(vv)), fc - f1);
          double q = ge0(vv) ? f1 : fc;
          if (shifted) q = q + posdef;
          fy = mul_rn(vv, q);
        }

        // B: low-order solution of row J-1
        if (m1 & kIP) {
          const long long kc = dkey(f1), kw = dkey(Q(G::F, s1, fl & kW ? -1 : 0)), ke = dkey(Q(G::F, s1, fl & kE ? 1 : 0)),
                          ks = fl & kS ? dkey(f2) : kc, kn = fl & kN ? dkey(fc) : kc;
          kx1 = max(max(max(max(kc, kw), ke), ks), kn);
          kn1 = min(min(min(min(kc, kw), ke), ks), kn);
          double c = f1;
          if (shifted) {
            kx1 = dkey(from_dkey(kx1) + posdef);
            kn1 = dkey(from_dkey(kn1) + posdef);
            c = c + posdef;
          }
          fdv = mul_rn(mul_rn((Q(G::FX, p1, 1) - Q(G::FX, p1)) + (fy - fy1), dt2), S(G::SCI, (J - 1) & 7));
          const double q = mul_rn(c, S(G::HO, p1)) - fdv;
          lo1 = from_dkey(max(kn1, min(kx1, dkey(div_by(q, S(G::HN, (J - 1) & 7), U2(G::RQ, (J - 1) & 7).x)))));
        }

        if (MP) {
          // C: antidiffusive fluxes of row J-2
          const uint32_t w2 = fl >> 8;
          const double fd2 = Q(G::FD, p0);
          if (w2 & kIU)
            ax = tx2 - div_by(S(G::U, (J - 2) & 7) * (fd2 + Q(G::FD, p0, -1)), S(G::DX, p0), U2(G::RD, p0).x);
          if (w2 & kIV) ay = ty2 - div_by(v2 * (fd2 + fd3), S(G::DY, p0), U2(G::RD, p0).y);
          af = f32_away(ay);

          // D: ratios of row J-3, bounded in FP32 as the FCT kernel's
          const uint32_t w3 = fl >> 16;
          const int s3 = (J - 3) & 3;
          double rp = 1.0, rm = 1.0;
          if (w3 & kIP) {
            const double dmx = from_dkey(kx3) - lo3, dmn = lo3 - from_dkey(kn3);
            const float xa = FAF(s3), xb = FAF(s3, 1);
            const float qf = __uint_as_float(U2(G::RQ, (J - 3) & 7).y), eps = 0.99e-8f, inf = __int_as_float(0x7F800000);
            const float in = ((fmaxf(xa, 0.0f) - fminf(xb, 0.0f)) + (fmaxf(af3, 0.0f) - fminf(af, 0.0f))) + eps;
            const float ou = ((fmaxf(xb, 0.0f) - fminf(xa, 0.0f)) + (fmaxf(af, 0.0f) - fminf(af3, 0.0f))) + eps;
            bool ex = !(f32_below(dmx) * qf > in * 1.000004f), en = !(f32_below(dmn) * qf > ou * 1.000004f);
            if (ex && __double_as_longlong(dmx) == 0 && qf > 0.0f && in < inf) ex = false, rp = 0.0;
            if (en && __double_as_longlong(dmn) == 0 && qf > 0.0f && ou < inf) en = false, rm = 0.0;
            if (ex || en) {
              const double fs = S(G::FCN, s3) * S(G::SCL, (J - 3) & 7);
              const double fx0 = Q(G::AX, s3), fx1 = Q(G::AX, s3, 1);
              // dm the distance to the bound; p and r the faces whose positive flux counts
              auto ratio = [&](double dm, double p, double q, double r, double s) {
                return kmin(1.0, div_rn(dm * fs, (kOnemu + ((pos0(p) - neg0(q)) + (pos0(r) - neg0(s)))) * dt2));
              };
              // one side a lane: few lanes have both
              const double r = ratio(ex ? dmx : dmn, ex ? fx0 : fx1, ex ? fx1 : fx0, ex ? ay3 : ay, ex ? ay : ay3);
              if (ex) rp = r; else rm = r;
              if (ex && en) rm = ratio(dmn, fx1, fx0, ay, ay3);
            }
          }

          // E: limited fluxes, x of row J-4 and y of face J-3
          const double rp4 = Q(G::RP, p0), rm4 = Q(G::RM, p0);
          double xl = 0.0;
          if (fl >> 24 & kIU) {
            const double f = Q(G::AX, s0);
            const bool neg = lt0(f);
            xl = limited(f, kmin(neg ? Q(G::RP, p0, -1) : rp4, neg ? rm4 : Q(G::RM, p0, -1)));
          }
          if (w3 & kIV) {
            const bool neg = lt0(ay3);
            yl = limited(ay3, kmin(neg ? rp4 : rp, neg ? rm : rm4));
          }

          // F: corrected update of row J-5
          if ((fl5 & kIP) && stored) {
            const double ch = ((Q(G::XL, p1, 1) - Q(G::XL, p1)) + (yl4 - yl5)) * dt2 * S(G::SCI, j & 7);
            double res = from_dkey(max(kn5, min(kx5, dkey(lo5 - div_by(ch, S(G::HN, j & 7), U2(G::RQ, j & 7).x)))));
            if (shifted) res = res - posdef;
            out[(long long)(j + nb - 1) * ld1] = res;
          }
          Q(G::AX, (J - 2) & 3) = ax;
          FAF((J - 2) & 3) = f32_away(ax);
          Q(G::FD, p1) = fdv;
          Q(G::RP, p1) = rp;
          Q(G::RM, p1) = rm;
          Q(G::XL, p0) = xl;
          fd3 = fd2;
        } else if ((m1 & kIP) && stored) {
          out[(long long)(j + nb - 1) * ld1] = lo1;
        }
        Q(G::FX, p0) = fx;
      }
      // land keeps the old value
      if (stored && !((MP ? fl5 : fl) & kIP)) out[(long long)(j + nb - 1) * ld1] = fn[(long long)(j + nb - 1) * ld1];

      f2 = f1, f1 = fc;
      fy1 = fy;
      if (MP) {
        tx2 = tx1, tx1 = tx, ty2 = ty1, ty1 = ty;
        v2 = v1, v1 = vv;
        ay3 = ay, af3 = af;
        lo5 = lo4, lo4 = lo3, lo3 = lo2, lo2 = lo1;
        kx5 = kx4, kx4 = kx3, kx3 = kx2, kx2 = kx1;
        kn5 = kn4, kn4 = kn3, kn3 = kn2, kn2 = kn1;
        yl5 = yl4, yl4 = yl;
      }
    }
    m2 = m1, m1 = m0;
    arrive(J + 2, mnext);
  }
}

// grid: (strips, segments, layers * field groups), the groups of a layer
// next to each other
template <int SCHEME, int NT, int NG>
__global__ void __launch_bounds__(NT *NG, 512 / (NT * NG)) march_kernel(const TileArgs A, int nrow) {
  after_previous();
  extern __shared__ __align__(16) char smc[];
  const int ngrp = (A.nfld + NG - 1) / NG;
  const int k = blockIdx.z / ngrp, q = blockIdx.z - k * ngrp;
  const int j0 = 1 + blockIdx.y * nrow;
  if constexpr (SCHEME == kFCT2 || SCHEME == kFCT4)
    march_body<SCHEME, NT, NG>(A, A.f, blockIdx.x, j0, min(nrow, A.jj + 1 - j0), k, q * NG, smc);
  else
    march1_body<SCHEME, NT, NG>(A, A.f, blockIdx.x, j0, min(nrow, A.jj + 1 - j0), k, q * NG, smc);
}

// Persistent form for an ensemble of basins: CTAs take work items (basin,
// strip * kMaxMarchGroups + field group, first row, layer) from a queue until
// it is empty.  The item's basin is staged in shared memory but for its fields: the
// full TileArgs would leave room for three CTAs on an SM instead of four.
template <int SCHEME, int NT, int NG>
__global__ void __launch_bounds__(NT *NG, 512 / (NT * NG))
    march_queue_kernel(const TileArgs *__restrict__ basins, const int4 *__restrict__ items, int nitems, int *head) {
  extern __shared__ __align__(16) char smc[];
  __shared__ int cur;
  __shared__ __align__(8) int sa[offsetof(TileArgs, f) / 4];
  int basin = -1;
  for (;;) {
    __syncthreads();  // every thread has read cur
    if (threadIdx.x == 0) cur = atomicAdd(head, 1);
    __syncthreads();
    const int it = cur;
    if (it >= nitems) break;
    const int4 w = items[it];
    if (w.x != basin) {  // the previous item's readers of sa passed the barriers above
      basin = w.x;
      const int *src = reinterpret_cast<const int *>(basins + basin);
      for (int q = threadIdx.x; q < (int)(offsetof(TileArgs, f) / 4); q += NT * NG) sa[q] = src[q];
      __syncthreads();
    }
    const TileArgs &A = *reinterpret_cast<const TileArgs *>(sa);
    const int strip = w.y / kMaxMarchGroups, q = w.y - strip * kMaxMarchGroups;
    march_body<SCHEME, NT, NG>(A, basins[basin].f, strip, w.z, min(A.seg, A.jj + 1 - w.z), w.w, q * NG, smc);
  }
}

}  // namespace hyc
