// hyc_tsdff.cu -- lateral diffusion at the end of tsadvc (mod_tsadvc.F90:
// 2138-2230; tsdff_2x :2262-2350, tsdff_1x :2352-2440) and the density
// update of the diffused layers through the 17-term equation of state
// (stmt_fns.h:183-218, :249-263, :496-505; EOS_17T with EOS_SIG2).
//
// The reference diffuses field after field, layer after layer: the
// face fluxes of the whole slice first (margin 1), then the in-place update
// of the sea cells (margin 0).  Every (field, layer) is independent, so one
// launch covers all of them: a CTA owns a 31x32 tile of one layer, computes
// the face factors temdf2*aspux*scuy*harmonc(h(i-1),h(i)) once for all the
// layer's fields, and writes each field's new values into a scratch slice
// (a neighbouring tile still reads the old values as its halo).  A second
// launch copies the new values into level n and recomputes th3d from the
// new temperature and salinity.
//
// FP64, built without FMA contraction, in the reference's operation order:
// the results equal the oracle's bit for bit.  The path is bound by the FP64
// pipe, not by HBM, so divisions, the square root and the products that need
// no neighbouring FP64 operation run on the integer pipes (hyc_div.cuh).  T
// and S, 1500x1100x10: tile kernel 1.15 -> 0.92 ms (FP64 pipe 83 -> 56 %,
// issue slots 24 -> 48 %: latency now), store kernel 1.01 -> 0.54 ms (issue
// slots 70 %).
#include <cuda_runtime.h>

#include <cstdint>

#include "hyc_args.h"
#include "hyc_device.cuh"
#include "hyc_eos.cuh"
#include "hyc_internal.h"

namespace hyc {

namespace {

constexpr int kTX = 31, kTY = 32;        // tile (cells); lane 31 carries the east face of column 30
constexpr int kBX = kTX + 2, kBY = kTY + 2;  // tile plus a one-cell ring
constexpr int kRows = 4;                 // rows of one column a thread owns
constexpr int kThreads = 32 * kTY / kRows;
constexpr double kEpsHar = 1.0e-20;      // eps_har, mod_tsadvc.F90:1762-1763

// harmonic means, mod_tsadvc.F90:1770-1771 (max on the integer pipes,
// kmax/pos0 of hyc_device.cuh)
__device__ __forceinline__ double harmonz(double a, double b) { return div_rn(mul_rn(twice_of(a), b), kmax((a + b), 2.0 * kEpsHar)); }
__device__ __forceinline__ double harmonc(double aa, double bb) { return harmonz(pos0(aa), pos0(bb)); }

__device__ __forceinline__ long long cell(const TsdffArgs &A, int i, int j) {
  return (long long)(i + A.nb - 1) + (long long)(j + A.nb - 1) * A.ld1;
}

// temdf2*asp*sc*harmonc(ha, hb) of a face (tsdff_2x :2274-2287): products and
// division on the integer pipes.  A real call: inlined at the nine faces of a
// thread it overflows the instruction cache.
static __device__ __noinline__ double face_factor(double temdf2, double asp, double sc, double ha, double hb) {
  return mul_rn(mul_rn(mul_rn(temdf2, asp), sc), harmonc(ha, hb));
}

// One (31x32 tile, layer) per CTA; every field of the layer.  A thread owns
// four rows of a column: the factors and fluxes of its west faces and of the
// five y-faces around them stay in registers, an east face's flux comes from
// the lane to the east, and so each face is computed once (the y-faces 5/4
// times) where a thread per cell computes all four of its faces.  The fluxes'
// products stay on the FP64 pipe: on the integer pipes too 1.27 ms.
__global__ void __launch_bounds__(kThreads) tsdff_tile_kernel(const TsdffArgs A, int ntx) {
  __shared__ double sh[kBY][kBX];      // dp(k,n)*onetamas(n) on the tile and its ring
  __shared__ double sf[kBY][kBX];      // the field being diffused (old values)
  __shared__ uint8_t sm[kBY][kBX];     // masks
  const int k = blockIdx.y;
  const int i0 = 1 + (int)(blockIdx.x % ntx) * kTX, j0 = 1 + (int)(blockIdx.x / ntx) * kTY;
  const int tid = threadIdx.x;
  const long long lk = (long long)k * A.slice;
  // box cells i0-1..i0+31, j0-1..j0+32 that any needed face touches: i <= ii+1, j <= jj+1
  const int bi1 = min(kBX, A.ii + 2 - (i0 - 1)), bj1 = min(kBY, A.jj + 2 - (j0 - 1));
  int any = 0;
  for (int t = tid; t < kBX * kBY; t += kThreads) {
    const int bj = t / kBX, bi = t - bj * kBX;
    uint8_t m = 0;
    double h = 0.0;
    if (bi < bi1 && bj < bj1) {
      const long long c = cell(A, i0 - 1 + bi, j0 - 1 + bj);
      m = A.msk[c];
      if (m & kIP) h = mul_rn(A.dpn[lk + c], A.oneta[c]);  // land cells touch no open face
    }
    sh[bj][bi] = h;
    sm[bj][bi] = m;
    any |= m;
  }
  if (!__syncthreads_or(any)) return;  // land
  // lane a: the cell (and its west and south faces) at column i0 + a, box column a + 1
  const int a = tid & 31, b0 = (tid >> 5) * kRows, i = i0 + a;
  double fu[kRows], fv[kRows + 1], fac[kRows];  // face factors (tsdff_2x :2274-2287), update factors (:2335-2336)
  uint32_t ou = 0, ov = 0, sea = 0;             // open faces, cells to update
#pragma unroll
  for (int r = 0; r <= kRows; r++) {
    const int b = b0 + r, m = sm[b + 1][a + 1];
    const long long c = cell(A, i, j0 + b);
    const double h = sh[b + 1][a + 1];
    fv[r] = 0.0;
    if ((m & kIV) && a < kTX) {
      fv[r] = face_factor(A.temdf2, A.aspvy[c], A.scvx[c], sh[b][a + 1], h);
      ov |= 1u << r;
    }
    if (r == kRows) break;
    fu[r] = fac[r] = 0.0;
    if (m & kIU) {
      fu[r] = face_factor(A.temdf2, A.aspux[c], A.scuy[c], sh[b + 1][a], h);
      ou |= 1u << r;
    }
    if (i <= A.ii && j0 + b <= A.jj && (m & kIP) && a < kTX) {
      fac[r] = div_rn(-A.delt1, mul_rn(A.scp2[c], kmax(h, kEpsHar)));
      sea |= 1u << r;
    }
  }
  for (int q = 0; q < A.nfld; q++) {
    const double *f = A.fld[q] + lk;
    __syncthreads();  // sf free
    for (int t = tid; t < kBX * kBY; t += kThreads) {
      const int bj = t / kBX, bi = t - bj * kBX;
      sf[bj][bi] = (bi < bi1 && bj < bj1) ? f[cell(A, i0 - 1 + bi, j0 - 1 + bj)] : 0.0;
    }
    __syncthreads();
    double *out = A.out + ((long long)q * A.kdm + k) * A.slice;
    if (!__any_sync(0xffffffffu, ou | ov | sea)) continue;  // the warp's cells are land
    double fc = sf[b0 + 1][a + 1];
    double vs = 0.0;
    if (ov & 1u) vs = fv[0] * (sf[b0][a + 1] - fc);
#pragma unroll
    for (int r = 0; r < kRows; r++) {
      const int b = b0 + r;
      const double fn = sf[b + 2][a + 1];
      double uw = 0.0, vn = 0.0;
      if (ou >> r & 1u) uw = fu[r] * (sf[b + 1][a] - fc);
      if (ov >> (r + 1) & 1u) vn = fv[r + 1] * (fc - fn);
      const double ue = __shfl_down_sync(0xffffffffu, uw, 1);
      if (sea >> r & 1u) out[cell(A, i, j0 + b)] = fc + ((ue - uw) + (vn - vs)) * fac[r];
      fc = fn;
      vs = vn;
    }
  }
}

// New values into level n at the sea cells of the interior; th3d from the
// new temperature and salinity (:2199-2229, the ldtemp branch).
__global__ void tsdff_store_kernel(const TsdffArgs A) {
  const int k = blockIdx.y;
  const long long lk = (long long)k * A.slice;
  const long long n = (long long)A.ii * A.jj;
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
    const int j = 1 + (int)(t / A.ii), i = 1 + (int)(t - (long long)(j - 1) * A.ii);
    const long long c = cell(A, i, j);
    if (!(A.msk[c] & kIP)) continue;
    double tn = 0.0, sn = 0.0;
    for (int q = 0; q < A.nfld; q++) {
      const double v = A.out[((long long)q * A.kdm + k) * A.slice + c];
      A.fld[q][lk + c] = v;
      if (q == A.eos_t) tn = v;
      if (q == A.eos_s) sn = v;
    }
    if (A.eos_t >= 0) A.th3d[lk + c] = sig17(tn, sn) - A.thbase;
  }
}

}  // namespace

cudaError_t launch_tsdff(const TsdffArgs &a, cudaStream_t s) {
  if (a.nfld < 1 || a.nfld > kMaxFields || a.kdm < 1 || a.kdm > 65535) return cudaErrorInvalidValue;
  const int ntx = (a.ii + kTX - 1) / kTX, nty = (a.jj + kTY - 1) / kTY;
  tsdff_tile_kernel<<<dim3((unsigned)(ntx * nty), (unsigned)a.kdm), kThreads, 0, s>>>(a, ntx);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  const long long n = (long long)a.ii * a.jj;
  long long bx = (n + 255) / 256;
  if (bx > 4096) bx = 4096;
  tsdff_store_kernel<<<dim3((unsigned)bx, (unsigned)a.kdm), 256, 0, s>>>(a);
  return cudaGetLastError();
}

}  // namespace hyc
