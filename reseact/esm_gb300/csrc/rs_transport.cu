// rs_transport.cu -- SSPRK43 flux-form transport: monotone PPM face fluxes and the stage kernel.
//
// Transport RHS (CWC mixing-ratio form of reseact.esm:2083, continuity reseact.esm:1535):
//   dq/dt = ( -(Dx(Mx q) + Dy(My q) + Dz(Mz q)) + q * (Dx Mx + Dy My + Dz Mz) ) / m
//   dm/dt = -(Dx Mx + Dy My + Dz Mz)
// with finite-volume divergences on the unit sphere (Dx = (F_e - F_w) dphi/(dlon dS),
// Dy = (F_n cos phi_n - F_s cos phi_s)/dS, Dz = F_top - F_bottom) and face values from the
// upwind cell's CW84-limited parabola (eqs. 1.6-1.8, 1.10; nonuniform-dp form vertically).
// At q == 1 every slope is 0, every face value is exactly 1 and each tracer flux equals the
// air-mass flux bit for bit, so dq/dt == 0 exactly (the CWC freestream gate of
// prototypes/transport_3d/transport_3d.esm and tools/cwc_gate.jl).
//
// SSPRK43 attempt (rx_traced_integrator.jl:362-400): 4 stages, each = 3 face-flux kernels
// (x, y, z) + 1 stage kernel; the 4th stage kernel also forms the embedded error and the
// fixed-tree partial sums of the hairer norm.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "rs_device.cuh"
#include "rs_kernels.h"

namespace rs {

constexpr double kOneSixth = 1.0 / 6.0;
#if RS_STRICT
constexpr int kFluxThreads = 256;
#else
constexpr int kLineThreads = 64;
#endif

// (the limit 2 min(|d0|, |d1|) equals min(2|d0|, 2|d1|) exactly: scaling by 2 is exact)
__device__ __forceinline__ double slope_u(double am, double a, double ap) {
  double d0 = a - am, d1 = ap - a;
  if (d1 * d0 > 0.0) {
    double da = 0.5 * (ap - am);
    double lim = 2.0 * fmin(fabs(d0), fabs(d1));
    return copysign(fmin(fabs(da), lim), da);
  }
  return 0.0;
}
__device__ __forceinline__ double slope_n(double am, double a, double ap, double sA, double sB) {
  double d0 = a - am, d1 = ap - a;
  if (d1 * d0 > 0.0) {
    double da = sA * d1 + sB * d0;
    double lim = 2.0 * fmin(fabs(d0), fabs(d1));
    return copysign(fmin(fabs(da), lim), da);
  }
  return 0.0;
}
__device__ __forceinline__ void limit(double a, double& aL, double& aR) {
  if ((aR - a) * (a - aL) <= 0.0) {
    aL = a;
    aR = a;
  } else {
    double dA = aR - aL;
    double a6 = 6.0 * (a - 0.5 * (aL + aR));
    if (dA * a6 > dA * dA) aL = 3.0 * a - 2.0 * aR;
    else if (-(dA * dA) > dA * a6) aR = 3.0 * a - 2.0 * aL;
  }
}
// ---- production-build forms of the slopes: the same slopes, with the sign tests and the exact
// power-of-two scalings done on the sign and exponent bits in the integer pipes (FP64 issues at
// ~2 lanes per SM per clock on this GPU):
//   d1*d0 > 0            <=>  d0, d1 nonzero with equal signs       (unless the product underflows)
//   0.5*s, 2*m           =    exponent field -1 / +1                 (normal operands)
//   fmin of magnitudes   =    integer min of the magnitude bits
// bit-identical to the FP forms for normal operands (where a product of differences could
// underflow, or an operand is subnormal, the FP form decides).
// copysign(min(|da|, 2 min(|d0|, |d1|)), da), or 0 where d0, d1 are not nonzero with equal
// signs, on the 32-bit halves of the bit patterns.  (Written on 64-bit masks of reinterpreted
// doubles, the same arithmetic was partly emitted as FP64 adds -- three per slope, measured with
// ncu -- so everything here stays in 32-bit integer operations.)  `half`: |da| = |span| / 2.
__device__ __forceinline__ double slope_pick32(double d0, double d1, double da, bool half) {
  const unsigned hs = (unsigned)__double2hiint(da);
  const unsigned hd = (hs & 0x7fffffffu) - (half ? (1u << 20) : 0u), ld = (unsigned)__double2loint(da);
  const unsigned h0 = (unsigned)__double2hiint(d0) & 0x7fffffffu, l0 = (unsigned)__double2loint(d0);
  const unsigned h1 = (unsigned)__double2hiint(d1) & 0x7fffffffu, l1 = (unsigned)__double2loint(d1);
  const bool p1 = mag_lt(h1, l1, h0, l0);
  const unsigned hm = (p1 ? h1 : h0) + (1u << 20), lm = p1 ? l1 : l0;  // 2 min(|d0|, |d1|)
  const bool binds = mag_lt(hm, lm, hd, ld);
  const unsigned hr = (binds ? hm : hd) | (hs & 0x80000000u), lr = binds ? lm : ld;
  const bool live = ((__double2hiint(d0) ^ __double2hiint(d1)) >= 0) & ((h0 | l0) != 0u) &
                    ((h1 | l1) != 0u);
  return __hiloint2double(live ? (int)hr : 0, live ? (int)lr : 0);
}
// slopes from the neighbour differences d0 = a - am, d1 = ap - a
#if RS_STRICT
// (am, ap: the oracle forms the centred slope from the values)
__device__ __forceinline__ double slope_ud(double d0, double d1, double am, double ap) {
  if (d1 * d0 > 0.0) {
    double da = 0.5 * (ap - am);
    double lim = 2.0 * fmin(fabs(d0), fabs(d1));
    return copysign(fmin(fabs(da), lim), da);
  }
  return 0.0;
}
#else
__device__ __forceinline__ double slope_ud(double d0, double d1) {
  if (prod_may_underflow(d0, d1)) {
    if (d1 * d0 > 0.0) {
      double da = 0.5 * (d0 + d1);
      double lim = 2.0 * fmin(fabs(d0), fabs(d1));
      return copysign(fmin(fabs(da), lim), da);
    }
    return 0.0;
  }
  return slope_pick32(d0, d1, d0 + d1, true);
}
#endif
__device__ __forceinline__ double slope_nd(double d0, double d1, double sA, double sB) {
#if !RS_STRICT
  if (!prod_may_underflow(d0, d1)) return slope_pick32(d0, d1, sA * d1 + sB * d0, false);
#endif
  if (d1 * d0 > 0.0) {
    double da = sA * d1 + sB * d0;
    double lim = 2.0 * fmin(fabs(d0), fabs(d1));
    return copysign(fmin(fabs(da), lim), da);
  }
  return 0.0;
}

// split a double into hi + lo floats (used only for boundary ghosts in the flux kernels)
__device__ __forceinline__ void split_d(double x, float& hi, float& lo) {
  hi = (float)x;
  lo = (float)(x - (double)hi);
}

// Bounds-check build (-DRS_BOUNDS_CHECK=1): the pencil kernels check every shared-memory row
// index, every halo / ghost load and every bulk-copy box start against its array.  An index
// outside [0, n) sets bit 2 of the handle's staging word (T.tma_err) and is replaced by 0, so
// the access stays inside the array; the host reports RS_ERR_INVALID after the step.  The
// other builds compile the checks away.
#ifndef RS_BOUNDS_CHECK
#define RS_BOUNDS_CHECK 0
#endif
__device__ __forceinline__ long long bck(const DevTransport<double>& T, long long i, long long n) {
#if RS_BOUNDS_CHECK
  if (i < 0 || i >= n) {
    if (T.tma_err) atomicOr(T.tma_err, 2);
    return 0;
  }
#endif
  return i;
}

// Stage input selection: inside an adaptive attempt the field and the time factor come from
// the device-resident controller (input U[cur] for stage 1, S1/S2/S3 for stages 2-4, g from
// ctl->g[stage-1]); for a single RHS evaluation they are given directly.
struct StageSel {
  const Ctl* ctl;
  int stage;
  const double* U0;
  const double* U1;
  const double* S1;
  const double* S2;
  const double* S3;
  const double* Q;  // direct evaluation
  double g;
};
__device__ __forceinline__ bool resolve_stage(const StageSel& s, const double*& Q, double& g) {
  if (!s.ctl) {
    Q = s.Q;
    g = s.g;
    return true;
  }
  if (s.ctl->done) return false;
  g = s.ctl->g[s.stage - 1];
  Q = s.stage == 1 ? (s.ctl->cur ? s.U1 : s.U0)
                   : (s.stage == 2 ? s.S1 : (s.stage == 3 ? s.S2 : s.S3));
  return true;
}

// ------------------------------------------------------------------ face fluxes (strict build)
// The oracle's flux form, expression by expression; the production build's kernels are in
// rs_adv64.cuh.
#if RS_STRICT
__device__ __forceinline__ double ppm_face_u(const double* v, bool right) {
  double dm1 = slope_u(v[0], v[1], v[2]);
  double d0 = slope_u(v[1], v[2], v[3]);
  double dp1 = slope_u(v[2], v[3], v[4]);
  double aL = v[1] + 0.5 * (v[2] - v[1]) - (d0 - dm1) * kOneSixth;
  double aR = v[2] + 0.5 * (v[3] - v[2]) - (dp1 - d0) * kOneSixth;
  limit(v[2], aL, aR);
  return right ? aR : aL;
}

// x faces: (i_f in 0..nlon, j, k), i_f fastest
__global__ void __launch_bounds__(kFluxThreads) k_flux_x(DevTransport<double> T, StageSel sel) {
  const double* Q;
  double g;
  if (!resolve_stage(sel, Q, g)) return;
  const int nf = T.nlon + 1;
  long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  long long total = (long long)nf * T.nlat * T.nlev;
  if (idx >= total) return;
  int i = (int)(idx % nf);
  int j = (int)((idx / nf) % T.nlat);
  int k = (int)(idx / ((long long)nf * T.nlat));
  const size_t nc = (size_t)T.nlon * T.nlat * T.nlev;
  const size_t row = ((size_t)k * T.nlat + j) * T.nlon;
  double M = g * T.mx[((size_t)k * T.nlat + j) * nf + i];
  bool right = M > 0.0;
  int up = right ? i - 1 : i;
  int ii[5];
  bool ghost[5];
  for (int o = 0; o < 5; ++o) {
    int q = up - 2 + o;
    ghost[o] = false;
    if (q < 0 || q >= T.nlon) {
      if (T.lon_bc == 0) q = ((q % T.nlon) + T.nlon) % T.nlon;
      else ghost[o] = true;
    }
    ii[o] = q;
  }
  for (int s = 0; s < T.ntr; ++s) {
    const double* q = Q + (size_t)s * nc + row;
    double v[5];
    for (int o = 0; o < 5; ++o) {
      if (ghost[o]) {
        const double* b = ii[o] < 0 ? T.qw : T.qe;
        v[o] = b[((size_t)s * T.nlev + k) * T.nlat + j];
      } else {
        v[o] = q[ii[o]];
      }
    }
    T.fx[((size_t)s * T.nlev * T.nlat + (size_t)k * T.nlat + j) * nf + i] = M * ppm_face_u(v, right);
  }
}

// y faces: (i, j_f in 0..nlat, k), i fastest
__global__ void __launch_bounds__(kFluxThreads) k_flux_y(DevTransport<double> T, StageSel sel) {
  const double* Q;
  double g;
  if (!resolve_stage(sel, Q, g)) return;
  const int nf = T.nlat + 1;
  long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  long long total = (long long)T.nlon * nf * T.nlev;
  if (idx >= total) return;
  int i = (int)(idx % T.nlon);
  int j = (int)((idx / T.nlon) % nf);
  int k = (int)(idx / ((long long)T.nlon * nf));
  const size_t nc = (size_t)T.nlon * T.nlat * T.nlev;
  const size_t fbase = ((size_t)k * nf + j) * T.nlon + i;
  const size_t fplane = (size_t)T.nlev * nf * T.nlon;
  if (T.lat_bc != 1 && (j == 0 || j == T.nlat)) {
    for (int s = 0; s < T.ntr; ++s) T.fy[(size_t)s * fplane + fbase] = 0.0;
    return;
  }
  double M = g * T.my[fbase];
  bool right = M > 0.0;
  int up = right ? j - 1 : j;
  int jj[5];
  bool ghost[5];
  for (int o = 0; o < 5; ++o) {
    int q = up - 2 + o;
    ghost[o] = false;
    if (q < 0 || q >= T.nlat) {
      if (T.lat_bc == 1) ghost[o] = true;
      else q = q < 0 ? -1 - q : 2 * T.nlat - 1 - q;
    }
    jj[o] = q;
  }
  for (int s = 0; s < T.ntr; ++s) {
    const double* q = Q + (size_t)s * nc + (size_t)k * T.nlat * T.nlon + i;
    double v[5];
    for (int o = 0; o < 5; ++o) {
      if (ghost[o]) {
        const double* b = jj[o] < 0 ? T.qs : T.qn;
        v[o] = b[((size_t)s * T.nlev + k) * T.nlon + i];
      } else {
        v[o] = q[(size_t)jj[o] * T.nlon];
      }
    }
    T.fy[(size_t)s * fplane + fbase] = M * ppm_face_u(v, right);
  }
}

// z faces: (i, j, k_f in 0..nlev), i fastest; nonuniform (dp-weighted) CW84 reconstruction
__global__ void __launch_bounds__(kFluxThreads) k_flux_z(DevTransport<double> T, StageSel sel) {
  const double* Q;
  double g;
  if (!resolve_stage(sel, Q, g)) return;
  const int nf = T.nlev + 1;
  const size_t ncol = (size_t)T.nlon * T.nlat;
  long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  long long total = (long long)ncol * nf;
  if (idx >= total) return;
  size_t col = (size_t)(idx % (long long)ncol);
  int kf = (int)(idx / (long long)ncol);
  const size_t nc = ncol * T.nlev;
  const size_t fplane = ncol * nf;
  if (kf == 0 || kf == T.nlev) {
    for (int s = 0; s < T.ntr; ++s) T.fz[(size_t)s * fplane + (size_t)kf * ncol + col] = 0.0;
    return;
  }
  double M = g * T.mz[(size_t)kf * ncol + col];
  bool right = M > 0.0;
  int up = right ? kf - 1 : kf;
  int kk[5];
  for (int o = 0; o < 5; ++o) {
    int q = up - 2 + o;
    kk[o] = q < 0 ? -1 - q : (q >= T.nlev ? 2 * T.nlev - 1 - q : q);
  }
  // coefficient rows: slope cells up-1..up+1 (stored from cell -1), edges up and up+1
  double sA0 = T.vsA[(size_t)(up) * ncol + col], sB0 = T.vsB[(size_t)(up) * ncol + col];
  double sA1 = T.vsA[(size_t)(up + 1) * ncol + col], sB1 = T.vsB[(size_t)(up + 1) * ncol + col];
  double sA2 = T.vsA[(size_t)(up + 2) * ncol + col], sB2 = T.vsB[(size_t)(up + 2) * ncol + col];
  double eLab = T.veAB[(size_t)up * ncol + col], eLc = T.veC[(size_t)up * ncol + col],
         eLd = T.veD[(size_t)up * ncol + col];
  double eRab = T.veAB[(size_t)(up + 1) * ncol + col], eRc = T.veC[(size_t)(up + 1) * ncol + col],
         eRd = T.veD[(size_t)(up + 1) * ncol + col];
  for (int s = 0; s < T.ntr; ++s) {
    const double* q = Q + (size_t)s * nc + col;
    double v[5];
    for (int o = 0; o < 5; ++o) v[o] = q[(size_t)kk[o] * ncol];
    double dm1 = slope_n(v[0], v[1], v[2], sA0, sB0);
    double d0 = slope_n(v[1], v[2], v[3], sA1, sB1);
    double dp1 = slope_n(v[2], v[3], v[4], sA2, sB2);
    double aL = v[1] + eLab * (v[2] - v[1]) + eLc * d0 + eLd * dm1;
    double aR = v[2] + eRab * (v[3] - v[2]) + eRc * dp1 + eRd * d0;
    limit(v[2], aL, aR);
    const double face = right ? aR : aL;
    T.fz[(size_t)s * fplane + (size_t)kf * ncol + col] = M * face;
  }
}

// ------------------------------------------------------------------ fused pencil kernels
// FP64 face fluxes with each cell's monotone slope and each edge value computed ONCE per
// stage (the per-face kernels above recompute three slopes and two edges for every face):
// a block stages whole pencils (a lon row; or 32 adjacent columns of a lat line / vertical
// column) in shared memory, then slopes, then edges, then the upwind limiter and flux of
// each face.  Same expressions in the same order as ppm_face_u / the vertical branch, so the
// fluxes are bit-identical to the per-face kernels.
__global__ void __launch_bounds__(256) k_flux_x_fused(DevTransport<double> T, StageSel sel) {
  const double* Q;
  double g;
  if (!resolve_stage(sel, Q, g)) return;
  extern __shared__ double smx[];
  const int n = T.nlon, nf = n + 1, L = n + 6;
  double* V = smx;            // V[p+3], p in [-3, n+2]
  double* Dd = smx + L;       // Dd[p+3] = v(p+1) - v(p), p in [-3, n+1]
  double* D = smx + 2 * L;    // D[p+3], slopes p in [-2, n+1]
  double* E = smx + 3 * L;    // strict: E[f+3], edge between f-1 and f, f in [-1, n+1];
                              // production: E[p+3] = 6 x right-edge deviation of cell p
  double* Mf = smx + 4 * L;   // Mf[f], the face's air-mass flux g*mx (shared by all tracers)
  const int row = blockIdx.x;  // (k, j)
  const int j = row % T.nlat, k = row / T.nlat;
  const size_t nc = (size_t)T.nlon * T.nlat * T.nlev;
  const size_t rbase = ((size_t)k * T.nlat + j) * n;
  for (int f = threadIdx.x; f <= n; f += blockDim.x) Mf[bck(T, f, nf)] = g * T.mx[((size_t)k * T.nlat + j) * nf + f];
  const int s0 = (int)((long long)blockIdx.y * T.ntr / gridDim.y);  // this block's tracers
  const int s1 = (int)((long long)(blockIdx.y + 1) * T.ntr / gridDim.y);
  for (int s = s0; s < s1; ++s) {
    const double* q = Q + (size_t)s * nc + rbase;
    auto val = [&](int p) -> double {
      if (p < 0 || p >= n) {
        if (T.lon_bc == 0) return q[bck(T, ((p % n) + n) % n, n)];
        return (p < 0 ? T.qw : T.qe)[bck(T, ((size_t)s * T.nlev + k) * T.nlat + j, (long long)T.ntr * T.nlev * T.nlat)];
      }
      return q[bck(T, p, n)];
    };
    for (int p = threadIdx.x - 3; p <= n + 2; p += blockDim.x) {
      const double v = val(p);
      V[bck(T, p + 3, L)] = v;
      if (p <= n + 1) Dd[bck(T, p + 3, L)] = val(p + 1) - v;
    }
    __syncthreads();
    for (int p = threadIdx.x - 2; p <= n + 1; p += blockDim.x)
      D[bck(T, p + 3, L)] = slope_ud(Dd[bck(T, p + 2, L)], Dd[bck(T, p + 3, L)], V[bck(T, p + 2, L)], V[bck(T, p + 4, L)]);
    __syncthreads();
    for (int f = threadIdx.x - 1; f <= n + 1; f += blockDim.x)
      E[bck(T, f + 3, L)] = V[bck(T, f + 2, L)] + 0.5 * Dd[bck(T, f + 2, L)] - (D[bck(T, f + 3, L)] - D[bck(T, f + 2, L)]) * kOneSixth;
    __syncthreads();
    for (int f = threadIdx.x; f <= n; f += blockDim.x) {
      const double M = Mf[bck(T, f, nf)];
      const bool right = __double_as_longlong(M) > 0;  // M > 0 for every non-NaN M
      int up = right ? f - 1 : f;
      double aL = E[bck(T, up + 3, L)], aR = E[bck(T, up + 4, L)];
      limit(V[bck(T, up + 3, L)], aL, aR);
      const double face = right ? aR : aL;
      T.fx[((size_t)s * T.nlev * T.nlat + (size_t)k * T.nlat + j) * nf + f] = M * face;
    }
    __syncthreads();
  }
}

// y: block = PW adjacent i at one level, all j; threads (PW, rows)
template <int kPencil>
__global__ void __launch_bounds__(512) k_flux_y_fused(DevTransport<double> T, StageSel sel) {
  const double* Q;
  double g;
  if (!resolve_stage(sel, Q, g)) return;
  extern __shared__ double smy[];
  const int n = T.nlat, nfj = n + 1, L = n + 6;
  double* V = smy;                    // [L][kPencil]
  double* Dd = smy + L * kPencil;     // neighbour differences v(p+1) - v(p)
  double* D = smy + 2 * L * kPencil;
  double* E = smy + 3 * L * kPencil;
  double* Mf = smy + 4 * L * kPencil;  // [n+1][kPencil] face air-mass fluxes g*my
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int ntile = (T.nlon + kPencil - 1) / kPencil;
  const int k = blockIdx.x / ntile;
  const int i = (blockIdx.x % ntile) * kPencil + tx;
  const bool live = i < T.nlon;
  const size_t nc = (size_t)T.nlon * T.nlat * T.nlev;
  const size_t fplane = (size_t)T.nlev * nfj * T.nlon;
  const bool open = T.lat_bc == 1;
  if (live)
    for (int f = ty; f <= n; f += blockDim.y)
      Mf[bck(T, f * kPencil + tx, (long long)(n + 1) * kPencil)] = g * T.my[((size_t)k * nfj + f) * T.nlon + i];
#define RS_P(a, p) a[bck(T, ((p) + 3) * kPencil + tx, (long long)L * kPencil)]
  const int s0 = (int)((long long)blockIdx.y * T.ntr / gridDim.y);  // this block's tracers
  const int s1 = (int)((long long)(blockIdx.y + 1) * T.ntr / gridDim.y);
  for (int s = s0; s < s1; ++s) {
    const double* q = Q + (size_t)s * nc + (size_t)k * T.nlat * T.nlon;
    auto val = [&](int p) -> double {
      if (!live) return 0.0;
      if (p < 0 || p >= n) {
        if (open) return (p < 0 ? T.qs : T.qn)[bck(T, ((size_t)s * T.nlev + k) * T.nlon + i, (long long)T.ntr * T.nlev * T.nlon)];
        return q[bck(T, (size_t)(p < 0 ? -1 - p : 2 * n - 1 - p) * T.nlon + i, (long long)T.nlat * T.nlon)];
      }
      return q[bck(T, (size_t)p * T.nlon + i, (long long)T.nlat * T.nlon)];
    };
    for (int p = (int)ty - 3; p <= n + 2; p += blockDim.y) {
      const double v = val(p);
      RS_P(V, p) = v;
      if (p <= n + 1) RS_P(Dd, p) = val(p + 1) - v;
    }
    __syncthreads();
    for (int p = (int)ty - 2; p <= n + 1; p += blockDim.y)
      RS_P(D, p) = slope_ud(RS_P(Dd, p - 1), RS_P(Dd, p), RS_P(V, p - 1), RS_P(V, p + 1));
    __syncthreads();
    for (int f = (int)ty - 1; f <= n + 1; f += blockDim.y)
      RS_P(E, f) = RS_P(V, f - 1) + 0.5 * RS_P(Dd, f - 1) - (RS_P(D, f) - RS_P(D, f - 1)) * kOneSixth;
    __syncthreads();
    if (live) {
      for (int f = ty; f <= n; f += blockDim.y) {
        size_t fb = ((size_t)k * nfj + f) * T.nlon + i;
        if (!open && (f == 0 || f == n)) {
          T.fy[(size_t)s * fplane + fb] = 0.0;
          continue;
        }
        const double M = Mf[bck(T, f * kPencil + tx, (long long)(n + 1) * kPencil)];
        const bool right = __double_as_longlong(M) > 0;
        int up = right ? f - 1 : f;
        double aL = RS_P(E, up), aR = RS_P(E, up + 1);
        limit(RS_P(V, up), aL, aR);
        const double face = right ? aR : aL;
        T.fy[(size_t)s * fplane + fb] = M * face;
      }
    }
    __syncthreads();
  }
}

// z: block = PW adjacent columns, all levels; dp-weighted coefficients
template <int kPencil>
__global__ void __launch_bounds__(512) k_flux_z_fused(DevTransport<double> T, StageSel sel) {
  const double* Q;
  double g;
  if (!resolve_stage(sel, Q, g)) return;
  extern __shared__ double smz[];
  const int n = T.nlev, L = n + 6;
  double* V = smz;
  double* Dd = smz + L * kPencil;
  double* D = smz + 2 * L * kPencil;
  double* E = smz + 3 * L * kPencil;
  double* Mf = smz + 4 * L * kPencil;  // [n+1][kPencil] face air-mass fluxes g*mz
  const int tx = threadIdx.x, ty = threadIdx.y;
  const size_t ncol = (size_t)T.nlon * T.nlat;
  const size_t col = (size_t)blockIdx.x * kPencil + tx;
  const bool live = col < ncol;
  const size_t nc = ncol * n;
  const size_t fplane = ncol * (n + 1);
  if (live)
    for (int kf = ty; kf <= n; kf += blockDim.y) Mf[bck(T, kf * kPencil + tx, (long long)(n + 1) * kPencil)] = g * T.mz[(size_t)kf * ncol + col];
  const int s0 = (int)((long long)blockIdx.y * T.ntr / gridDim.y);  // this block's tracers
  const int s1 = (int)((long long)(blockIdx.y + 1) * T.ntr / gridDim.y);
  for (int s = s0; s < s1; ++s) {
    const double* q = Q + (size_t)s * nc;
    auto val = [&](int p) -> double {
      const int pp = p < 0 ? -1 - p : (p >= n ? 2 * n - 1 - p : p);
      return live ? q[bck(T, (size_t)pp * ncol + col, (long long)nc)] : 0.0;
    };
    for (int p = (int)ty - 3; p <= n + 2; p += blockDim.y) {
      const double v = val(p);
      RS_P(V, p) = v;
      if (p <= n + 1) RS_P(Dd, p) = val(p + 1) - v;
    }
    __syncthreads();
    for (int p = (int)ty - 1; p <= n; p += blockDim.y) {  // slopes of cells -1..n
      double sA = live ? T.vsA[bck(T, (size_t)(p + 1) * ncol + col, (long long)(n + 2) * ncol)] : 0.0;
      double sB = live ? T.vsB[bck(T, (size_t)(p + 1) * ncol + col, (long long)(n + 2) * ncol)] : 0.0;
      RS_P(D, p) = slope_nd(RS_P(Dd, p - 1), RS_P(Dd, p), sA, sB);
    }
    __syncthreads();
    for (int e = ty; e <= n; e += blockDim.y) {  // edges 0..n (cells e-1 | e)
      double eab = live ? T.veAB[bck(T, (size_t)e * ncol + col, (long long)(n + 1) * ncol)] : 0.0;
      double ec = live ? T.veC[bck(T, (size_t)e * ncol + col, (long long)(n + 1) * ncol)] : 0.0;
      double ed = live ? T.veD[bck(T, (size_t)e * ncol + col, (long long)(n + 1) * ncol)] : 0.0;
      RS_P(E, e) = RS_P(V, e - 1) + eab * RS_P(Dd, e - 1) + ec * RS_P(D, e) + ed * RS_P(D, e - 1);
    }
    __syncthreads();
    if (live) {
      for (int kf = ty; kf <= n; kf += blockDim.y) {
        if (kf == 0 || kf == n) {
          T.fz[(size_t)s * fplane + (size_t)kf * ncol + col] = 0.0;
          continue;
        }
        const double M = Mf[bck(T, kf * kPencil + tx, (long long)(n + 1) * kPencil)];
        const bool right = __double_as_longlong(M) > 0;
        int up = right ? kf - 1 : kf;
        double aL = RS_P(E, up), aR = RS_P(E, up + 1);
        limit(RS_P(V, up), aL, aR);
        const double face = right ? aR : aL;
        T.fz[(size_t)s * fplane + (size_t)kf * ncol + col] = M * face;
      }
    }
    __syncthreads();
  }
#undef RS_P
}
#endif  // RS_STRICT

// ------------------------------------------------------------------ mixed precision
// Compensated FP32 transport.  Every transport value is carried as a double-float pair
// (value = h + l, |l| <= ulp(h)/2: two FP32 numbers, about 48 significant bits) and combined
// with error-free transformations (Knuth's TwoSum for sums, FMA-based TwoProduct for products),
// so the reconstruction runs on the FP32 pipe at FP64-class accuracy.  The face terms are written
// in advective form: for cell c and face f with air-mass flux M_f, the CWC tendency
//   m dq/dt = -div(M q) + q div(M) = sum_f sigma_f G_f M_f (q_c - q_f)
// (sigma_f = +1 on the east / north / top face, -1 on the west / south / bottom face, G_f the
// face's metric factor) needs only differences: q_c - q_f is minus the edge deviation when c is
// upwind, or minus (neighbour difference + edge deviation) when it is not.  With
//   Phi_f = M_f (q_f - q_L),  Psi_f = M_f (q_R - q_f)      (L / R: the cells below / above f)
// a cell's tendency is -G (Phi_e + Psi_w) along x, -(G_n Phi_n + G_s Psi_s) along y and
// -(Phi_t + Psi_b) vertically.  No term is of the size of q itself, so a value far smaller
// than its neighbours keeps its relative accuracy (an FP32 reconstruction of deviations does
// not: its error scales with the neighbour difference).  q == const gives exactly zero.
//
// Each direction's pencil adds its part of m dq/dt into a per-cell double-float accumulator
// (x writes it, y and z add), and the stage kernel turns it into the stage update in FP64.
// The state, the air mass, the stage combinations and the error norm stay FP64.
struct df {
  float h, l;
};
__device__ __forceinline__ df df_two_sum(float a, float b) {  // a + b = s + e exactly
  const float s = a + b, bb = s - a;
  return {s, (a - (s - bb)) + (b - bb)};
}
// Sum of pairs: TwoSum of the high parts, the low parts added to its error, then the fast
// renormalisation (h = s + e, l = e - (h - s)).  The renormalisation is exact unless the high
// parts cancel below the low parts; its error is then below 2^-46 max(|a|, |b|), a few times
// the operands' own representation error, so the sum keeps the pairs' accuracy at 11
// operations instead of the 14 of a second TwoSum.
__device__ __forceinline__ df df_add(df a, df b) {
  const df s = df_two_sum(a.h, b.h);
  const float e = s.l + (a.l + b.l);
  const float h = s.h + e;
  return {h, e - (h - s.h)};
}
__device__ __forceinline__ df df_neg(df a) { return {-a.h, -a.l}; }
__device__ __forceinline__ df df_sub(df a, df b) { return df_add(a, df_neg(b)); }
__device__ __forceinline__ df df_mul(df a, df b) {
  const float p = a.h * b.h;
  const float e = fmaf(a.h, b.l, fmaf(a.l, b.h, fmaf(a.h, b.h, -p)));
  const float s = p + e;
  return {s, e - (s - p)};
}
__device__ __forceinline__ df df_scale(df a, float pow2) { return {a.h * pow2, a.l * pow2}; }
__device__ __forceinline__ df df_ld(const float* H, const float* L, long long x) {
  return {H[x], L[x]};
}
__device__ __forceinline__ df df_ld2(const float2* p, size_t x) {
  const float2 v = p[x];
  return {v.x, v.y};
}
// 1/6 as a pair (hi = fl(1/6), lo = fl(1/6 - hi))
constexpr float kSixthH = (float)(1.0 / 6.0);
constexpr float kSixthL = (float)(1.0 / 6.0 - (double)(float)(1.0 / 6.0));

// |a| < |b| for pairs of the same sign (sg = +1 or -1 their sign)
__device__ __forceinline__ bool df_absless(df a, df b, float sg) {
  return (fabsf(a.h) < fabsf(b.h)) || (a.h == b.h && sg * a.l < sg * b.l);
}
// CW84 eq. 1.8 monotonised slope from the neighbour differences d0 (left) and d1 (right):
// 0 unless they have the same strict sign, else the smallest in magnitude of the centred
// slope da and 2 d0, 2 d1 (all three share that sign)
__device__ __forceinline__ df mc_pick(df d0, df d1, df da) {
  const bool same = (d0.h > 0.0f && d1.h > 0.0f) || (d0.h < 0.0f && d1.h < 0.0f);
  const float sg = d0.h > 0.0f ? 1.0f : -1.0f;
  df m = da;
  const df t0 = df_scale(d0, 2.0f), t1 = df_scale(d1, 2.0f);
  if (df_absless(t0, m, sg)) m = t0;
  if (df_absless(t1, m, sg)) m = t1;
  return same ? m : df{0.0f, 0.0f};
}
__device__ __forceinline__ df mc_slope(df d0, df d1) {
  return mc_pick(d0, d1, df_scale(df_add(d0, d1), 0.5f));
}
__device__ __forceinline__ df mc_slope_n(df d0, df d1, df sA, df sB) {  // dp-weighted centre
  return mc_pick(d0, d1, df_add(df_mul(sA, d1), df_mul(sB, d0)));
}
// CW84 eq. 1.10 limiter on the upwind cell's edge deviations (aL, aR) from its own value
// (a = 0): flatten unless aL and aR have strictly opposite signs, else steepen where the
// parabola overshoots; the tests dA a6 > dA^2 and -dA^2 > dA a6 of the FP64 form become sign
// tests of aL + 2 aR and 2 aL + aR.  Returns the limited right (M > 0) or left edge.
__device__ __forceinline__ df lim_pick(df aL, df aR, bool right) {
  const bool opp = (aR.h > 0.0f && aL.h < 0.0f) || (aR.h < 0.0f && aL.h > 0.0f);
  const float sR = aR.h > 0.0f ? 1.0f : -1.0f;
  const df t1 = df_add(aL, df_scale(aR, 2.0f));
  const df t2 = df_add(df_scale(aL, 2.0f), aR);
  const bool c1 = sR * t1.h < 0.0f;
  const bool c2 = !c1 && sR * t2.h > 0.0f;
  df r = right ? (c2 ? df_scale(aL, -2.0f) : aR) : (c1 ? df_scale(aR, -2.0f) : aL);
  return opp ? r : df{0.0f, 0.0f};
}
// Edge term E_p of cell p (the deviation of edge p+1/2 from cell p, unlimited), uniform grid:
// E_p = D_p / 2 - (S_{p+1} - S_p) / 6; the left edge of cell p is E_{p-1} - D_{p-1}.
__device__ __forceinline__ df edge_u(df Dp, df Sp, df Sp1) {
  return df_sub(df_scale(Dp, 0.5f), df_mul(df_sub(Sp1, Sp), df{kSixthH, kSixthL}));
}
// dp-weighted: E_p = ab D_p + c S_{p+1} + d S_p with the coefficients of edge p+1
__device__ __forceinline__ df edge_n(df Dp, df Sp, df Sp1, df ab, df c, df d) {
  return df_add(df_add(df_mul(ab, Dp), df_mul(c, Sp1)), df_mul(d, Sp));
}
// A cell's two faces along one direction: w (below, flux Mw) and e (above, flux Me).
// E(o), D(o) give E_{p+o}, D_{p+o}.  Returns {Psi_w, Phi_e}; a face with M == 0 (a wall)
// contributes exactly 0.
template <class FE, class FD>
__device__ __forceinline__ void cell_faces(df Mw, df Me, FE E, FD D, df& psi, df& phi) {
  psi = df{0.0f, 0.0f};
  phi = df{0.0f, 0.0f};
  if (Mw.h > 0.0f) {  // upwind p-1: its right edge
    const df dev = lim_pick(df_sub(E(-2), D(-2)), E(-1), true);
    psi = df_mul(Mw, df_sub(D(-1), dev));
  } else if (Mw.h < 0.0f) {  // upwind p: its left edge
    const df dev = lim_pick(df_sub(E(-1), D(-1)), E(0), false);
    psi = df_mul(Mw, df_neg(dev));
  }
  if (Me.h > 0.0f) {  // upwind p: its right edge
    const df dev = lim_pick(df_sub(E(-1), D(-1)), E(0), true);
    phi = df_mul(Me, dev);
  } else if (Me.h < 0.0f) {  // upwind p+1: its left edge
    const df dev = lim_pick(df_sub(E(0), D(0)), E(1), false);
    phi = df_mul(Me, df_add(D(0), dev));
  }
}
// split a double into a pair: production build with integer operations (split_bits below,
// truncating: hi + lo = v to 2^-47), strict build with conversions
__device__ __forceinline__ df split_df(double v);
// float -> double by re-biasing the exponent in the integer pipes (exact; zero kept, subnormal,
// inf and NaN convert)
__device__ __forceinline__ double f2d_bits(float x) {
  const unsigned u = __float_as_uint(x);
  const unsigned fe = (u >> 23) & 0xffu;
  if ((u << 1) == 0u) return __hiloint2double((int)(u & 0x80000000u), 0);
  if (fe == 0u || fe == 255u) return (double)x;
  return __hiloint2double((int)((u & 0x80000000u) | ((fe + 896u) << 20) | ((u & 0x7fffffu) >> 3)),
                          (int)(u << 29));
}
__device__ __forceinline__ double df_to_d(float2 v) {
#if RS_STRICT
  return (double)v.x + (double)v.y;
#else
  return f2d_bits(v.x) + f2d_bits(v.y);
#endif
}

// ---- bulk-copy staging (TMA): mbarrier with a transaction count, one elected issuing thread.
// Every wait is bounded: after kSpinLimit polls the block records the failure, stops the
// adaptive solve it belongs to, waits (bounded again) for its own copies and returns.
struct MixedTmaps {
  CUtensorMap yh[2], yl[2];  // lat pencils over qhi / qlo, box {pw, nlat, 1}; [0]: pw 16, [1]: 32
  CUtensorMap zh[2], zl[2];  // vertical pencils, box {pw, nlev, 1}
  bool x_ok, y_ok, z_ok;
};
constexpr int kSpinLimit = 1 << 24;
constexpr size_t kSmemAlignPad = 128;  // the launch adds this so the layout can start 128-aligned

__device__ __forceinline__ float* align128(unsigned char* p) {
  return reinterpret_cast<float*>((reinterpret_cast<uintptr_t>(p) + 127) & ~(uintptr_t)127);
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(unsigned long long* b) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(b)) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long* b, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(b)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_wait_bounded(unsigned long long* b, uint32_t parity) {
  for (int i = 0; i < kSpinLimit; ++i) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(smem_u32(b)), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* m, int c0, int c1, int c2,
                                            unsigned long long* b) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(m)), "r"(c0), "r"(c1), "r"(c2), "r"(smem_u32(b))
      : "memory");
}
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes,
                                          unsigned long long* b) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
          "r"(smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(b))
      : "memory");
}
// A staging wait ran out: flag it, stop the solve (every later kernel of the attempt returns on
// `done` and the controller ends the loop), then give this block's copies a bounded chance to
// land before the block's shared memory is released.
__device__ __noinline__ void staging_abort(int* err, const Ctl* ctl, unsigned long long* bar,
                                           int uses0, int uses1) {
  if (threadIdx.x == 0 && threadIdx.y == 0) {
    atomicOr(err, 1);
    if (ctl) atomicExch(const_cast<int*>(&ctl->done), 1);
    if (uses0 > 0) mbar_wait_bounded(bar, (uint32_t)((uses0 - 1) & 1));
    if (uses1 > 0) mbar_wait_bounded(bar + 1, (uint32_t)((uses1 - 1) & 1));
  }
}

// Shared-memory layout of the mixed pencils (floats, 128-byte aligned rows so that bulk copies
// can land in them): the staged hi / lo rows (two sets with bulk copies, so the next tracer's
// copy overlaps this tracer's work), then the pair rows of the neighbour differences D and the
// slopes S (interior cell p at row p + kHo), then the face air-mass fluxes as pairs.  After the
// differences are formed the current hi / lo rows hold the edge terms E.
constexpr int kHoX = 32;  // lon rows: interior starts 128 bytes into each row
constexpr int kHoP = 8;   // lat / vertical pencils: interior starts 8 pencil rows in
__host__ __device__ inline int mixed_rows_x(int n) { return (n + kHoX + 3 + 31) / 32 * 32; }
__host__ __device__ inline int mixed_rows_p(int n) { return (n + kHoP + 3 + 1) / 2 * 2; }
__host__ __device__ inline int mixed_frows(int n) { return (n + 1 + 31) / 32 * 32; }

// Lon rows: one block per (lat, level) row, blockIdx.y a group of sper tracers.
template <bool kTma>
__global__ void __launch_bounds__(256) k_adv_x_mixed(DevTransport<double> T, StageSel sel, int sper) {
  const double* Q;
  double g;
  if (!resolve_stage(sel, Q, g)) return;
  const df gd = split_df(g);  // the stage time factor as a pair
  const int s0 = blockIdx.y * sper, s1 = min(T.ntr, s0 + sper);  // this block's tracers
  extern __shared__ __align__(16) unsigned char smx32_raw[];
  float* smx32 = align128(smx32_raw);
  __shared__ __align__(8) unsigned long long bar[2];
  const int n = T.nlon, nf = n + 1, L = mixed_rows_x(n);
  float* const H0 = smx32;  // H[p + kHoX], p in [-3, n+2]
  float* const L0 = smx32 + L;
  float* const H1 = smx32 + (kTma ? 2 * L : 0);
  float* const L1 = smx32 + (kTma ? 3 * L : L);
  float* const Dh = smx32 + (kTma ? 4 : 2) * L;  // D[p] = q(p+1) - q(p), p in [-3, n+1]
  float* const Dl = Dh + L;
  float* const Sh = Dl + L;  // slopes of cells [-2, n+1]
  float* const Sl = Sh + L;
  float* const Mh = Sl + L;  // face fluxes [0, n] as pairs
  float* const Ml = Mh + mixed_frows(n);
  const int row = blockIdx.x;
  const int j = row % T.nlat, k = row / T.nlat;
  const size_t nc = (size_t)T.nlon * T.nlat * T.nlev;
  const long long nall = (long long)T.ntr * nc;
  const size_t rbase = ((size_t)k * T.nlat + j) * n;
  const bool periodic = T.lon_bc == 0;
  const int tid = threadIdx.x;
  const df G = df_ld2(T.gx2, j);
  auto X = [&](int p) { return bck(T, p + kHoX, L); };  // row index of cell p
  int uses0 = 0, uses1 = 0;  // copies issued per buffer
  auto issue = [&](int s, int b) {  // one tracer's interior hi / lo rows (n floats each)
    const size_t pb = (size_t)bck(T, (size_t)s * nc + rbase, nall - n + 1);
    fence_proxy_async();
    mbar_expect_tx(bar + b, (uint32_t)(2 * n * sizeof(float)));
    bulk_load((b ? H1 : H0) + kHoX, T.qhi + pb, (uint32_t)(n * sizeof(float)), bar + b);
    bulk_load((b ? L1 : L0) + kHoX, T.qlo + pb, (uint32_t)(n * sizeof(float)), bar + b);
  };
  if (kTma) {
    if (tid == 0) {
      mbar_init(bar);
      mbar_init(bar + 1);
      fence_mbar_init();
    }
    __syncthreads();
    if (tid == 0 && s0 < s1) issue(s0, 0);
    uses0 = s0 < s1;
  }
  for (int f = tid; f <= n; f += blockDim.x) {
    const df M = df_mul(gd, df_ld2(T.mx2, ((size_t)k * T.nlat + j) * nf + f));
    Mh[bck(T, f, mixed_frows(n))] = M.h;
    Ml[bck(T, f, mixed_frows(n))] = M.l;
  }
  for (int s = s0; s < s1; ++s) {
    const int it = s - s0, b = kTma ? (it & 1) : 0;
    float* H = b ? H1 : H0;
    float* Lo = b ? L1 : L0;
    const size_t pb = (size_t)s * nc + rbase;
    auto ghost = [&](int p, float& h, float& l) {  // p outside 0..n-1
      if (periodic) {
        const int q = ((p % n) + n) % n;
        h = T.qhi[bck(T, pb + q, nall)];
        l = T.qlo[bck(T, pb + q, nall)];
      } else {
        split_d((p < 0 ? T.qw : T.qe)[bck(T, ((size_t)s * T.nlev + k) * T.nlat + j,
                                          (long long)T.ntr * T.nlev * T.nlat)], h, l);
      }
    };
    if (kTma) {
      if (s + 1 < s1) {
        if (tid == 0) issue(s + 1, b ^ 1);
        if (b) uses0 += 1;
        else uses1 += 1;
      }
      if (tid < 6) {  // the three ghost cells on each side
        const int p = tid < 3 ? tid - 3 : n + tid - 3;
        float h, l;
        ghost(p, h, l);
        H[X(p)] = h;
        Lo[X(p)] = l;
      }
      const bool ok = mbar_wait_bounded(bar + b, (uint32_t)(((it >> 1)) & 1));
      if (__syncthreads_or(!ok)) {
        staging_abort(T.tma_err, sel.ctl, bar, uses0, uses1);
        return;
      }
    } else {
      for (int p = tid - 3; p <= n + 2; p += blockDim.x) {
        float h, l;
        if (p < 0 || p >= n) {
          ghost(p, h, l);
        } else {
          h = T.qhi[bck(T, pb + p, nall)];
          l = T.qlo[bck(T, pb + p, nall)];
        }
        H[X(p)] = h;
        Lo[X(p)] = l;
      }
      __syncthreads();
    }
    for (int p = tid - 3; p <= n + 1; p += blockDim.x) {
      const df d = df_sub(df_ld(H, Lo, X(p + 1)), df_ld(H, Lo, X(p)));
      Dh[X(p)] = d.h;
      Dl[X(p)] = d.l;
    }
    __syncthreads();
    for (int p = tid - 2; p <= n + 1; p += blockDim.x) {
      const df sl = mc_slope(df_ld(Dh, Dl, X(p - 1)), df_ld(Dh, Dl, X(p)));
      Sh[X(p)] = sl.h;
      Sl[X(p)] = sl.l;
    }
    __syncthreads();
    for (int p = tid - 2; p <= n; p += blockDim.x) {  // edge terms over the staged values
      const df e = edge_u(df_ld(Dh, Dl, X(p)), df_ld(Sh, Sl, X(p)), df_ld(Sh, Sl, X(p + 1)));
      H[X(p)] = e.h;
      Lo[X(p)] = e.l;
    }
    __syncthreads();
    for (int p = tid; p < n; p += blockDim.x) {
      df psi, phi;
      cell_faces(df{Mh[bck(T, p, nf)], Ml[bck(T, p, nf)]},
                 df{Mh[bck(T, p + 1, nf)], Ml[bck(T, p + 1, nf)]},
                 [&](int o) { return df_ld(H, Lo, X(p + o)); },
                 [&](int o) { return df_ld(Dh, Dl, X(p + o)); }, psi, phi);
      const df a = df_neg(df_mul(G, df_add(phi, psi)));
      T.acc[bck(T, pb + p, nall)] = make_float2(a.h, a.l);
    }
    __syncthreads();
  }
}

// Lat (DIR 1) and vertical (DIR 2) pencils: kPencil columns per block (threadIdx.x), the
// pencil's cells along threadIdx.y; rows [L][kPencil].  The lat pencils use the uniform
// reconstruction with the metric factors of the south and north faces, the vertical ones the
// dp-weighted coefficients; both add their part into the accumulator.
template <int DIR, int kPencil, bool kTma>
__global__ void __launch_bounds__(512) k_adv_yz_mixed(DevTransport<double> T, StageSel sel, int sper,
                                                      const __grid_constant__ CUtensorMap mh,
                                                      const __grid_constant__ CUtensorMap ml) {
  const double* Q;
  double g;
  if (!resolve_stage(sel, Q, g)) return;
  const df gd = split_df(g);  // the stage time factor as a pair
  const int s0 = blockIdx.y * sper, s1 = min(T.ntr, s0 + sper);  // this block's tracers
  extern __shared__ __align__(16) unsigned char smp32_raw[];
  float* smp32 = align128(smp32_raw);
  __shared__ __align__(8) unsigned long long bar[2];
  const int n = DIR == 1 ? T.nlat : T.nlev, L = mixed_rows_p(n);
  const int R = L * kPencil;  // one row set [L][kPencil], cell p at row p + kHoP
  float* const H0 = smp32;
  float* const L0 = smp32 + R;
  float* const H1 = smp32 + (kTma ? 2 * R : 0);
  float* const L1 = smp32 + (kTma ? 3 * R : R);
  float* const Dh = smp32 + (kTma ? 4 : 2) * R;
  float* const Dl = Dh + R;
  float* const Sh = Dl + R;
  float* const Sl = Sh + R;
  float* const Mh = Sl + R;  // [n+1][kPencil]
  float* const Ml = Mh + (n + 1) * kPencil;
  const int tx = threadIdx.x, ty = threadIdx.y;
  const bool lead = tx == 0 && ty == 0;
  const size_t ncol = (size_t)T.nlon * T.nlat;
  const size_t nc = ncol * T.nlev;
  const long long nall = (long long)T.ntr * nc;
  const long long mb = (long long)(n + 1) * kPencil;
  // DIR 1: blockIdx.x = (lon tile, level); DIR 2: blockIdx.x = column tile
  const int ntile = (T.nlon + kPencil - 1) / kPencil;
  const int k = DIR == 1 ? (int)(blockIdx.x / ntile) : 0;
  const int i0 = DIR == 1 ? (int)(blockIdx.x % ntile) * kPencil : 0;
  const size_t col0 = DIR == 2 ? (size_t)blockIdx.x * kPencil : 0;
  const int i = i0 + tx;
  const size_t col = col0 + tx;
  const bool live = DIR == 1 ? i < T.nlon : col < ncol;
  const size_t stride = DIR == 1 ? (size_t)T.nlon : ncol;  // cell p to p+1
  const size_t cbase = DIR == 1 ? (size_t)k * ncol + i : col;  // cell 0 of the pencil
  const bool open = DIR == 1 && T.lat_bc == 1;
  int uses0 = 0, uses1 = 0;  // copies issued per buffer
  auto issue = [&](int s, int b) {  // interior rows 0..n-1: box {kPencil, n, 1}
    if (RS_BOUNDS_CHECK) {  // box starts inside the tensor
      bck(T, DIR == 1 ? i0 : (long long)col0, DIR == 1 ? T.nlon : (long long)ncol);
      bck(T, DIR == 1 ? k + s * T.nlev : s, DIR == 1 ? (long long)T.nlev * T.ntr : T.ntr);
    }
    fence_proxy_async();
    mbar_expect_tx(bar + b, (uint32_t)(2 * n * kPencil * sizeof(float)));
    if (DIR == 1) {
      tma_load_3d((b ? H1 : H0) + kHoP * kPencil, &mh, i0, 0, k + s * T.nlev, bar + b);
      tma_load_3d((b ? L1 : L0) + kHoP * kPencil, &ml, i0, 0, k + s * T.nlev, bar + b);
    } else {
      tma_load_3d((b ? H1 : H0) + kHoP * kPencil, &mh, (int)col0, 0, s, bar + b);
      tma_load_3d((b ? L1 : L0) + kHoP * kPencil, &ml, (int)col0, 0, s, bar + b);
    }
  };
  if (kTma) {
    if (lead) {
      mbar_init(bar);
      mbar_init(bar + 1);
      fence_mbar_init();
    }
    __syncthreads();
    if (lead && s0 < s1) issue(s0, 0);
    uses0 = s0 < s1;
  }
#define RS_P(a, p) a[bck(T, ((p) + kHoP) * kPencil + tx, R)]
  if (live)
    for (int f = ty; f <= n; f += blockDim.y) {
      df M{0.0f, 0.0f};
      if (DIR == 1) {
        if (open || (f > 0 && f < n))  // closed walls: no flux through the poles
          M = df_mul(gd, df_ld2(T.my2, ((size_t)k * (n + 1) + f) * T.nlon + i));
      } else if (f > 0 && f < n) {  // no flux through the surface and the model top
        M = df_mul(gd, df_ld2(T.mz2, (size_t)f * ncol + col));
      }
      Mh[bck(T, f * kPencil + tx, mb)] = M.h;
      Ml[bck(T, f * kPencil + tx, mb)] = M.l;
    }
  for (int s = s0; s < s1; ++s) {
    const int it = s - s0, b = kTma ? (it & 1) : 0;
    float* H = b ? H1 : H0;
    float* Lo = b ? L1 : L0;
    const size_t pb = (size_t)s * nc + cbase;
    auto cell = [&](int p, float& h, float& l) {  // a ghost (p outside 0..n-1) or interior cell
      h = 0.0f;
      l = 0.0f;
      if (!live) return;
      if (p < 0 || p >= n) {
        if (open) {
          split_d((p < 0 ? T.qs : T.qn)[bck(T, ((size_t)s * T.nlev + k) * T.nlon + i,
                                            (long long)T.ntr * T.nlev * T.nlon)], h, l);
          return;
        }
        p = p < 0 ? -1 - p : 2 * n - 1 - p;  // mirror ghosts at the walls
      }
      h = T.qhi[bck(T, pb + (size_t)p * stride, nall)];
      l = T.qlo[bck(T, pb + (size_t)p * stride, nall)];
    };
    if (kTma) {
      if (s + 1 < s1) {
        if (lead) issue(s + 1, b ^ 1);
        if (b) uses0 += 1;
        else uses1 += 1;
      }
      for (int r = ty; r < 6; r += blockDim.y) {
        const int p = r < 3 ? r - 3 : n + r - 3;
        float h, l;
        cell(p, h, l);
        RS_P(H, p) = h;
        RS_P(Lo, p) = l;
      }
      const bool ok = mbar_wait_bounded(bar + b, (uint32_t)((it >> 1) & 1));
      if (__syncthreads_or(!ok)) {
        staging_abort(T.tma_err, sel.ctl, bar, uses0, uses1);
        return;
      }
    } else {
      for (int p = (int)ty - 3; p <= n + 2; p += blockDim.y) {
        float h, l;
        cell(p, h, l);
        RS_P(H, p) = h;
        RS_P(Lo, p) = l;
      }
      __syncthreads();
    }
    for (int p = (int)ty - 3; p <= n + 1; p += blockDim.y) {
      const df d = df_sub(df{RS_P(H, p + 1), RS_P(Lo, p + 1)}, df{RS_P(H, p), RS_P(Lo, p)});
      RS_P(Dh, p) = d.h;
      RS_P(Dl, p) = d.l;
    }
    __syncthreads();
    for (int p = (int)ty - 2; p <= n + 1; p += blockDim.y) {
      const df d0{RS_P(Dh, p - 1), RS_P(Dl, p - 1)}, d1{RS_P(Dh, p), RS_P(Dl, p)};
      df sl{0.0f, 0.0f};
      if (DIR == 1) {
        sl = mc_slope(d0, d1);
      } else if (p >= -1 && p <= n && live) {  // slopes of cells -1..n (coefficient row p+1)
        const size_t x = bck(T, (size_t)(p + 1) * ncol + col, (long long)(n + 2) * ncol);
        sl = mc_slope_n(d0, d1, df_ld2(T.vsA2, x), df_ld2(T.vsB2, x));
      }
      RS_P(Sh, p) = sl.h;
      RS_P(Sl, p) = sl.l;
    }
    __syncthreads();
    // edge terms over the staged values: cells -2..n (uniform), -1..n-1 (coefficient rows
    // 0..n of the dp-weighted edges)
    for (int p = (int)ty - 2; p <= n; p += blockDim.y) {
      const df Dp{RS_P(Dh, p), RS_P(Dl, p)};
      const df Sp{RS_P(Sh, p), RS_P(Sl, p)}, Sp1{RS_P(Sh, p + 1), RS_P(Sl, p + 1)};
      df e{0.0f, 0.0f};
      if (DIR == 1) {
        e = edge_u(Dp, Sp, Sp1);
      } else if (p >= -1 && p <= n - 1 && live) {
        const size_t x = bck(T, (size_t)(p + 1) * ncol + col, (long long)(n + 1) * ncol);
        e = edge_n(Dp, Sp, Sp1, df_ld2(T.veAB2, x), df_ld2(T.veC2, x), df_ld2(T.veD2, x));
      }
      RS_P(H, p) = e.h;
      RS_P(Lo, p) = e.l;
    }
    __syncthreads();
    if (live) {
      for (int p = ty; p < n; p += blockDim.y) {
        df psi, phi;
        cell_faces(df{Mh[bck(T, p * kPencil + tx, mb)], Ml[bck(T, p * kPencil + tx, mb)]},
                   df{Mh[bck(T, (p + 1) * kPencil + tx, mb)], Ml[bck(T, (p + 1) * kPencil + tx, mb)]},
                   [&](int o) { return df{RS_P(H, p + o), RS_P(Lo, p + o)}; },
                   [&](int o) { return df{RS_P(Dh, p + o), RS_P(Dl, p + o)}; }, psi, phi);
        df a;
        if (DIR == 1)
          a = df_neg(df_add(df_mul(df_ld2(T.gyhi2, p), phi), df_mul(df_ld2(T.gylo2, p), psi)));
        else
          a = df_neg(df_add(phi, psi));
        const size_t x = bck(T, pb + (size_t)p * stride, nall);
        const float2 o = T.acc[x];
        const df t = df_add(df{o.x, o.y}, a);
        T.acc[x] = make_float2(t.h, t.l);
      }
    }
    __syncthreads();
  }
#undef RS_P
}

// ---- streaming forms of the mixed pencils (no shared memory, no barriers).  The same pair
// operations in the same order as k_adv_x_mixed / k_adv_yz_mixed, so the accumulators are bit
// for bit those of the pencils; rs_autotune picks per direction.
//
// Lon rows: one warp per segment of kSegX = 26 cells of a row; lane l holds cell
// p = base - 3 + l, and the neighbour values the stencil needs move between lanes by shuffles.
// Lane l computes the limited deviation of face p (its west face); cells at lanes 3..28 have
// all of D(p-2..p), E(p-2..p+1) and their east face's Phi from lane l+1.
constexpr int kSegX = 26;
__device__ __forceinline__ df shfl_up_df(df v, int d) {
  return {__shfl_up_sync(0xffffffffu, v.h, d), __shfl_up_sync(0xffffffffu, v.l, d)};
}
__device__ __forceinline__ df shfl_down_df(df v, int d) {
  return {__shfl_down_sync(0xffffffffu, v.h, d), __shfl_down_sync(0xffffffffu, v.l, d)};
}
// Face f's two pair terms from the upwind cell's edges: Psi_f (for cell f) and Phi_f (for cell
// f-1).  E(o), D(o) give E_{f+o}, D_{f+o}.  The expressions of cell_faces, so the same bits.
template <class FE, class FD>
__device__ __forceinline__ void face_terms(df M, FE E, FD D, df& psi, df& phi) {
  psi = df{0.0f, 0.0f};
  phi = df{0.0f, 0.0f};
  if (M.h > 0.0f) {  // upwind f-1: its right edge
    const df dev = lim_pick(df_sub(E(-2), D(-2)), E(-1), true);
    psi = df_mul(M, df_sub(D(-1), dev));
    phi = df_mul(M, dev);
  } else if (M.h < 0.0f) {  // upwind f: its left edge
    const df dev = lim_pick(df_sub(E(-1), D(-1)), E(0), false);
    psi = df_mul(M, df_neg(dev));
    phi = df_mul(M, df_add(D(-1), dev));
  }
}

__global__ void __launch_bounds__(128) k_adv_x_stream(DevTransport<double> T, StageSel sel,
                                                      int sper) {
  const double* Q;
  double g;
  if (!resolve_stage(sel, Q, g)) return;
  const df gd = split_df(g);  // the stage time factor as a pair
  const int n = T.nlon, nf = n + 1;
  const int nseg = (n + kSegX - 1) / kSegX;
  const int lane = threadIdx.x & 31;
  const long long wg = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (wg >= (long long)nseg * T.nlat * T.nlev) return;  // whole warps leave together
  const int row = (int)(wg / nseg), seg = (int)(wg % nseg);
  const int j = row % T.nlat, k = row / T.nlat;
  const int p = seg * kSegX - 3 + lane;  // this lane's cell (and west face)
  const size_t nc = (size_t)T.nlon * T.nlat * T.nlev;
  const long long nall = (long long)T.ntr * nc;
  const size_t rbase = ((size_t)k * T.nlat + j) * n;
  const bool periodic = T.lon_bc == 0;
  const df G = df_ld2(T.gx2, j);
  const df M = (p >= 0 && p <= n) ? df_mul(gd, df_ld2(T.mx2, ((size_t)k * T.nlat + j) * nf + p))
                                   : df{0.0f, 0.0f};
  const bool out = lane >= 3 && lane <= 28 && p >= 0 && p < n;
  const int s0 = blockIdx.y * sper, s1 = min(T.ntr, s0 + sper);
  for (int s = s0; s < s1; ++s) {
    const size_t pb = (size_t)s * nc + rbase;
    df q;
    if (p >= 0 && p < n) {
      q = df{T.qhi[bck(T, pb + p, nall)], T.qlo[bck(T, pb + p, nall)]};
    } else if (periodic) {
      const int w = ((p % n) + n) % n;
      q = df{T.qhi[bck(T, pb + w, nall)], T.qlo[bck(T, pb + w, nall)]};
    } else {
      split_d((p < 0 ? T.qw : T.qe)[bck(T, ((size_t)s * T.nlev + k) * T.nlat + j,
                                        (long long)T.ntr * T.nlev * T.nlat)], q.h, q.l);
    }
    const df D = df_sub(shfl_down_df(q, 1), q);                 // D(p), lanes 0..30
    const df S = mc_slope(shfl_up_df(D, 1), D);                 // S(p), lanes 1..30
    const df E = edge_u(D, S, shfl_down_df(S, 1));              // E(p), lanes 1..29
    const df Dm1 = shfl_up_df(D, 1), Dm2 = shfl_up_df(D, 2);
    const df Em1 = shfl_up_df(E, 1), Em2 = shfl_up_df(E, 2);
    df psi, phi;
    face_terms(M, [&](int o) { return o == 0 ? E : (o == -1 ? Em1 : Em2); },
               [&](int o) { return o == -1 ? Dm1 : Dm2; }, psi, phi);
    const df phie = shfl_down_df(phi, 1);  // the east face's Phi, computed by lane + 1
    if (out) {
      const df a = df_neg(df_mul(G, df_add(phie, psi)));
      T.acc[bck(T, pb + p, nall)] = make_float2(a.h, a.l);
    }
  }
}

// Lat (DIR 1) and vertical (DIR 2) lines: one thread per line (consecutive lon points at one
// level, or consecutive columns), walking the line once per tracer with a register window:
// when q(p) arrives, D(p-1), S(p-1), E(p-2) are formed and face p-2 is complete; its Phi
// closes cell p-3 and its Psi opens cell p-2.
template <int DIR>
__global__ void __launch_bounds__(128) k_adv_yz_stream(DevTransport<double> T, StageSel sel,
                                                       int sper) {
  const double* Q;
  double g;
  if (!resolve_stage(sel, Q, g)) return;
  const df gd = split_df(g);  // the stage time factor as a pair
  const int n = DIR == 1 ? T.nlat : T.nlev;
  const size_t ncol = (size_t)T.nlon * T.nlat;
  const size_t nc = ncol * T.nlev;
  const long long nall = (long long)T.ntr * nc;
  const int ntile = (T.nlon + (int)blockDim.x - 1) / (int)blockDim.x;
  const int k = DIR == 1 ? (int)(blockIdx.x / ntile) : 0;
  const int i = DIR == 1 ? (int)(blockIdx.x % ntile) * (int)blockDim.x + (int)threadIdx.x : 0;
  const size_t col = DIR == 2 ? (size_t)blockIdx.x * blockDim.x + threadIdx.x : 0;
  if (DIR == 1 ? i >= T.nlon : col >= ncol) return;
  const size_t stride = DIR == 1 ? (size_t)T.nlon : ncol;
  const size_t cbase = DIR == 1 ? (size_t)k * ncol + i : col;
  const bool open = DIR == 1 && T.lat_bc == 1;
  auto flux = [&](int f) -> df {  // face f's air-mass flux, zero through closed walls
    if (DIR == 1) {
      if (open || (f > 0 && f < n)) return df_mul(gd, df_ld2(T.my2, ((size_t)k * (n + 1) + f) * T.nlon + i));
    } else if (f > 0 && f < n) {
      return df_mul(gd, df_ld2(T.mz2, (size_t)f * ncol + col));
    }
    return df{0.0f, 0.0f};
  };
  const int s0 = blockIdx.y * sper, s1 = min(T.ntr, s0 + sper);
  for (int s = s0; s < s1; ++s) {
    const size_t pb = (size_t)s * nc + cbase;
    auto load = [&](int p) -> df {
      if (p < 0 || p >= n) {
        if (open) {
          df v;
          split_d((p < 0 ? T.qs : T.qn)[bck(T, ((size_t)s * T.nlev + k) * T.nlon + i,
                                            (long long)T.ntr * T.nlev * T.nlon)], v.h, v.l);
          return v;
        }
        p = p < 0 ? -1 - p : 2 * n - 1 - p;  // mirror ghosts at the walls
      }
      const size_t x = bck(T, pb + (size_t)p * stride, nall);
      return df{T.qhi[x], T.qlo[x]};
    };
    const df z{0.0f, 0.0f};
    // window: qp = q(p-1); D4..D1 = D(p-4..p-1); S2, S1 = S(p-2), S(p-1); E4..E2 = E(p-4..p-2)
    df qp = load(-3), D4 = z, D3 = z, D2 = z, D1 = z, S2 = z, S1 = z, E4 = z, E3 = z, E2 = z;
    df psi_prev = z;  // Psi of the previous face (the open cell's west face)
    // one iteration ahead: q(p), the flux of face p-2 and the accumulator of cell p-3
    df q_nx = load(-2), m_nx = z;
    float2 a_nx = make_float2(0.0f, 0.0f);
    for (int p = -2; p <= n + 2; ++p) {
      const df qn = q_nx, Mf = m_nx;
      const float2 o = a_nx;
      if (p < n + 2) q_nx = load(p + 1);
      if (p - 1 >= 0 && p - 1 <= n) m_nx = flux(p - 1);
      if (p - 2 >= 0 && p - 2 < n) a_nx = T.acc[bck(T, pb + (size_t)(p - 2) * stride, nall)];
      D4 = D3; D3 = D2; D2 = D1;
      D1 = df_sub(qn, qp);  // D(p-1)
      qp = qn;
      S2 = S1;
      const int ps = p - 1;  // the slope formed now
      if (DIR == 1) {
        S1 = mc_slope(D2, D1);
      } else if (ps >= -1 && ps <= n) {  // slopes of cells -1..n (coefficient row ps+1)
        const size_t x = bck(T, (size_t)(ps + 1) * ncol + col, (long long)(n + 2) * ncol);
        S1 = mc_slope_n(D2, D1, df_ld2(T.vsA2, x), df_ld2(T.vsB2, x));
      } else {
        S1 = z;
      }
      E4 = E3; E3 = E2;
      const int pe = p - 2;  // the edge term formed now: E(pe) from D(pe), S(pe), S(pe+1)
      if (DIR == 1) {
        E2 = edge_u(D2, S2, S1);
      } else if (pe >= -1 && pe <= n - 1) {
        const size_t x = bck(T, (size_t)(pe + 1) * ncol + col, (long long)(n + 1) * ncol);
        E2 = edge_n(D2, S2, S1, df_ld2(T.veAB2, x), df_ld2(T.veC2, x), df_ld2(T.veD2, x));
      } else {
        E2 = z;
      }
      const int f = p - 2;  // the face now complete (needs E(f-2..f), D(f-2..f-1))
      if (f < 0 || f > n) continue;
      df psi, phi;
      face_terms(Mf, [&](int o) { return o == 0 ? E2 : (o == -1 ? E3 : E4); },
                 [&](int o) { return o == -1 ? D3 : D4; }, psi, phi);
      if (f >= 1) {  // cell f-1 is complete: its east face f, west face f-1
        const int c = f - 1;
        df a;
        if (DIR == 1)
          a = df_neg(df_add(df_mul(df_ld2(T.gyhi2, c), phi), df_mul(df_ld2(T.gylo2, c), psi_prev)));
        else
          a = df_neg(df_add(phi, psi_prev));
        const size_t x = bck(T, pb + (size_t)c * stride, nall);
        const df t = df_add(df{o.x, o.y}, a);
        T.acc[x] = make_float2(t.h, t.l);
      }
      psi_prev = psi;
    }
  }
}

// ------------------------------------------------------------------ stage kernel
#if !RS_STRICT
// hi + lo split without FP64-pipe conversions (production build): hi = v truncated to 24
// significant bits, lo = the next 24 bits of the remainder, truncated -- hi + lo = v to 2^-47
// relative.  Values outside [2^-74, 2^127) (zero, subnormals, inf, NaN included) convert.
__device__ __forceinline__ void split_bits(double v, float& hi, float& lo) {
  const unsigned h = (unsigned)__double2hiint(v), l = (unsigned)__double2loint(v);
  const int e = (int)((h >> 20) & 0x7ff);
  if (e < 949 || e > 1150) {
    hi = (float)v;
    lo = (float)(v - (double)hi);
    return;
  }
  const unsigned sign = h & 0x80000000u;
  hi = __uint_as_float(sign | ((unsigned)(e - 896) << 23) | ((h & 0xfffffu) << 3) | (l >> 29));
  const unsigned r = l & 0x1fffffffu;  // the 29 mantissa bits below hi
  if (r == 0) {
    lo = 0.0f;
    return;
  }
  const int t = 31 - __clz((int)r);  // leading bit of r, 0..28
  const unsigned mant = t >= 23 ? (r >> (t - 23)) : (r << (23 - t));
  lo = __uint_as_float(sign | ((unsigned)(e - 948 + t) << 23) | (mant & 0x7fffffu));
}
#endif
__device__ __forceinline__ void split_store(const DevTransport<double>& T, size_t x, double v) {
  float hi, lo;
#if RS_STRICT
  hi = (float)v;
  lo = (float)(v - (double)hi);
#else
  split_bits(v, hi, lo);
#endif
  T.qhi[x] = hi;
  T.qlo[x] = lo;
}
__device__ __forceinline__ df split_df(double v) {
  df r;
#if RS_STRICT
  r.h = (float)v;
  r.l = (float)(v - (double)r.h);
#else
  split_bits(v, r.h, r.l);
#endif
  return r;
}

// (hi, lo) pairs of a double array (the air-mass face fluxes of the mixed kernels)
__global__ void k_make_pairs(const double* __restrict__ src, float2* __restrict__ dst, size_t n) {
  const size_t x = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (x < n) {
    const df v = split_df(src[x]);
    dst[x] = make_float2(v.h, v.l);
  }
}
void launch_make_pairs(cudaStream_t st, const double* src, float2* dst, size_t n) {
  if (n) k_make_pairs<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(src, dst, n);
}

// split the attempt's input state U[cur] (stage 1's RHS argument) into hi/lo planes
__global__ void __launch_bounds__(kRedThreads) k_split_input(DevTransport<double> T,
                                                             const Ctl* __restrict__ ctl,
                                                             const double* __restrict__ U0,
                                                             const double* __restrict__ U1,
                                                             const double* __restrict__ Qd) {
  const double* U;
  if (ctl) {
    if (ctl->done) return;
    U = ctl->cur ? U1 : U0;
  } else {
    U = Qd;
  }
  // four elements per thread, a block's 4 x 256 consecutive values: the loads go out
  // together
  const size_t n = (size_t)T.ntr * T.nlon * T.nlat * T.nlev;
  const size_t x0 = (size_t)blockIdx.x * (4 * blockDim.x) + threadIdx.x;
  double v[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const size_t x = x0 + (size_t)r * blockDim.x;
    v[r] = x < n ? U[x] : 0.0;
  }
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const size_t x = x0 + (size_t)r * blockDim.x;
    if (x < n) split_store(T, x, v[r]);
  }
}
// Divergence of the air-mass flux at cell (i,j,k) at time factor g.
struct CellGeo {
  double gx, gylo, gyhi;
};
// The six air-mass face fluxes of cell (i,j,k) at time factor g, zero through closed walls.
struct MassFluxes {
  double w, e, s, n, b, t;
};
__device__ __forceinline__ MassFluxes mass_fluxes(const DevTransport<double>& T, int i, int j,
                                                  int k, double g) {
  const int nf = T.nlon + 1;
  const size_t ncol = (size_t)T.nlon * T.nlat, col = (size_t)j * T.nlon + i;
  MassFluxes F;
  F.w = g * T.mx[((size_t)k * T.nlat + j) * nf + i];
  F.e = g * T.mx[((size_t)k * T.nlat + j) * nf + i + 1];
  F.s = (T.lat_bc != 1 && j == 0) ? 0.0 : g * T.my[((size_t)k * (T.nlat + 1) + j) * T.nlon + i];
  F.n = (T.lat_bc != 1 && j + 1 == T.nlat) ? 0.0
      : g * T.my[((size_t)k * (T.nlat + 1) + j + 1) * T.nlon + i];
  F.b = (k == 0) ? 0.0 : g * T.mz[(size_t)k * ncol + col];
  F.t = (k + 1 == T.nlev) ? 0.0 : g * T.mz[(size_t)(k + 1) * ncol + col];
  return F;
}
// horizontal (DxM + DyM) and vertical (DzM) parts of the air-mass flux divergence
__device__ __forceinline__ void div_parts(const MassFluxes& F, const CellGeo& G, double& hz,
                                          double& vz) {
  double DxM = (F.e - F.w) * G.gx;
  double DyM = F.n * G.gyhi - F.s * G.gylo;
  hz = DxM + DyM;
  vz = F.t - F.b;
}
__device__ __forceinline__ void div_parts(const DevTransport<double>& T, int i, int j, int k,
                                          double g, const CellGeo& G, double& hz, double& vz) {
  div_parts(mass_fluxes(T, i, j, k, g), G, hz, vz);
}
#if RS_STRICT
__device__ __forceinline__ double div_m(const DevTransport<double>& T, int i, int j, int k,
                                        double g, const CellGeo& G) {
  double hz, vz;
  div_parts(T, i, j, k, g, G, hz, vz);
  return hz + vz;
}
#endif
// air-mass tendency: -divM, or with the pressure fixer -((divh + corr) + DzM)
__device__ __forceinline__ double dm_dt(const DevTransport<double>& T, int i, int j, int k,
                                        double g, const CellGeo& G, size_t c) {
  double hz, vz;
  div_parts(T, i, j, k, g, G, hz, vz);
  return T.mcorr ? -((hz + T.mcorr[c]) + vz) : -(hz + vz);
}

// Full PBL mixing (reseact.esm Transport3D pbl_sum_* / pbl_mean_*): per tracer and column the
// PBL mean qbar = sum_k w_k q_k / den, summed from the surface up as the reference's column
// aggregate; the stage kernels add pbl_f * (qbar - q) / tau to each tracer tendency.
__global__ void __launch_bounds__(kRedThreads) k_pbl_mean(DevTransport<double> T, StageSel sel) {
  const double* Q;
  double g;
  if (!resolve_stage(sel, Q, g)) return;
  const size_t ncol = (size_t)T.nlon * T.nlat, nc = ncol * T.nlev;
  const size_t id = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (id >= (size_t)T.ntr * ncol) return;
  const size_t s = id / ncol, col = id % ncol;
  const double* q = Q + s * nc + col;
  double acc = 0.0;
  if (T.mixed) {  // the stage input is the pencils' (hi, lo) planes
    for (int k = 0; k < T.nlev; ++k) {
      const size_t x = s * nc + (size_t)k * ncol + col;
      acc = acc + T.pbl_w[(size_t)k * ncol + col] * df_to_d(make_float2(T.qhi[x], T.qlo[x]));
    }
  } else {
    for (int k = 0; k < T.nlev; ++k) acc = acc + T.pbl_w[(size_t)k * ncol + col] * q[(size_t)k * ncol];
  }
  T.pbl_qbar[id] = acc / T.pbl_den[col];
}

__device__ __forceinline__ double pbl_term(const DevTransport<double>& T, size_t c, size_t col,
                                           int s, double q) {
  const double pb = T.pbl_f[c] * (T.pbl_qbar[(size_t)s * T.nlon * T.nlat + col] - q);
#if RS_STRICT
  return pb / T.pbl_tau;
#else
  return pb * T.pbl_rtau;
#endif
}

static void launch_pbl_mean(cudaStream_t st, const DevTransport<double>& T, const StageSel& sel) {
  size_t n = (size_t)T.ntr * T.nlon * T.nlat;
  k_pbl_mean<<<(unsigned)((n + kRedThreads - 1) / kRedThreads), kRedThreads, 0, st>>>(T, sel);
}

#if RS_STRICT
// stage in 1..4.  Qin: the field whose fluxes were computed (RHS argument).
//   1: S1 = U + dt/2 f(U)           2: S2 = S1 + dt/2 f(S1)
//   3: S1 = u3 = S2 + dt/2 f(S2), S3 = u4 = 2/3 U + 1/3 u3
//   4: unew = S3 + dt/2 f(S3); err = 1/2 (1/3 U + 2/3 u3 - unew); candidate = clamp(unew)
template <int STAGE>
__global__ void __launch_bounds__(kRedThreads) k_stage(DevTransport<double> T,
                                                       const Ctl* __restrict__ ctl,
                                                       TransportBufs B, double rtol,
                                                       double atol, int clamp) {
  __shared__ double sm[kRedThreads];
  if (ctl->done) return;
  const double g = ctl->g[STAGE - 1];
  const int cur = ctl->cur;
  const double* U = cur ? B.U1 : B.U0;
  double* Un = cur ? B.U0 : B.U1;
  const double dt = ctl->dtc;
  const double dt_2 = dt / 2;
  const double* Qin = STAGE == 1 ? U : (STAGE == 2 ? B.S1 : (STAGE == 3 ? B.S2 : B.S3));
  const size_t nc = (size_t)T.nlon * T.nlat * T.nlev;
  size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  // transport stage tape (recording): this stage's tendency at Fo, its output state (stages
  // 1-3: V1, V2, V4) at Vo, in the slot of the accepted count
  double* Fo = nullptr;
  double* Vo = nullptr;
  if (ctl->ftape) {
    const int slot = (int)ctl->nacc;
    if (slot >= 0 && slot < ctl->fcap) {
      const size_t nst = nc * (size_t)T.nsp;
      double* rec = ctl->ftape + (size_t)slot * 7 * nst;
      Fo = rec + (size_t)(STAGE - 1) * nst;
      if (STAGE < 4) Vo = rec + (size_t)(3 + STAGE) * nst;
    }
  }
  double e = 0.0;
  if (c < nc) {
    int i = (int)(c % T.nlon);
    int j = (int)((c / T.nlon) % T.nlat);
    int k = (int)(c / ((size_t)T.nlon * T.nlat));
    CellGeo G{T.gx[j], T.gylo[j], T.gyhi[j]};
    // the air-mass divergence, once per cell: tracers and the air-mass row
    const MassFluxes F = mass_fluxes(T, i, j, k, g);
    double hz, vz;
    div_parts(F, G, hz, vz);
    const double divM = hz + vz;
    const double dmdt = T.mcorr ? -((hz + T.mcorr[c]) + vz) : -(hz + vz);  // = dm_dt(...)
    double m = Qin[(size_t)(T.nsp - 1) * nc + c];
    const int nfx = T.nlon + 1, nfy = T.nlat + 1;
    const size_t ncol = (size_t)T.nlon * T.nlat, col = (size_t)j * T.nlon + i;
    const size_t fxp = (size_t)T.nlev * T.nlat * nfx, fyp = (size_t)T.nlev * nfy * T.nlon,
                 fzp = ncol * (T.nlev + 1);
    const size_t fxi = ((size_t)k * T.nlat + j) * nfx + i;
    const size_t fyi = ((size_t)k * nfy + j) * T.nlon + i;
    const size_t fzi = (size_t)k * ncol + col;
    for (int s = 0; s < T.nsp; ++s) {
      size_t x = (size_t)s * nc + c;
      double q = Qin[x];
      // the stage's new value is q + dt/2 * f: nx = q + dt_2 * du (strict: the oracle's
      // expression order); the production build forms it as fma(du, scale, q), folding 1/m
      // into the scale when no PBL term is added
      double du;
      if (s < T.ntr) {
        double fw = T.fx[s * fxp + fxi], fe = T.fx[s * fxp + fxi + 1];
        double fs = T.fy[s * fyp + fyi], fn = T.fy[s * fyp + fyi + T.nlon];
        double fb = T.fz[s * fzp + fzi], ft = T.fz[s * fzp + fzi + ncol];
        double Dx = (fe - fw) * G.gx;
        double Dy = fn * G.gyhi - fs * G.gylo;
        double Dz = ft - fb;
        double a = -((Dx + Dy) + Dz);
        double b = q * divM;
        du = (a + b) / m;
        if (T.pbl) du = du + pbl_term(T, c, col, s, q);
      } else {
        du = dmdt;
      }
      const double nx = q + dt_2 * du;
      if (Fo) Fo[x] = du;
      if (STAGE == 1) {
        B.S1[x] = nx;
        if (Vo) Vo[x] = nx;
      } else if (STAGE == 2) {
        B.S2[x] = nx;
        if (Vo) Vo[x] = nx;
      } else if (STAGE == 3) {
        double u3 = nx;
        double u0 = U[x];
        B.S1[x] = u3;
        double u4 = (2.0 / 3.0) * u0 + (1.0 / 3.0) * u3;
        B.S3[x] = u4;
        if (Vo) Vo[x] = u4;
      } else {
        double u0 = U[x];
        double u3 = B.S1[x];
        double un = nx;
        double ut = (1.0 / 3.0) * u0 + (2.0 / 3.0) * u3;
        double err = 0.5 * (ut - un);
        double am = fmax(fabs(u0), fabs(un));
        double den = am * rtol + atol;
        double at = err / den;
        e = e + at * at;
        Un[x] = clamp ? fmax(un, 0.0) : un;
      }
    }
  }
  if (STAGE == 4) {
    double tot = block_tree256(e, sm);
    if (threadIdx.x == 0) B.partial[blockIdx.x] = tot;
  }
}
#endif  // RS_STRICT
#include "rs_adv64.cuh"

// Compensated-FP32 stage kernel (mixed precision).  The tracers of stages 1-3 stay pairs:
// the stage input is the pencils' own (hi, lo) planes, the update q + dt/2 * (m dq/dt) / m is
// formed in pairs and written back into those planes (in place: the update is pointwise), u3
// is kept as pairs in the tracer part of S1; only stage 4 returns to FP64 -- the candidate
// state, the embedded error and the hairer norm, as the benchmark spec keeps them.  The air-mass
// row is the FP64 scheme's, stage by stage (m in the air-mass planes of U, S1, S2, S3).
//   1: P = U + dt/2 f(U)          2: P = P + dt/2 f(P)
//   3: u3 = P + dt/2 f(P) -> S1 (pairs), P = u4 = 2/3 U + 1/3 u3
//   4: unew = P + dt/2 f(P); err = 1/2 (1/3 U + 2/3 u3 - unew); candidate = clamp(unew)
constexpr float kTwoThirdsH = (float)(2.0 / 3.0);
constexpr float kTwoThirdsL = (float)(2.0 / 3.0 - (double)(float)(2.0 / 3.0));
constexpr float kThirdH = (float)(1.0 / 3.0);
constexpr float kThirdL = (float)(1.0 / 3.0 - (double)(float)(1.0 / 3.0));
template <int STAGE>
__global__ void __launch_bounds__(kRedThreads) k_stage_mixed(DevTransport<double> T,
                                                             const Ctl* __restrict__ ctl,
                                                             TransportBufs B, double rtol,
                                                             double atol, int clamp) {
  __shared__ double sm[kRedThreads];
  if (ctl->done) return;
  const double g = ctl->g[STAGE - 1];
  const int cur = ctl->cur;
  const double* U = cur ? B.U1 : B.U0;
  double* Un = cur ? B.U0 : B.U1;
  const double dt_2 = ctl->dtc / 2;
  // air mass of the stage input
  const double* Qm = STAGE == 1 ? U : (STAGE == 2 ? B.S1 : (STAGE == 3 ? B.S2 : B.S3));
  const size_t nc = (size_t)T.nlon * T.nlat * T.nlev;
  float2* u3p = reinterpret_cast<float2*>(B.S1);  // u3 of the tracers as pairs, [ntr][nc]
  const df c23{kTwoThirdsH, kTwoThirdsL}, c13{kThirdH, kThirdL};
  const size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  double e = 0.0;
  if (c < nc) {
    const int i = (int)(c % T.nlon);
    const int j = (int)((c / T.nlon) % T.nlat);
    const int k = (int)(c / ((size_t)T.nlon * T.nlat));
    const CellGeo G{T.gx[j], T.gylo[j], T.gyhi[j]};
    const MassFluxes F = mass_fluxes(T, i, j, k, g);
    double hz, vz;
    div_parts(F, G, hz, vz);
    const double dmdt = T.mcorr ? -((hz + T.mcorr[c]) + vz) : -(hz + vz);
    const size_t xm = (size_t)(T.nsp - 1) * nc + c;
    const double m = Qm[xm];
#if RS_STRICT
    const double rm = 1.0 / m;
#else
    const double rm = rcp_nr(m);  // m > 0
#endif
    const df sc = split_df(dt_2 * rm);  // the tracer increment is (m dq/dt) * dt/2 / m
    const size_t col = (size_t)j * T.nlon + i;
    // the air-mass row, in FP64 as the FP64 scheme forms it
    const double mn = fma(dmdt, dt_2, m);
    if (STAGE == 1) B.S1[xm] = mn;
    if (STAGE == 2) B.S2[xm] = mn;
    if (STAGE == 3) {
      B.S1[xm] = mn;
      B.S3[xm] = (2.0 / 3.0) * U[xm] + (1.0 / 3.0) * mn;
    }
    if (STAGE == 4) {
      const double u0 = U[xm], u3 = B.S1[xm];
      const double err = fma(2.0 / 3.0, u3, fma(1.0 / 3.0, u0, -mn));
      const double den = fma(amax_bits(u0, mn), rtol, atol);
      const double at = err * rcp_nr1(den);
      e = fma(at, at, e);
      Un[xm] = (clamp && __double2hiint(mn) < 0) ? 0.0 : mn;
    }
    // one tracer from its loaded inputs (q, the accumulator, and for stages 3-4 the attempt's
    // input u0 and stage 4's u3); the norm terms are added in tracer order
    auto tracer = [&](int s, size_t x, df q, float2 a, double u0, float2 u3) {
      df nx;
      if (T.pbl) {  // with full PBL mixing the tendency is formed in FP64 (rare combination)
        const double qd = df_to_d(make_float2(q.h, q.l));
        const double du = fma(df_to_d(a), rm, pbl_term(T, c, col, s, qd));
        nx = split_df(fma(du, dt_2, qd));
      } else {
        nx = df_add(q, df_mul(df{a.x, a.y}, sc));
      }
      if (STAGE == 1 || STAGE == 2) {
        T.qhi[x] = nx.h;
        T.qlo[x] = nx.l;
      } else if (STAGE == 3) {
        u3p[x] = make_float2(nx.h, nx.l);
        const df u4 = df_add(df_mul(c23, split_df(u0)), df_mul(c13, nx));
        T.qhi[x] = u4.h;
        T.qlo[x] = u4.l;
      } else {
        const double un = df_to_d(make_float2(nx.h, nx.l));
        // (1/3 u0 + 2/3 u3) - un in pairs, then FP64 for the norm; its factor 1/2 goes onto
        // the cell's sum as an exact 1/4
        const df ut = df_add(df_mul(c13, split_df(u0)), df_mul(c23, df{u3.x, u3.y}));
        const df d = df_sub(ut, nx);
        const double err = df_to_d(make_float2(d.h, d.l));
        const double den = fma(amax_bits(u0, un), rtol, atol);
        const double at = err * rcp_nr1(den);  // den >= atol > 0
        e = fma(at, at, e);
        Un[x] = (clamp && __double2hiint(un) < 0) ? 0.0 : un;
      }
    };
    // tracers in groups of four: every load of a group is issued before its arithmetic, so a
    // thread keeps four tracers' loads in flight (the same arithmetic, in the same order)
    constexpr int kGrp = 4;
    int s = 0;
    for (; s + kGrp <= T.ntr; s += kGrp) {
      df q[kGrp];
      float2 a[kGrp], u3[kGrp];
      double u0[kGrp];
#pragma unroll
      for (int r = 0; r < kGrp; ++r) {
        const size_t x = (size_t)(s + r) * nc + c;
        q[r] = df{T.qhi[x], T.qlo[x]};
        a[r] = T.acc[x];
        u0[r] = STAGE >= 3 ? U[x] : 0.0;
        u3[r] = STAGE == 4 ? u3p[x] : make_float2(0.0f, 0.0f);
      }
#pragma unroll
      for (int r = 0; r < kGrp; ++r) tracer(s + r, (size_t)(s + r) * nc + c, q[r], a[r], u0[r], u3[r]);
    }
    for (; s < T.ntr; ++s) {
      const size_t x = (size_t)s * nc + c;
      tracer(s, x, df{T.qhi[x], T.qlo[x]}, T.acc[x], STAGE >= 3 ? U[x] : 0.0,
             STAGE == 4 ? u3p[x] : make_float2(0.0f, 0.0f));
    }
  }
  if (STAGE == 4) {
    const double tot = block_tree256(0.25 * e, sm);
    if (threadIdx.x == 0) B.partial[blockIdx.x] = tot;
  }
}

// Plain RHS evaluation for the rs_rhs_transport hook: du = f(U) at time factor g.
__global__ void __launch_bounds__(kRedThreads) k_rhs_eval(DevTransport<double> T,
                                                          const double* __restrict__ Qin,
                                                          double* __restrict__ dU, double g,
                                                          double* __restrict__ dUadv) {
  const size_t nc = (size_t)T.nlon * T.nlat * T.nlev;
  size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= nc) return;
  int i = (int)(c % T.nlon);
  int j = (int)((c / T.nlon) % T.nlat);
  int k = (int)(c / ((size_t)T.nlon * T.nlat));
  CellGeo G{T.gx[j], T.gylo[j], T.gyhi[j]};
  const size_t ncol = (size_t)T.nlon * T.nlat, col = (size_t)j * T.nlon + i;
  const double m = Qin[(size_t)(T.nsp - 1) * nc + c];
#if RS_STRICT
  double divM = div_m(T, i, j, k, g, G);
  const int nfx = T.nlon + 1, nfy = T.nlat + 1;
  const size_t fxp = (size_t)T.nlev * T.nlat * nfx, fyp = (size_t)T.nlev * nfy * T.nlon,
               fzp = ncol * (T.nlev + 1);
  const size_t fxi = ((size_t)k * T.nlat + j) * nfx + i;
  const size_t fyi = ((size_t)k * nfy + j) * T.nlon + i;
  const size_t fzi = (size_t)k * ncol + col;
#endif
  for (int s = 0; s < T.nsp; ++s) {
    size_t x = (size_t)s * nc + c;
    if (s < T.ntr) {
      double adv;
      if (T.mixed) {  // the kernels accumulated m dq/dt as a pair
        adv = df_to_d(T.acc[x]) / m;
      } else {
#if RS_STRICT
        double fw = T.fx[s * fxp + fxi], fe = T.fx[s * fxp + fxi + 1];
        double fs = T.fy[s * fyp + fyi], fn = T.fy[s * fyp + fyi + T.nlon];
        double fb = T.fz[s * fzp + fzi], ft = T.fz[s * fzp + fzi + ncol];
        double Dx = (fe - fw) * G.gx;
        double Dy = fn * G.gyhi - fs * G.gylo;
        double Dz = ft - fb;
        double a = -((Dx + Dy) + Dz);
        double b = Qin[x] * divM;
        adv = (a + b) / m;
#else
        adv = -(g * T.acc64[x]) / m;
#endif
      }
      dU[x] = T.pbl ? adv + pbl_term(T, c, col, s, Qin[x]) : adv;
      if (dUadv) dUadv[x] = adv;
    } else {
      const double dm = dm_dt(T, i, j, k, g, G, c);
      dU[x] = dm;
      if (dUadv) dUadv[x] = dm;
    }
  }
}

// allow > 48 KB of dynamic shared memory for long pencils (once per process)
constexpr int kPencilSmemCap = 200 * 1024;
static void allow_big_smem() {
  static bool done = false;
  if (done) return;
  const int cap = kPencilSmemCap;
#if RS_STRICT
  cudaFuncSetAttribute(k_flux_x_fused, cudaFuncAttributeMaxDynamicSharedMemorySize, cap);
  cudaFuncSetAttribute(k_flux_y_fused<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, cap);
  cudaFuncSetAttribute(k_flux_y_fused<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, cap);
  cudaFuncSetAttribute(k_flux_y_fused<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, cap);
  cudaFuncSetAttribute(k_flux_z_fused<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, cap);
  cudaFuncSetAttribute(k_flux_z_fused<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, cap);
  cudaFuncSetAttribute(k_flux_z_fused<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, cap);
#else
  cudaFuncSetAttribute(k_adv_x_rows, cudaFuncAttributeMaxDynamicSharedMemorySize, cap);
  cudaFuncSetAttribute(k_adv_pencil<1, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize, cap);
  cudaFuncSetAttribute(k_adv_pencil<1, 16>, cudaFuncAttributeMaxDynamicSharedMemorySize, cap);
  cudaFuncSetAttribute(k_adv_pencil<1, 32>, cudaFuncAttributeMaxDynamicSharedMemorySize, cap);
  cudaFuncSetAttribute(k_adv_pencil<2, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize, cap);
  cudaFuncSetAttribute(k_adv_pencil<2, 16>, cudaFuncAttributeMaxDynamicSharedMemorySize, cap);
  cudaFuncSetAttribute(k_adv_pencil<2, 32>, cudaFuncAttributeMaxDynamicSharedMemorySize, cap);
#endif
  cudaFuncSetAttribute(k_adv_x_mixed<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, cap);
  cudaFuncSetAttribute(k_adv_x_mixed<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, cap);
  cudaFuncSetAttribute(k_adv_yz_mixed<1, 16, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, cap);
  cudaFuncSetAttribute(k_adv_yz_mixed<1, 16, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, cap);
  cudaFuncSetAttribute(k_adv_yz_mixed<1, 32, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, cap);
  cudaFuncSetAttribute(k_adv_yz_mixed<1, 32, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, cap);
  cudaFuncSetAttribute(k_adv_yz_mixed<2, 16, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, cap);
  cudaFuncSetAttribute(k_adv_yz_mixed<2, 16, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, cap);
  cudaFuncSetAttribute(k_adv_yz_mixed<2, 32, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, cap);
  cudaFuncSetAttribute(k_adv_yz_mixed<2, 32, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, cap);
  done = true;
}

#if RS_STRICT
// Launch shape of the fused pencil kernels: V, Dd, D, E rows (n+6 each) plus the n+1 face fluxes,
// per pencil.  Lat / vertical blocks are (pencil width 8, 16 or 32) x rows threads, at most 512;
// the tuned width drops to 16 where 32 does not fit; a direction whose pencils do not fit even
// at 16 uses the per-face FP64 kernel (the same fluxes, bit for bit).  Lon rows take 64..256
// threads in steps of 32.
struct FluxShape {
  int pw, rows, xt;
  int gx, gyz;  // tracer groups (grid y) of the lon and of the lat / vertical pencils
  size_t shx, shy, shz;
  bool fx, fy, fz;  // fused kernel used for x / y / z
};
static size_t pencil_bytes(int n, int pw) { return (size_t)(4 * (n + 6) + (n + 1)) * pw * sizeof(double); }
static FluxShape flux_shape(const DevTransport<double>& T) {
  FluxShape f;
  f.pw = (T.pencil == 8 || T.pencil == 16) ? T.pencil : 32;
  if (f.pw == 32 && (pencil_bytes(T.nlat, f.pw) > (size_t)kPencilSmemCap ||
                     pencil_bytes(T.nlev, f.pw) > (size_t)kPencilSmemCap))
    f.pw = 16;
  f.rows = (T.rows == 4 || T.rows == 16 || T.rows == 32) ? T.rows : 8;
  if (f.pw * f.rows > 512) f.rows = 512 / f.pw;
  f.xt = (T.xthreads >= 64 && T.xthreads <= 256 && T.xthreads % 32 == 0) ? T.xthreads : 128;
  const int ntr = T.ntr > 0 ? T.ntr : 1;
  f.gx = T.xgroups < 1 ? 1 : (T.xgroups > ntr ? ntr : T.xgroups);
  f.gyz = T.yzgroups < 1 ? 1 : (T.yzgroups > ntr ? ntr : T.yzgroups);
  f.shx = pencil_bytes(T.nlon, 1);
  f.shy = pencil_bytes(T.nlat, f.pw);
  f.shz = pencil_bytes(T.nlev, f.pw);
  f.fx = f.shx <= (size_t)kPencilSmemCap;
  f.fy = f.shy <= (size_t)kPencilSmemCap;
  f.fz = f.shz <= (size_t)kPencilSmemCap;
  return f;
}

static void launch_flux_one(cudaStream_t st, const DevTransport<double>& T, const StageSel& sel,
                            const FluxShape& f, int dir) {
  size_t ncol = (size_t)T.nlon * T.nlat;
  if (dir == 0) {
    if (f.fx) {
      k_flux_x_fused<<<dim3((unsigned)(T.nlat * T.nlev), (unsigned)f.gx), f.xt, f.shx, st>>>(T, sel);
    } else {
      long long nx = (long long)(T.nlon + 1) * T.nlat * T.nlev;
      k_flux_x<<<(unsigned)((nx + kFluxThreads - 1) / kFluxThreads), kFluxThreads, 0, st>>>(T, sel);
    }
  } else if (dir == 1) {
    if (f.fy) {
      unsigned ntile = (unsigned)((T.nlon + f.pw - 1) / f.pw);
      const dim3 grid(ntile * (unsigned)T.nlev, (unsigned)f.gyz);
      if (f.pw == 8) k_flux_y_fused<8><<<grid, dim3(8, f.rows), f.shy, st>>>(T, sel);
      else if (f.pw == 16) k_flux_y_fused<16><<<grid, dim3(16, f.rows), f.shy, st>>>(T, sel);
      else k_flux_y_fused<32><<<grid, dim3(32, f.rows), f.shy, st>>>(T, sel);
    } else {
      long long ny = (long long)T.nlon * (T.nlat + 1) * T.nlev;
      k_flux_y<<<(unsigned)((ny + kFluxThreads - 1) / kFluxThreads), kFluxThreads, 0, st>>>(T, sel);
    }
  } else {
    if (f.fz) {
      const dim3 grid((unsigned)((ncol + f.pw - 1) / f.pw), (unsigned)f.gyz);
      if (f.pw == 8) k_flux_z_fused<8><<<grid, dim3(8, f.rows), f.shz, st>>>(T, sel);
      else if (f.pw == 16) k_flux_z_fused<16><<<grid, dim3(16, f.rows), f.shz, st>>>(T, sel);
      else k_flux_z_fused<32><<<grid, dim3(32, f.rows), f.shz, st>>>(T, sel);
    } else {
      long long nz = (long long)T.nlon * T.nlat * (T.nlev + 1);
      k_flux_z<<<(unsigned)((nz + kFluxThreads - 1) / kFluxThreads), kFluxThreads, 0, st>>>(T, sel);
    }
  }
}
void launch_scale_fluxes(cudaStream_t, const DevTransport<double>&, double*, double*, double*) {}
#else
// Launch shape of the FP64 kernels.  Lat / vertical pencil blocks are (pencil width 8, 16 or 32) x
// up to `rows` threads, at most 512; a line of n cells takes n + 5 entries per phase, dealt evenly
// over the passes it needs (51 entries at rows 32: two passes of 26, not 32 + 19).  The tuned
// width drops to 8 where the pencils do not fit; lines that do not fit even then take the
// thread-per-line kernel, lon rows that do not fit the thread-per-cell kernel -- the same bits.
struct FluxShape {
  int pw, rows, xt, xr;  // xr: lon rows per block
  int gx, gyz;           // tracer groups (grid y)
  size_t shx, shy, shz;
  bool fx, fy, fz;       // shared-memory kernel used for x / y / z
};
static size_t pencil_bytes(int n, int pw, int nm) {
  return (size_t)(4 * (n + 6) + nm * (n + 1)) * pw * sizeof(double);
}
static int even_rows(int n, int rows) {  // threads along the line for the fewest passes
  const int passes = (n + 5 + rows - 1) / rows;
  return (n + 5 + passes - 1) / passes;
}
static FluxShape flux_shape(const DevTransport<double>& T) {
  FluxShape f;
  const size_t cap = (size_t)kPencilSmemCap;
  const int ntr = T.ntr > 0 ? T.ntr : 1;
  // Shapes not set by hand or by the autotuner follow the grid (measured with 12 tracers on
  // 36x18x10, 67x45x37, 72x46x47, 144x91x47 and 30 on 180x91x72):
  // - lat / vertical: a thread per line once there are 2,000 warps of them in both directions
  //   (315 against 335 us on 144x91x47 with 2,538 lat warps, but 100 against 94 us on 72x46x47 with
  //   1,242: under three warps per sub-partition the last wave is too coarse), else pencils 8 wide
  //   with up to 32 threads along the line (every grid's fastest pencils);
  // - pencils: tracer groups for 16 blocks per SM of the smaller direction, as a divisor of the
  //   tracer count (36x18x10: 49 us in one group, 16 in 12; 72x46x47: 109 in one, 94 in 6);
  // - lon rows: a row and its halo in whole warps, 128-256 threads (144x91x47: 160 threads 142 us,
  //   128 156 us, 256 149 us), one tracer per block up to 12 groups (133 us against 142 in one).
  const size_t ncol = (size_t)T.nlon * T.nlat;
  const size_t warps = std::min((size_t)T.nlon * T.nlev, ncol) * ntr / 32;
  const bool line = T.yzline < 0 ? (T.pencil == 0 && T.rows == 0 && warps >= 2000) : T.yzline != 0;
  f.pw = T.pencil == 16 || T.pencil == 32 ? T.pencil : 8;
  while (f.pw > 8 && (pencil_bytes(T.nlat, f.pw, 2) > cap || pencil_bytes(T.nlev, f.pw, 1) > cap)) f.pw /= 2;
  f.rows = (T.rows == 4 || T.rows == 8 || T.rows == 16) ? T.rows : 32;
  if (f.pw * f.rows > 512) f.rows = 512 / f.pw;
  const int fit = std::max(128, std::min(256, (T.nlon + 6 + 31) / 32 * 32));
  f.xt = (T.xthreads >= 64 && T.xthreads <= 256 && T.xthreads % 32 == 0) ? T.xthreads : fit;
  f.gx = T.xgroups < 1 ? std::min(ntr, 12) : std::min(T.xgroups, ntr);
  f.gyz = std::min(T.yzgroups, ntr);
  if (f.gyz < 1) {
    const size_t tiles = std::min((size_t)((T.nlon + f.pw - 1) / f.pw) * T.nlev, (ncol + f.pw - 1) / f.pw);
    f.gyz = 1;
    while (f.gyz < ntr && (ntr % f.gyz != 0 || tiles * f.gyz < (size_t)16 * 152)) ++f.gyz;
  }
  // lon rows per block: the fewest (up to 8, within 48 KB) whose entries fill the block's last
  // pass to within 4 %, as long as the grid still has four blocks per SM (152 SMs)
  const int nrows = T.nlat * T.nlev, len = T.nlon + 6;
  f.xr = 1;
  double best = 1e30;
  for (int r = 1; r <= 8; ++r) {
    if (r > 1 && ((size_t)5 * len * r * sizeof(double) > 48 * 1024 || (long long)((nrows + r - 1) / r) * f.gx < 4 * 152)) break;
    const double waste = (double)((r * len + f.xt - 1) / f.xt * f.xt) / (r * len);
    if (waste < best - 0.04) {
      best = waste;
      f.xr = r;
    }
  }
  f.shx = (size_t)5 * len * f.xr * sizeof(double);
  f.shy = pencil_bytes(T.nlat, f.pw, 2);
  f.shz = pencil_bytes(T.nlev, f.pw, 1);
  f.fx = f.shx <= cap;
  f.fy = f.shy <= cap && !line;
  f.fz = f.shz <= cap && !line;
  return f;
}
template <int DIR>
static void launch_adv_yz(cudaStream_t st, const DevTransport<double>& T, const StageSel& sel,
                          const FluxShape& f) {
  const size_t ncol = (size_t)T.nlon * T.nlat;
  if (!(DIR == 1 ? f.fy : f.fz)) {
    const size_t lines = DIR == 1 ? (size_t)T.nlon * T.nlev : ncol;
    k_adv_line<DIR><<<dim3((unsigned)((lines + kLineThreads - 1) / kLineThreads), (unsigned)T.ntr), kLineThreads, 0, st>>>(T, sel);
    return;
  }
  const unsigned tiles = DIR == 1 ? (unsigned)((T.nlon + f.pw - 1) / f.pw) * (unsigned)T.nlev
                                  : (unsigned)((ncol + f.pw - 1) / f.pw);
  const dim3 grid(tiles, (unsigned)f.gyz), block(f.pw, even_rows(DIR == 1 ? T.nlat : T.nlev, f.rows));
  const size_t sh = DIR == 1 ? f.shy : f.shz;
  if (f.pw == 8) k_adv_pencil<DIR, 8><<<grid, block, sh, st>>>(T, sel);
  else if (f.pw == 16) k_adv_pencil<DIR, 16><<<grid, block, sh, st>>>(T, sel);
  else k_adv_pencil<DIR, 32><<<grid, block, sh, st>>>(T, sel);
}
static void launch_flux_one(cudaStream_t st, const DevTransport<double>& T, const StageSel& sel,
                            const FluxShape& f, int dir) {
  if (dir == 1) launch_adv_yz<1>(st, T, sel, f);
  else if (dir == 2) launch_adv_yz<2>(st, T, sel, f);
  else if (f.fx)
    k_adv_x_rows<<<dim3((unsigned)((T.nlat * T.nlev + f.xr - 1) / f.xr), (unsigned)f.gx), f.xt, f.shx, st>>>(T, sel, f.xr);
  else
    k_adv_x_cell<<<dim3((unsigned)(((size_t)T.nlon * T.nlat * T.nlev + 255) / 256), (unsigned)T.ntr), 256, 0, st>>>(T, sel);
}
void launch_scale_fluxes(cudaStream_t st, const DevTransport<double>& T, double* mx6, double* myn6,
                         double* mys6) {
  const size_t n = (size_t)T.nlev * std::max((size_t)T.nlat * (T.nlon + 1), (size_t)(T.nlat + 1) * T.nlon);
  k_scale_fluxes<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(T, mx6, myn6, mys6);
}
#endif

// Mixed-precision pencils: the staged hi / lo rows (four with the second set of the bulk-copy
// staging), the pair rows of the differences and slopes, and the face fluxes as pairs.
size_t mixed_pencil_bytes(int n, int pw, bool tma) {
  const int rows = tma ? 8 : 6;
  if (pw == 1)
    return (size_t)rows * mixed_rows_x(n) * sizeof(float) + 2 * (size_t)mixed_frows(n) * sizeof(float) +
           kSmemAlignPad;
  return ((size_t)rows * mixed_rows_p(n) + 2 * (size_t)(n + 1)) * pw * sizeof(float) + kSmemAlignPad;
}
size_t mixed_pencil_cap() { return (size_t)kPencilSmemCap; }

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link to the driver
// library); null when the entry point is unavailable.
static PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static bool tried = false;
  if (!tried) {
    tried = true;
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q{};
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault,
                                         &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    else
      cudaGetLastError();
  }
  return fn;
}

// 3-D FP32 tensor {d0, d1, d2} (d0 contiguous) with box {b0, b1, 1}; false if rejected.
static bool encode_f32_3d(CUtensorMap* m, float* base, uint64_t d0, uint64_t d1, uint64_t d2,
                          uint32_t b0, uint32_t b1) {
  auto enc = tensor_map_encoder();
  if (!enc) return false;
  const cuuint64_t dims[3] = {d0, d1, d2};
  const cuuint64_t strides[2] = {d0 * sizeof(float), d0 * d1 * sizeof(float)};
  const cuuint32_t box[3] = {b0, b1, 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, base, dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
             CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

MixedTmaps* mixed_tmaps_create(const DevTransport<double>& T, const char** why) {
  *why = nullptr;
  if (!T.qhi || !T.qlo) {
    *why = "no split planes (FP64 transport)";
    return nullptr;
  }
  auto* m = new MixedTmaps();
  const uint64_t ncol = (uint64_t)T.nlon * T.nlat;
  // 1-D bulk copies of lon rows: 16-byte aligned starts and sizes need nlon % 4 == 0
  const size_t cap = (size_t)kPencilSmemCap;
  m->x_ok = T.nlon % 4 == 0 && mixed_pencil_bytes(T.nlon, 1, true) <= cap;
  // tensor strides must be multiples of 16 bytes; boxes at most 256 rows
  m->y_ok = T.nlon % 4 == 0 && T.nlat <= 256 && mixed_pencil_bytes(T.nlat, 16, true) <= cap;
  m->z_ok = ncol % 4 == 0 && T.nlev <= 256 && mixed_pencil_bytes(T.nlev, 16, true) <= cap;
  for (int w = 0; w < 2 && m->y_ok; ++w) {
    const uint32_t pw = w ? 32 : 16;
    m->y_ok = encode_f32_3d(&m->yh[w], T.qhi, T.nlon, T.nlat, (uint64_t)T.nlev * T.ntr, pw, T.nlat) &&
              encode_f32_3d(&m->yl[w], T.qlo, T.nlon, T.nlat, (uint64_t)T.nlev * T.ntr, pw, T.nlat);
  }
  for (int w = 0; w < 2 && m->z_ok; ++w) {
    const uint32_t pw = w ? 32 : 16;
    m->z_ok = encode_f32_3d(&m->zh[w], T.qhi, ncol, T.nlev, T.ntr, pw, T.nlev) &&
              encode_f32_3d(&m->zl[w], T.qlo, ncol, T.nlev, T.ntr, pw, T.nlev);
  }
  if (!m->x_ok && !m->y_ok && !m->z_ok) {
    *why = "grid does not meet the bulk-copy alignment rules";
    delete m;
    return nullptr;
  }
  return m;
}

void mixed_tmaps_destroy(MixedTmaps* m) { delete m; }
bool mixed_tmaps_dir_ok(const MixedTmaps* m, int dir) {
  return m && (dir == 0 ? m->x_ok : (dir == 1 ? m->y_ok : m->z_ok));
}

static void launch_fluxes_mixed(cudaStream_t st, const DevTransport<double>& T, const StageSel& sel,
                                int only_dir = -1) {
  int pw = T.mpencil == 16 ? 16 : 32;
  const MixedTmaps* tm = T.tma;
  const bool tx = tm && tm->x_ok && T.mbulk_x, ty = tm && tm->y_ok && T.mbulk_yz,
             tz = tm && tm->z_ok && T.mbulk_yz;
  if (mixed_pencil_bytes(T.nlat, pw, ty) > (size_t)kPencilSmemCap ||
      mixed_pencil_bytes(T.nlev, pw, tz) > (size_t)kPencilSmemCap)
    pw = 16;
  const int w = pw == 32;
  const int rows = (T.mrows == 4 || T.mrows == 16) ? T.mrows : 8;
  const int xt = (T.mxthreads == 64 || T.mxthreads == 256) ? T.mxthreads : 128;
  auto groups = [&](int sper) { return (unsigned)((T.ntr + sper - 1) / sper); };
  const int sx = std::max(1, std::min(T.ntr, T.msper_x)), syz = std::max(1, std::min(T.ntr, T.msper_yz));
  const size_t ncol = (size_t)T.nlon * T.nlat;
  const size_t shx = mixed_pencil_bytes(T.nlon, 1, tx), shy = mixed_pencil_bytes(T.nlat, pw, ty),
               shz = mixed_pencil_bytes(T.nlev, pw, tz);
  static const CUtensorMap kNoMap{};  // placeholder argument of the plain-load variants
  // rs_create refuses mixed precision on grids whose pencils do not fit at width 16
  if ((only_dir < 0 || only_dir == 0) && T.mstream_x) {
    const long long warps = (long long)((T.nlon + kSegX - 1) / kSegX) * T.nlat * T.nlev;
    k_adv_x_stream<<<dim3((unsigned)((warps + 3) / 4), groups(sx)), 128, 0, st>>>(T, sel, sx);
  } else if (only_dir < 0 || only_dir == 0) {
    dim3 grid((unsigned)(T.nlat * T.nlev), groups(sx));
    if (tx) k_adv_x_mixed<true><<<grid, xt, shx, st>>>(T, sel, sx);
    else k_adv_x_mixed<false><<<grid, xt, shx, st>>>(T, sel, sx);
  }
  if (T.mstream_yz) {
    if (only_dir < 0 || only_dir == 1)
      k_adv_yz_stream<1><<<dim3((unsigned)((T.nlon + 127) / 128) * (unsigned)T.nlev, groups(syz)),
                           128, 0, st>>>(T, sel, syz);
    if (only_dir < 0 || only_dir == 2)
      k_adv_yz_stream<2><<<dim3((unsigned)((ncol + 127) / 128), groups(syz)), 128, 0, st>>>(
          T, sel, syz);
    return;
  }
  if (only_dir < 0 || only_dir == 1) {
    dim3 grid((unsigned)((T.nlon + pw - 1) / pw) * (unsigned)T.nlev, groups(syz));
    const CUtensorMap& mh = ty ? tm->yh[w] : kNoMap;
    const CUtensorMap& ml = ty ? tm->yl[w] : kNoMap;
    if (pw == 16) {
      if (ty) k_adv_yz_mixed<1, 16, true><<<grid, dim3(16, rows), shy, st>>>(T, sel, syz, mh, ml);
      else k_adv_yz_mixed<1, 16, false><<<grid, dim3(16, rows), shy, st>>>(T, sel, syz, mh, ml);
    } else {
      if (ty) k_adv_yz_mixed<1, 32, true><<<grid, dim3(32, rows), shy, st>>>(T, sel, syz, mh, ml);
      else k_adv_yz_mixed<1, 32, false><<<grid, dim3(32, rows), shy, st>>>(T, sel, syz, mh, ml);
    }
  }
  if (only_dir < 0 || only_dir == 2) {
    dim3 grid((unsigned)((ncol + pw - 1) / pw), groups(syz));
    const CUtensorMap& mh = tz ? tm->zh[w] : kNoMap;
    const CUtensorMap& ml = tz ? tm->zl[w] : kNoMap;
    if (pw == 16) {
      if (tz) k_adv_yz_mixed<2, 16, true><<<grid, dim3(16, rows), shz, st>>>(T, sel, syz, mh, ml);
      else k_adv_yz_mixed<2, 16, false><<<grid, dim3(16, rows), shz, st>>>(T, sel, syz, mh, ml);
    } else {
      if (tz) k_adv_yz_mixed<2, 32, true><<<grid, dim3(32, rows), shz, st>>>(T, sel, syz, mh, ml);
      else k_adv_yz_mixed<2, 32, false><<<grid, dim3(32, rows), shz, st>>>(T, sel, syz, mh, ml);
    }
  }
}

static void launch_fluxes(cudaStream_t st, const DevTransport<double>& T, const StageSel& sel) {
  allow_big_smem();
  if (T.mixed) {
    launch_fluxes_mixed(st, T, sel);
    return;
  }
  const FluxShape f = flux_shape(T);
  for (int dir = 0; dir < 3; ++dir) launch_flux_one(st, T, sel, f, dir);
}

// one direction of the mixed-precision flux computation on a given field (used by the
// autotuner); the hi/lo planes of Q are split first
void launch_flux_dir_mixed(cudaStream_t st, const DevTransport<double>& T, const double* Q, int dir,
                           bool split) {
  StageSel sel{nullptr, 0, nullptr, nullptr, nullptr, nullptr, nullptr, Q, 1.0};
  allow_big_smem();
  if (split) {
    size_t n = (size_t)T.ntr * T.nlon * T.nlat * T.nlev;
    k_split_input<<<(unsigned)((n + 4 * kRedThreads - 1) / (4 * kRedThreads)), kRedThreads, 0, st>>>(
        T, nullptr, nullptr, nullptr, Q);
  }
  launch_fluxes_mixed(st, T, sel, dir);
}

// one direction of the flux computation on a given field (used by the autotuner)
void launch_flux_dir(cudaStream_t st, const DevTransport<double>& T, const double* Q, int dir) {
  StageSel sel{nullptr, 0, nullptr, nullptr, nullptr, nullptr, nullptr, Q, 1.0};
  DevTransport<double> T1 = T;
  T1.mixed = 0;
  allow_big_smem();
  launch_flux_one(st, T1, sel, flux_shape(T1), dir);
}

void launch_ssprk43_attempt(cudaStream_t st, const DevTransport<double>& T, const Ctl* ctl,
                            const TransportBufs& B, double rtol, double atol, int clamp) {
  size_t nc = (size_t)T.nlon * T.nlat * T.nlev;
  unsigned nb = (unsigned)((nc + kRedThreads - 1) / kRedThreads);
  StageSel sel{ctl, 1, B.U0, B.U1, B.S1, B.S2, B.S3, nullptr, 1.0};
  if (T.mixed) {
    size_t n = (size_t)T.ntr * nc;
    k_split_input<<<(unsigned)((n + 4 * kRedThreads - 1) / (4 * kRedThreads)), kRedThreads, 0, st>>>(
        T, ctl, B.U0, B.U1, nullptr);
  }
  if (T.mixed) {  // compensated FP32: the stages stay pairs until stage 4
    launch_fluxes(st, T, sel);
    if (T.pbl) launch_pbl_mean(st, T, sel);
    k_stage_mixed<1><<<nb, kRedThreads, 0, st>>>(T, ctl, B, rtol, atol, clamp);
    sel.stage = 2;
    launch_fluxes(st, T, sel);
    if (T.pbl) launch_pbl_mean(st, T, sel);
    k_stage_mixed<2><<<nb, kRedThreads, 0, st>>>(T, ctl, B, rtol, atol, clamp);
    sel.stage = 3;
    launch_fluxes(st, T, sel);
    if (T.pbl) launch_pbl_mean(st, T, sel);
    k_stage_mixed<3><<<nb, kRedThreads, 0, st>>>(T, ctl, B, rtol, atol, clamp);
    sel.stage = 4;
    launch_fluxes(st, T, sel);
    if (T.pbl) launch_pbl_mean(st, T, sel);
    k_stage_mixed<4><<<nb, kRedThreads, 0, st>>>(T, ctl, B, rtol, atol, clamp);
    return;
  }
  launch_fluxes(st, T, sel);
  if (T.pbl) launch_pbl_mean(st, T, sel);
  k_stage<1><<<nb, kRedThreads, 0, st>>>(T, ctl, B, rtol, atol, clamp);
  sel.stage = 2;
  launch_fluxes(st, T, sel);
  if (T.pbl) launch_pbl_mean(st, T, sel);
  k_stage<2><<<nb, kRedThreads, 0, st>>>(T, ctl, B, rtol, atol, clamp);
  sel.stage = 3;
  launch_fluxes(st, T, sel);
  if (T.pbl) launch_pbl_mean(st, T, sel);
  k_stage<3><<<nb, kRedThreads, 0, st>>>(T, ctl, B, rtol, atol, clamp);
  sel.stage = 4;
  launch_fluxes(st, T, sel);
  if (T.pbl) launch_pbl_mean(st, T, sel);
  k_stage<4><<<nb, kRedThreads, 0, st>>>(T, ctl, B, rtol, atol, clamp);
}

void launch_transport_rhs(cudaStream_t st, const DevTransport<double>& T, const double* U,
                          double g, double* dU, double* dUadv) {
  StageSel sel{nullptr, 0, nullptr, nullptr, nullptr, nullptr, nullptr, U, g};
  size_t nc = (size_t)T.nlon * T.nlat * T.nlev;
  if (T.mixed) {
    size_t n = (size_t)T.ntr * nc;
    k_split_input<<<(unsigned)((n + 4 * kRedThreads - 1) / (4 * kRedThreads)), kRedThreads, 0, st>>>(
        T, nullptr, nullptr, nullptr, U);
  }
  launch_fluxes(st, T, sel);
  if (T.pbl) launch_pbl_mean(st, T, sel);
  k_rhs_eval<<<(unsigned)((nc + kRedThreads - 1) / kRedThreads), kRedThreads, 0, st>>>(T, U, dU, g,
                                                                                     dUadv);
}

}  // namespace rs
