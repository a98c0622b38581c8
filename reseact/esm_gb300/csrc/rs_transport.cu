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
// Start of a kernel that `behind` launches: waits for the grid before it, lets the next one be launched.
// What the grids before it write (the controller record, states, partial sums) may change until
// then, so no kernel that calls this takes those by __restrict__ pointers: those promise memory that
// is read-only for the whole kernel, and loads through them may move above the wait.
__device__ __forceinline__ void await_previous() {
#if !RS_STRICT
  asm volatile("griddepcontrol.wait;\n\tgriddepcontrol.launch_dependents;" ::: "memory");
#endif
}
#if !RS_STRICT
// The kernels of an attempt depend on each other in a row.  Launched one by one from the host on a
// small grid, each goes programmatically behind the one before, as soon as that one's blocks have
// started, and waits in await_previous: the launches' latency is hidden (the hook calls of 36x18x10
// 184 -> 173 us).  Not inside a graph, whose launches are already queued on the device, and not on
// larger grids, where the waiting blocks take room from the running ones (180x91x72: 25.5 -> 25.8 ms).
template <typename... P, typename... A>
static void behind(const DevTransport<double>& T, void (*k)(P...), dim3 grid, dim3 block, size_t smem,
                   cudaStream_t st, A&&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusActive;
  if ((long long)T.nlon * T.nlat * T.nlev <= 152 * 128) cudaStreamIsCapturing(st, &cap);
  cfg.numAttrs = cap == cudaStreamCaptureStatusNone ? 1 : 0;
  cudaLaunchKernelEx(&cfg, k, P(std::forward<A>(args))...);
}
#else
template <typename... P, typename... A>
static void behind(const DevTransport<double>&, void (*k)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
  k<<<grid, block, smem, st>>>(std::forward<A>(args)...);
}
#endif
__device__ __forceinline__ bool resolve_stage(const StageSel& s, const double*& Q, double& g) {
  await_previous();
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
  double* E = smx + 3 * L;    // E[f+3], edge between f-1 and f, f in [-1, n+1]
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
// so the reconstruction runs on the FP32 pipe at FP64-class accuracy.  The face terms are in
// advective form on edge deviations, as in rs_adv64.cuh: for cell c and face f with air-mass flux
// M_f, m dq/dt is -(sum over its faces of G_f M_f times A or B), where A = q_f - q_{f-1} goes to
// the cell below the face, B = D - A to the one above, and q_f - q of the upwind cell is its limited
// edge deviation -- its own sign with min(|e|, 2 |the opposite edge's|), 0 unless the two edges
// have strictly opposite signs.  No term is of the size of q itself, so a value far smaller than
// its neighbours keeps its relative accuracy.  q == const gives exactly zero.
//
// The uniform directions carry 12 x the deviations (with slopes doubled, so that every scaling is
// exact): 12 E_p = 6 D_p - (S'_{p+1} - S'_p), 12 eL_p = -(6 D_{p-1} + (S'_p - S'_{p-1})); the 1/12
// and the cells' metric are folded into the air-mass fluxes once per forcing, the vertical slope
// and edge coefficients carry the 2 and 1/2.  Comparisons of pairs are the sign of a difference
// (three FP32 operations), so they ride the FP32 pipe too.
//
// Each direction adds its part into a per-cell pair accumulator (x writes it, y and z add), and
// the stage kernel turns it into the stage update, whose error norm is formed in pairs as well.  The
// state, the air mass and the step-size control stay FP64.
//
// What bounds it: issue slots and the FP32 / integer pipes.  Packed f32x2 operations do two
// tracers per instruction at the scalar rate of flops, so the streaming kernels carry a pair of
// tracers per thread: half the FP32 issue slots, and the fluxes, vertical coefficients and
// addresses once for two.  FV<1> and FV<2> form the same values bit for bit (every operation is
// rounded to nearest on its own; subtraction of packed values is an exact multiply-add with -1).
// A stage at 360x181x72 with 30 tracers (144x91x47 with 12), one tracer per thread and flux-form
// pairs before -> now: lon rows 1.20 -> 0.74 ms (85 -> 52 us; of the 0.33 ms its bytes take), lat
// lines 1.29 -> 0.78 ms (137 -> 65 us; 0.49 ms), vertical lines 2.16 -> 1.04 ms (128 -> 77 us;
// 0.55 ms).  Doing stages 1-3's update inside the vertical line kernel (one read and one write of
// the accumulator less) was slower, 1.35 ms and an air-mass kernel of 0.23 against 1.04 + 0.57.
template <int N>
struct FV;
template <>
struct FV<1> {
  float v;
};
template <>
struct FV<2> {
  unsigned long long v;
};
__device__ __forceinline__ unsigned long long pack2(float a, float b) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float half(FV<1> a, int) { return a.v; }
__device__ __forceinline__ float half(FV<2> a, int i) {
  float x, y;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.v));
  return i ? y : x;
}
template <int N>
__device__ __forceinline__ FV<N> splat(float a) {
  if constexpr (N == 1) return {a};
  else return {pack2(a, a)};
}
__device__ __forceinline__ FV<1> vadd(FV<1> a, FV<1> b) { return {__fadd_rn(a.v, b.v)}; }
__device__ __forceinline__ FV<1> vsub(FV<1> a, FV<1> b) { return {__fsub_rn(a.v, b.v)}; }
__device__ __forceinline__ FV<1> vmul(FV<1> a, FV<1> b) { return {__fmul_rn(a.v, b.v)}; }
__device__ __forceinline__ FV<1> vfma(FV<1> a, FV<1> b, FV<1> c) { return {__fmaf_rn(a.v, b.v, c.v)}; }
__device__ __forceinline__ FV<2> vadd(FV<2> a, FV<2> b) {
  FV<2> r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ FV<2> vmul(FV<2> a, FV<2> b) {
  FV<2> r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ FV<2> vfma(FV<2> a, FV<2> b, FV<2> c) {
  FV<2> r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
__device__ __forceinline__ FV<2> vsub(FV<2> a, FV<2> b) { return vfma(b, splat<2>(-1.0f), a); }
// halves of a where m[i], of b otherwise
template <int N>
struct Mask {
  bool m[N];
};
template <int N>
__device__ __forceinline__ FV<N> vsel(const Mask<N>& k, FV<N> a, FV<N> b) {
  if constexpr (N == 1) return {k.m[0] ? a.v : b.v};
  else return {pack2(k.m[0] ? half(a, 0) : half(b, 0), k.m[1] ? half(a, 1) : half(b, 1))};
}
// x and y have the same sign bit (one logic instruction that sets the predicate)
template <int N>
__device__ __forceinline__ Mask<N> same_sign(FV<N> x, FV<N> y) {
  Mask<N> r;
#pragma unroll
  for (int i = 0; i < N; ++i)
    r.m[i] = ((__float_as_uint(half(x, i)) ^ __float_as_uint(half(y, i))) & 0x80000000u) == 0u;
  return r;
}

template <int N>
struct DF {
  FV<N> h, l;
};
using df = DF<1>;
__device__ __forceinline__ df mkdf(float h, float l) { return {{h}, {l}}; }
// the pair (h, l) in both halves
template <int N>
__device__ __forceinline__ DF<N> splat_df(float h, float l) {
  return {splat<N>(h), splat<N>(l)};
}
// (h, l) from a leading part s and a small correction e
template <int N>
__device__ __forceinline__ DF<N> df_renorm(DF<N> a) {
  const FV<N> h = vadd(a.h, a.l);
  return {h, vsub(a.l, vsub(h, a.h))};
}
// Sums of pairs: TwoSum of the high parts, the low parts added to its error.  Exact but for the
// roundings of the low parts, 2^-48 of the operands.  The _raw forms leave the result
// unnormalised (l may be a few ulp of h, more where the high parts cancel); that is enough for
// an operand of another sum or product, while a pair whose sign or size is looked at is normalised
// unless its parts cannot cancel.
template <int N>
__device__ __forceinline__ DF<N> add_raw(DF<N> a, DF<N> b) {
  const FV<N> s = vadd(a.h, b.h), bb = vsub(s, a.h);
  return {s, vadd(vadd(vsub(a.h, vsub(s, bb)), vsub(b.h, bb)), vadd(a.l, b.l))};
}
template <int N>
__device__ __forceinline__ DF<N> sub_raw(DF<N> a, DF<N> b) {
  const FV<N> s = vsub(a.h, b.h), bb = vsub(s, a.h);
  return {s, vadd(vsub(vsub(a.h, vsub(s, bb)), vadd(b.h, bb)), vsub(a.l, b.l))};
}
// a + b and a - b for |a| > |b| or a = b = 0: the shorter FastTwoSum
template <int N>
__device__ __forceinline__ DF<N> add_big(DF<N> a, DF<N> b) {
  const FV<N> s = vadd(a.h, b.h);
  return {s, vadd(vadd(vsub(a.h, s), b.h), vadd(a.l, b.l))};
}
template <int N>
__device__ __forceinline__ DF<N> sub_big(DF<N> a, DF<N> b) {
  const FV<N> s = vsub(a.h, b.h);
  return {s, vadd(vsub(vsub(a.h, s), b.h), vsub(a.l, b.l))};
}
template <int N>
__device__ __forceinline__ DF<N> df_add(DF<N> a, DF<N> b) { return df_renorm(add_raw(a, b)); }
template <int N>
__device__ __forceinline__ DF<N> df_sub(DF<N> a, DF<N> b) { return df_renorm(sub_raw(a, b)); }
template <int N>
__device__ __forceinline__ DF<N> df_scale(DF<N> a, float pow2) {
  return {vmul(a.h, splat<N>(pow2)), vmul(a.l, splat<N>(pow2))};
}
template <int N>
__device__ __forceinline__ DF<N> mul_raw(DF<N> a, DF<N> b) {
  const FV<N> p = vmul(a.h, b.h);
  return {p, vfma(a.h, b.l, vfma(a.l, b.h, vfma(a.h, b.h, vmul(p, splat<N>(-1.0f)))))};
}
template <int N>
__device__ __forceinline__ DF<N> fma_raw(DF<N> a, DF<N> b, DF<N> c) {  // a b + c
  const DF<N> p = mul_raw(a, b);
  const FV<N> s = vadd(c.h, p.h), bb = vsub(s, c.h);
  return {s, vadd(vadd(vsub(c.h, vsub(s, bb)), vsub(p.h, bb)), vadd(c.l, p.l))};
}
template <int N>
__device__ __forceinline__ DF<N> df_fma(DF<N> a, DF<N> b, DF<N> c) { return df_renorm(fma_raw(a, b, c)); }
template <int N>
__device__ __forceinline__ DF<N> times6(DF<N> a) {  // unnormalised
  const FV<N> k = splat<N>(6.0f), p = vmul(a.h, k);
  return {p, vfma(a.l, k, vfma(a.h, k, vmul(p, splat<N>(-1.0f))))};
}
template <int N>
__device__ __forceinline__ DF<N> df_sel(const Mask<N>& k, DF<N> a, DF<N> b) {
  return {vsel(k, a.h, b.h), vsel(k, a.l, b.l)};
}
template <int N>
__device__ __forceinline__ FV<N> df_diff(DF<N> a, DF<N> b) {  // a - b, exact in sign
  return vadd(vsub(a.h, b.h), vsub(a.l, b.l));
}
__device__ __forceinline__ df df_ld(const float* H, const float* L, long long x) { return mkdf(H[x], L[x]); }
__device__ __forceinline__ df df_ldp(const PairPlanes& P, size_t x) { return mkdf(P.h[x], P.l[x]); }
template <int N>
__device__ __forceinline__ DF<N> df_ldc(const PairPlanes& P, size_t x) {  // one value for all tracers
  return splat_df<N>(P.h[x], P.l[x]);
}

// k where a and b have the same sign, else 0 (a zero counts by its sign bit: the limited values
// below are 0 either way)
template <int N>
__device__ __forceinline__ FV<N> live(DF<N> a, DF<N> b, float k) {
  const Mask<N> m = same_sign(a.h, b.h);
  if constexpr (N == 1) return {m.m[0] ? k : 0.0f};
  else return {pack2(m.m[0] ? k : 0.0f, m.m[1] ? k : 0.0f)};
}
// the smaller in magnitude of `self` and k `other`, which have one sign wherever k is not 0
template <int N>
__device__ __forceinline__ DF<N> limit(DF<N> self, DF<N> other, FV<N> k) {
  const DF<N> m{vmul(other.h, k), vmul(other.l, k)};
  return df_sel(same_sign(df_diff(self, m), self.h), m, self);
}
// Twice the CW84 eq. 1.8 monotonised slope from the neighbour differences d0 (left), d1 (right) and
// twice the centred slope w: 0 unless d0, d1 have the same sign (k4 = live(d0, d1, 4)), else the
// smallest in magnitude of w, 4 d0, 4 d1.
template <int N>
__device__ __forceinline__ DF<N> slope2(DF<N> d0, DF<N> d1, DF<N> w, FV<N> k4) {
  return limit(w, df_sel(same_sign(df_diff(d0, d1), d0.h), d1, d0), k4);
}
// The two face terms A, B of a face from x, the limited q_f - q_{f-1} (upwind below) or q_f' of
// the cell above, and y, the rest of the neighbour difference
template <int N>
__device__ __forceinline__ void face_terms(DF<N> x, DF<N> y, bool right, DF<N>& A, DF<N>& B) {
  A = right ? x : y;
  B = right ? y : x;
}
// Uniform directions: 6 D, 12 E_p = 6 D_p - (S'_{p+1} - S'_p) and 12 L_{p+1} = 6 D_p + (S'_{p+1} -
// S'_p), L = -eL.  Both slopes are limited by 4 D_p and have its sign, so |dS'| <= 4 |D_p|: no
// cancellation, E_p and L_{p+1} have the sign of D_p and need no normalisation.
template <int N>
__device__ __forceinline__ void edges_u(DF<N> D, DF<N> S0, DF<N> S1, DF<N>& t, DF<N>& E, DF<N>& Lnext) {
  t = times6(D);
  const DF<N> ds = sub_raw(S1, S0);
  E = sub_big(t, ds);
  Lnext = add_big(t, ds);
}
// x = 12 (limited deviation) lies between 0 and 10 D: the rest of 12 D does not cancel
template <int N>
__device__ __forceinline__ DF<N> rest_u(DF<N> t, DF<N> x) { return sub_big(df_scale(t, 2.0f), x); }
// dp-weighted: E_p = ab D_p + c S_{p+1} + d S_p with the coefficients of edge p+1; L = D - E of
// the cell before
template <int N>
__device__ __forceinline__ DF<N> edge_n(DF<N> D, DF<N> S0, DF<N> S1, DF<N> ab, DF<N> c, DF<N> d) {
  return df_fma(d, S0, fma_raw(c, S1, mul_raw(ab, D)));
}
template <int N>
__device__ __forceinline__ DF<N> centre_n(DF<N> d0, DF<N> d1, DF<N> sA, DF<N> sB) {  // twice the centred slope
  return df_fma(sA, d1, mul_raw(sB, d0));
}
// the upwind cell is the one below the face: sign of g M (gs: the bits of g's high word)
__device__ __forceinline__ bool upwind_lo(float M, int gs) { return (__float_as_int(M) ^ gs) >= 0; }
// split a double into a pair: production build with integer operations (split_bits below, hi + lo = v
// to 2^-49), strict build with conversions
__device__ __forceinline__ df split_df(double v);
// The conversions of values outside the integer forms' range are calls: as short branches they are
// predicated, and an FP64-pipe instruction holds the pipe for its 64 cycles with no lane active too
// (57 of the 88 such instructions of a cell's stage 4 with 12 tracers were of this kind).
__device__ __noinline__ double f2d_convert(float x) { return (double)x; }
__device__ __noinline__ float2 split_convert(double v) {
  const float h = (float)v;
  return make_float2(h, (float)(v - (double)h));
}
// float -> double by re-biasing the exponent in the integer pipes (exact; zero kept, subnormal,
// inf and NaN convert)
__device__ __forceinline__ double f2d_bits(float x) {
  const unsigned u = __float_as_uint(x);
  const unsigned fe = (u >> 23) & 0xffu;
  if ((u << 1) == 0u) return __hiloint2double((int)(u & 0x80000000u), 0);
  if (fe == 0u || fe == 255u) return f2d_convert(x);
  return __hiloint2double((int)((u & 0x80000000u) | ((fe + 896u) << 20) | ((u & 0x7fffffu) >> 3)),
                          (int)(u << 29));
}
__device__ __forceinline__ double df_to_d(df v) {
#if RS_STRICT
  return (double)v.h.v + (double)v.l.v;
#else
  return f2d_bits(v.h.v) + f2d_bits(v.l.v);
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
  const int gs = __double2hiint(g);  // only its sign is needed here
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
    const df M = df_ldp(T.mx12, ((size_t)k * T.nlat + j) * nf + f);
    Mh[bck(T, f, mixed_frows(n))] = M.h.v;
    Ml[bck(T, f, mixed_frows(n))] = M.l.v;
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
      Dh[X(p)] = d.h.v;
      Dl[X(p)] = d.l.v;
    }
    __syncthreads();
    for (int p = tid - 2; p <= n + 1; p += blockDim.x) {
      const df d0 = df_ld(Dh, Dl, X(p - 1)), d1 = df_ld(Dh, Dl, X(p));
      const df sl = slope2(d0, d1, df_add(d0, d1), live(d0, d1, 4.0f));
      Sh[X(p)] = sl.h.v;
      Sl[X(p)] = sl.l.v;
    }
    __syncthreads();
    for (int p = tid - 2; p <= n; p += blockDim.x) {  // edge terms over the staged values
      df t, e, lnext;
      edges_u(df_ld(Dh, Dl, X(p)), df_ld(Sh, Sl, X(p)), df_ld(Sh, Sl, X(p + 1)), t, e, lnext);
      H[X(p)] = e.h.v;
      Lo[X(p)] = e.l.v;
    }
    __syncthreads();
    auto face = [&](int f, df& A, df& B) {
      const bool right = upwind_lo(Mh[bck(T, f, nf)], gs);
      const int up = right ? f - 1 : f;
      const df Dm = df_ld(Dh, Dl, X(up - 1)), Er = df_ld(H, Lo, X(up));
      df t, e, l;
      edges_u(Dm, df_ld(Sh, Sl, X(up - 1)), df_ld(Sh, Sl, X(up)), t, e, l);
      const df x = limit(right ? Er : l, right ? l : Er, live(Dm, df_ld(Dh, Dl, X(up)), 2.0f));
      face_terms(x, rest_u(times6(df_ld(Dh, Dl, X(f - 1))), x), right, A, B);
    };
    for (int p = tid; p < n; p += blockDim.x) {
      df A, B, o;
      face(p, o, B);
      face(p + 1, A, o);
      const df a = fma_raw(mkdf(Mh[bck(T, p + 1, nf)], Ml[bck(T, p + 1, nf)]), A,
                           mul_raw(mkdf(Mh[bck(T, p, nf)], Ml[bck(T, p, nf)]), B));
      T.acc.h[bck(T, pb + p, nall)] = a.h.v;
      T.acc.l[bck(T, pb + p, nall)] = a.l.v;
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
  const int gs = __double2hiint(g);  // only its sign is needed here
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
  // the fluxes as the cell below the face sees them, [n+1][kPencil] (those of the cell above a lat
  // face come from the cache: staging them too would shrink the largest grid that fits)
  float* const Nh = Sl + R;
  float* const Nl = Nh + (n + 1) * kPencil;
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
  const bool inside = DIR == 1 ? i < T.nlon : col < ncol;
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
  if (inside)
    for (int f = ty; f <= n; f += blockDim.y) {
      const long long m = bck(T, f * kPencil + tx, mb);
      if (DIR == 1) {  // zero through closed walls
        const size_t x = ((size_t)k * (n + 1) + f) * T.nlon + i;
        Nh[m] = T.myn12.h[x];
        Nl[m] = T.myn12.l[x];
      } else {  // no flux through the surface and the model top
        const bool in = f > 0 && f < n;
        Nh[m] = in ? T.mz2.h[(size_t)f * ncol + col] : 0.0f;
        Nl[m] = in ? T.mz2.l[(size_t)f * ncol + col] : 0.0f;
      }
    }
  for (int s = s0; s < s1; ++s) {
    const int it = s - s0, b = kTma ? (it & 1) : 0;
    float* H = b ? H1 : H0;
    float* Lo = b ? L1 : L0;
    const size_t pb = (size_t)s * nc + cbase;
    auto cell = [&](int p, float& h, float& l) {  // a ghost (p outside 0..n-1) or interior cell
      h = 0.0f;
      l = 0.0f;
      if (!inside) return;
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
      const df d = df_sub(mkdf(RS_P(H, p + 1), RS_P(Lo, p + 1)), mkdf(RS_P(H, p), RS_P(Lo, p)));
      RS_P(Dh, p) = d.h.v;
      RS_P(Dl, p) = d.l.v;
    }
    __syncthreads();
#define RS_PP(a, b, p) mkdf(RS_P(a, p), RS_P(b, p))
    for (int p = (int)ty - 2; p <= n + 1; p += blockDim.y) {
      const df d0 = RS_PP(Dh, Dl, p - 1), d1 = RS_PP(Dh, Dl, p);
      df sl = mkdf(0.0f, 0.0f);
      if (DIR == 1) {
        sl = slope2(d0, d1, df_add(d0, d1), live(d0, d1, 4.0f));
      } else if (p >= -1 && p <= n && inside) {  // slopes of cells -1..n (coefficient row p+1)
        const size_t x = bck(T, (size_t)(p + 1) * ncol + col, (long long)(n + 2) * ncol);
        sl = slope2(d0, d1, centre_n(d0, d1, df_ldp(T.vsA2, x), df_ldp(T.vsB2, x)), live(d0, d1, 4.0f));
      }
      RS_P(Sh, p) = sl.h.v;
      RS_P(Sl, p) = sl.l.v;
    }
    __syncthreads();
    // edge terms over the staged values: cells -2..n (uniform), -1..n-1 (coefficient rows
    // 0..n of the dp-weighted edges)
    for (int p = (int)ty - 2; p <= n; p += blockDim.y) {
      const df Dp = RS_PP(Dh, Dl, p), Sp = RS_PP(Sh, Sl, p), Sp1 = RS_PP(Sh, Sl, p + 1);
      df e = mkdf(0.0f, 0.0f), l, t;
      if (DIR == 1) {
        edges_u(Dp, Sp, Sp1, t, e, l);
      } else if (p >= -1 && p <= n - 1 && inside) {
        const size_t x = bck(T, (size_t)(p + 1) * ncol + col, (long long)(n + 1) * ncol);
        e = edge_n(Dp, Sp, Sp1, df_ldp(T.veAB2, x), df_ldp(T.veC2, x), df_ldp(T.veD2, x));
      }
      RS_P(H, p) = e.h.v;
      RS_P(Lo, p) = e.l.v;
    }
    __syncthreads();
    auto face = [&](int f, df& A, df& B) {
      A = B = mkdf(0.0f, 0.0f);
      if (DIR == 2 && (f == 0 || f == n)) return;
      const bool right = upwind_lo(Nh[bck(T, f * kPencil + tx, mb)], gs);
      const int up = right ? f - 1 : f;
      const df Dm = RS_PP(Dh, Dl, up - 1), D = RS_PP(Dh, Dl, f - 1), Er = RS_PP(H, Lo, up);
      df t, e, l, x, y;
      if (DIR == 1) {
        edges_u(Dm, RS_PP(Sh, Sl, up - 1), RS_PP(Sh, Sl, up), t, e, l);
        x = limit(right ? Er : l, right ? l : Er, live(Dm, RS_PP(Dh, Dl, up), 2.0f));
        y = rest_u(times6(D), x);
      } else {
        l = df_sub(Dm, RS_PP(H, Lo, up - 1));
        x = limit(right ? Er : l, right ? l : Er, live(l, Er, 2.0f));
        y = sub_raw(D, x);
      }
      face_terms(x, y, right, A, B);
    };
    if (inside) {
      for (int p = ty; p < n; p += blockDim.y) {
        df A, B, o;
        face(p, o, B);
        face(p + 1, A, o);
        const size_t x = bck(T, pb + (size_t)p * stride, nall);
        const long long ms = bck(T, p * kPencil + tx, mb), mn = bck(T, (p + 1) * kPencil + tx, mb);
        const df Ms = DIR == 1 ? df_ldp(T.mys12, ((size_t)k * (n + 1) + p) * T.nlon + i) : mkdf(Nh[ms], Nl[ms]);
        const df t = fma_raw(mkdf(Nh[mn], Nl[mn]), A, fma_raw(Ms, B, mkdf(T.acc.h[x], T.acc.l[x])));
        T.acc.h[x] = t.h.v;
        T.acc.l[x] = t.l.v;
      }
    }
    __syncthreads();
  }
#undef RS_PP
#undef RS_P
}

// ---- streaming forms of the mixed pencils (no shared memory, no barriers).  The same pair
// operations in the same order as k_adv_x_mixed / k_adv_yz_mixed, so the accumulators are bit
// for bit those of the pencils; rs_autotune picks per direction.  N tracers side by side in the
// halves of packed operations (an odd last tracer runs beside a copy of itself that is not
// stored).
template <int N>
struct Tracers {  // this block's tracers s .. s + N - 1, of which the second may not count
  size_t off[N];
  bool two;
  __device__ __forceinline__ Tracers(int s, int s1, size_t nc) : two(N == 2 && s + 1 < s1) {
#pragma unroll
    for (int i = 0; i < N; ++i) off[i] = (size_t)min(s + i, s1 - 1) * nc;
  }
  // the plane offsets are the same for the whole block, the cell's is 32 bits: addresses then cost
  // no 64-bit arithmetic per thread
  __device__ __forceinline__ DF<N> load(const float* H, const float* L, unsigned x) const {
    if constexpr (N == 1) return {{(H + off[0])[x]}, {(L + off[0])[x]}};
    else return {{pack2((H + off[0])[x], (H + off[1])[x])}, {pack2((L + off[0])[x], (L + off[1])[x])}};
  }
  __device__ __forceinline__ void store(float* H, float* L, unsigned x, const DF<N>& v) const {
    (H + off[0])[x] = half(v.h, 0);
    (L + off[0])[x] = half(v.l, 0);
    if constexpr (N == 2)
      if (two) {
        (H + off[1])[x] = half(v.h, 1);
        (L + off[1])[x] = half(v.l, 1);
      }
  }
};
// an open wall's ghost: the prescribed boundary values of the thread's tracers
template <int N>
__device__ __forceinline__ DF<N> ghost_df(const DevTransport<double>& T, const double* b, int s, int s1,
                                          size_t plane, size_t x, long long n) {
  float h[2], l[2];
#pragma unroll
  for (int i = 0; i < N; ++i) split_d(b[bck(T, (size_t)min(s + i, s1 - 1) * plane + x, n)], h[i], l[i]);
  if constexpr (N == 1) return {{h[0]}, {l[0]}};
  else return {{pack2(h[0], h[1])}, {pack2(l[0], l[1])}};
}

// Lon rows: one warp per segment of kSegX = 26 cells of a row; lane l holds cell
// p = base - 3 + l, and the neighbour values the stencil needs move between lanes by shuffles.
// Each lane limits both edges of its own cell, so that its west face takes the neighbour's right
// deviation or its own left one; cells at lanes 3..28 have their east face's A from lane l+1.
constexpr int kSegX = 26;
template <int N>
__device__ __forceinline__ FV<N> shfl_up_v(FV<N> v, int d) {
  if constexpr (N == 1) return {__shfl_up_sync(0xffffffffu, v.v, d)};
  else return {pack2(__shfl_up_sync(0xffffffffu, half(v, 0), d), __shfl_up_sync(0xffffffffu, half(v, 1), d))};
}
template <int N>
__device__ __forceinline__ FV<N> shfl_down_v(FV<N> v, int d) {
  if constexpr (N == 1) return {__shfl_down_sync(0xffffffffu, v.v, d)};
  else return {pack2(__shfl_down_sync(0xffffffffu, half(v, 0), d), __shfl_down_sync(0xffffffffu, half(v, 1), d))};
}
template <int N>
__device__ __forceinline__ DF<N> shfl_up_df(DF<N> v, int d) { return {shfl_up_v(v.h, d), shfl_up_v(v.l, d)}; }
template <int N>
__device__ __forceinline__ DF<N> shfl_down_df(DF<N> v, int d) { return {shfl_down_v(v.h, d), shfl_down_v(v.l, d)}; }

template <int N>
__global__ void __launch_bounds__(128) k_adv_x_stream(DevTransport<double> T, StageSel sel,
                                                      int sper) {
  const double* Q;
  double g;
  if (!resolve_stage(sel, Q, g)) return;
  const int gs = __double2hiint(g);  // only its sign is needed here
  const int n = T.nlon, nf = n + 1;
  const int nseg = (n + kSegX - 1) / kSegX;
  const int lane = threadIdx.x & 31;
  const int ngrp = (T.ntr + sper - 1) / sper;  // the tracer groups are the fastest grid dimension
  const long long wg = (long long)(blockIdx.x / ngrp) * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (wg >= (long long)nseg * T.nlat * T.nlev) return;  // whole warps leave together
  const int row = (int)(wg / nseg), seg = (int)(wg % nseg);
  const int p = seg * kSegX - 3 + lane;  // this lane's cell (and west face)
  const size_t nc = (size_t)T.nlon * T.nlat * T.nlev;
  const size_t rbase = (size_t)row * n;
  const bool periodic = T.lon_bc == 0;
  const df M1 = (p >= 0 && p <= n) ? df_ldp(T.mx12, (size_t)row * nf + p) : mkdf(0.0f, 0.0f);
  const bool right = upwind_lo(M1.h.v, gs);
  const DF<N> Mw = splat_df<N>(M1.h.v, M1.l.v);
  const df E1 = shfl_down_df(M1, 1);
  const DF<N> Me = splat_df<N>(E1.h.v, E1.l.v);
  const bool out = lane >= 3 && lane <= 28 && p >= 0 && p < n;
  const int pw = periodic ? ((p % n) + n) % n : p;
  const int s0 = (int)(blockIdx.x % ngrp) * sper, s1 = min(T.ntr, s0 + sper);
  for (int s = s0; s < s1; s += N) {
    const Tracers<N> tr(s, s1, nc);
    DF<N> q;
    if (pw >= 0 && pw < n) q = tr.load(T.qhi, T.qlo, (unsigned)(rbase + bck(T, pw, n)));
    else q = ghost_df<N>(T, p < 0 ? T.qw : T.qe, s, s1, (size_t)T.nlev * T.nlat, row, (long long)T.ntr * T.nlev * T.nlat);
    const DF<N> D = df_sub(shfl_down_df(q, 1), q);              // D(p), lanes 0..30
    const DF<N> Dm = shfl_up_df(D, 1);                          // D(p-1)
    const FV<N> k4 = live(Dm, D, 4.0f);
    const DF<N> S = slope2(Dm, D, df_add(Dm, D), k4);           // lanes 1..30
    DF<N> t, E, Ln;
    edges_u(D, S, shfl_down_df(S, 1), t, E, Ln);                // E(p), L(p+1), lanes 1..29
    const DF<N> L = shfl_up_df(Ln, 1), tm = shfl_up_df(t, 1);   // lanes 2..30
    const FV<N> k2 = vmul(k4, splat<N>(0.5f));
    const DF<N> xRm = shfl_up_df(limit(E, L, k2), 1);           // of cell p-1, lanes 3..30
    const DF<N> x = right ? xRm : limit(L, E, k2);
    DF<N> A, B;
    face_terms(x, rest_u(tm, x), right, A, B);
    const DF<N> Ae = shfl_down_df(A, 1);  // the east face's A, formed by lane + 1
    if (out) tr.store(T.acc.h, T.acc.l, (unsigned)(rbase + p), fma_raw(Me, Ae, mul_raw(Mw, B)));
  }
}

// Lat (DIR 1) and vertical (DIR 2) lines: one thread per line (consecutive lon points over all
// levels, or consecutive columns), walking the line once per N tracers with a register window:
// when q(p) arrives, D(p-1), S(p-1), E(p-2), L(p-1) are formed and face p-2 is complete; its A
// closes cell p-3 and its B opens cell p-2.  The tracer groups are the fastest grid dimension:
// the fluxes and coefficients of a set of lines are read from DRAM once and come from L2 for the
// other groups.
constexpr int kLine32 = 64;  // threads per block of the line kernels
// Blocks per SM (168 registers) and iterations that a line's loads run ahead.  Both directions
// together, 360x181x72 / 144x91x47: 6 x 4 1.84 ms / 145 us, 6 x 3 1.81 / 143, 6 x 2 1.86 / 141,
// 8 x 2 (128 registers, spilling) 1.75 / 145, no bound and 4 ahead (192-220 registers, a second wave
// of a few blocks) 2.13 / 176.
constexpr int kLineBlocks = 6;
constexpr int kAhead = 3;
template <int DIR, int N>
__global__ void __launch_bounds__(kLine32, kLineBlocks) k_adv_yz_stream(DevTransport<double> T, StageSel sel,
                                                           int sper) {
  const double* Q;
  double g;
  if (!resolve_stage(sel, Q, g)) return;
  const int gs = __double2hiint(g);  // only its sign is needed here
  const int n = DIR == 1 ? T.nlat : T.nlev;
  const unsigned ncol = (unsigned)(T.nlon * T.nlat);
  const size_t nc = (size_t)ncol * T.nlev;
  const unsigned ngrp = (unsigned)((T.ntr + sper - 1) / sper);
  const unsigned id = blockIdx.x / ngrp * blockDim.x + threadIdx.x;
  if (id >= (DIR == 1 ? (unsigned)(T.nlon * T.nlev) : ncol)) return;
  const unsigned k = DIR == 1 ? id / T.nlon : 0, i = DIR == 1 ? id % T.nlon : 0;
  const unsigned stride = DIR == 1 ? (unsigned)T.nlon : ncol;
  const unsigned cbase = DIR == 1 ? k * ncol + i : id;
  const unsigned fb = DIR == 1 ? k * (unsigned)(n + 1) * T.nlon + i : id;  // face 0 of the line
  const bool open = DIR == 1 && T.lat_bc == 1;
  const int s0 = (int)(blockIdx.x % ngrp) * sper, s1 = min(T.ntr, s0 + sper);
  for (int s = s0; s < s1; s += N) {
    const Tracers<N> tr(s, s1, nc);
    auto cell = [&](int p) { return cbase + (unsigned)bck(T, p, n) * stride; };
    auto value = [&](int p, bool edge) -> DF<N> {
      if (edge && (p < 0 || p >= n)) {
        if (open)
          return ghost_df<N>(T, p < 0 ? T.qs : T.qn, s, s1, (size_t)T.nlev * T.nlon, (size_t)k * T.nlon + i,
                             (long long)T.ntr * T.nlev * T.nlon);
        p = p < 0 ? -1 - p : 2 * n - 1 - p;  // mirror ghosts at the walls
      }
      return tr.load(T.qhi, T.qlo, cell(p));
    };
    const DF<N> z = splat_df<N>(0.0f, 0.0f);
    const FV<N> z1 = splat<N>(0.0f);
    // what iteration p reads: q(p), face p-2's fluxes, the accumulator of the cell above that face,
    // the coefficients of slope p-1 and edge p-2.  kAhead iterations are in flight.
    struct In {
      DF<N> q, a;
      df mn, ms, sA, sB, ab, c, d;
    };
    auto fetch = [&](int p, bool edge, In& in) {
      const int f = p - 2;
      if (!edge || p <= n + 2) in.q = value(p, edge);
      if (!edge || (f >= 0 && f <= n)) {
        const unsigned x = fb + (unsigned)f * stride;
        if (DIR == 1) {
          in.mn = df_ldp(T.myn12, x);
          in.ms = df_ldp(T.mys12, x);
        } else {
          in.mn = !edge || (f > 0 && f < n) ? df_ldp(T.mz2, x) : mkdf(0.0f, 0.0f);
        }
        if (!edge || f < n) in.a = tr.load(T.acc.h, T.acc.l, cell(f));
      }
      if (DIR == 2) {
        if (!edge || (p >= 0 && p <= n + 1)) {  // slopes of cells -1..n (coefficient row of cell + 1)
          const unsigned x = (unsigned)bck(T, p, n + 2) * ncol + id;
          in.sA = df_ldp(T.vsA2, x);
          in.sB = df_ldp(T.vsB2, x);
        }
        if (!edge || (f >= -1 && f <= n - 1)) {  // right edges of cells -1..n-1 (row f+1)
          const unsigned x = (unsigned)bck(T, f + 1, n + 1) * ncol + id;
          in.ab = df_ldp(T.veAB2, x);
          in.c = df_ldp(T.veC2, x);
          in.d = df_ldp(T.veD2, x);
        }
      }
    };
    auto both = [](df v) { return splat_df<N>(v.h.v, v.l.v); };
    // window: qp = q(p-1); D3, D2 = D(p-3), D(p-2), t3, t2 = 6 D; S1 = S(p-1); E3, E2 = E(p-3),
    // E(p-2); L3, L2, L1 and k3, k2, k1 (live) of cells p-3, p-2, p-1; ac the open cell's
    // accumulator
    DF<N> qp = value(-2, true), D3 = z, D2 = df_sub(qp, value(-3, true)), t3 = z, t2 = z, S1 = z;
    DF<N> E3 = z, E2 = z, L3 = z, L2 = z, L1 = z, ac = z;
    FV<N> k3 = z1, k2 = z1, k1 = z1;
    auto step = [&](int p, bool edge, const In& in) {  // edge: near a wall, every range is checked
      const int f = p - 2;
      const DF<N> D1 = df_sub(in.q, qp);  // D(p-1)
      qp = in.q;
      const DF<N> S2 = S1;
      E3 = E2;
      L3 = L2;
      k3 = k2;
      if (DIR == 1) {
        const FV<N> k4 = live(D2, D1, 4.0f);
        S1 = slope2(D2, D1, df_add(D2, D1), k4);  // S(p-1)
        t3 = t2;
        L2 = L1;
        k2 = k1;
        k1 = vmul(k4, splat<N>(0.5f));
        edges_u(D2, S2, S1, t2, E2, L1);
      } else {
        if (!edge || (p >= 0 && p <= n + 1))
          S1 = slope2(D2, D1, centre_n(D2, D1, both(in.sA), both(in.sB)), live(D2, D1, 4.0f));
        if (!edge || (f >= -1 && f <= n - 1)) {
          E2 = edge_n(D2, S2, S1, both(in.ab), both(in.c), both(in.d));
          L2 = df_sub(D3, E3);
        }
      }
      if (!edge || f >= 0) {  // the face now complete
        DF<N> A = z, B = z;
        if (DIR == 1 || !edge || (f > 0 && f < n)) {
          const bool right = upwind_lo(in.mn.h.v, gs);
          const DF<N> self = right ? E3 : L2, other = right ? L3 : E2;
          DF<N> x, y;
          if (DIR == 1) {
            x = limit(self, other, right ? k3 : k2);
            y = rest_u(t3, x);
          } else {
            x = limit(self, other, live(other, self, 2.0f));
            y = sub_raw(D3, x);
          }
          face_terms(x, y, right, A, B);
        }
        if (!edge || f >= 1)  // cell f-1 is complete
          tr.store(T.acc.h, T.acc.l, cell(f - 1), fma_raw(both(in.mn), A, ac));
        ac = fma_raw(both(DIR == 1 ? in.ms : in.mn), B, in.a);
      }
      D3 = D2;
      D2 = D1;
    };
    In buf[kAhead];
#pragma unroll
    for (int j = 0; j < kAhead; ++j) fetch(-1 + j, true, buf[j]);
    for (int p = -1; p <= n + 2; p += kAhead) {
      if (p >= 3 && p + 2 * kAhead <= n) {  // this group and the one it fetches are inside
#pragma unroll
        for (int j = 0; j < kAhead; ++j) {
          const In in = buf[j];
          fetch(p + kAhead + j, false, buf[j]);
          step(p + j, false, in);
        }
      } else {
#pragma unroll
        for (int j = 0; j < kAhead; ++j) {
          const In in = buf[j];
          fetch(p + kAhead + j, true, buf[j]);
          if (p + j <= n + 2) step(p + j, true, in);
        }
      }
    }
  }
}

// ------------------------------------------------------------------ stage kernel
#if !RS_STRICT
// hi + lo split without FP64-pipe conversions (production build): hi = v rounded to 24
// significant bits, lo = the remainder rounded to 24 -- hi + lo = v to 2^-49 relative, without
// bias, and |lo| <= ulp(hi) / 2 as the sums of pairs expect.  (Truncating both, the error of every
// state had the sign of the state and lo was up to a whole ulp: one transport step was off by 5.3e-16
// rms of a tracer's largest value and 2.7e-14 of each value at most, now 3.1e-16 and 1.4e-14.)
// Values outside [2^-74, 2^126) (zero, subnormals, inf, NaN included) convert.
__device__ __forceinline__ void split_bits(double v, float& hi, float& lo) {
  const unsigned h = (unsigned)__double2hiint(v), l = (unsigned)__double2loint(v);
  const int e = (int)((h >> 20) & 0x7ff);
  if (e < 949 || e > 1148) {
    const float2 p = split_convert(v);
    hi = p.x;
    lo = p.y;
    return;
  }
  const unsigned sign = h & 0x80000000u;
  // the 29 mantissa bits below hi, as a signed remainder: from half an ulp on hi goes up by one
  const int r = (int)(l << 3) >> 3;
  const unsigned up = (l >> 28) & 1u;
  hi = __uint_as_float(sign | ((((unsigned)(e - 896) << 23) | ((h & 0xfffffu) << 3) | (l >> 29)) + up));
  const float d = __fmul_rn(__int2float_rn(r), __uint_as_float((unsigned)(e - 948) << 23));
  lo = __uint_as_float(__float_as_uint(d) ^ sign);
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
  float h, l;
#if RS_STRICT
  h = (float)v;
  l = (float)(v - (double)h);
#else
  split_bits(v, h, l);
#endif
  return mkdf(h, l);
}

// hi and lo planes of scale times a double array (the air-mass face fluxes of the mixed kernels)
__global__ void k_make_pairs(const double* __restrict__ src, double scale, float* __restrict__ hi,
                             float* __restrict__ lo, size_t n) {
  const size_t x = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (x < n) {
    const df v = split_df(src[x] * scale);
    hi[x] = v.h.v;
    lo[x] = v.l.v;
  }
}
void launch_make_pairs(cudaStream_t st, const double* src, double scale, float* dst, size_t n) {
  if (n) k_make_pairs<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(src, scale, dst, dst + n, n);
}

// The air-mass fluxes with the cells' metric and the uniform edges' 1/6 folded in: mx6 (both
// cells of a lon face share the row's factor), myn6 / mys6 (as the cell south / north of a lat face
// sees it; zero through closed walls; the south-most open face has no cell south of it, its myn6
// serves the upwind direction only).  Once per forcing change.
__global__ void k_scale_fluxes(DevTransport<double> T, double* __restrict__ mx6,
                               double* __restrict__ myn6, double* __restrict__ mys6) {
  const size_t x = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const size_t nx = (size_t)T.nlev * T.nlat * (T.nlon + 1), ny = (size_t)T.nlev * (T.nlat + 1) * T.nlon;
  if (x < nx) mx6[x] = T.mx[x] * (T.gx[(x / (T.nlon + 1)) % T.nlat] * kOneSixth);
  if (x < ny) {
    const int f = (int)((x / T.nlon) % (T.nlat + 1));
    const bool wall = T.lat_bc != 1 && (f == 0 || f == T.nlat);
    const double m = T.my[x];
    myn6[x] = wall ? 0.0 : m * ((f > 0 ? T.gyhi[f - 1] : T.gylo[0]) * kOneSixth);
    mys6[x] = wall || f == T.nlat ? 0.0 : m * (T.gylo[f] * kOneSixth);
  }
}

// split the attempt's input state U[cur] (stage 1's RHS argument) into hi/lo planes
__global__ void __launch_bounds__(kRedThreads) k_split_input(DevTransport<double> T,
                                                             const Ctl* ctl, const double* U0,
                                                             const double* U1, const double* Qd) {
  const double* U;
  await_previous();
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
// The air-mass flux divergence of every cell at time factor 1, once per forcing change: formed by the
// stage kernels it was 16 of their 26 FP64 instructions per cell, four times per attempt.
__global__ void k_air_divergence(DevTransport<double> T, double* __restrict__ mdiv) {
  const size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= (size_t)T.nlon * T.nlat * T.nlev) return;
  const int i = (int)(c % T.nlon), j = (int)((c / T.nlon) % T.nlat);
  double hz, vz;
  div_parts(T, i, j, (int)(c / ((size_t)T.nlon * T.nlat)), 1.0, CellGeo{T.gx[j], T.gylo[j], T.gyhi[j]}, hz, vz);
  mdiv[c] = hz + vz;
}
void launch_air_divergence(cudaStream_t st, const DevTransport<double>& T, double* mdiv) {
  const size_t nc = (size_t)T.nlon * T.nlat * T.nlev;
  k_air_divergence<<<(unsigned)((nc + 255) / 256), 256, 0, st>>>(T, mdiv);
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
      acc = acc + T.pbl_w[(size_t)k * ncol + col] * df_to_d(mkdf(T.qhi[x], T.qlo[x]));
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
//   4: unew = S3 + dt/2 f(S3); err = 1/2 ((U - u3) / 3 + (u3 - unew)); candidate = clamp(unew)
template <int STAGE>
__global__ void __launch_bounds__(kRedThreads) k_stage(DevTransport<double> T,
                                                       const Ctl* ctl,
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
constexpr float kThirdH = (float)(1.0 / 3.0);
constexpr float kThirdL = (float)(1.0 / 3.0 - (double)(float)(1.0 / 3.0));
__device__ __forceinline__ df df_abs(df a) {  // of a normalised pair
  const unsigned sg = __float_as_uint(a.h.v) & 0x80000000u;
  return mkdf(fabsf(a.h.v), __uint_as_float(__float_as_uint(a.l.v) ^ sg));
}
// a / b: the quotient of the leading parts and one correction from the exact remainder
__device__ __forceinline__ df df_div(df a, df b) {
  float r;
  asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(b.h.v));
  const float q = __fmul_rn(a.h.v, r);
  const float rem = __fmaf_rn(-q, b.l.v, __fadd_rn(__fmaf_rn(-q, b.h.v, a.h.v), a.l.v));
  return df_renorm(df{{q}, {__fmul_rn(rem, r)}});
}
// one tracer's squared error ratio in FP64, for what is outside the pairs' range (and NaN); a call
// for the reason given at f2d_convert
__device__ __noinline__ double error_fp64(float dh, float dl, double am, double rtol, double atol) {
  const double at = df_to_d(mkdf(dh, dl)) * rcp_nr1(fma(am, rtol, atol));  // den >= atol > 0
  return at * at;
}
// One tracer's error err against the tolerance of |u|: (err / (am rtol + atol))^2 added to the pair
// ep on the FP32 pipe, or to e in FP64 where the pairs' range does not hold it.  The split is
// branch-free: h the leading 24 bits, l the 29 below them rounded to 24 (fewer below 2^-74; 0 below
// 2^-126).
__device__ __forceinline__ df split_any(double v, unsigned& big) {
  const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
  const unsigned mag = hi & 0x7fffffffu;
  big = max(big, mag);
  const unsigned f = (__funnelshift_l(lo, hi, 3) ^ 0x40000000u) & 0x7fffffffu;  // exponent - 896
  const int sc = max((int)(f & 0x7f800000u) - (52 << 23), 0);
  const float l = __fmul_rn(__int2float_rn((int)(lo & 0x1fffffffu)), __int_as_float(sc));
  const unsigned sg = hi & 0x80000000u;
  const bool z = mag < (898u << 20);
  return mkdf(z ? 0.0f : __uint_as_float(f | sg), z ? 0.0f : __uint_as_float(__float_as_uint(l) ^ sg));
}
__device__ __noinline__ double error_term(double err, double am, double rtol, double atol) {
  const double at = err * rcp_nr1(fma(am, rtol, atol));  // den >= atol > 0
  return at * at;
}
__device__ __forceinline__ void add_error(double err, double am, double rtol, double atol, df rt, df at0,
                                          bool pairs, df& ep, double& e) {
  unsigned big = 0;
  const df t = df_div(split_any(err, big), df_fma(split_any(am, big), rt, at0));
  if (pairs && big < (1126u << 20) && fabsf(t.h.v) < 0x1p60f) ep = df_fma(t, t, ep);
  else e += error_term(err, am, rtol, atol);
}
#include "rs_adv64.cuh"

// Compensated-FP32 stage kernel (mixed precision).  The tracers of stages 1-3 stay pairs:
// the stage input is the (hi, lo) planes, the update q + dt/2 * (m dq/dt) / m is formed in pairs
// and written back into those planes (in place: the update is pointwise), u3 is kept as hi and lo
// planes in the tracer part of S1; stage 4 returns to FP64 with the candidate state.  Its embedded
// error and the hairer norm are formed in pairs as well (relative error ~1e-13 after the one
// cancellation, which the pairs of the states carry anyway; the FP64 form's one-step reciprocal has
// 1e-12): eight FP64 instructions per cell and tracer, 64 cycles each, had made this stage five
// times as long as the others (144x91x47: 211 us against 41, now 86; 360x181x72 with 30 tracers
// 3.47 ms).  Stages 1-2 take 32 us there, close to the 30 us of their bytes.
// The air-mass row is the FP64 scheme's, stage by stage (m in the air-mass planes of U, S1, S2, S3).
//   1: P = U + dt/2 f(U)          2: P = P + dt/2 f(P)
//   3: u3 = P + dt/2 f(P) -> S1 (pairs), P = u4 = U + (u3 - U) / 3
//   4: unew = P + dt/2 f(P); err = 1/2 ((U - u3) / 3 + (u3 - unew)); candidate = clamp(unew)
template <int STAGE>
__global__ void __launch_bounds__(kRedThreads) k_stage_mixed(DevTransport<double> T,
                                                             const Ctl* ctl,
                                                             TransportBufs B, double rtol,
                                                             double atol, int clamp) {
  __shared__ double sm[kRedThreads];
  await_previous();
  if (ctl->done) return;
  const double g = ctl->g[STAGE - 1];
  const int cur = ctl->cur;
  const double* U = cur ? B.U1 : B.U0;
  double* Un = cur ? B.U0 : B.U1;
  const double dt_2 = ctl->dtc / 2;
  // air mass of the stage input
  const double* Qm = STAGE == 1 ? U : (STAGE == 2 ? B.S1 : (STAGE == 3 ? B.S2 : B.S3));
  const size_t nc = (size_t)T.nlon * T.nlat * T.nlev;
  float* u3h = reinterpret_cast<float*>(B.S1);  // u3 of the tracers, hi and lo planes [ntr][nc]
  float* u3l = u3h + (size_t)T.ntr * nc;
  const df c13 = mkdf(kThirdH, kThirdL);
  const df rt = split_df(rtol), at0 = split_df(atol);
  const bool pairs = atol >= 0x1p-100 && atol <= 0x1p100 && rtol >= 0x1p-60;  // else the norm in FP64
  const size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  double e = 0.0;
  df ep = mkdf(0.0f, 0.0f);
  if (c < nc) {
    const double dmdt = T.mcorr ? -fma(g, T.mdiv[c], T.mcorr[c]) : -(g * T.mdiv[c]);
    const size_t xm = (size_t)(T.nsp - 1) * nc + c;
    const double m = Qm[xm];
#if RS_STRICT
    const double rmg = g / m;
#else
    const double rmg = g * rcp_nr(m);  // m > 0
#endif
    const df sc = split_df(-dt_2 * rmg);  // the tracer increment is acc * sc
    const size_t col = c % ((size_t)T.nlon * T.nlat);
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
    auto tracer = [&](int s, size_t x, df q, df a, double u0, df u3) {
      df nx;
      if (T.pbl) {  // with full PBL mixing the tendency is formed in FP64 (rare combination)
        const double qd = df_to_d(q);
        const double du = fma(-df_to_d(a), rmg, pbl_term(T, c, col, s, qd));
        nx = split_df(fma(du, dt_2, qd));
      } else {
        nx = df_fma(a, sc, q);
      }
      if (STAGE == 1 || STAGE == 2) {
        T.qhi[x] = nx.h.v;
        T.qlo[x] = nx.l.v;
      } else if (STAGE == 3) {
        u3h[x] = nx.h.v;
        u3l[x] = nx.l.v;
        const df u0p = split_df(u0);
        const df u4 = df_fma(c13, df_sub(nx, u0p), u0p);  // u0 + (u3 - u0) / 3
        T.qhi[x] = u4.h.v;
        T.qlo[x] = u4.l.v;
      } else {
        const double un = df_to_d(nx);
        // (1/3 u0 + 2/3 u3) - un from the two increments, so that no rounding is of the size of u;
        // its factor 1/2 goes onto the cell's sum as an exact 1/4
        const df u0p = split_df(u0);
        const df d = df_fma(c13, df_sub(u0p, u3), df_sub(u3, nx));
        // the larger of |U| and |unew|: signs off, then the sign of the difference
        const df a0 = df_abs(u0p), a1 = df_abs(nx);
        const df t = df_div(d, df_fma(df_diff(a0, a1).v < 0.0f ? a1 : a0, rt, at0));
        if (pairs && fabsf(t.h.v) < 0x1p60f) ep = df_fma(t, t, ep);
        else e += error_fp64(d.h.v, d.l.v, amax_bits(u0, un), rtol, atol);
        Un[x] = (clamp && __double2hiint(un) < 0) ? 0.0 : un;
      }
    };
    // tracers in groups of four: every load of a group is issued before its arithmetic, so a
    // thread keeps four tracers' loads in flight (the same arithmetic, in the same order)
    constexpr int kGrp = 4;
    const df zero = mkdf(0.0f, 0.0f);
    int s = 0;
    for (; s + kGrp <= T.ntr; s += kGrp) {
      df q[kGrp], a[kGrp], u3[kGrp];
      double u0[kGrp];
#pragma unroll
      for (int r = 0; r < kGrp; ++r) {
        const size_t x = (size_t)(s + r) * nc + c;
        q[r] = mkdf(T.qhi[x], T.qlo[x]);
        a[r] = mkdf(T.acc.h[x], T.acc.l[x]);
        u0[r] = STAGE >= 3 ? U[x] : 0.0;
        u3[r] = STAGE == 4 ? mkdf(u3h[x], u3l[x]) : zero;
      }
#pragma unroll
      for (int r = 0; r < kGrp; ++r) tracer(s + r, (size_t)(s + r) * nc + c, q[r], a[r], u0[r], u3[r]);
    }
    for (; s < T.ntr; ++s) {
      const size_t x = (size_t)s * nc + c;
      tracer(s, x, mkdf(T.qhi[x], T.qlo[x]), mkdf(T.acc.h[x], T.acc.l[x]), STAGE >= 3 ? U[x] : 0.0,
             STAGE == 4 ? mkdf(u3h[x], u3l[x]) : zero);
    }
  }
  if (STAGE == 4) {
    const double tot = block_tree256(0.25 * (e + df_to_d(ep)), sm);
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
        adv = -(g * df_to_d(mkdf(T.acc.h[x], T.acc.l[x]))) / m;
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
    behind(T, k_adv_line<DIR>, dim3((unsigned)((lines + kLineThreads - 1) / kLineThreads), (unsigned)T.ntr), kLineThreads, 0, st, T, sel);
    return;
  }
  const unsigned tiles = DIR == 1 ? (unsigned)((T.nlon + f.pw - 1) / f.pw) * (unsigned)T.nlev
                                  : (unsigned)((ncol + f.pw - 1) / f.pw);
  const dim3 grid(tiles, (unsigned)f.gyz), block(f.pw, even_rows(DIR == 1 ? T.nlat : T.nlev, f.rows));
  const size_t sh = DIR == 1 ? f.shy : f.shz;
  if (f.pw == 8) behind(T, k_adv_pencil<DIR, 8>, grid, block, sh, st, T, sel);
  else if (f.pw == 16) behind(T, k_adv_pencil<DIR, 16>, grid, block, sh, st, T, sel);
  else behind(T, k_adv_pencil<DIR, 32>, grid, block, sh, st, T, sel);
}
static void launch_flux_one(cudaStream_t st, const DevTransport<double>& T, const StageSel& sel,
                            const FluxShape& f, int dir) {
  if (dir == 1) launch_adv_yz<1>(st, T, sel, f);
  else if (dir == 2) launch_adv_yz<2>(st, T, sel, f);
  else if (f.fx)
    behind(T, k_adv_x_rows, dim3((unsigned)((T.nlat * T.nlev + f.xr - 1) / f.xr), (unsigned)f.gx), f.xt, f.shx, st, T, sel, f.xr);
  else
    behind(T, k_adv_x_cell, dim3((unsigned)(((size_t)T.nlon * T.nlat * T.nlev + 255) / 256), (unsigned)T.ntr), 256, 0, st, T, sel);
}
#endif

void launch_scale_fluxes(cudaStream_t st, const DevTransport<double>& T, double* mx6, double* myn6,
                         double* mys6) {
  const size_t n = (size_t)T.nlev * std::max((size_t)T.nlat * (T.nlon + 1), (size_t)(T.nlat + 1) * T.nlon);
  k_scale_fluxes<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(T, mx6, myn6, mys6);
}

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
  // rs_create refuses mixed precision on grids whose pencils do not fit at width 16; the streaming
  // kernels count the cells and faces of a tracer in 32 bits
  const bool small = (long long)(T.nlev + 2) * (T.nlat + 1) * (T.nlon + 1) < (1LL << 31);
  if ((only_dir < 0 || only_dir == 0) && T.mstream_x && small) {
    const long long warps = (long long)((T.nlon + kSegX - 1) / kSegX) * T.nlat * T.nlev;
    const unsigned grid = (unsigned)((warps + 3) / 4) * groups(sx);
    if (sx > 1) behind(T, k_adv_x_stream<2>, grid, 128, 0, st, T, sel, sx);
    else behind(T, k_adv_x_stream<1>, grid, 128, 0, st, T, sel, sx);
  } else if (only_dir < 0 || only_dir == 0) {
    dim3 grid((unsigned)(T.nlat * T.nlev), groups(sx));
    if (tx) k_adv_x_mixed<true><<<grid, xt, shx, st>>>(T, sel, sx);
    else k_adv_x_mixed<false><<<grid, xt, shx, st>>>(T, sel, sx);
  }
  if (T.mstream_yz && small) {
    const size_t lines = (size_t)T.nlon * T.nlev;
    const unsigned gy = (unsigned)((lines + kLine32 - 1) / kLine32) * groups(syz),
                   gz = (unsigned)((ncol + kLine32 - 1) / kLine32) * groups(syz);
    if (only_dir < 0 || only_dir == 1) {
      if (syz > 1) behind(T, k_adv_yz_stream<1, 2>, gy, kLine32, 0, st, T, sel, syz);
      else behind(T, k_adv_yz_stream<1, 1>, gy, kLine32, 0, st, T, sel, syz);
    }
    if (only_dir < 0 || only_dir == 2) {
      if (syz > 1) behind(T, k_adv_yz_stream<2, 2>, gz, kLine32, 0, st, T, sel, syz);
      else behind(T, k_adv_yz_stream<2, 1>, gz, kLine32, 0, st, T, sel, syz);
    }
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
    behind(T, k_stage_mixed<1>, nb, kRedThreads, 0, st, T, ctl, B, rtol, atol, clamp);
    sel.stage = 2;
    launch_fluxes(st, T, sel);
    if (T.pbl) launch_pbl_mean(st, T, sel);
    behind(T, k_stage_mixed<2>, nb, kRedThreads, 0, st, T, ctl, B, rtol, atol, clamp);
    sel.stage = 3;
    launch_fluxes(st, T, sel);
    if (T.pbl) launch_pbl_mean(st, T, sel);
    behind(T, k_stage_mixed<3>, nb, kRedThreads, 0, st, T, ctl, B, rtol, atol, clamp);
    sel.stage = 4;
    launch_fluxes(st, T, sel);
    if (T.pbl) launch_pbl_mean(st, T, sel);
    behind(T, k_stage_mixed<4>, nb, kRedThreads, 0, st, T, ctl, B, rtol, atol, clamp);
    return;
  }
  launch_fluxes(st, T, sel);
  if (T.pbl) launch_pbl_mean(st, T, sel);
  behind(T, k_stage<1>, nb, kRedThreads, 0, st, T, ctl, B, rtol, atol, clamp);
  sel.stage = 2;
  launch_fluxes(st, T, sel);
  if (T.pbl) launch_pbl_mean(st, T, sel);
  behind(T, k_stage<2>, nb, kRedThreads, 0, st, T, ctl, B, rtol, atol, clamp);
  sel.stage = 3;
  launch_fluxes(st, T, sel);
  if (T.pbl) launch_pbl_mean(st, T, sel);
  behind(T, k_stage<3>, nb, kRedThreads, 0, st, T, ctl, B, rtol, atol, clamp);
  sel.stage = 4;
  launch_fluxes(st, T, sel);
  if (T.pbl) launch_pbl_mean(st, T, sel);
  behind(T, k_stage<4>, nb, kRedThreads, 0, st, T, ctl, B, rtol, atol, clamp);
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
