// rs_adv64.cuh -- FP64 transport of the production build: PPM face terms in advective form on
// edge deviations, one accumulator per cell, and the stage kernels that turn it into the SSPRK43
// update (included by rs_transport.cu; the strict build keeps the oracle's flux form there).
//
// What bounds it: the FP64 pipe.  It issues one warp instruction per 64 cycles and SM
// sub-partition here, whatever the instruction-level parallelism or the number of active lanes,
// while the integer and load pipes are nearly idle; so FP64 instructions per cell are the time.
//
// With D_p = v(p+1) - v(p) and S_p the limited slope, the deviation of cell p's right edge is
// eR = D_p/2 - (S_{p+1} - S_p)/6 and that of its left edge eL = E_{p-1} - D_{p-1} (E the right
// deviations).  On these the CW84 limiter (eq. 1.10) needs no arithmetic: it flattens unless eL
// and eR have strictly opposite signs, and
//   dA a6 >  dA^2  <=>  |eL| > 2 |eR|   (eL <- -2 eR)
//   dA a6 < -dA^2  <=>  |eR| > 2 |eL|   (eR <- -2 eL),
// so the limited deviation of an edge is its own sign with min(|e|, 2 |the other|): sign tests,
// magnitude compares and an exact doubling on the integer pipes.
//
// The CWC tendency of cell c, m dq/dt = -div(M q) + q div(M), is a sum over its faces of
// G M (q_c - q_f), which needs differences only: with dev the limited deviation of the upwind
// cell's edge, face f (between cells f-1 and f) adds
//   to cell f-1:  G M A,  A = q_f - q_{f-1} =  dev (upwind f-1) or D + dev (upwind f)
//   to cell f:    G M B,  B = q_f' - ...    =  D - dev             or -dev       (A + B = D)
// and m dq/dt = -(sum).  The metric G, the 1/6 of the uniform edges and nothing else are folded
// into the air-mass fluxes once per forcing (mx6, myn6, mys6); the stage's time factor g is the
// same for all three directions, so it goes into the stage update's scale and only its sign is
// needed here.  The uniform directions carry 6 x the deviations: 6 E_p = 3 D_p - (S_{p+1} - S_p).
// FP64 instructions per cell and tracer: 8 (lon, lat: D, slope span, slope difference, edge, left
// edge, the other face term, two accumulating FMAs) and 10 (vertical, dp-weighted), and 1 for the
// stage update; the flux form on the same deviations took 7, 7, 9 and 7.  A uniform field gives
// exactly 0.  Measured on 144x91x47 with 12 tracers against that flux form: lon 125 -> 133 us, lat +
// vertical 275 -> 315 us, stage kernels 112-194 -> 53-100 us, one attempt 2.25 -> 2.13 ms; the
// transport macro step of 180x91x72 with 30 tracers 29.1 -> 26.7 ms.  FP64 pipe 80-85 % busy.
#pragma once

#if !RS_STRICT

// ------------------------------------------------------------------ per-face arithmetic
__device__ __forceinline__ double edge6_u(double D, double S0, double S1) {
  return fma(3.0, D, -(S1 - S0));
}
__device__ __forceinline__ double left6_u(double Em, double Dm) { return fma(-6.0, Dm, Em); }
__device__ __forceinline__ double edge_nd(double D, double S0, double S1, double ab, double c,
                                          double d) {
  return fma(d, S0, fma(c, S1, ab * D));
}
// The limited deviation of the right (right) or left edge from the unlimited eL, eR (times 6 if
// UNI).  Where their product could underflow (the limiter's extremum test in FP64 then sees 0), the
// FP form decides.
template <bool UNI>
__device__ __forceinline__ double limited_dev(double eL, double eR, bool right) {
  if (prod_may_underflow(eL, eR)) {
    double l = UNI ? eL * kOneSixth : eL, r = UNI ? eR * kOneSixth : eR;
    limit(0.0, l, r);
    const double v = right ? r : l;
    return UNI ? 6.0 * v : v;
  }
  const int hL = __double2hiint(eL), hR = __double2hiint(eR);
  const unsigned lL = (unsigned)__double2loint(eL), lR = (unsigned)__double2loint(eR);
  const unsigned mL = (unsigned)hL & 0x7fffffffu, mR = (unsigned)hR & 0x7fffffffu;
  const unsigned ms = right ? mR : mL, ls = right ? lR : lL;                 // the edge itself
  const unsigned mo = (right ? mL : mR) + (1u << 20), lo = right ? lL : lR;  // 2 |the other|
  const bool binds = mag_lt(mo, lo, ms, ls);
  const unsigned sg = (unsigned)(right ? hR : hL) & 0x80000000u;
  const bool opp = ((hL ^ hR) < 0) & ((mL | lL) != 0u) & ((mR | lR) != 0u);
  return __hiloint2double(opp ? (int)((binds ? mo : ms) | sg) : 0,
                          opp ? (int)(binds ? lo : ls) : 0);
}
// The two face terms A (for the cell below) and B (for the cell above) from the neighbour
// difference across the face and the limited deviation (times 6 if UNI).
template <bool UNI>
__device__ __forceinline__ void face_terms64(double D, double dev, bool right, double& A, double& B) {
  const double x = right ? dev : __hiloint2double(__double2hiint(dev) ^ (int)0x80000000, __double2loint(dev));
  const double y = UNI ? fma(6.0, D, -x) : D - x;
  A = sel_d(right, x, y);
  B = sel_d(right, y, x);
}
// the upwind cell is the one below the face: sign of g M
__device__ __forceinline__ bool upwind_below(double M, int gsign) {
  return (__double2hiint(M) ^ gsign) >= 0;
}

// ------------------------------------------------------------------ lon rows
// R consecutive lon rows per block in shared memory, blockIdx.y a group of tracers.  Entry o of a
// row (of n + 6) stands for cell p = o - 3 or face f = o - 3; the rows' entries are dealt to the
// threads as one list, so that a row length that is no multiple of the block leaves no idle warps,
// and every array is indexed by the list position e (neighbours at e - 1, e + 1).  Writes the
// accumulator.
__global__ void __launch_bounds__(256) k_adv_x_rows(DevTransport<double> T, StageSel sel, int R) {
  const double* Q;
  double g;
  if (!resolve_stage(sel, Q, g)) return;
  extern __shared__ double smx[];
  const int n = T.nlon, L = n + 6;
  double* D = smx;           // differences v(p+1) - v(p), p in [-3, n+1]
  double* S = D + R * L;     // slopes, p in [-2, n+1]; then A of the faces
  double* E = S + R * L;     // 6 x right-edge deviations, p in [-2, n]
  double* B = E + R * L;     // B of the faces
  double* M = B + R * L;     // scaled air-mass fluxes of the faces
  const int nrows = T.nlat * T.nlev, r0 = blockIdx.x * R, nr = min(R, nrows - r0), ne = nr * L;
  const size_t nc = (size_t)nrows * n;
  const int gs = __double2hiint(g);
  const int rt = threadIdx.x / L, ot = threadIdx.x - rt * L;  // this thread's first entry
  const int dr = blockDim.x / L, dO = blockDim.x - dr * L;    // and the step to its next
  auto each = [&](int lo, int hi, auto f) {  // f(list position, row, entry) for entries lo..hi
    for (int e = threadIdx.x, r = rt, o = ot; e < ne; e += blockDim.x) {
      if (o >= lo && o <= hi) f(e, r, o);
      r += dr;
      o += dO;
      if (o >= L) {
        o -= L;
        ++r;
      }
    }
  };
#define RS_X(a, e) a[bck(T, e, (long long)R * L)]
  each(3, n + 3, [&](int e, int r, int o) { RS_X(M, e) = T.mx6[(size_t)(r0 + r) * (n + 1) + o - 3]; });
  const int s0 = (int)((long long)blockIdx.y * T.ntr / gridDim.y);
  const int s1 = (int)((long long)(blockIdx.y + 1) * T.ntr / gridDim.y);
  for (int s = s0; s < s1; ++s) {
    const double* q = Q + (size_t)s * nc + (size_t)r0 * n;
    auto val = [&](int r, int p) -> double {
      if (p < 0 || p >= n) {
        if (T.lon_bc == 0) p = p < 0 ? p + n : p - n;
        else return (p < 0 ? T.qw : T.qe)[bck(T, (size_t)s * nrows + r0 + r, (long long)T.ntr * nrows)];
      }
      return q[bck(T, r * n + p, (long long)nr * n)];
    };
    each(0, n + 4, [&](int e, int r, int o) { RS_X(D, e) = val(r, o - 2) - val(r, o - 3); });
    __syncthreads();
    each(1, n + 4, [&](int e, int, int) { RS_X(S, e) = slope_ud(RS_X(D, e - 1), RS_X(D, e)); });
    __syncthreads();
    each(1, n + 3, [&](int e, int, int) { RS_X(E, e) = edge6_u(RS_X(D, e), RS_X(S, e), RS_X(S, e + 1)); });
    __syncthreads();
    each(3, n + 3, [&](int e, int, int) {
      const bool right = upwind_below(RS_X(M, e), gs);
      const int up = right ? e - 1 : e;
      const double dev = limited_dev<true>(left6_u(RS_X(E, up - 1), RS_X(D, up - 1)), RS_X(E, up), right);
      double a, b;
      face_terms64<true>(RS_X(D, e - 1), dev, right, a, b);
      RS_X(S, e) = a;
      RS_X(B, e) = b;
    });
    __syncthreads();
    double* acc = T.acc64 + (size_t)s * nc + (size_t)r0 * n;
    each(3, n + 2, [&](int e, int r, int o) {
      acc[bck(T, r * n + o - 3, (long long)nr * n)] = fma(RS_X(M, e + 1), RS_X(S, e + 1), RS_X(M, e) * RS_X(B, e));
    });
  }
#undef RS_X
}

// One thread per cell (lon rows too long for shared memory): both faces from seven values, the
// same operations.
__global__ void __launch_bounds__(256) k_adv_x_cell(DevTransport<double> T, StageSel sel) {
  const double* Q;
  double g;
  if (!resolve_stage(sel, Q, g)) return;
  const int n = T.nlon, nrows = T.nlat * T.nlev;
  const size_t nc = (size_t)nrows * n;
  const size_t x = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (x >= nc) return;
  const int row = (int)(x / n), c = (int)(x % n);
  const int gs = __double2hiint(g);
  const double Mw = T.mx6[(size_t)row * (n + 1) + c], Me = T.mx6[(size_t)row * (n + 1) + c + 1];
  for (int s = blockIdx.y; s < T.ntr; s += gridDim.y) {
    const double* q = Q + (size_t)s * nc + (size_t)row * n;
    double v[7], D[6], S[5], E[4];
#pragma unroll
    for (int o = 0; o < 7; ++o) {
      int p = c - 3 + o;
      if (p < 0 || p >= n) {
        if (T.lon_bc == 0) p = p < 0 ? p + n : p - n;
        else {
          v[o] = (p < 0 ? T.qw : T.qe)[bck(T, (size_t)s * nrows + row, (long long)T.ntr * nrows)];
          continue;
        }
      }
      v[o] = q[bck(T, p, n)];
    }
#pragma unroll
    for (int o = 0; o < 6; ++o) D[o] = v[o + 1] - v[o];               // D of cell c-3+o
#pragma unroll
    for (int o = 0; o < 5; ++o) S[o] = slope_ud(D[o], D[o + 1]);      // S of cell c-2+o
#pragma unroll
    for (int o = 0; o < 4; ++o) E[o] = edge6_u(D[o + 1], S[o], S[o + 1]);  // E of cell c-2+o
    const bool rw = upwind_below(Mw, gs), re = upwind_below(Me, gs);
    double a, b, be;
    face_terms64<true>(D[2], limited_dev<true>(rw ? left6_u(E[0], D[1]) : left6_u(E[1], D[2]), rw ? E[1] : E[2], rw), rw, be, b);
    face_terms64<true>(D[3], limited_dev<true>(re ? left6_u(E[1], D[2]) : left6_u(E[2], D[3]), re ? E[2] : E[3], re), re, a, be);
    T.acc64[(size_t)s * nc + x] = fma(Me, a, Mw * b);
  }
}

// ------------------------------------------------------------------ lat / vertical pencils
// PW adjacent lines per block in shared memory (lat lines at one level, or columns), the line's
// cells along threadIdx.y.  Adds to the accumulator.
template <int DIR, int PW>
__global__ void __launch_bounds__(512) k_adv_pencil(DevTransport<double> T, StageSel sel) {
  const double* Q;
  double g;
  if (!resolve_stage(sel, Q, g)) return;
  extern __shared__ double smp[];
  const int n = DIR == 1 ? T.nlat : T.nlev, L = n + 6;
  double* D = smp;               // [p+3][PW]
  double* S = D + L * PW;        // slopes; then A of face f at f+3
  double* E = S + L * PW;
  double* B = E + L * PW;
  double* Mn = B + L * PW;       // [f][PW]: the flux as seen by the cell below the face
  double* Ms = DIR == 1 ? Mn + (n + 1) * PW : Mn;  // and by the cell above
  const int tx = threadIdx.x, ty = threadIdx.y, ny = blockDim.y;
  const size_t ncol = (size_t)T.nlon * T.nlat, nc = ncol * T.nlev;
  const int ntile = (T.nlon + PW - 1) / PW;
  const int k = DIR == 1 ? (int)(blockIdx.x / ntile) : 0;
  const int i = DIR == 1 ? (int)(blockIdx.x % ntile) * PW + tx : 0;
  const size_t col = DIR == 2 ? (size_t)blockIdx.x * PW + tx : 0;
  const bool live = DIR == 1 ? i < T.nlon : col < ncol;
  const size_t stride = DIR == 1 ? (size_t)T.nlon : ncol;
  const size_t cbase = DIR == 1 ? (size_t)k * ncol + i : col;  // cell 0 of the line
  const bool open = DIR == 1 && T.lat_bc == 1;
  const int gs = __double2hiint(g);
  const long long mb = (long long)(n + 1) * PW;
#define RS_P(a, p) a[bck(T, ((p) + 3) * PW + tx, (long long)L * PW)]
  for (int f = ty; f <= n; f += ny) {
    if (DIR == 1) {
      const size_t fb = ((size_t)k * (n + 1) + f) * T.nlon + i;
      Mn[bck(T, f * PW + tx, mb)] = live ? T.myn6[fb] : 0.0;
      Ms[bck(T, f * PW + tx, mb)] = live ? T.mys6[fb] : 0.0;
    } else {
      Mn[bck(T, f * PW + tx, mb)] = live && f > 0 && f < n ? T.mz[(size_t)f * ncol + col] : 0.0;
    }
  }
  const int s0 = (int)((long long)blockIdx.y * T.ntr / gridDim.y);
  const int s1 = (int)((long long)(blockIdx.y + 1) * T.ntr / gridDim.y);
  for (int s = s0; s < s1; ++s) {
    const double* q = Q + (size_t)s * nc + cbase;
    auto val = [&](int p) -> double {
      if (!live) return 0.0;
      if (p < 0 || p >= n) {
        if (open) return (p < 0 ? T.qs : T.qn)[bck(T, ((size_t)s * T.nlev + k) * T.nlon + i, (long long)T.ntr * T.nlev * T.nlon)];
        p = p < 0 ? -1 - p : 2 * n - 1 - p;  // mirror ghosts at the walls
      }
      return q[(size_t)bck(T, p, n) * stride];
    };
    for (int p = ty - 3; p <= n + 1; p += ny) RS_P(D, p) = val(p + 1) - val(p);
    __syncthreads();
    if (DIR == 1) {
      for (int p = ty - 2; p <= n + 1; p += ny) RS_P(S, p) = slope_ud(RS_P(D, p - 1), RS_P(D, p));
      __syncthreads();
      for (int p = ty - 2; p <= n; p += ny) RS_P(E, p) = edge6_u(RS_P(D, p), RS_P(S, p), RS_P(S, p + 1));
    } else {
      for (int p = ty - 1; p <= n; p += ny) {  // slopes of cells -1..n (coefficient row p+1)
        const size_t x = bck(T, (size_t)(p + 1) * ncol + (live ? col : 0), (long long)(n + 2) * ncol);
        RS_P(S, p) = slope_nd(RS_P(D, p - 1), RS_P(D, p), T.vsA[x], T.vsB[x]);
      }
      __syncthreads();
      for (int p = ty - 1; p <= n - 1; p += ny) {  // right edges of cells -1..n-1 (row p+1)
        const size_t x = bck(T, (size_t)(p + 1) * ncol + (live ? col : 0), (long long)(n + 1) * ncol);
        RS_P(E, p) = edge_nd(RS_P(D, p), RS_P(S, p), RS_P(S, p + 1), T.veAB[x], T.veC[x], T.veD[x]);
      }
    }
    __syncthreads();
    for (int f = ty; f <= n; f += ny) {
      double a = 0.0, b = 0.0;
      if (DIR == 1 || (f > 0 && f < n)) {
        const bool right = upwind_below(Mn[bck(T, f * PW + tx, mb)], gs);
        const int up = right ? f - 1 : f;
        const double eL = DIR == 1 ? left6_u(RS_P(E, up - 1), RS_P(D, up - 1)) : RS_P(E, up - 1) - RS_P(D, up - 1);
        const double dev = limited_dev<DIR == 1>(eL, RS_P(E, up), right);
        face_terms64<DIR == 1>(RS_P(D, f - 1), dev, right, a, b);
      }
      RS_P(S, f) = a;
      RS_P(B, f) = b;
    }
    __syncthreads();
    if (live) {
      double* acc = T.acc64 + (size_t)s * nc + cbase;
      for (int c = ty; c < n; c += ny) {
        const long long m = bck(T, c * PW + tx, mb - PW);
        double* o = acc + (size_t)c * stride;
        *o = fma(Mn[m + PW], RS_P(S, c + 1), fma(Ms[m], RS_P(B, c), *o));
      }
    }
  }
#undef RS_P
}

// ------------------------------------------------------------------ lat / vertical lines
// One thread per line and tracer, walking it with a register window (no shared memory, no
// barriers): when q(p) arrives, D(p-1), S(p-1) and E(p-2) are formed, face p-2 is complete, its A
// closes cell p-3 and its B opens cell p-2.  The same operations in the same order as the pencils.
// One warp per sub-partition already fills the FP64 pipe, so few warps suffice; against the pencils
// on lat + vertical together: 315 to 335 us on 144x91x47, 1.31 to 1.48 ms on 180x91x72 with 30
// tracers, but 100 to 94 us on 72x46x47 (two warps per sub-partition: a coarse last wave).
template <int DIR>
__global__ void __launch_bounds__(128) k_adv_line(DevTransport<double> T, StageSel sel) {
  const double* Q;
  double g;
  if (!resolve_stage(sel, Q, g)) return;
  const int n = DIR == 1 ? T.nlat : T.nlev;
  const size_t ncol = (size_t)T.nlon * T.nlat, nc = ncol * T.nlev;
  const size_t id = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (id >= (DIR == 1 ? (size_t)T.nlon * T.nlev : ncol)) return;
  const int k = DIR == 1 ? (int)(id / T.nlon) : 0, i = DIR == 1 ? (int)(id % T.nlon) : 0;
  const size_t stride = DIR == 1 ? (size_t)T.nlon : ncol;
  const size_t cbase = DIR == 1 ? (size_t)k * ncol + i : id;
  const bool open = DIR == 1 && T.lat_bc == 1;
  const int gs = __double2hiint(g);
  const size_t fb = DIR == 1 ? (size_t)k * (n + 1) * T.nlon + i : id;  // face 0 of the line
  for (int s = blockIdx.y; s < T.ntr; s += gridDim.y) {
    const double* q = Q + (size_t)s * nc + cbase;
    double* acc = T.acc64 + (size_t)s * nc + cbase;
    auto val = [&](int p) -> double {
      if (p < 0 || p >= n) {
        if (open) return (p < 0 ? T.qs : T.qn)[bck(T, ((size_t)s * T.nlev + k) * T.nlon + i, (long long)T.ntr * T.nlev * T.nlon)];
        p = p < 0 ? -1 - p : 2 * n - 1 - p;
      }
      return q[(size_t)bck(T, p, n) * stride];
    };
    // window: qp = q(p-1), D2, D1 = D(p-2), D(p-1), S1 = S(p-1), E3, E2 = E(p-3), E(p-2),
    // L3, L2 their left deviations; ac the open cell's accumulator
    double qp = val(-2), D3 = 0.0, D2 = qp - val(-3), D1 = 0.0;
    double S2 = 0.0, S1 = 0.0, E3 = 0.0, E2 = 0.0, L3 = 0.0, L2 = 0.0, ac = 0.0;
    // one iteration ahead: q(p), the face's fluxes and the accumulator of the cell above it
    double q_nx = val(-1), mn_nx = 0.0, ms_nx = 0.0, a_nx = 0.0;
    for (int p = -1; p <= n + 2; ++p) {
      const double qn = q_nx, Mn = mn_nx, Ms = DIR == 1 ? ms_nx : mn_nx, ao = a_nx;
      const int f = p - 2;
      if (p < n + 2) q_nx = val(p + 1);
      if (f + 1 >= 0) {
        if (DIR == 1) {
          if (f + 1 <= n) {
            mn_nx = T.myn6[fb + (size_t)(f + 1) * stride];
            ms_nx = T.mys6[fb + (size_t)(f + 1) * stride];
          }
        } else {
          mn_nx = f + 1 > 0 && f + 1 < n ? T.mz[fb + (size_t)(f + 1) * stride] : 0.0;
        }
        if (f + 1 < n) a_nx = acc[(size_t)bck(T, f + 1, n) * stride];
      }
      D1 = qn - qp;  // D(p-1)
      qp = qn;
      S2 = S1;
      E3 = E2;
      L3 = L2;
      if (DIR == 1) {
        S1 = slope_ud(D2, D1);            // S(p-1)
        E2 = edge6_u(D2, S2, S1);         // E(p-2)
        L2 = left6_u(E3, D3);             // left deviation of cell p-2
      } else {
        const int ps = p - 1, pe = p - 2;
        if (ps >= -1 && ps <= n) {
          const size_t x = bck(T, (size_t)(ps + 1) * ncol + id, (long long)(n + 2) * ncol);
          S1 = slope_nd(D2, D1, T.vsA[x], T.vsB[x]);
        }
        if (pe >= -1 && pe <= n - 1) {
          const size_t x = bck(T, (size_t)(pe + 1) * ncol + id, (long long)(n + 1) * ncol);
          E2 = edge_nd(D2, S2, S1, T.veAB[x], T.veC[x], T.veD[x]);
          L2 = E3 - D3;
        }
      }
      if (f >= 0) {
        double a = 0.0, b = 0.0;
        if (DIR == 1 || (f > 0 && f < n)) {
          const bool right = upwind_below(Mn, gs);
          const double dev = limited_dev<DIR == 1>(sel_d(right, L3, L2), sel_d(right, E3, E2), right);
          face_terms64<DIR == 1>(D3, dev, right, a, b);
        }
        if (f >= 1) acc[(size_t)bck(T, f - 1, n) * stride] = fma(Mn, a, ac);
        ac = fma(Ms, b, ao);
      }
      D3 = D2;
      D2 = D1;
    }
  }
}

// ------------------------------------------------------------------ stage kernels
// stage in 1..4 of one attempt from the accumulator acc (m dq/dt = -g acc):
//   1: S1 = U + dt/2 f(U)           2: S2 = S1 + dt/2 f(S1)
//   3: S1 = u3 = S2 + dt/2 f(S2), S3 = u4 = 2/3 U + 1/3 u3
//   4: unew = S3 + dt/2 f(S3); err = 1/2 (1/3 U + 2/3 u3 - unew); candidate = clamp(unew)
// One thread per cell; the tracers in groups of four whose loads are issued together.  Stage 4's
// norm divides and sums in float pairs (relative error ~1e-13; the one-step reciprocal it replaces
// has 1e-12): five of its eight FP64 instructions per cell and tracer (144x91x47: 147 -> 92 us).
// the recorded tendency; a call, as predicated the multiplication holds the FP64 pipe on every
// unrecorded step too (12 of the 34 FP64-pipe instructions of a cell's stage 1 with 12 tracers)
__device__ __noinline__ double tendency(double a, double rmg) { return -a * rmg; }
template <int STAGE>
__global__ void __launch_bounds__(kRedThreads) k_stage(DevTransport<double> T,
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
  const double* Qin = STAGE == 1 ? U : (STAGE == 2 ? B.S1 : (STAGE == 3 ? B.S2 : B.S3));
  const size_t nc = (size_t)T.nlon * T.nlat * T.nlev;
  const size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
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
  df ep = mkdf(0.0f, 0.0f), rt = ep, at0 = ep;
  bool pairs = false;
  if (STAGE == 4) {
    rt = split_df(rtol);
    at0 = split_df(atol);
    pairs = atol >= 0x1p-40 && atol <= 0x1p100 && rtol >= 0x1p-60 && rtol <= 0x1p60;
  }
  if (c < nc) {
    const double dmdt = T.mcorr ? -fma(g, T.mdiv[c], T.mcorr[c]) : -(g * T.mdiv[c]);
    const size_t col = c % ((size_t)T.nlon * T.nlat), xm = (size_t)(T.nsp - 1) * nc + c;
    const double m = Qin[xm];
    const double rmg = g * rcp_nr(m);  // m > 0
    const double sc = -dt_2 * rmg;     // the tracer increment is acc * sc without PBL mixing
    // one species' update: its new value nx from the stage input q, the step's start u0 (stages
    // 3-4) and u3 (stage 4); the norm terms are added in species order
    auto finish = [&](size_t x, double du, double nx, double u0, double u3) {
      if (Fo) Fo[x] = du;
      if (STAGE == 1) {
        B.S1[x] = nx;
        if (Vo) Vo[x] = nx;
      } else if (STAGE == 2) {
        B.S2[x] = nx;
        if (Vo) Vo[x] = nx;
      } else if (STAGE == 3) {
        B.S1[x] = nx;
        const double u4 = (2.0 / 3.0) * u0 + (1.0 / 3.0) * nx;
        B.S3[x] = u4;
        if (Vo) Vo[x] = u4;
      } else {
        // (1/3 u0 + 2/3 u3) - nx in two FMAs; the factor 1/2 of the error goes onto the
        // cell's sum as an exact 1/4
        const double err = fma(2.0 / 3.0, u3, fma(1.0 / 3.0, u0, -nx));
        add_error(err, amax_bits(u0, nx), rtol, atol, rt, at0, pairs, ep, e);
        // clamp at 0 on the sign bit (integer pipe); a NaN candidate fails the norm anyway
        Un[x] = (clamp && __double2hiint(nx) < 0) ? 0.0 : nx;
      }
    };
    auto tracer = [&](int s, size_t x, double q, double a, double u0, double u3) {
      if (T.pbl) {
        const double du = fma(-a, rmg, pbl_term(T, c, col, s, q));
        finish(x, du, fma(du, dt_2, q), u0, u3);
      } else {
        finish(x, Fo ? tendency(a, rmg) : 0.0, fma(a, sc, q), u0, u3);
      }
    };
    constexpr int kGrp = 4;
    int s = 0;
    for (; s + kGrp <= T.ntr; s += kGrp) {
      double q[kGrp], a[kGrp], u0[kGrp], u3[kGrp];
#pragma unroll
      for (int r = 0; r < kGrp; ++r) {
        const size_t x = (size_t)(s + r) * nc + c;
        q[r] = Qin[x];
        a[r] = T.acc64[x];
        u0[r] = STAGE >= 3 ? U[x] : 0.0;
        u3[r] = STAGE == 4 ? B.S1[x] : 0.0;
      }
#pragma unroll
      for (int r = 0; r < kGrp; ++r) tracer(s + r, (size_t)(s + r) * nc + c, q[r], a[r], u0[r], u3[r]);
    }
    for (; s < T.ntr; ++s) {
      const size_t x = (size_t)s * nc + c;
      tracer(s, x, Qin[x], T.acc64[x], STAGE >= 3 ? U[x] : 0.0, STAGE == 4 ? B.S1[x] : 0.0);
    }
    finish(xm, dmdt, fma(dmdt, dt_2, m), STAGE >= 3 ? U[xm] : 0.0, STAGE == 4 ? B.S1[xm] : 0.0);
  }
  if (STAGE == 4) {
    const double tot = block_tree256(0.25 * (e + df_to_d(ep)), sm);
    if (threadIdx.x == 0) B.partial[blockIdx.x] = tot;
  }
}

#endif  // !RS_STRICT
