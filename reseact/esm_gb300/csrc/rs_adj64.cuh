// rs_adj64.cuh -- VJP of the FP64 transport tendency in the production build (included by
// rs_adjoint.cu): the forward kernels' advective form (rs_adv64.cuh) swept backwards.
//
// What bounds it: the FP64 pipe, one warp instruction per 64 cycles and SM sub-partition.  Carrying
// the weights of every slope (3), edge (4) and face (5) as the adjoint of the flux form does costs 42
// to 46 FP64 instructions per cell, tracer and direction; propagating the adjoint of each quantity
// to the quantities it was formed from costs about 20, because every frozen limiter decision is one
// selected source with an exact factor:
//   acc(f-1) += Mn A, acc(f) += Ms B      ->  A', B' = Mn G', Ms G' (G' = -g fbar / m)
//   A, B = x, 6 D - x                     ->  x' = +-(A' - B'), (6 D)' = the other one's
//   x = L, E, 2 E, 2 L or 0 of the upwind cell
//   E_p = 3 D_p - (S_{p+1} - S_p), L_{p+1} = 6 D_p - E_p
//   S_p = (D_{p-1} + D_p) / 2, 2 D_{p-1}, 2 D_p or 0
//   D_p = v(p+1) - v(p)
// (times 6 in the uniform directions; L = -eL.)  Each quantity gathers from the at most two or four
// that used it, in a fixed order: no atomics, the same bits on every run.  The decisions are the
// forward kernels'.  The tendency contains differences of q only, so there is no term in div(M).
//
// The entries of a block's lines -- rows of n + 6 for the lon direction, [n + 6][PW] for PW adjacent
// lat or vertical lines -- are dealt to the threads as one list, so only the last warp of a phase is
// partly idle.  72x46x47, 12 tracers: lon 252 -> 105 us, lat 198 -> 101, vertical 224 -> 102, the cell
// kernel 90 -> 14; FP64 pipe 80 % busy.
#pragma once

#if !RS_STRICT

// which source a limited slope took: 0 none (zero), 1 the centred one, 2 / 3 twice the left / right
// difference -- the forward kernels' slope with its decision
__device__ __noinline__ double slope_code_tiny(double d0, double d1, double da, int& code) {
  code = 0;
  if (!(d1 * d0 > 0.0)) return 0.0;
  const double lim = 2.0 * fmin(fabs(d0), fabs(d1));
  code = lim < fabs(da) ? (fabs(d1) < fabs(d0) ? 3 : 2) : 1;
  return copysign(fmin(fabs(da), lim), da);
}
__device__ __forceinline__ double slope_code(double d0, double d1, double da, bool half, int& code) {
  if (prod_may_underflow(d0, d1)) return slope_code_tiny(d0, d1, half ? 0.5 * da : da, code);
  const unsigned hs = (unsigned)__double2hiint(da);
  const unsigned hd = (hs & 0x7fffffffu) - (half ? (1u << 20) : 0u), ld = (unsigned)__double2loint(da);
  const unsigned h0 = (unsigned)__double2hiint(d0) & 0x7fffffffu, l0 = (unsigned)__double2loint(d0);
  const unsigned h1 = (unsigned)__double2hiint(d1) & 0x7fffffffu, l1 = (unsigned)__double2loint(d1);
  const bool p1 = mag_lt(h1, l1, h0, l0);
  const unsigned hm = (p1 ? h1 : h0) + (1u << 20), lm = p1 ? l1 : l0;  // 2 min(|d0|, |d1|)
  const bool binds = mag_lt(hm, lm, hd, ld);
  const bool live = ((__double2hiint(d0) ^ __double2hiint(d1)) >= 0) & ((h0 | l0) != 0u) &
                    ((h1 | l1) != 0u);
  code = live ? (binds ? (p1 ? 3 : 2) : 1) : 0;
  return __hiloint2double(live ? (int)((binds ? hm : hd) | (hs & 0x80000000u)) : 0,
                          live ? (int)(binds ? lm : ld) : 0);
}
// which source the limited deviation of the right or left edge took: 0 none, 1 its own, 2 twice the
// other
__device__ __noinline__ int dev_code_tiny(double eL, double eR, bool right) {
  if (eR * -eL <= 0.0) return 0;
  const double dA = eR - eL, a6 = -3.0 * (eL + eR);
  if (dA * a6 > dA * dA) return right ? 1 : 2;     // eL <- -2 eR
  if (-(dA * dA) > dA * a6) return right ? 2 : 1;  // eR <- -2 eL
  return 1;
}
__device__ __forceinline__ int dev_code(double eL, double eR, bool right) {
  if (prod_may_underflow(eL, eR)) return dev_code_tiny(eL, eR, right);
  const int hL = __double2hiint(eL), hR = __double2hiint(eR);
  const unsigned lL = (unsigned)__double2loint(eL), lR = (unsigned)__double2loint(eR);
  const unsigned mL = (unsigned)hL & 0x7fffffffu, mR = (unsigned)hR & 0x7fffffffu;
  const bool binds = right ? mag_lt(mL + (1u << 20), lL, mR, lR) : mag_lt(mR + (1u << 20), lR, mL, lL);
  const bool opp = ((hL ^ hR) < 0) & ((mL | lL) != 0u) & ((mR | lR) != 0u);
  return opp ? (binds ? 2 : 1) : 0;
}
__device__ __forceinline__ double twice(double x) {  // exact, in the integer pipes (x finite)
  const unsigned h = (unsigned)__double2hiint(x), l = (unsigned)__double2loint(x);
  if ((h & 0x7ff00000u) == 0u)  // zero or subnormal
    return __hiloint2double((int)((h & 0x80000000u) | (h << 1 & 0x7fffffffu) | l >> 31), (int)(l << 1));
  return __hiloint2double((int)(h + ((h & 0x7ff00000u) != 0x7ff00000u ? 1u << 20 : 0u)), (int)l);
}

// per cell: G = fbar / m, mbar = -sum G f.  One reciprocal per cell (a division per tracer took 10 of
// 22 FP64 instructions per cell and tracer).
__global__ void __launch_bounds__(256) k_adj_cell_dev(DevTransport<double> T, const double* __restrict__ U,
                                                      const double* __restrict__ F,
                                                      const double* __restrict__ fbar,
                                                      double* __restrict__ ubar, double* __restrict__ G) {
  const size_t nc = (size_t)T.nlon * T.nlat * T.nlev;
  const size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= nc) return;
  const double rm = rcp_nr(U[(size_t)T.ntr * nc + c]);  // m > 0
  double mb = 0.0;
#pragma unroll 4
  for (int s = 0; s < T.ntr; ++s) {
    const size_t x = (size_t)s * nc + c;
    const double gs = fbar[x] * rm;
    G[x] = gs;
    mb = fma(-gs, F[x], mb);
  }
  ubar[(size_t)T.ntr * nc + c] = mb;
}

constexpr int kAdjThreads = 256;
// six doubles and two bytes per entry
__host__ __device__ inline size_t adj_dev_bytes(size_t entries) { return entries * (6 * sizeof(double) + 2); }

// One tracer (blockIdx.y) of R lon rows (DIR 0) or PW adjacent lat (1) or vertical (2) lines.  DIR 0
// writes ubar, the other two add to it.
template <int DIR, int PW>
__global__ void __launch_bounds__(kAdjThreads) k_adj_dev(DevTransport<double> T, const double* __restrict__ U,
                                                         const double* __restrict__ G,
                                                         double* __restrict__ ubar, double g, int R) {
  extern __shared__ double sma[];
  constexpr bool UNI = DIR != 2;
  const int n = DIR == 0 ? T.nlon : (DIR == 1 ? T.nlat : T.nlev), L = n + 6;
  const int bc = DIR == 0 ? T.lon_bc : (DIR == 1 ? (T.lat_bc == 1 ? 1 : 2) : 2);
  constexpr int ST = DIR == 0 ? 1 : PW;  // from an entry to the next of its line
  const int N = DIR == 0 ? R * L : L * PW;
  double* D = sma;    // differences; then their adjoints
  double* S = D + N;  // slopes; then their adjoints
  double* E = S + N;  // right-edge deviations; then the adjoint E' - L' of an edge
  double* X = E + N;  // x' of the faces, with the factor 2 of code 2
  double* Y = X + N;  // the adjoint of a face's D term
  double* H = Y + N;  // G' of the cells
  unsigned char* ks = reinterpret_cast<unsigned char*>(H + N);  // slope codes
  unsigned char* kf = ks + N;  // faces: code, 4 = upwind below, 8 = carries a flux
  const size_t ncol = (size_t)T.nlon * T.nlat, nc = ncol * T.nlev;
  const int nrows = T.nlat * T.nlev, s = blockIdx.y;
  const int r0 = DIR == 0 ? blockIdx.x * R : 0, nr = DIR == 0 ? min(R, nrows - r0) : 0;
  const int ntile = (T.nlon + PW - 1) / PW;
  const int k = DIR == 1 ? (int)(blockIdx.x / ntile) : 0;
  const int i0 = DIR == 1 ? (int)(blockIdx.x % ntile) * PW : 0;
  const size_t col0 = DIR == 2 ? (size_t)blockIdx.x * PW : 0;
  const int gs = __double2hiint(g);
  // f(list index, line, entry o of the line) for o in [lo, hi]; entry o is cell or face o - 3
  const int rt = threadIdx.x / L, ot = threadIdx.x - rt * L;
  const int dr = blockDim.x / L, dO = blockDim.x - dr * L;
  auto each = [&](int lo, int hi, auto f) {
    if (DIR == 0) {
      for (int e = threadIdx.x, r = rt, o = ot; e < nr * L; e += blockDim.x) {
        if (o >= lo && o <= hi) f(e, r, o);
        r += dr;
        o += dO;
        if (o >= L) {
          o -= L;
          ++r;
        }
      }
    } else {
      for (int e = lo * PW + (int)threadIdx.x; e < (hi + 1) * PW; e += blockDim.x) f(e, e % PW, e / PW);
    }
  };
  auto live = [&](int ln) {
    return DIR == 0 ? true : (DIR == 1 ? i0 + ln < T.nlon : col0 + ln < ncol);
  };
  auto cell = [&](int ln, int p) -> size_t {
    if (DIR == 0) return (size_t)(r0 + ln) * n + p;
    if (DIR == 1) return ((size_t)k * n + p) * T.nlon + i0 + ln;
    return (size_t)p * ncol + col0 + ln;
  };
  const double* q = U + (size_t)s * nc;
  auto val = [&](int ln, int p) -> double {
    const int m = map_pos(p, n, bc);
    if (m >= 0) return q[cell(ln, m)];
    if (DIR == 0) return (p < 0 ? T.qw : T.qe)[(size_t)s * nrows + r0 + ln];
    return (p < 0 ? T.qs : T.qn)[((size_t)s * T.nlev + k) * T.nlon + i0 + ln];
  };
  // ---- forward: differences, slopes and their decisions, edges
  each(0, n + 5, [&](int e, int ln, int o) {
    const int p = o - 3;
    ks[e] = kf[e] = 0;
    D[e] = live(ln) && o <= n + 4 ? val(ln, p + 1) - val(ln, p) : 0.0;
    if (p >= 0 && p < n) H[e] = live(ln) ? -g * G[(size_t)s * nc + cell(ln, p)] : 0.0;
  });
  __syncthreads();
  each(1, n + 4, [&](int e, int ln, int o) {
    const double d0 = D[e - ST], d1 = D[e];
    int code = 0;
    double v = 0.0;
    if (UNI) {
      v = slope_code(d0, d1, d0 + d1, true, code);
    } else if (o >= 2 && o <= n + 3 && live(ln)) {  // cells -1..n (coefficient row of cell + 1)
      const size_t x = (size_t)(o - 2) * ncol + col0 + ln;
      v = slope_code(d0, d1, T.vsA[x] * d1 + T.vsB[x] * d0, false, code);
    }
    S[e] = v;
    ks[e] = (unsigned char)code;
  });
  __syncthreads();
  each(1, n + 3, [&](int e, int ln, int o) {
    double v = 0.0;
    if (UNI) {
      v = fma(3.0, D[e], -(S[e + ST] - S[e]));
    } else if (o >= 2 && o <= n + 2 && live(ln)) {  // cells -1..n-1 (row of cell + 1)
      const size_t x = (size_t)(o - 2) * ncol + col0 + ln;
      v = fma(T.veD[x], S[e], fma(T.veC[x], S[e + ST], T.veAB[x] * D[e]));
    }
    E[e] = v;
  });
  __syncthreads();
  // ---- faces: the limiter's decision and the adjoints of x and of the D term
  each(3, n + 3, [&](int e, int ln, int o) {
    const int f = o - 3;
    if (!live(ln) || (DIR == 1 && bc == 2 && (f == 0 || f == n)) || (DIR == 2 && (f == 0 || f == n))) return;
    double Mn, Ms;
    if (DIR == 0) {
      Mn = Ms = T.mx6[(size_t)(r0 + ln) * (n + 1) + f];
    } else if (DIR == 1) {
      const size_t x = ((size_t)k * (n + 1) + f) * T.nlon + i0 + ln;
      Mn = T.myn6[x];
      Ms = T.mys6[x];
    } else {
      Mn = Ms = T.mz[(size_t)f * ncol + col0 + ln];
    }
    const bool right = (__double2hiint(Mn) ^ gs) >= 0;
    const int up = right ? e - ST : e;
    const double Em = E[up - ST], Dm = D[up - ST];
    const int code = dev_code(UNI ? fma(-6.0, Dm, Em) : Em - Dm, E[up], right);
    const double a = f > 0 ? Mn * H[e - ST] : 0.0, b = f < n ? Ms * H[e] : 0.0;
    const double x = right ? a - b : b - a;
    X[e] = code == 2 ? twice(x) : x;
    Y[e] = right ? b : a;
    kf[e] = (unsigned char)(code | (right ? 4 : 0) | 8);
  });
  __syncthreads();
  // ---- edges: E_p feeds x of face p (upwind above, doubled) and p + 1 (upwind below); L_{p+1} those
  // of face p + 1 (upwind above) and p + 2 (upwind below, doubled)
  each(0, n + 4, [&](int e, int ln, int o) {
    double d = 0.0, ep = 0.0;
    if (o >= 1 && o <= n + 3) {
      const int f0 = kf[e], f1 = kf[e + ST], f2 = o <= n + 2 ? kf[e + 2 * ST] : 0;
      const double eb = ((f0 & 7) == 2 ? X[e] : 0.0) + ((f1 & 7) == 5 ? X[e + ST] : 0.0);
      const double lb = ((f1 & 7) == 1 ? X[e + ST] : 0.0) + ((f2 & 7) == 6 ? X[e + 2 * ST] : 0.0);
      ep = eb - lb;
      d = lb + (f1 & 8 ? Y[e + ST] : 0.0);
      if (UNI) d = fma(6.0, d, 3.0 * ep);
      else if (o >= 2 && o <= n + 2 && live(ln)) d = fma(T.veAB[(size_t)(o - 2) * ncol + col0 + ln], ep, d);
    }
    E[e] = ep;
    D[e] = d;
  });
  __syncthreads();
  // ---- slopes: S_p feeds E_p and E_{p-1}
  each(0, n + 5, [&](int e, int ln, int o) {
    double v = 0.0;
    if (o >= 1 && o <= n + 4) {
      if (UNI) {
        v = E[e] - E[e - ST];
      } else if (live(ln)) {
        const size_t x = (size_t)(o - 2) * ncol + col0 + ln;  // the row of cell o - 3's own edge
        if (o >= 2 && o <= n + 2) v = T.veD[x] * E[e];
        if (o >= 3 && o <= n + 3) v = fma(T.veC[x - ncol], E[e - ST], v);
      }
    }
    S[e] = v;
  });
  __syncthreads();
  // ---- differences: D_p is the right one of cell p's slope and the left one of cell p + 1's
  each(0, n + 4, [&](int e, int ln, int o) {
    const int c0 = ks[e], c1 = ks[e + ST];
    double wr = c0 == 3 ? 2.0 : 0.0, wl = c1 == 2 ? 2.0 : 0.0;
    if (UNI) {
      if (c0 == 1) wr = 0.5;
      if (c1 == 1) wl = 0.5;
    } else {  // (a centred slope's cell lies in the coefficient rows)
      if (c0 == 1) wr = T.vsA[(size_t)(o - 2) * ncol + col0 + ln];
      if (c1 == 1) wl = T.vsB[(size_t)(o - 1) * ncol + col0 + ln];
    }
    D[e] = fma(wl, S[e + ST], fma(wr, S[e], D[e]));
  });
  __syncthreads();
  // ---- values: q(p) is in D_{p-1} and D_p; ghost positions belong to the cells they mirror
  each(3, n + 2, [&](int e, int ln, int o) {
    if (!live(ln)) return;
    const int p = o - 3;
    double v = D[e - ST] - D[e];
    if (bc != 1 && (p < 3 || p > n - 4)) {
      const int e0 = e - o * ST;  // the line's first entry
      for (int r = 0; r < 6; ++r) {
        const int gp = r < 3 ? r - 3 : n + r - 3;
        if (map_pos(gp, n, bc) != p) continue;
        const int go = gp + 3;
        v += (go > 0 ? D[e0 + (go - 1) * ST] : 0.0) - (go <= n + 4 ? D[e0 + go * ST] : 0.0);
      }
    }
    double* out = ubar + (size_t)s * nc + cell(ln, p);
    if (DIR == 0) *out = v;
    else *out += v;
  });
}

constexpr size_t kAdjDevCap = 110 * 1024;
template <int DIR, int PW>
static void adj_dev_launch(cudaStream_t st, const DevTransport<double>& T, const double* U, const double* G,
                           double* ubar, double g, dim3 grid, int R, size_t smem) {
  if (smem > 48 * 1024)
    cudaFuncSetAttribute(k_adj_dev<DIR, PW>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kAdjDevCap);
  k_adj_dev<DIR, PW><<<grid, kAdjThreads, smem, st>>>(T, U, G, ubar, g, R);
}
// All three directions, or false (nothing launched) when a line is too long for shared memory (the
// face and gather kernels then take the whole call).
static bool launch_adj_dev(cudaStream_t st, const DevTransport<double>& T, const double* U, const double* F,
                           const double* fbar, double* ubar, double* G, double g) {
  const size_t ncol = (size_t)T.nlon * T.nlat, nc = ncol * T.nlev;
  // the widest tile of lines that leaves room for five blocks per SM, else for two
  auto width = [](int n) {
    for (size_t cap : {(size_t)44 * 1024, kAdjDevCap})
      for (int pw : {16, 8, 4})
        if (adj_dev_bytes((size_t)(n + 6) * pw) <= cap) return pw;
    return 0;
  };
  const int wy = width(T.nlat), wz = width(T.nlev);
  if (!wy || !wz || adj_dev_bytes((size_t)T.nlon + 6) > kAdjDevCap) return false;
  k_adj_cell_dev<<<(unsigned)((nc + 255) / 256), 256, 0, st>>>(T, U, F, fbar, ubar, G);
  {  // about 512 entries per block
    const int R = std::max(1, 512 / (T.nlon + 6)), nrows = T.nlat * T.nlev;
    adj_dev_launch<0, 1>(st, T, U, G, ubar, g, dim3((unsigned)((nrows + R - 1) / R), (unsigned)T.ntr), R,
                         adj_dev_bytes((size_t)R * (T.nlon + 6)));
  }
  {
    const dim3 grid((unsigned)((T.nlon + wy - 1) / wy) * (unsigned)T.nlev, (unsigned)T.ntr);
    const size_t b = adj_dev_bytes((size_t)(T.nlat + 6) * wy);
    if (wy == 16) adj_dev_launch<1, 16>(st, T, U, G, ubar, g, grid, 0, b);
    else if (wy == 8) adj_dev_launch<1, 8>(st, T, U, G, ubar, g, grid, 0, b);
    else adj_dev_launch<1, 4>(st, T, U, G, ubar, g, grid, 0, b);
  }
  {
    const dim3 grid((unsigned)((ncol + wz - 1) / wz), (unsigned)T.ntr);
    const size_t b = adj_dev_bytes((size_t)(T.nlev + 6) * wz);
    if (wz == 16) adj_dev_launch<2, 16>(st, T, U, G, ubar, g, grid, 0, b);
    else if (wz == 8) adj_dev_launch<2, 8>(st, T, U, G, ubar, g, grid, 0, b);
    else adj_dev_launch<2, 4>(st, T, U, G, ubar, g, grid, 0, b);
  }
  return true;
}
#endif  // !RS_STRICT
