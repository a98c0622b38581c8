// rs_jit.cu -- generator and NVRTC loader of the mechanism-specialised chemistry kernels.
//
// The generated kernels compute exactly what the table-walking kernels of rs_chem.cu compute
// (ROS23 attempt, rx_traced_integrator.jl:279-349; blocksolve :110-135; hairer norm
// :329-347; per-cell PI controller :455-507), term for term in the same association:
//   v_r   = k_r * x_a * x_a * x_b ...             (reactant entries in table order)
//   f_s   = sum_r net[r,s] v_r (+ emission_s)     (reactions ascending; x*1 and x*(-1) folded)
//   P_p   = d v_r / d x_q                          (same product order as the tables)
//   W     = I - dtgamma * J on the LU fill pattern
//   LU    natural-order pivot-free elimination, zero updates skipped
// so that a strict build (no FMA contraction, divides where the reference divides) is still
// bit-compatible with the CPU restatement.  The only freedom taken is the sign of an exact
// zero (an off-diagonal W entry is written -(dtgamma*acc) instead of 0.0 - dtgamma*acc).
//
// NVRTC is loaded with dlopen so that the library itself loads without it; a handle whose
// kernels cannot be generated keeps the table-walking kernels (also CUDA).
#include <cuda_runtime.h>
#include <dlfcn.h>
#include <nvrtc.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstddef>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <memory>
#include <mutex>
#include <sstream>
#include <string>
#include <type_traits>
#include <vector>

#include "rs_jit.h"
#include "rs_kernels.h"
#include "rs_units.h"

namespace rs {

static_assert(sizeof(PerCellArgs) == 128 && offsetof(PerCellArgs, clamp) == 112 &&
                  offsetof(PerCellArgs, totals) == 120,
              "PerCellArgs layout is restated in the generated source");

namespace {

// ------------------------------------------------------------------ NVRTC entry points
struct Nvrtc {
  decltype(&nvrtcCreateProgram) create = nullptr;
  decltype(&nvrtcCompileProgram) compile = nullptr;
  decltype(&nvrtcGetProgramLogSize) log_size = nullptr;
  decltype(&nvrtcGetProgramLog) log = nullptr;
  decltype(&nvrtcGetCUBINSize) cubin_size = nullptr;
  decltype(&nvrtcGetCUBIN) cubin = nullptr;
  decltype(&nvrtcDestroyProgram) destroy = nullptr;
  decltype(&nvrtcGetErrorString) err = nullptr;
  std::string why;
  bool ok() const { return why.empty(); }
};

const Nvrtc& nvrtc() {
  static const Nvrtc api = [] {
    Nvrtc a;
    std::vector<std::string> names = {"libnvrtc.so.13", "libnvrtc.so"};
    if (const char* ch = std::getenv("CUDA_HOME")) names.push_back(std::string(ch) + "/lib64/libnvrtc.so.13");
    names.push_back("/usr/local/cuda/lib64/libnvrtc.so.13");
    void* h = nullptr;
    for (const auto& n : names)
      if ((h = dlopen(n.c_str(), RTLD_NOW | RTLD_LOCAL))) break;
    if (!h) {
      a.why = "libnvrtc.so.13 not found";
      return a;
    }
    auto sym = [&](auto& fp, const char* name) {
      fp = reinterpret_cast<std::remove_reference_t<decltype(fp)>>(dlsym(h, name));
      if (!fp && a.why.empty()) a.why = std::string("libnvrtc lacks ") + name;
    };
    sym(a.create, "nvrtcCreateProgram");
    sym(a.compile, "nvrtcCompileProgram");
    sym(a.log_size, "nvrtcGetProgramLogSize");
    sym(a.log, "nvrtcGetProgramLog");
    sym(a.cubin_size, "nvrtcGetCUBINSize");
    sym(a.cubin, "nvrtcGetCUBIN");
    sym(a.destroy, "nvrtcDestroyProgram");
    sym(a.err, "nvrtcGetErrorString");
    return a;
  }();
  return api;
}

// ------------------------------------------------------------------ source generation
std::string lit(double v) {  // exact hex-float literal
  char b[64];
  std::snprintf(b, sizeof b, "%a", v);
  return std::signbit(v) ? "(" + std::string(b) + ")" : std::string(b);
}

// W storage: shared-memory variant only while NLU doubles per thread fit for the largest block
constexpr int kBlock = 256;
constexpr int kJitUnits = 8;  // RS_IN units of the generated source
constexpr size_t kSmemCap = 227 * 1024 - kBlock * sizeof(double);

// Whether the global-dt attempts form their error estimate in float pairs.  The pairs' splits and
// sums take registers: beyond this many LU slots they spill more than the FP64 instructions they save
// are worth.  Attempt in us, pairs / FP64 estimate (both with W in registers): 94 slots 132 / 136 on
// 40,960 cells, 315 / 320 on 150,528, 1,126 / 1,181 on 614,400; 122 slots 169 / 171, 394 / 403, 1,616 /
// 1,524; 162 slots 215 / 212, 535 / 509, 2,266 / 1,926; 242 slots 353 / 300, 886 / 732, 3,676 / 2,791.
constexpr int kPairSlots = 108;
bool jit_pairs(const MechTables& T, bool strict) { return !strict && T.nlu <= kPairSlots; }

size_t smem_bytes(const MechTables& T) { return (size_t)T.nlu * kBlock * sizeof(double); }
// "split" variant: the last split_slots(T) LU slots of W in shared memory, the others in
// registers, two 256-thread blocks per SM (each block's shared part within half an SM's
// 228 KB, its static reduction array and the per-block reserve included)
int split_slots(const MechTables& T) {
  const int cap = (int)((113 * 1024 - 3 * 1024) / (kBlock * sizeof(double)));  // 55
  return T.nlu >= 16 ? (T.nlu < cap ? T.nlu : cap) : 0;
}

struct Gen {
  const MechTables& T;
  bool strict;
  std::ostringstream o;

  void vel(const char* x) {
    for (int r = 0; r < T.nr; ++r) {
      std::ostringstream e;
      e << "K(" << r << ")";
      for (int q = T.rptr[r]; q < T.rptr[r + 1]; ++q)
        for (int t = 0; t < T.rnu[q]; ++t) e << "*" << x << "[" << T.rsp[q] << "]";
      o << "  v[" << r << "] = " << e.str() << ";\n";
    }
  }
  // acc = sum c_t * a[i_t], first term without the leading 0.0 +, +-1 coefficients folded
  static void sum_terms(std::ostringstream& e, bool first, double c, const std::string& term) {
    if (first) {
      if (c == 1.0) e << term;
      else if (c == -1.0) e << "-" << term;
      else e << lit(c) << "*" << term;
    } else {
      // fold into the running sum: e is rebuilt around the previous expression
      std::string prev = e.str();
      e.str("");
      if (c == 1.0) e << prev << " + " << term;
      else if (c == -1.0) e << prev << " - " << term;
      else e << "RS_FMA(" << lit(c) << ", " << term << ", " << prev << ")";
    }
  }
  void rhs(const char* f) {
    for (int s = 0; s < T.ns; ++s) {
      std::ostringstream e;
      bool first = true;
      for (int t = T.rhs_ptr[s]; t < T.rhs_ptr[s + 1]; ++t) {
        sum_terms(e, first, T.rhs_c[t], "v[" + std::to_string(T.rhs_r[t]) + "]");
        first = false;
      }
      std::string ex = first ? std::string("0.0") : e.str();
      o << "  { const double a_ = " << ex << "; " << f << "[" << s << "] = HE ? a_ + EM(" << s
        << ") : a_; }\n";
    }
  }
  // f = RHS at state x.  Strict build: the rates v_r, then each species' sum of c * v_r (the
  // oracle's order).  Production build: per reaction the head u_r = K_r * (all factors but
  // the last) once, and each term as one FMA of u_r with the last factor into the species'
  // sum -- one instruction fewer per reaction than a rate product followed by adds.
  void rates_rhs(const char* x, const char* f) {
    if (strict) {
      vel(x);
      rhs(f);
      return;
    }
    o << "  {\n";  // the heads are local to this evaluation
    std::vector<std::string> last(T.nr);
    for (int r = 0; r < T.nr; ++r) {
      std::vector<int> fac;
      for (int q = T.rptr[r]; q < T.rptr[r + 1]; ++q)
        for (int t = 0; t < T.rnu[q]; ++t) fac.push_back(T.rsp[q]);
      std::ostringstream h;
      h << "K(" << r << ")";
      for (size_t i = 0; i + 1 < fac.size(); ++i) h << "*" << x << "[" << fac[i] << "]";
      o << "  const double u" << r << "_ = " << h.str() << ";\n";
      last[r] = fac.empty() ? std::string() : std::string(x) + "[" + std::to_string(fac.back()) + "]";
    }
    // Sums that two species have in common (one's loss is the other's production) are formed once:
    // n shared terms cost n + 2 instructions instead of 2 n.  Rows are lists of (term, coefficient);
    // term r < nr is reaction r, nr + k the k-th shared sum; the pair with the most in common first.
    typedef std::vector<std::pair<int, double>> Row;
    std::vector<Row> rows(T.ns);
    for (int sp = 0; sp < T.ns; ++sp)
      for (int t = T.rhs_ptr[sp]; t < T.rhs_ptr[sp + 1]; ++t) rows[sp].push_back({T.rhs_r[t], T.rhs_c[t]});
    for (;;) {
      size_t most = 2;
      int bi = -1, bj = -1;
      double brho = 1.0;
      auto common = [&](int i, int j, double rho) {
        Row v;
        for (auto& x : rows[i])
          for (auto& y : rows[j])
            if (x.first == y.first && y.second == rho * x.second) v.push_back(x);
        return v;
      };
      for (int i = 0; i < (int)rows.size(); ++i)
        for (int j = i + 1; j < (int)rows.size(); ++j)
          for (double rho : {1.0, -1.0}) {
            const size_t n = common(i, j, rho).size();
            if (n > most) most = n, bi = i, bj = j, brho = rho;
          }
      if (bi < 0) break;
      const Row shared = common(bi, bj, brho);
      for (int k : {bi, bj}) {
        Row rest;
        for (auto& x : rows[k])
          if (std::none_of(shared.begin(), shared.end(), [&](const std::pair<int, double>& y) { return y.first == x.first; }))
            rest.push_back(x);
        rest.insert(rest.begin(), {T.nr + (int)rows.size() - T.ns, k == bi ? 1.0 : brho});
        rows[k] = rest;
      }
      rows.push_back(shared);
    }
    auto sum = [&](const Row& row) {
      std::string acc;
      for (auto& tc : row) {
        const int r = tc.first;
        const double cf = tc.second;
        const std::string u = r < T.nr ? "u" + std::to_string(r) + "_" : "g" + std::to_string(r - T.nr) + "_";
        const std::string lf = r < T.nr ? last[r] : std::string();
        std::string term;  // the product c * v_r, for a first term
        if (lf.empty()) term = cf == 1.0 ? u : (cf == -1.0 ? "(-" + u + ")" : lit(cf) + "*" + u);
        else if (cf == 1.0) term = u + "*" + lf;
        else if (cf == -1.0) term = "(-" + u + ")*" + lf;
        else term = lit(cf) + "*(" + u + "*" + lf + ")";
        if (acc.empty()) {
          acc = term;
        } else if (lf.empty()) {
          acc = cf == 1.0 ? acc + " + " + u : (cf == -1.0 ? acc + " - " + u : "RS_FMA(" + lit(cf) + ", " + u + ", " + acc + ")");
        } else if (cf == 1.0) {
          acc = "RS_FMA(" + u + ", " + lf + ", " + acc + ")";
        } else if (cf == -1.0) {
          acc = "RS_FMA(-" + u + ", " + lf + ", " + acc + ")";
        } else {
          acc = "RS_FMA(" + lit(cf) + ", " + u + "*" + lf + ", " + acc + ")";
        }
      }
      return acc.empty() ? std::string("0.0") : acc;
    };
    for (int k = (int)rows.size() - 1; k >= T.ns; --k)  // a shared sum may hold later ones
      o << "  const double g" << k - T.ns << "_ = " << sum(rows[k]) << ";\n";
    for (int sp = 0; sp < T.ns; ++sp)
      o << "  { const double a_ = " << sum(rows[sp]) << "; " << f << "[" << sp << "] = HE ? a_ + EM(" << sp
        << ") : a_; }\n";
    o << "  }\n";
  }
  // Partial derivatives dv_r/dx_q of the rates at xa; `scaled` forms them from kd<r>_ =
  // -dtg * K_r (declared by build_w_scaled) instead of K_r.
  void partials(const char* xa = "x", const char* Pa = "P", bool scaled = false) {
    for (int p = 0; p < T.npart; ++p) {
      int r = T.part_r[p], qs = T.part_q[p];
      std::ostringstream d;
      if (scaled) d << "kd" << r << "_";
      else d << "K(" << r << ")";
      for (int q = T.rptr[r]; q < T.rptr[r + 1]; ++q) {
        int s = T.rsp[q], nu = T.rnu[q];
        if (s == qs) {
          if (nu >= 2) {
            std::ostringstream f;
            f << lit((double)nu);
            for (int t = 1; t < nu; ++t) f << "*" << xa << "[" << s << "]";
            d << "*(" << f.str() << ")";
          }
        } else {
          for (int t = 0; t < nu; ++t) d << "*" << xa << "[" << s << "]";
        }
      }
      o << "  " << Pa << "[" << p << "] = " << d.str() << ";\n";
    }
  }
  void build_w() {
    std::vector<std::string> w(T.nlu, "0.0");
    for (int i = 0; i < T.ns; ++i) w[T.lu_diag[i]] = "1.0";
    for (int e = 0; e < T.njac; ++e) {
      std::ostringstream acc;
      bool first = true;
      for (int t = T.jac_ptr[e]; t < T.jac_ptr[e + 1]; ++t) {
        sum_terms(acc, first, T.jac_coef[t], "P[" + std::to_string(T.jac_part[t]) + "]");
        first = false;
      }
      std::string a = first ? std::string("0.0") : acc.str();
      w[T.jac_slot[e]] = T.jac_diag[e] ? "RS_FMA(-dtg, (" + a + "), 1.0)" : "-(dtg*(" + a + "))";
    }
    for (int e = 0; e < T.nlu; ++e) o << "  WV(" << e << ") = " << w[e] << ";\n";
  }
  // Production attempt: W = I - dtg*J with -dtg folded once into each reaction's rate
  // constant (kd_r = -dtg * K_r) before the partials at x are formed, so each Jacobian entry of
  // W is its plain sum of scaled partials (plus 1 on the diagonal): one multiply per reaction
  // instead of one per entry.
  // the off-diagonal Jacobian entry whose terms are those of diagonal entry d, negated, or -1
  int negated_entry(int d) const {
    const int n = T.jac_ptr[d + 1] - T.jac_ptr[d];
    for (int e = 0; e < T.njac; ++e) {
      if (T.jac_diag[e] || n < 2 || T.jac_ptr[e + 1] - T.jac_ptr[e] != n) continue;
      bool eq = true;
      for (int t = 0; t < n && eq; ++t)
        eq = T.jac_part[T.jac_ptr[e] + t] == T.jac_part[T.jac_ptr[d] + t] &&
             T.jac_coef[T.jac_ptr[e] + t] == -T.jac_coef[T.jac_ptr[d] + t];
      if (eq) return e;
    }
    return -1;
  }
  // pivot k is exactly 1: no Jacobian entry on its diagonal and no elimination update
  bool unit_pivot(int k) const {
    for (int e = 0; e < T.njac; ++e)
      if (T.jac_diag[e] && T.jac_slot[e] == T.lu_diag[k] && T.jac_ptr[e + 1] > T.jac_ptr[e]) return false;
    for (int dst : T.upd_dst)
      if (dst == T.lu_diag[k]) return false;
    return true;
  }
  void build_w_scaled() {
    std::vector<char> used(T.nr, 0);
    for (int p = 0; p < T.npart; ++p) used[T.part_r[p]] = 1;
    o << "  {\n";
    for (int r = 0; r < T.nr; ++r)
      if (used[r]) o << "  const double kd" << r << "_ = -dtg * K(" << r << ");\n";
    partials("x", "P", true);
    std::vector<std::string> w(T.nlu, "0.0"), tail(T.nlu);
    std::vector<int> late;  // slots formed from another slot
    for (int i = 0; i < T.ns; ++i) w[T.lu_diag[i]] = "1.0";
    for (int e = 0; e < T.njac; ++e) {
      std::ostringstream acc;
      bool first = true;
      for (int t = T.jac_ptr[e]; t < T.jac_ptr[e + 1]; ++t) {
        sum_terms(acc, first, T.jac_coef[t], "P[" + std::to_string(T.jac_part[t]) + "]");
        first = false;
      }
      if (first) continue;
      // a loss that is another entry's production, term by term: one sum for both (negation is exact)
      const int same = T.jac_diag[e] ? negated_entry(e) : -1;
      if (same >= 0) w[T.jac_slot[e]] = "1.0 - WV(" + std::to_string(T.jac_slot[same]) + ")", late.push_back(T.jac_slot[e]);
      else w[T.jac_slot[e]] = T.jac_diag[e] ? "1.0 + (" + acc.str() + ")" : acc.str();
    }
    for (int sl : late) std::swap(w[sl], tail[sl]);
    for (int e = 0; e < T.nlu; ++e)
      if (tail[e].empty()) o << "  WV(" << e << ") = " << w[e] << ";\n";
    for (int e = 0; e < T.nlu; ++e)
      if (!tail[e].empty()) o << "  WV(" << e << ") = " << tail[e] << ";\n";
    o << "  }\n";
  }
  // (eh, el) <- W^-1 (eh, el) in float pairs from the FP64 factors, split entry by entry
  void solve_pairs() {
    for (int k = 0; k < T.ns; ++k)
      for (int e = T.low_ptr[k]; e < T.low_ptr[k + 1]; ++e)
        o << "  pair_msub(" << T.low_row[e] << ", " << T.low_slot[e] << ", " << T.ord[k] << ")\n";
    for (int i = T.ns - 1; i >= 0; --i) {
      for (int e = T.up_ptr[i]; e < T.up_ptr[i + 1]; ++e)
        o << "  pair_msub(" << T.ord[i] << ", " << T.up_slot[e] << ", " << T.up_col[e] << ")\n";
      o << "  pair_scale(" << T.ord[i] << ", " << i << ")\n";
    }
  }
  void lu_factor() {
    int m = 0;
    for (int k = 0; k < T.ns; ++k) {
      if (strict)
        o << "  pv[" << k << "] = 1.0 / WV(" << T.lu_diag[k] << ");\n";
      else if (unit_pivot(k))
        o << "  pv[" << k << "] = 1.0;\n";
      else
        o << "  pv[" << k << "] = rcp_nr(WV(" << T.lu_diag[k] << "));\n";
      for (int ii = T.elim_ptr[k]; ii < T.elim_ptr[k + 1]; ++ii, ++m) {
        int sl = T.elim_lik[ii];
        o << "  { const double mu_ = WV(" << sl << ") * pv[" << k << "];\n";
        for (int u = T.upd_ptr[m]; u < T.upd_ptr[m + 1]; ++u)
          o << "    WV(" << T.upd_dst[u] << ") = RS_FMA(-mu_, WV(" << T.upd_src[u] << "), WV("
            << T.upd_dst[u] << "));\n";
        o << "    WV(" << sl << ") = mu_; }\n";
      }
    }
  }
  // W^T x = b in place with the same factors: U^T then L^T (the table kernels' lu_solve_T)
  void lu_solve_T(const char* b) {
    for (int j = 0; j < T.ns; ++j) {
      const int sj = T.ord[j];
      if (strict)
        o << "  { const double tj = " << b << "[" << sj << "] / WV(" << T.lu_diag[j] << ");\n";
      else
        o << "  { const double tj = " << b << "[" << sj << "] * pv[" << j << "];\n";
      o << "    " << b << "[" << sj << "] = tj;\n";
      for (int e = T.up_ptr[j]; e < T.up_ptr[j + 1]; ++e)
        o << "    " << b << "[" << T.up_col[e] << "] = RS_FMA(-WV(" << T.up_slot[e] << "), tj, " << b
          << "[" << T.up_col[e] << "]);\n";
      o << "  }\n";
    }
    for (int k = T.ns - 1; k >= 0; --k) {
      const int sk = T.ord[k];
      std::string acc = std::string(b) + "[" + std::to_string(sk) + "]";
      for (int e = T.low_ptr[k]; e < T.low_ptr[k + 1]; ++e)
        acc = "RS_FMA(-WV(" + std::to_string(T.low_slot[e]) + "), " + b + "[" +
              std::to_string(T.low_row[e]) + "], " + acc + ")";
      o << "  " << b << "[" << sk << "] = " << acc << ";\n";
    }
  }
  // a_r = sum_s net[r,s] y_s, species ascending within each reaction (the tables' order)
  void reaction_sums(const char* y, const char* a) {
    std::vector<std::vector<std::pair<int, double>>> per(T.nr);
    for (int sp = 0; sp < T.ns; ++sp)
      for (int t = T.rhs_ptr[sp]; t < T.rhs_ptr[sp + 1]; ++t)
        per[T.rhs_r[t]].push_back({sp, T.rhs_c[t]});
    for (int r = 0; r < T.nr; ++r) {
      std::ostringstream e;
      bool first = true;
      for (auto& tc : per[r]) {
        sum_terms(e, first, tc.second, std::string(y) + "[" + std::to_string(tc.first) + "]");
        first = false;
      }
      o << "  " << a << "[" << r << "] = " << (first ? std::string("0.0") : e.str()) << ";\n";
    }
  }
  // out += J^T y from the partials Pa (a: scratch for the reaction sums)
  void jt_apply(const char* Pa, const char* y, const char* a, const char* out) {
    reaction_sums(y, a);
    for (int p = 0; p < T.npart; ++p)
      o << "  " << out << "[" << T.part_q[p] << "] = RS_FMA(" << a << "[" << T.part_r[p] << "], "
        << Pa << "[" << p << "], " << out << "[" << T.part_q[p] << "]);\n";
  }
  // exact mass-action Hessian term of the ROS23 VJP: for every reaction r and reactant entries
  // j, q: ub_q += dtg (a1_r z2_j + a0_r k1_j) d2v_r/dx_j dx_q (structural zeros skipped)
  void hessian() {
    for (int r = 0; r < T.nr; ++r)
      for (int ea = T.rptr[r]; ea < T.rptr[r + 1]; ++ea) {
        const int j = T.rsp[ea];
        bool any = false;
        std::ostringstream body;
        for (int eb = T.rptr[r]; eb < T.rptr[r + 1]; ++eb) {
          const int q = T.rsp[eb];
          std::ostringstream d;
          d << "K(" << r << ")";
          bool zero = false;
          for (int e = T.rptr[r]; e < T.rptr[r + 1]; ++e) {
            const int sp = T.rsp[e], nu = T.rnu[e];
            const int order = (sp == j) + (sp == q);
            if (order > nu) { zero = true; break; }
            double cst = 1.0;
            for (int t = 0; t < order; ++t) cst *= (double)(nu - t);
            const int m = nu - order;
            if (cst == 1.0 && m == 0) continue;
            std::ostringstream c;
            if (cst != 1.0) c << lit(cst);
            for (int t = 0; t < m; ++t) c << ((cst != 1.0 || t > 0) ? "*" : "") << "x[" << sp << "]";
            d << "*(" << c.str() << ")";
          }
          if (zero) continue;
          any = true;
          body << "    ub[" << q << "] = RS_FMA(gj, " << d.str() << ", ub[" << q << "]);\n";
        }
        if (!any) continue;
        o << "  { const double gj = dtg * RS_FMA(a0[" << r << "], k1[" << j << "], a1[" << r
          << "] * z2[" << j << "]);\n" << body.str() << "  }\n";
      }
  }

  // pivots in elimination order, vector entries by species index (T.ord maps the two)
  void lu_solve(const char* b) {
    for (int k = 0; k < T.ns; ++k)
      for (int e = T.low_ptr[k]; e < T.low_ptr[k + 1]; ++e)
        o << "  " << b << "[" << T.low_row[e] << "] = RS_FMA(-WV(" << T.low_slot[e] << "), " << b
          << "[" << T.ord[k] << "], " << b << "[" << T.low_row[e] << "]);\n";
    for (int i = T.ns - 1; i >= 0; --i) {
      const int si = T.ord[i];
      std::string acc = std::string(b) + "[" + std::to_string(si) + "]";
      for (int e = T.up_ptr[i]; e < T.up_ptr[i + 1]; ++e)
        acc = "RS_FMA(-WV(" + std::to_string(T.up_slot[e]) + "), " + b + "[" +
              std::to_string(T.up_col[e]) + "], " + acc + ")";
      if (strict)
        o << "  " << b << "[" << si << "] = (" << acc << ") / WV(" << T.lu_diag[i] << ");\n";
      else
        o << "  " << b << "[" << si << "] = (" << acc << ") * pv[" << i << "];\n";
    }
  }
};

const char* kPrelude = R"(
typedef unsigned long long u64;
struct PCA {
  double t0, t1, dt0, rtol, atol, maxiters;
  double beta1, beta2, invqmin, invqmax, gamma, qsmin, qsmax, qoldinit;
  int clamp;
  double* totals;
};
static_assert(sizeof(PCA) == 128, "PerCellArgs layout");

// Reciprocal from the hardware approximation r (PTX rcp.approx.ftz.f64) by one third-order
// correction: with e = 1 - d r, 1/d = r / (1 - e) = r (1 + e + e^2 + ...), so r (1 + e + e^2)
// leaves e^3 -- below an ulp for the approximation's |e| -- in three FMAs.  Used by the
// production build in place of IEEE division; d > 0 and normal on every call site (LU pivots
// 1 - dtgamma*J_ii, error-norm denominators >= atol).
__device__ __forceinline__ double rcp_nr(double d) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
  const double e = fma(-d, r, 1.0);
  return fma(r, fma(e, e, e), r);
}
// one Newton step: relative error ~1e-12 or better -- enough for error-norm denominators, whose
// only use is the step-size controller
__device__ __forceinline__ double rcp_nr1(double d) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
  return fma(r, fma(-d, r, 1.0), r);
}
// max(|a|, |b|) as the larger magnitude bit pattern, on 32-bit halves (integer pipe; NaN stays
// NaN)
__device__ __forceinline__ double amax_bits(double a, double b) {
  const unsigned ha = (unsigned)__double2hiint(a) & 0x7fffffffu, la = (unsigned)__double2loint(a);
  const unsigned hb = (unsigned)__double2hiint(b) & 0x7fffffffu, lb = (unsigned)__double2loint(b);
  const bool bl = ha < hb || (ha == hb && la < lb);
  return __hiloint2double((int)(bl ? hb : ha), (int)(bl ? lb : la));
}

// ---- float pairs (value = h + l, about 47 bits) for the error estimate
struct fp2 {
  float h, l;
};
// A double as a pair, on the integer pipe (an FP64 conversion costs an FP64 instruction): h the
// leading 24 bits, l the 29 below them rounded to 24.  Below 2^-74 l loses bits, below 2^-126 the
// value counts as 0; `big` collects the magnitudes so that the caller can refuse values from
// 2^127 on, infinities and NaN.
__device__ __forceinline__ fp2 split_pair(double v, unsigned& big) {
  const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
  const unsigned mag = hi & 0x7fffffffu;
  big = big > mag ? big : mag;
  const unsigned f = (__funnelshift_l(lo, hi, 3) ^ 0x40000000u) & 0x7fffffffu;  // exponent - 896
  const int sc = max((int)(f & 0x7f800000u) - (52 << 23), 0);
  const float l = __int2float_rn((int)(lo & 0x1fffffffu)) * __int_as_float(sc);
  const unsigned sg = hi & 0x80000000u;
  const bool z = mag < (898u << 20);
  return {z ? 0.0f : __uint_as_float(f | sg), z ? 0.0f : __uint_as_float(__float_as_uint(l) ^ sg)};
}
constexpr unsigned kPairBig = 1150u << 20;
__device__ __forceinline__ fp2 pair_renorm(float s, float e) {
  const float h = s + e;
  return {h, e - (h - s)};
}
__device__ __forceinline__ fp2 pair_mul(fp2 a, fp2 b) {
  const float p = a.h * b.h;
  return pair_renorm(p, fmaf(a.h, b.l, fmaf(a.l, b.h, fmaf(a.h, b.h, -p))));
}
__device__ __forceinline__ fp2 pair_add(fp2 a, fp2 b) {
  const float s = a.h + b.h, bb = s - a.h;
  return pair_renorm(s, ((a.h - (s - bb)) + (b.h - bb)) + (a.l + b.l));
}
__device__ __forceinline__ fp2 pair_fnma(fp2 a, fp2 b, fp2 c) {  // c - a b
  const float p = a.h * b.h;
  const float pe = fmaf(a.h, b.l, fmaf(a.l, b.h, fmaf(a.h, b.h, -p)));
  const float s = c.h - p, bb = s - c.h;
  return pair_renorm(s, ((c.h - (s - bb)) + (-p - bb)) + (c.l - pe));
}
// a / b: the quotient of the leading parts and one correction from the exact remainder
__device__ __forceinline__ fp2 pair_div(fp2 a, fp2 b) {
  float r;
  asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(b.h));
  const float q = a.h * r;
  const float rem = fmaf(-q, b.l, fmaf(-q, b.h, a.h) + a.l);
  return pair_renorm(q, rem * r);
}
__device__ __forceinline__ double pair_to_d(fp2 a) { return (double)a.h + (double)a.l; }

// Per-cell step sizes are rounded down to 4 fraction bits (16 sizes per octave): a perturbation
// of the inputs then changes a cell's step sequence only where a proposal sits within the
// perturbation of a lattice point, so per-cell trajectories stay within roundoff of each other
// under roundoff-sized changes.
__device__ __forceinline__ double quant_dt(double d) {
  return __longlong_as_double(__double_as_longlong(d) & ~((1ll << 48) - 1));
}

// block total of v in thread 0: strict build (256 threads), the oracle's pairwise tree v[t] +=
// v[t+s] for s = 128 ... 1; production build, a shuffle tree per warp and the warps' sums in
// order (whole warps, at most 8)
__device__ __forceinline__ double block_total(double v, double* sm) {
  const int t = threadIdx.x;
#if !RS_STRICT
  for (int s = 16; s > 0; s >>= 1) v += __shfl_down_sync(0xffffffffu, v, s);
  if ((t & 31) == 0) sm[t >> 5] = v;
  __syncthreads();
  for (int w = 1; w < (int)(blockDim.x >> 5); ++w) v += sm[w];
  return v;
#else
  sm[t] = v;
  __syncthreads();
  for (int s = 128; s >= 32; s >>= 1) {
    if (t < s) sm[t] = sm[t] + sm[t + s];
    __syncthreads();
  }
  double a = sm[t];
  if (t < 32) {
    for (int s = 16; s > 0; s >>= 1) {
      const double o = __shfl_down_sync(0xffffffffu, a, s);
      if (t < s) a = a + o;
    }
  }
  __syncthreads();
  return a;
#endif
}
)";

std::string generate(const MechTables& T, double ros_d, double ros_c32, bool strict,
                     bool with_smem) {
  const int nsplit = split_slots(T);
  Gen g{T, strict, {}};
  auto& o = g.o;
  o << "// generated: " << T.ns << " species, " << T.nr << " reactions, " << T.nlu
    << " LU slots\n";
  o << "#define NS " << T.ns << "\n#define NRA " << (T.nr > 0 ? T.nr : 1) << "\n#define NPA "
    << (T.npart > 0 ? T.npart : 1) << "\n#define NLU " << T.nlu << "\n#define NLU_R "
    << (T.nlu - nsplit) << "  // LU slots in registers in the split variant\n";
  o << "#define ROS_D " << lit(ros_d) << "\n#define ROS_C32 " << lit(ros_c32) << "\n";
  o << "#define OFF_DONE " << offsetof(Ctl, done) << "\n#define OFF_CUR " << offsetof(Ctl, cur)
    << "\n#define OFF_DTC " << offsetof(Ctl, dtc) << "\n#define OFF_DTO2 "
    << offsetof(Ctl, dto2) << "\n#define OFF_DTO6 " << offsetof(Ctl, dto6)
    << "\n#define OFF_DTG " << offsetof(Ctl, dtgamma)
    << "\n#define OFF_ITERS "
    << offsetof(Ctl, iters) << "\n#define OFF_NACC " << offsetof(Ctl, nacc)
    << "\n#define OFF_KZ " << offsetof(Ctl, kz) << "\n#define OFF_KZCAP "
    << offsetof(Ctl, kzcap) << "\n";
  // the kernels in units that compile side by side (RS_UNIT 0: all of them)
  o << "#ifndef RS_UNIT\n#define RS_UNIT 0\n#endif\n#define RS_IN(k) (RS_UNIT == 0 || RS_UNIT == (k))\n";
  // about the FP64 instructions of an attempt (two right-hand sides, the Jacobian, W, its LU, two
  // solves, the updates) at 64 cycles of 0.48 ns
  const size_t ops = 2 * (T.rhs_r.size() + T.nr) + T.nr + T.npart + T.jac_part.size() + T.upd_dst.size() +
                     T.elim_lik.size() + 2 * T.nlu + 11 * T.ns;
  o << "#define RS_WARP_NS " << ops * 31 << "u\n";
  o << "#define RS_STRICT " << (strict ? 1 : 0) << "\n#define RS_PAIRS " << (jit_pairs(T, strict) ? 1 : 0) << "\n" << kPrelude << R"(
// The first wave's warps of one SM sub-partition (`depth` of them fit; 152 SMs with four each) start
// apart, over the FP64 time of one warp (RS_WARP_NS).  Started together they stay in lock step: all
// load, convert and miss the instruction cache at once and leave the FP64 pipe idle, and they
// finish together, so that what is left over runs as a whole extra wave.  One warp alone keeps the
// pipe busy, so the wait costs nothing once the grid has more than one wave (615,888 cells: 910 ->
// 886 us per attempt, 314,496: 497 -> 479, 155,664: 271 -> 255, 111,555: 186 -> 178).
__device__ __forceinline__ void stagger(unsigned depth) {
  const unsigned wpb = blockDim.x >> 5, w = blockIdx.x * wpb / 608u;
  if (w > 0u && w < depth && gridDim.x * wpb > depth * 608u) __nanosleep(w * RS_WARP_NS / (depth - 1u));
}
)";
  // Every multiply-add is written out: RS_FMA fuses in the production build and keeps the
  // multiply and the add separate in the strict build; both builds compile with --fmad=false,
  // so no compiler contraction decides anything and all variants compute the same bits.
  o << (strict ? "#define RS_FMA(a, b, c) ((a) * (b) + (c))\n"
                 "#define RS_VDECL double v[NRA];  // the rates of the oracle-order RHS\n"
               : "#define RS_FMA(a, b, c) fma((a), (b), (c))\n"
                 "#define RS_VDECL  // the fused RHS keeps no rate array\n");
  // One ROS23 attempt of one cell: xn (unclamped) and the cell's sum of squared scaled errors.
  // f0 = f(x) is computed here unless the caller already holds it (have_f0): after an
  // accepted attempt whose clamp left the state bit for bit unchanged, f(x_new) is exactly
  // the third RHS evaluation f2 of that attempt.  fout (global layout, may be null) receives
  // f2 when the clamp leaves xn unchanged and a NaN marker in plane 0 otherwise; with KEEP
  // the caller also gets f2 in registers.
  o << R"(
// the stage-tape slot of the attempt a controller is running (null when it keeps no tape):
// slot = the accepted count, [2][NS][N] doubles per slot, slots below the controller's kzcap
// a field of the controller record, which the grid before this one may still be writing until the
// wait: a coherent load that stays in program order
template <class V>
__device__ __forceinline__ V ctl_field(const unsigned char* ctl, int off) {
  return *(const volatile V*)(ctl + off);
}
__device__ __forceinline__ double* stage_slot(const unsigned char* ctl, u64 N) {
  double* kz = ctl_field<double*>(ctl, OFF_KZ);
  const int cap = ctl_field<int>(ctl, OFF_KZCAP);
  const int slot = (int)ctl_field<double>(ctl, OFF_NACC);
  return (kz && slot >= 0 && slot < cap) ? kz + (u64)slot * 2 * NS * N : nullptr;
}
// SOL: the step's solution only (a replay along recorded accepted steps needs no error norm).
// W storage: LU slots e < KR in the register array W, the others in shared memory at
// WSM[(e - KR) * 64] (this thread's column of a [slot][thread] array per 64 threads of the block, see
// w_column); every slot index is a compile-time constant, so each access resolves to one of the two
// when compiled.
// un, fin (may be null): where the clamped new state and, unless have_f0, f(x) go in global
// memory -- written as soon as they are final, so that neither stays live through the error solve.
// PAIRS: the error estimate in float pairs; returns a negative value where the pairs' range does
// not hold it (the caller forms the estimate again without PAIRS).
template <bool HE, int KR, bool KEEP, bool SOL = false, bool PAIRS = false>
__device__ __forceinline__ double ros23_cell(const double* __restrict__ kr,
    const double* __restrict__ em, u64 N, int c, const double* x, double* xn, double* W,
    double* WSM, double* f0, bool have_f0, double* __restrict__ fout, int clamp, double* f2,
    double dt, double dto2, double dto6, double dtg, double rtol, double atol,
    double* __restrict__ kzo, double* __restrict__ un = nullptr,
    double* __restrict__ fin = nullptr) {
#define K(r) __ldg(kr + (u64)(r) * N + c)
#define EM(s) __ldg(em + (u64)(s) * N + c)
#define WV(e) (*((e) < KR ? &W[(e)] : &WSM[((e) - KR) * 64]))
  RS_VDECL
  double P[NPA], k1[NS], f1[NS], k2[NS], b[NS], pv[NS];
  if (!have_f0) {
)";
  g.rates_rhs("x", "f0");
  o << "  }\n";
  if (g.strict) {
    g.partials();
    g.build_w();
  } else {
    g.build_w_scaled();
  }
  g.lu_factor();
  o << "#pragma unroll\n  for (int s = 0; s < NS; ++s) k1[s] = f0[s];\n";
  g.lu_solve("k1");
  o << "  if (kzo) {  // stage tape: k1\n#pragma unroll\n    for (int s = 0; s < NS; ++s) "
       "kzo[(u64)s * N + c] = k1[s];\n  }\n";
  o << "#pragma unroll\n  for (int s = 0; s < NS; ++s) xn[s] = RS_FMA(dto2, k1[s], x[s]);\n";
  g.rates_rhs("xn", "f1");
  o << "#pragma unroll\n  for (int s = 0; s < NS; ++s) k2[s] = f1[s] - k1[s];\n";
  g.lu_solve("k2");
  o << "  if (kzo) {  // stage tape: z2, the solve's result before k1 is added\n#pragma unroll\n"
       "    for (int s = 0; s < NS; ++s) kzo[(u64)(NS + s) * N + c] = k2[s];\n  }\n";
  o << "#pragma unroll\n  for (int s = 0; s < NS; ++s) k2[s] = k2[s] + k1[s];\n";
  o << "#pragma unroll\n  for (int s = 0; s < NS; ++s) xn[s] = RS_FMA(dt, k2[s], x[s]);\n";
  o << "  if constexpr (SOL) return 0.0;\n";
  g.rates_rhs("xn", "b");
  o << R"(  if (fout) {
    bool same = true;
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      const double cl = clamp ? fmax(xn[s], 0.0) : xn[s];
      same = same && (__double_as_longlong(cl) == __double_as_longlong(xn[s]));
    }
    if (same) {
#pragma unroll
      for (int s = 0; s < NS; ++s) fout[(u64)s * N + c] = b[s];
    } else {
      fout[c] = __longlong_as_double(0x7ff8000000000000LL);
    }
  }
  if constexpr (KEEP) {
#pragma unroll
    for (int s = 0; s < NS; ++s) f2[s] = b[s];
  }
)";
  o << R"(  if (fin && !have_f0) {  // f(x), for a retry of this state after a rejection
#pragma unroll
    for (int s = 0; s < NS; ++s) fin[(u64)s * N + c] = f0[s];
  }
)";
  const char* store_un = R"(  if (un) {
#pragma unroll
    for (int s = 0; s < NS; ++s) un[(u64)s * N + c] = clamp ? fmax(xn[s], 0.0) : xn[s];
  }
)";
  if (!g.strict) {
    // The error estimate dt/6 (k1 - 2 k2 + k3).  With W k1 = f0 and W k2 = f1 - k1 + f0 the third
    // stage's equation becomes W (k1 - 2 k2 + k3) = (f2 - 2 f1 + f0) - c32 (k2 - f1): one solve for
    // the whole estimate, whose right-hand side takes the cancellation in FP64.  Nothing after it
    // cancels, and the norm only steers the step size, so on large grids solve and norm run in
    // float pairs on the FP32 pipe (relative error ~1e-13; the FP64 norm's one-step reciprocal
    // has 1e-12): 131 FP64 instructions of 64 cycles each become ~2,900 instructions on pipes that
    // stand idle beside them.  Where one warp per sub-partition runs alone (attempt_fp64_norm) the
    // FP64 form's shorter chain wins.
    o << R"(#pragma unroll
  for (int s = 0; s < NS; ++s)
    b[s] = fma(-ROS_C32, k2[s] - f1[s], fma(-2.0, f1[s], b[s]) + f0[s]);
  if constexpr (PAIRS) {
  unsigned big = 0;
  float eh[NS], el[NS], dh[NS], dl[NS];
  const fp2 rt = split_pair(rtol, big), at0 = split_pair(atol, big);
#pragma unroll
  for (int s = 0; s < NS; ++s) {
    const fp2 v = split_pair(b[s], big);
    const fp2 den = pair_add(pair_mul(split_pair(amax_bits(x[s], xn[s]), big), rt), at0);
    eh[s] = v.h;
    el[s] = v.l;
    dh[s] = den.h;
    dl[s] = den.l;
  }
)" << store_un << R"(#define pair_msub(i, slot, k)                                                              \
  {                                                                                        \
    const fp2 v_ = pair_fnma(split_pair(WV(slot), big), fp2{eh[k], el[k]}, fp2{eh[i], el[i]}); \
    eh[i] = v_.h;                                                                          \
    el[i] = v_.l;                                                                          \
  }
#define pair_scale(i, q)                                                                   \
  {                                                                                        \
    const fp2 v_ = pair_mul(fp2{eh[i], el[i]}, split_pair(pv[q], big));                    \
    eh[i] = v_.h;                                                                          \
    el[i] = v_.l;                                                                          \
  }
)";
    g.solve_pairs();
    o << R"(#undef pair_msub
#undef pair_scale
  fp2 sum = {0.0f, 0.0f};
#pragma unroll
  for (int s = 0; s < NS; ++s) {
    const fp2 q = pair_div(fp2{eh[s], el[s]}, fp2{dh[s], dl[s]});
    sum = pair_add(sum, pair_mul(q, q));
  }
  // a square beyond FP32, or an overflow on the way, leaves an infinity or a NaN in the sum
  return fabsf(sum.h) < 0x1p126f && big < kPairBig ? pair_to_d(sum) * (dto6 * dto6) : -1.0;
  } else {
)" << store_un;
    g.lu_solve("b");
    o << R"(  double acc = 0.0;
#pragma unroll
  for (int s = 0; s < NS; ++s) {
    const double at = b[s] * rcp_nr1(fma(amax_bits(x[s], xn[s]), rtol, atol));
    acc = fma(at, at, acc);
  }
  return acc * (dto6 * dto6);
  }
)";
  } else {
    o << store_un << R"(#pragma unroll
  for (int s = 0; s < NS; ++s)
    b[s] = RS_FMA(-2.0, k1[s] - f0[s], RS_FMA(-ROS_C32, (k2[s] - f1[s]), b[s]));
)";
    g.lu_solve("b");
    o << R"(  double acc = 0.0;
#pragma unroll
  for (int s = 0; s < NS; ++s) {
    const double ut = dto6 * (RS_FMA(-2.0, k2[s], k1[s]) + b[s]);
    const double den = RS_FMA(fmax(fabs(x[s]), fabs(xn[s])), rtol, atol);
    const double at = ut / den;
    acc = RS_FMA(at, at, acc);
  }
  return acc;
)";
  }
  o << R"(#undef K
#undef EM
#undef WV
}

// global-dt attempt: every cell steps with the controller's dtc; one partial sum per block.
// F0/F1 (may be null) pair with U0/U1: F[cur] holds f(U[cur]) per cell (NaN in plane 0 where
// unknown); from the second attempt of a solve on, a cell reuses it instead of evaluating
// f(x) again (the first attempt of a solve starts from a state written elsewhere).
// MODE 0: W in registers; 1: W in shared memory; 2: split (NLU_R slots in registers)
#if !RS_STRICT
// the error estimate of one cell once more in FP64 (values outside the float pairs' range)
template <bool HE>
__device__ __noinline__ double attempt_error_fp64(const double* __restrict__ U,
    const double* __restrict__ kr, const double* __restrict__ em, u64 N, int c, double dt,
    double dto2, double dto6, double dtg, double rtol, double atol) {
  double x[NS], xn[NS], f0[NS], W[NLU];
  for (int s = 0; s < NS; ++s) x[s] = U[(u64)s * N + c];
  return ros23_cell<HE, NLU, false>(kr, em, N, c, x, xn, W, nullptr, f0, false, nullptr, 0,
                                    nullptr, dt, dto2, dto6, dtg, rtol, atol, nullptr);
}
#endif
// a thread's column of the shared part of W: 64 threads to a [slot][thread] array, so that a warp's
// accesses are contiguous, the strides constants and the shared memory that of the block's own threads
__device__ __forceinline__ double* w_column(double* wsm, int slots) {
  return wsm + (threadIdx.x >> 6) * (slots * 64) + (threadIdx.x & 63u);
}
template <bool HE, int MODE, bool PAIRS, int MINB>
__device__ __forceinline__ void attempt_body(const unsigned char* ctl, double* U0, double* U1,
    const double* __restrict__ kr, const double* __restrict__ em, double* partial, int nc, int nsp,
    double rtol, double atol, int clamp, double* F0, double* F1) {
  __shared__ double red[256];
#if !RS_STRICT
  // Programmatic launch: this grid was launched while the controller before it still ran, and lets the
  // controller after it be launched now, which waits here in turn: the launches' latency is hidden
  // (the 600 s window of 36x18x10: 7.71 -> 7.54 ms).  Until the wait the record, the states and F may
  // still change, so none of them is a __restrict__ pointer; kr and em are written before any overlap.
  asm volatile("griddepcontrol.wait;\n\tgriddepcontrol.launch_dependents;" ::: "memory");
#endif
  if (ctl_field<int>(ctl, OFF_DONE)) return;
  const double dt = ctl_field<double>(ctl, OFF_DTC);
  const double dto2 = ctl_field<double>(ctl, OFF_DTO2);
  const double dto6 = ctl_field<double>(ctl, OFF_DTO6);
  const double dtg = ctl_field<double>(ctl, OFF_DTG);
  const int cur = ctl_field<int>(ctl, OFF_CUR);
  const double iters = ctl_field<double>(ctl, OFF_ITERS);
  const double* U = cur ? U1 : U0;
  double* Un = cur ? U0 : U1;
  double* Fin = cur ? F1 : F0;
  double* Fout = cur ? F0 : F1;
  double* __restrict__ kzo = stage_slot(ctl, (u64)nc);
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  const u64 N = (u64)nc;
  double e = 0.0;
#if !RS_STRICT
  stagger(2 * MINB);
#endif
  if (c < nc) {
    double x[NS], xn[NS], f0[NS];
#pragma unroll
    for (int s = 0; s < NS; ++s) x[s] = U[(u64)s * N + c];
    bool have = false;
    if (F0 && iters > 0.0) {
#pragma unroll
      for (int s = 0; s < NS; ++s) f0[s] = Fin[(u64)s * N + c];
      have = f0[0] == f0[0];
    }
    if constexpr (MODE == 1) {
      extern __shared__ double wsm[];
      e = ros23_cell<HE, 0, false, false, PAIRS>(kr, em, N, c, x, xn, nullptr, w_column(wsm, NLU), f0, have,
                                   F0 ? Fout : nullptr, clamp, nullptr, dt, dto2, dto6, dtg,
                                   rtol, atol, kzo, Un, F0 ? Fin : nullptr);
    } else if constexpr (MODE == 2) {
      extern __shared__ double wsm[];
      double W[NLU_R > 0 ? NLU_R : 1];
      e = ros23_cell<HE, NLU_R, false, false, PAIRS>(kr, em, N, c, x, xn, W, w_column(wsm, NLU - NLU_R), f0, have,
                                       F0 ? Fout : nullptr, clamp, nullptr, dt, dto2, dto6,
                                       dtg, rtol, atol, kzo, Un, F0 ? Fin : nullptr);
    } else {
      double W[NLU];
      e = ros23_cell<HE, NLU, false, false, PAIRS>(kr, em, N, c, x, xn, W, nullptr, f0, have,
                                     F0 ? Fout : nullptr, clamp, nullptr, dt, dto2, dto6, dtg,
                                     rtol, atol, kzo, Un, F0 ? Fin : nullptr);
    }
#if !RS_STRICT
    if constexpr (PAIRS)
      if (e < 0.0) e = attempt_error_fp64<HE>(U, kr, em, N, c, dt, dto2, dto6, dtg, rtol, atol);
#endif
    for (int s = NS; s < nsp; ++s) {
      const double xv = U[(u64)s * N + c];
      Un[(u64)s * N + c] = clamp ? fmax(xv, 0.0) : xv;
    }
  }
  const double tot = block_total(e, red);
  if (threadIdx.x == 0) partial[blockIdx.x] = tot;
}

// per-cell adaptive form: persistent threads pull cells from a device work queue and
// integrate each over [t0, t1] with its own PI controller
template <bool HE>
__device__ __forceinline__ void per_cell_body(int nc, int nsp, double* __restrict__ U,
    const double* __restrict__ kr, const double* __restrict__ em,
    double* __restrict__ dt_cell, double* __restrict__ steps_cell,
    unsigned long long* __restrict__ queue, int* __restrict__ status, PCA a) {
  double x[NS], xn[NS], W[NLU], f0[NS], f2[NS];
  bool have = false;  // f0 == f(x) for the current cell
  double my_steps = 0.0, my_attempts = 0.0;
  double t = 0, dt = 0, qold = 0, iters = 0, nacc = 0;
  int c = -1;
  const u64 N = (u64)nc;
  const double tlim = a.t1 - 1.0e-9;
  for (;;) {
    if (c < 0) {
      const unsigned long long nxt = atomicAdd(queue, 1ull);
      if (nxt >= (unsigned long long)nc) break;
      c = (int)nxt;
#pragma unroll
      for (int s = 0; s < NS; ++s) x[s] = U[(u64)s * N + c];
      have = false;
      t = a.t0;
      dt = quant_dt(dt_cell[c] > 0.0 ? dt_cell[c] : a.dt0);
      qold = a.qoldinit;
      iters = 0;
      nacc = 0;
    }
    if ((t < tlim) && (iters < a.maxiters)) {
      const double dtc = fmin(dt, a.t1 - t);
      const double sse = ros23_cell<HE, NLU, true>(kr, em, N, c, x, xn, W, nullptr, f0, have, nullptr,
                                                 a.clamp, f2, dtc, dtc / 2, dtc / 6,
                                                 dtc * ROS_D, a.rtol, a.atol, nullptr);
      have = true;  // f0 == f(x) after the call; replaced below if x moves
      double EEst = sqrt(sse / (double)nsp);
      if (EEst != EEst) EEst = 1.0e10;
      const double q11 = pow(fmax(EEst, 1.0e-35), a.beta1);
      double q = q11 / pow(qold, a.beta2);
      q = fmax(a.invqmax, fmin(a.invqmin, q / a.gamma));
      if (EEst <= 1.0) {
        bool same = true;
#pragma unroll
        for (int s = 0; s < NS; ++s) {
          const double xs = a.clamp ? fmax(xn[s], 0.0) : xn[s];
          same = same && (__double_as_longlong(xs) == __double_as_longlong(xn[s]));
          x[s] = xs;
        }
        if (same) {
#pragma unroll
          for (int s = 0; s < NS; ++s) f0[s] = f2[s];
        }
        have = same;
        t = t + dtc;
        const bool insteady = (a.qsmin <= q) && (q <= a.qsmax);
        dt = quant_dt(dtc / (insteady ? 1.0 : q));
        qold = fmax(EEst, a.qoldinit);
        nacc += 1.0;
      } else {
        dt = quant_dt(dtc / fmin(a.invqmin, q11 / a.gamma));
      }
      iters += 1.0;
    } else {
      if (t < tlim) atomicOr(status, 1);
#pragma unroll
      for (int s = 0; s < NS; ++s) U[(u64)s * N + c] = x[s];
      dt_cell[c] = dt;
      if (steps_cell) steps_cell[c] = nacc;
      my_steps += nacc;
      my_attempts += iters;
      c = -1;
    }
  }
  if (a.totals) {
    atomicAdd(a.totals, my_steps);
    atomicAdd(a.totals + 1, my_attempts);
  }
}

#define RS_ATTEMPT(NAME, HE, MODE, MINB, PAIRS)                                                  \
  extern "C" __global__ void __launch_bounds__(256, MINB) NAME(                             \
      const unsigned char* ctl, double* U0, double* U1, const double* __restrict__ kr,      \
      const double* __restrict__ em, double* partial, int nc, int nsp, double rtol,         \
      double atol, int clamp, double* F0, double* F1) {                                     \
    attempt_body<HE, MODE, PAIRS, MINB>(ctl, U0, U1, kr, em, partial, nc, nsp, rtol, atol, clamp, F0,    \
                           F1);                                                             \
  }
#if RS_IN(1) && RS_PAIRS
RS_ATTEMPT(rs_jit_attempt_l0, false, 0, 1, false)
RS_ATTEMPT(rs_jit_attempt_l1, true, 0, 1, false)
#endif
#if RS_IN(2)
RS_ATTEMPT(rs_jit_attempt_r0, false, 0, 1, RS_PAIRS)
RS_ATTEMPT(rs_jit_attempt_r1, true, 0, 1, RS_PAIRS)
#endif
#if RS_IN(3)
RS_ATTEMPT(rs_jit_attempt_q0, false, 0, 2, RS_PAIRS)
RS_ATTEMPT(rs_jit_attempt_q1, true, 0, 2, RS_PAIRS)
#endif

// one accepted step at the controller's dtc without the error estimate: the attempt's own
// arithmetic up to the new state (the same bits), for the fixed-sequence replay of a recorded
// macro step
template <bool HE>
__device__ __forceinline__ void step_body(const unsigned char* __restrict__ ctl,
    double* __restrict__ U0, double* __restrict__ U1, const double* __restrict__ kr,
    const double* __restrict__ em, int nc, int nsp, int clamp) {
  if (*(const int*)(ctl + OFF_DONE)) return;
  const double dt = *(const double*)(ctl + OFF_DTC);
  const double dto2 = *(const double*)(ctl + OFF_DTO2);
  const double dtg = *(const double*)(ctl + OFF_DTG);
  const int cur = *(const int*)(ctl + OFF_CUR);
  const double* __restrict__ U = cur ? U1 : U0;
  double* __restrict__ Un = cur ? U0 : U1;
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= nc) return;
  const u64 N = (u64)nc;
  double x[NS], xn[NS], f0[NS], W[NLU];
#pragma unroll
  for (int s = 0; s < NS; ++s) x[s] = U[(u64)s * N + c];
  ros23_cell<HE, NLU, false, true>(kr, em, N, c, x, xn, W, nullptr, f0, false, nullptr, clamp, nullptr,
                                 dt, dto2, 0.0, dtg, 0.0, 0.0, stage_slot(ctl, N));
#pragma unroll
  for (int s = 0; s < NS; ++s) Un[(u64)s * N + c] = clamp ? fmax(xn[s], 0.0) : xn[s];
  for (int s = NS; s < nsp; ++s) {
    const double xv = U[(u64)s * N + c];
    Un[(u64)s * N + c] = clamp ? fmax(xv, 0.0) : xv;
  }
}
#define RS_STEP(NAME, HE)                                                                   \
  extern "C" __global__ void __launch_bounds__(256, 2) NAME(                                \
      const unsigned char* __restrict__ ctl, double* __restrict__ U0,                       \
      double* __restrict__ U1, const double* __restrict__ kr,                               \
      const double* __restrict__ em, int nc, int nsp, int clamp) {                          \
    step_body<HE>(ctl, U0, U1, kr, em, nc, nsp, clamp);                                     \
  }
#if RS_IN(6)
RS_STEP(rs_jit_step_0, false)
RS_STEP(rs_jit_step_1, true)
#endif
)";
  if (with_smem)
    o << "#if RS_IN(4)\nRS_ATTEMPT(rs_jit_attempt_s0, false, 1, 1, RS_PAIRS)\nRS_ATTEMPT(rs_jit_attempt_s1, true, 1, 1, RS_PAIRS)\n#endif\n";
  if (nsplit > 0)
    o << "#if RS_IN(5)\nRS_ATTEMPT(rs_jit_attempt_h0, false, 2, 2, RS_PAIRS)\nRS_ATTEMPT(rs_jit_attempt_h1, true, 2, 2, RS_PAIRS)\n#endif\n";
  o << R"(
#define RS_PER_CELL(NAME, HE)                                                                \
  extern "C" __global__ void __launch_bounds__(256) NAME(int nc, int nsp,                   \
      double* __restrict__ U, const double* __restrict__ kr, const double* __restrict__ em,  \
      double* __restrict__ dt_cell, double* __restrict__ steps_cell,                         \
      unsigned long long* __restrict__ queue, int* __restrict__ status, PCA a) {             \
    per_cell_body<HE>(nc, nsp, U, kr, em, dt_cell, steps_cell, queue, status, a);            \
  }
#if RS_IN(7)
RS_PER_CELL(rs_jit_per_cell_0, false)
RS_PER_CELL(rs_jit_per_cell_1, true)
#endif

// VJP of one ROS23 step at a recorded dt (the table kernel k_ros23_vjp, specialised): forward
// recompute of the live stages, then lam_out = (d unew / d u)^T lam and ebar += d J / d emission.
// KZ: k1 and z2 come from the stage tape (kzi, [2][NS][nc]) written by the step's forward, so
// the two RHS evaluations and forward solves are skipped; the partials, W and its LU are
// recomputed either way.
template <bool HE, bool KZ>
__device__ __forceinline__ void vjp_body(int nc, int nsp, const double* __restrict__ U,
    const double* __restrict__ Uout, const double* __restrict__ lam,
    double* __restrict__ lam_out, const double* __restrict__ kr,
    const double* __restrict__ em, double* __restrict__ ebar, double dt, int clamp,
    const double* __restrict__ kzi) {
#if !RS_STRICT
  stagger(3);
#endif
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= nc) return;
  const u64 N = (u64)nc;
  const double dto2 = dt / 2, dtg = dt * ROS_D;
#define K(r) __ldg(kr + (u64)(r) * N + c)
#define EM(s) __ldg(em + (u64)(s) * N + c)
#define WV(e) W[(e)]
  double x[NS], f0[NS], k1[NS], u1[NS], f1[NS], z2[NS], bb[NS], f0b[NS], f1b[NS], ub[NS], pv[NS];
  RS_VDECL
  double a0[NRA], a1[NRA], P[NPA], P1[NPA], W[NLU];
#pragma unroll
  for (int s = 0; s < NS; ++s) x[s] = U[(u64)s * N + c];
)";
  o << "  if constexpr (!KZ) {\n";
  g.rates_rhs("x", "f0");
  o << "  }\n";
  g.partials("x", "P");
  g.build_w();
  g.lu_factor();
  o << "  if constexpr (KZ) {\n#pragma unroll\n    for (int s = 0; s < NS; ++s) k1[s] = "
       "kzi[(u64)s * N + c];\n  } else {\n";
  o << "#pragma unroll\n  for (int s = 0; s < NS; ++s) k1[s] = f0[s];\n";
  g.lu_solve("k1");
  o << "  }\n";
  o << "#pragma unroll\n  for (int s = 0; s < NS; ++s) u1[s] = RS_FMA(dto2, k1[s], x[s]);\n";
  o << "  if constexpr (!KZ) {\n";
  g.rates_rhs("u1", "f1");
  o << "  }\n";
  g.partials("u1", "P1");
  o << "  if constexpr (KZ) {\n#pragma unroll\n    for (int s = 0; s < NS; ++s) z2[s] = "
       "kzi[(u64)(NS + s) * N + c];\n  } else {\n";
  o << "#pragma unroll\n  for (int s = 0; s < NS; ++s) z2[s] = f1[s] - k1[s];\n";
  g.lu_solve("z2");
  o << "  }\n";
  o << R"(#pragma unroll
  for (int s = 0; s < NS; ++s) {
    double l = lam[(u64)s * N + c];
    if (clamp && Uout && !(Uout[(u64)s * N + c] > 0.0)) l = 0.0;
    ub[s] = l;
    bb[s] = dt * l;
  }
)";
  g.lu_solve_T("bb");
  o << R"(#pragma unroll
  for (int s = 0; s < NS; ++s) {
    f1b[s] = bb[s];
    f0b[s] = RS_FMA(dt, ub[s], -bb[s]);
  }
  {
    double u1b[NS];
#pragma unroll
    for (int s = 0; s < NS; ++s) u1b[s] = 0.0;
)";
  g.jt_apply("P1", "f1b", "a0", "u1b");
  o << R"(#pragma unroll
    for (int s = 0; s < NS; ++s) {
      ub[s] = ub[s] + u1b[s];
      f0b[s] = RS_FMA(dto2, u1b[s], f0b[s]);
    }
  }
)";
  g.lu_solve_T("f0b");
  g.jt_apply("P", "f0b", "a0", "ub");
  g.reaction_sums("bb", "a1");
  g.reaction_sums("f0b", "a0");
  g.hessian();
  o << R"(#pragma unroll
  for (int s = 0; s < NS; ++s) {
    lam_out[(u64)s * N + c] = ub[s];
    if (ebar) ebar[(u64)s * N + c] += f0b[s] + f1b[s];
  }
  for (int s = NS; s < nsp; ++s) {
    double l = lam[(u64)s * N + c];
    if (clamp && Uout && !(Uout[(u64)s * N + c] > 0.0)) l = 0.0;
    lam_out[(u64)s * N + c] = l;
  }
#undef K
#undef EM
#undef WV
}
// 64-thread blocks at 168 registers, three warps per sub-partition: two macro steps' VJPs take 2.9 ms on
// 36x18x10, 4.2 on 48x30x20, 21.2 on 72x46x47, against 3.0, 5.1 and 22.2 with 128 threads and 255
// registers.
#define RS_VJP(NAME, HE, KZ)                                                                 \
  extern "C" __global__ void __launch_bounds__(64, 6) NAME(int nc, int nsp,                 \
      const double* __restrict__ U, const double* __restrict__ Uout,                        \
      const double* __restrict__ lam, double* __restrict__ lam_out,                         \
      const double* __restrict__ kr, const double* __restrict__ em,                         \
      double* __restrict__ ebar, double dt, int clamp, const double* __restrict__ kzi) {     \
    vjp_body<HE, KZ>(nc, nsp, U, Uout, lam, lam_out, kr, em, ebar, dt, clamp, kzi);          \
  }
#if RS_IN(8)
RS_VJP(rs_jit_vjp_0, false, false)
RS_VJP(rs_jit_vjp_1, true, false)
RS_VJP(rs_jit_vjpk_0, false, true)
RS_VJP(rs_jit_vjpk_1, true, true)
#endif

#if RS_IN(6)
// the production reciprocal applied elementwise (accuracy check against IEEE division)
extern "C" __global__ void rs_jit_rcp(const double* __restrict__ x, double* __restrict__ r,
                                      int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) r[i] = rcp_nr(x[i]);
}
#endif
)";
  return o.str();
}

// ------------------------------------------------------------------ wide mechanisms
// Mechanisms too large for the kernels above (their work arrays do not fit a thread's registers)
// get straight-line forms of the two table-walking kernels that run whole solves,
// k_ros23_attempt and k_chem_per_cell, with the same operations in the same order: the same bits.
// What they gain is the table walk itself (an index load in front of every operand) and where the
// work arrays live.  FP64 issues one warp instruction per 64 cycles and SM sub-partition, so two
// warps per sub-partition (one 256-thread block per SM) are enough, and at that occupancy
//   - the least-used LU slots of W, 111 of them, sit in shared memory ([slot][thread]) and the
//     others in registers or their spills: volatile accesses and compiler barriers keep the
//     compiler from promoting shared slots to registers and spilling those;
//   - f, the partials and the Jacobian are formed reaction by reaction (each sum still adds its
//     terms in ascending order), so no rate or partial outlives its reaction;
//   - rate constants are loaded in groups one group ahead.
// 30 species, 60 reactions, 290 slots (3,400 FP64 instructions an attempt, 5.4 ns per cell at the
// FP64 pipe's rate): 12.4 -> 6.8 ns per cell-attempt against k_ros23_attempt (128 threads per SM
// with 226 shared slots: 7.4 ns; W in registers and spills alone: 8.4 ns).  It holds to the largest
// accepted: 44 species 3.72 -> 1.99 ms per attempt on 155,648 cells, 64 species 3.26 -> 1.83, rs_create
// 2.8 s.
constexpr int kWideSlots = (int)((227 * 1024 - 2 * kBlock * sizeof(double)) / (kBlock * sizeof(double)));

bool wide_eligible(const MechTables& T) {
  if (T.ns < 1 || T.ns > 64 || T.nlu > 640 || T.nr > 256) return false;
  for (int e = 0; e < T.njac; ++e)  // the Jacobian's terms arrive with ascending partials
    for (int t = T.jac_ptr[e] + 1; t < T.jac_ptr[e + 1]; ++t)
      if (T.jac_part[t] <= T.jac_part[t - 1]) return false;
  return true;
}
int wide_reg_slots(const MechTables& T) { return T.nlu > kWideSlots ? T.nlu - kWideSlots : 0; }
size_t wide_smem_bytes(const MechTables& T) {
  return (size_t)(T.nlu - wide_reg_slots(T)) * kBlock * sizeof(double);
}

struct WideGen {
  const MechTables& T;
  bool per_cell;
  std::ostringstream o;
  std::vector<int> place;  // position of each slot, hottest first: < KR in a register
  int KR = 0;
  static constexpr int kGroup = 10;  // rate constants loaded together

  void rank_slots() {
    std::vector<long> use(T.nlu, 0);
    for (int k = 0; k < T.ns; ++k) use[T.lu_diag[k]] += 5;
    for (size_t m = 0; m < T.elim_lik.size(); ++m) {
      use[T.elim_lik[m]] += 2;
      for (int u = T.upd_ptr[m]; u < T.upd_ptr[m + 1]; ++u) {
        use[T.upd_dst[u]] += 2;
        use[T.upd_src[u]] += 1;
      }
    }
    for (int sl : T.low_slot) use[sl] += 3;
    for (int sl : T.up_slot) use[sl] += 3;
    std::vector<int> by(T.nlu);
    for (int i = 0; i < T.nlu; ++i) by[i] = i;
    std::stable_sort(by.begin(), by.end(), [&](int a, int b) { return use[a] > use[b]; });
    place.assign(T.nlu, 0);
    for (int i = 0; i < T.nlu; ++i) place[by[i]] = i;
    KR = wide_reg_slots(T);
  }
  std::string w(int slot) const {
    const int p = place[slot];
    return p < KR ? "W" + std::to_string(p) : "S[" + std::to_string((p - KR) * kBlock) + "]";
  }
  static std::string nm(const char* v, int s) { return v + std::to_string(s); }
  void fence() { o << "  RS_FENCE\n"; }
  void load_rates(int g) {
    for (int r = g; r < std::min(T.nr, g + kGroup); ++r) o << "  LDK(" << r << ")\n";
  }
  // one term of a running sum: dst = c * v or dst + c * v, as fma(c, v, dst) of the tables
  // (c = +-1: the same value as an add)
  static std::string term(const std::string& dst, bool first, double c, const char* v) {
    if (first) return dst + " = " + (c == 1.0 ? std::string(v) : c == -1.0 ? "-" + std::string(v) : lit(c) + " * " + v) + ";";
    if (c == 1.0) return dst + " = " + dst + " + " + v + ";";
    if (c == -1.0) return dst + " = " + dst + " - " + v + ";";
    return dst + " = fma(" + lit(c) + ", " + v + ", " + dst + ");";
  }
  void rhs(const char* x, const char* f) {
    std::vector<std::vector<std::pair<int, double>>> per(T.nr);
    for (int sp = 0; sp < T.ns; ++sp)
      for (int t = T.rhs_ptr[sp]; t < T.rhs_ptr[sp + 1]; ++t) per[T.rhs_r[t]].push_back({sp, T.rhs_c[t]});
    std::vector<char> seen(T.ns, 0);
    o << "  {\n";
    load_rates(0);
    for (int g = 0; g < T.nr; g += kGroup) {
      load_rates(g + kGroup);
      for (int r = g; r < std::min(T.nr, g + kGroup); ++r) {
        o << "  { const double v = K" << r;
        for (int q = T.rptr[r]; q < T.rptr[r + 1]; ++q)
          for (int t = 0; t < T.rnu[q]; ++t) o << " * " << nm(x, T.rsp[q]);
        o << ";\n";
        for (auto& sc : per[r]) {
          o << "    " << term(nm(f, sc.first), !seen[sc.first], sc.second, "v") << "\n";
          seen[sc.first] = 1;
        }
        o << "  }\n";
      }
    }
    for (int sp = 0; sp < T.ns; ++sp)
      if (!seen[sp]) o << "  " << nm(f, sp) << " = 0.0;\n";
    o << "  }\n  if (em) {\n";
    for (int sp = 0; sp < T.ns; ++sp) o << "  " << nm(f, sp) << " = " << nm(f, sp) << " + EM(" << sp << ");\n";
    o << "  }\n";
  }
  void build_w() {
    std::vector<std::vector<std::pair<int, double>>> per(T.npart);  // partial -> (entry, coefficient)
    for (int e = 0; e < T.njac; ++e)
      for (int t = T.jac_ptr[e]; t < T.jac_ptr[e + 1]; ++t) per[T.jac_part[t]].push_back({e, T.jac_coef[t]});
    std::vector<char> seen(T.njac, 0), is_jac(T.nlu, 0), is_diag(T.nlu, 0);
    for (int e = 0; e < T.njac; ++e) is_jac[T.jac_slot[e]] = 1;
    for (int k = 0; k < T.ns; ++k) is_diag[T.lu_diag[k]] = 1;
    o << "  {\n";
    load_rates(0);
    int p = 0;
    for (int g = 0; g < T.nr; g += kGroup) {
      load_rates(g + kGroup);
      for (int r = g; r < std::min(T.nr, g + kGroup); ++r) {
        for (; p < T.npart && T.part_r[p] == r; ++p) {
          o << "  { const double P = K" << r;
          for (int q = T.rptr[r]; q < T.rptr[r + 1]; ++q) {
            const int sp = T.rsp[q], nu = T.rnu[q];
            if (sp == T.part_q[p]) {
              if (nu < 2) continue;
              o << " * (" << lit((double)nu);
              for (int t = 1; t < nu; ++t) o << " * " << nm("x", sp);
              o << ")";
            } else {
              for (int t = 0; t < nu; ++t) o << " * " << nm("x", sp);
            }
          }
          o << ";\n";
          for (auto& ec : per[p]) {
            o << "    " << term(w(T.jac_slot[ec.first]), !seen[ec.first], ec.second, "P") << "\n";
            seen[ec.first] = 1;
          }
          o << "  }\n";
        }
        fence();
      }
    }
    for (int e = 0; e < T.nlu; ++e) {
      const char* d = is_diag[e] ? "1.0" : "0.0";
      if (is_jac[e]) o << "  " << w(e) << " = fma(-dtg, " << w(e) << ", " << d << ");\n";
      else o << "  " << w(e) << " = " << d << ";\n";
      if (e % 8 == 7) fence();
    }
    o << "  }\n";
  }
  // the pivot's reciprocal takes the place of U_kk, which nothing reads again
  void lu_factor() {
    int m = 0;
    for (int k = 0; k < T.ns; ++k) {
      fence();
      const std::string d = w(T.lu_diag[k]);
      o << "  { const double pk = rcp_nr(" << d << ");\n  " << d << " = pk;\n";
      for (int ii = T.elim_ptr[k]; ii < T.elim_ptr[k + 1]; ++ii, ++m) {
        const std::string l = w(T.elim_lik[ii]);
        o << "  { const double mu = " << l << " * pk;\n";
        for (int u = T.upd_ptr[m]; u < T.upd_ptr[m + 1]; ++u)
          o << "    " << w(T.upd_dst[u]) << " = fma(-mu, " << w(T.upd_src[u]) << ", " << w(T.upd_dst[u]) << ");\n";
        o << "    " << l << " = mu; }\n";
      }
      o << "  }\n";
    }
  }
  void solve(const char* b) {
    fence();
    for (int k = 0; k < T.ns; ++k) {
      if (k % 4 == 3) fence();
      for (int e = T.low_ptr[k]; e < T.low_ptr[k + 1]; ++e)
        o << "  " << nm(b, T.low_row[e]) << " = fma(-" << w(T.low_slot[e]) << ", " << nm(b, T.ord[k]) << ", "
          << nm(b, T.low_row[e]) << ");\n";
    }
    for (int i = T.ns - 1; i >= 0; --i) {
      if (i % 4 == 3) fence();
      const std::string bi = nm(b, T.ord[i]);
      for (int e = T.up_ptr[i]; e < T.up_ptr[i + 1]; ++e)
        o << "  " << bi << " = fma(-" << w(T.up_slot[e]) << ", " << nm(b, T.up_col[e]) << ", " << bi << ");\n";
      o << "  " << bi << " = " << bi << " * " << w(T.lu_diag[i]) << ";\n";
    }
  }
  void each(const std::string& text) {  // text with # for the species
    for (int sp = 0; sp < T.ns; ++sp) {
      std::string t = text;
      for (size_t i; (i = t.find('#')) != std::string::npos;) t.replace(i, 1, std::to_string(sp));
      o << "  " << t << "\n";
    }
  }
  void decl(const char* v, const char* init = "") {
    o << "  double ";
    for (int sp = 0; sp < T.ns; ++sp) o << (sp ? ", " : "") << nm(v, sp) << init;
    o << ";\n";
  }
  // one attempt from x: n (unclamped) and acc, with f0 = f(x) evaluated unless `have`
  void attempt() {
    for (int i = 0; i < KR; ++i) o << (i ? ", W" : "  double W") << i << (i + 1 == KR ? ";\n" : "");
    decl("k1_"); decl("f1_"); decl("k2_"); decl("n"); decl("b");
    o << "  if (!have) {\n";
    rhs("x", "f0_");
    o << "  }\n";
    build_w();
    lu_factor();
    each("k1_# = f0_#;");
    solve("k1_");
    each("n# = fma(dto2, k1_#, x#);");
    rhs("n", "f1_");
    each("k2_# = f1_# - k1_#;");
    solve("k2_");
    each("k2_# = k2_# + k1_#; n# = fma(dt, k2_#, x#);");
    rhs("n", "b");
    if (per_cell) each("f2_# = b#;");
    each("b# = fma(-2.0, k1_# - f0_#, fma(-ROS_C32, k2_# - f1_#, b#));");
    solve("b");
    o << "  double acc = 0.0;\n";
    each("{ const double ut = dto6 * (fma(-2.0, k2_#, k1_#) + b#); const double at = ut * "
         "rcp_nr1(fma(amax_bits(x#, n#), rtol, atol)); acc = fma(at, at, acc); }");
  }
};

std::string generate_wide(const MechTables& T, double ros_d, double ros_c32, bool per_cell) {
  WideGen g{T, per_cell, {}, {}, 0};
  g.rank_slots();
  auto& o = g.o;
  o << "// generated: " << T.ns << " species, " << T.nr << " reactions, " << T.nlu << " LU slots, " << g.KR
    << " of them in registers\n#define NS " << T.ns << "\n#define NRA " << (T.nr > 0 ? T.nr : 1)
    << "\n#define ROS_D " << lit(ros_d) << "\n#define ROS_C32 " << lit(ros_c32) << "\n#define OFF_DONE "
    << offsetof(Ctl, done) << "\n#define OFF_CUR " << offsetof(Ctl, cur) << "\n#define OFF_DTC "
    << offsetof(Ctl, dtc) << "\n#define OFF_DTO2 " << offsetof(Ctl, dto2) << "\n#define OFF_DTO6 "
    << offsetof(Ctl, dto6) << "\n#define OFF_DTG " << offsetof(Ctl, dtgamma) << "\n#define RS_STRICT 1\n"
    << kPrelude << "#define RS_FENCE asm volatile(\"\" ::: \"memory\");\n#define EM(s) __ldg(em + (u64)(s) * N + c)\n";
  if (!per_cell) {
    o << R"(#define LDK(r) double K##r; asm volatile("ld.global.nc.f64 %0, [%1];" : "=d"(K##r) : "l"(kr + (u64)(r) * N + c));
extern "C" __global__ void __launch_bounds__(256, 1) rs_wide_attempt(
    const unsigned char* __restrict__ ctl, double* U0, double* U1,
    const double* __restrict__ kr, const double* __restrict__ em, double* __restrict__ partial,
    int nc, int nsp, double rtol, double atol, int clamp) {
  extern __shared__ double wsm[];
  __shared__ double red[256];
  if (*(const int*)(ctl + OFF_DONE)) return;
  volatile double* S = wsm + threadIdx.x;
  const double dt = *(const double*)(ctl + OFF_DTC), dto2 = *(const double*)(ctl + OFF_DTO2);
  const double dto6 = *(const double*)(ctl + OFF_DTO6), dtg = *(const double*)(ctl + OFF_DTG);
  const int cur = *(const int*)(ctl + OFF_CUR);
  const double* U = cur ? U1 : U0;
  double* Un = cur ? U0 : U1;
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  const u64 N = (u64)nc;
  double e = 0.0;
  if (c < nc) {
  const bool have = false;
)";
    g.decl("f0_");
    g.each("const double x# = U[(u64)# * N + c];");
    g.attempt();
    g.each("Un[(u64)# * N + c] = clamp ? fmax(n#, 0.0) : n#;");
    o << R"(  for (int s = NS; s < nsp; ++s) {
    const double xv = U[(u64)s * N + c];
    Un[(u64)s * N + c] = clamp ? fmax(xv, 0.0) : xv;
  }
  e = acc;
  }
  const double tot = block_total(e, red);
  if (threadIdx.x == 0) partial[blockIdx.x] = tot;
}
)";
    return o.str();
  }
  o << R"(#define LDK(r) const double K##r = kc[r];
extern "C" __global__ void __launch_bounds__(256, 1) rs_wide_per_cell(int nc, int nsp,
    double* __restrict__ U, const double* __restrict__ kr, const double* __restrict__ em,
    double* __restrict__ dt_cell, double* __restrict__ steps_cell,
    unsigned long long* __restrict__ queue, int* __restrict__ status, PCA a) {
  extern __shared__ double wsm[];
  volatile double* S = wsm + threadIdx.x;
  volatile double kc[NRA];
  const u64 N = (u64)nc;
  const double rtol = a.rtol, atol = a.atol;
  double my_steps = 0.0, my_attempts = 0.0;
  double t = 0, dtn = 0, qold = 0, iters = 0, nacc = 0;
  bool have = false;
  int c = -1;
  const double tlim = a.t1 - 1.0e-9;
)";
  g.decl("x", " = 0.0");
  g.decl("f0_", " = 0.0");
  g.decl("f2_", " = 0.0");
  o << R"(  for (;;) {
  if (c < 0) {
    const unsigned long long nxt = atomicAdd(queue, 1ull);
    if (nxt >= (unsigned long long)nc) break;
    c = (int)nxt;
)";
  g.each("x# = U[(u64)# * N + c];");
  o << R"(#pragma unroll 4
    for (int r = 0; r < NRA; ++r) kc[r] = kr[(u64)r * N + c];
    have = false;
    t = a.t0;
    dtn = quant_dt(dt_cell[c] > 0.0 ? dt_cell[c] : a.dt0);
    qold = a.qoldinit;
    iters = 0;
    nacc = 0;
  }
  if ((t < tlim) && (iters < a.maxiters)) {
  const double dt = fmin(dtn, a.t1 - t), dto2 = dt / 2, dto6 = dt / 6, dtg = dt * ROS_D;
)";
  g.attempt();
  o << R"(  have = true;  // f0 == f(x); replaced below if x moves
  double EEst = sqrt(acc / (double)nsp);
  if (isnan(EEst)) EEst = 1.0e10;
  const double q11 = pow(fmax(EEst, 1.0e-35), a.beta1);
  double q = q11 / pow(qold, a.beta2);
  q = fmax(a.invqmax, fmin(a.invqmin, q / a.gamma));
  if (EEst <= 1.0) {
    bool same = true;  // the clamp left the candidate as it was: f(x) is f2
)";
  g.each("{ const double xs = a.clamp ? fmax(n#, 0.0) : n#; same = same && (__double_as_longlong(xs) == "
         "__double_as_longlong(n#)); x# = xs; }");
  o << "    if (same) {\n";
  g.each("f0_# = f2_#;");
  o << R"(    }
    have = same;
    t = t + dt;
    const bool insteady = (a.qsmin <= q) && (q <= a.qsmax);
    dtn = quant_dt(dt / (insteady ? 1.0 : q));
    qold = fmax(EEst, a.qoldinit);
    nacc += 1.0;
  } else {
    dtn = quant_dt(dt / fmin(a.invqmin, q11 / a.gamma));
  }
  iters += 1.0;
  } else {
    if (t < tlim) atomicOr(status, 1);
)";
  g.each("U[(u64)# * N + c] = x#;");
  o << R"(    dt_cell[c] = dtn;
    if (steps_cell) steps_cell[c] = nacc;
    my_steps += nacc;
    my_attempts += iters;
    c = -1;
  }
  }
  if (a.totals) {
    atomicAdd(a.totals, my_steps);
    atomicAdd(a.totals + 1, my_attempts);
  }
}
)";
  return o.str();
}

// ------------------------------------------------------------------ compile cache
struct Compiled {
  std::vector<cudaLibrary_t> libs;
  double ms = 0;
};
std::mutex g_mu;
std::map<std::string, Compiled> g_cache;  // source + options -> loaded library (process life)

}  // namespace

// NVRTC compile of generated source to an sm_103a cubin (no device needed).  With verbose
// the log carries ptxas's resource usage (registers, spill stores/loads, shared memory).
bool jit_compile(const std::string& src, bool strict, bool verbose, std::vector<char>* cubin,
                 std::string* log, int unit) {
  const Nvrtc& N = nvrtc();
  if (!N.ok()) {
    *log = N.why;
    return false;
  }
  nvrtcProgram prog = nullptr;
  nvrtcResult r = N.create(&prog, src.c_str(), "rs_chem_jit.cu", 0, nullptr, nullptr);
  if (r != NVRTC_SUCCESS) {
    *log = std::string("nvrtcCreateProgram: ") + N.err(r);
    return false;
  }
  (void)strict;  // the source itself differs between the builds (RS_FMA)
  std::vector<const char*> opts = {"-arch=sm_103a", "-std=c++17", "--fmad=false"};
  const std::string def = "-DRS_UNIT=" + std::to_string(unit);
  opts.push_back(def.c_str());
  if (verbose) opts.push_back("--ptxas-options=-v");
  r = N.compile(prog, (int)opts.size(), opts.data());
  size_t n = 0;
  N.log_size(prog, &n);
  std::string text(n, '\0');
  if (n) N.log(prog, &text[0]);
  while (!text.empty() && text.back() == '\0') text.pop_back();
  if (r != NVRTC_SUCCESS) {
    *log = std::string("nvrtcCompileProgram: ") + N.err(r) + "\n" + text;
    N.destroy(&prog);
    return false;
  }
  *log = text;
  if (cubin) {
    size_t nb = 0;
    N.cubin_size(prog, &nb);
    cubin->resize(nb);
    N.cubin(prog, cubin->data());
  }
  N.destroy(&prog);
  return true;
}

namespace {

// Compiles the source's units (1 .. units) in parallel threads -- NVRTC compiles a whole program
// in one -- and loads them; units = 0: the source is one unit.
bool compile_and_load(const std::string& src, bool strict, int units, Compiled* out, std::string* why) {
  auto t0 = std::chrono::steady_clock::now();
  const int n = std::max(1, units);
  std::vector<std::vector<char>> cubin(n);
  std::vector<std::string> log(n), thrown;
  std::vector<char> ok(n, 0);
  run_units(n, [&](int u) { ok[u] = jit_compile(src, strict, false, &cubin[u], &log[u], units ? u + 1 : 0); }, &thrown);
  for (int u = 0; u < n; ++u)
    if (!ok[u]) {
      *why = (thrown[u].empty() ? log[u] : "compiling a unit: " + thrown[u]).substr(0, 4000);
      return false;
    }
  for (int u = 0; u < n; ++u) {
    cudaLibrary_t lib = nullptr;
    cudaError_t e = cudaLibraryLoadData(&lib, cubin[u].data(), nullptr, nullptr, 0, nullptr, nullptr, 0);
    if (e != cudaSuccess) {
      *why = std::string("cudaLibraryLoadData: ") + cudaGetErrorString(e);
      for (auto l : out->libs) cudaLibraryUnload(l);
      out->libs.clear();
      return false;
    }
    out->libs.push_back(lib);
  }
  out->ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0)
                .count();
  return true;
}
cudaError_t find_kernel(const Compiled& c, cudaKernel_t* k, const char* name) {
  cudaError_t e = cudaErrorSymbolNotFound;
  for (auto lib : c.libs)
    if ((e = cudaLibraryGetKernel(k, lib, name)) == cudaSuccess) return e;
  cudaGetLastError();  // the units that do not hold it
  return e;
}

}  // namespace

const char* const kJitVariantNames[kJitVariants] = {"regs", "smem", "regs2", "split"};

bool jit_chem_eligible(const MechTables& T) {
  return T.ns >= 1 && T.ns <= 32 && T.nlu <= 256 && T.nr <= 160 && T.npart <= 320;
}

std::string jit_chem_source(const MechTables& T, bool strict) {
  return generate(T, 1.0 / (2.0 + std::sqrt(2.0)), 6.0 + std::sqrt(2.0), strict,
                  smem_bytes(T) <= kSmemCap);
}

std::shared_ptr<JitChem> jit_chem_build(const MechTables& T, double ros_d, double ros_c32,
                                        bool strict, std::string* why) {
  if (!jit_chem_eligible(T)) {
    *why = "mechanism too large for straight-line kernels";
    return nullptr;
  }
  const bool with_smem = smem_bytes(T) <= kSmemCap;
  std::string src = generate(T, ros_d, ros_c32, strict, with_smem);
  std::string key = src + (strict ? "|strict" : "|fast");
  Compiled cmp;
  double ms = 0;
  {
    std::lock_guard<std::mutex> lk(g_mu);
    auto it = g_cache.find(key);
    if (it != g_cache.end()) {
      cmp = it->second;
    } else {
      if (!compile_and_load(src, strict, kJitUnits, &cmp, why)) return nullptr;
      g_cache[key] = cmp;
      ms = cmp.ms;
    }
  }
  auto J = std::make_shared<JitChem>();
  J->compile_ms = ms;
  auto get = [&](cudaKernel_t* k, const char* name) {
    cudaError_t e = find_kernel(cmp, k, name);
    if (e != cudaSuccess && why->empty())
      *why = std::string("cudaLibraryGetKernel(") + name + "): " + cudaGetErrorString(e);
    return e == cudaSuccess;
  };
  bool ok = (!jit_pairs(T, strict) || (get(&J->fp64_norm[0], "rs_jit_attempt_l0") && get(&J->fp64_norm[1], "rs_jit_attempt_l1"))) &&
            get(&J->attempt[0][0], "rs_jit_attempt_r0") && get(&J->attempt[0][1], "rs_jit_attempt_r1") &&
            get(&J->attempt[2][0], "rs_jit_attempt_q0") && get(&J->attempt[2][1], "rs_jit_attempt_q1") &&
            get(&J->per_cell[0], "rs_jit_per_cell_0") && get(&J->per_cell[1], "rs_jit_per_cell_1") &&
            get(&J->rcp, "rs_jit_rcp") && get(&J->vjp[0], "rs_jit_vjp_0") &&
            get(&J->vjp[1], "rs_jit_vjp_1") && get(&J->step[0], "rs_jit_step_0") &&
            get(&J->step[1], "rs_jit_step_1") && get(&J->vjpk[0], "rs_jit_vjpk_0") &&
            get(&J->vjpk[1], "rs_jit_vjpk_1");
  if (!ok) return nullptr;
  // the shared-memory variants: their dynamic shared memory, or dropped where it cannot be set
  auto shared_variant = [&](int v, const char* n0, const char* n1, size_t bytes) {
    if (!get(&J->attempt[v][0], n0) || !get(&J->attempt[v][1], n1)) {
      J->attempt[v][0] = J->attempt[v][1] = nullptr;
      return;
    }
    J->attempt_smem[v] = bytes;
    for (int he = 0; he < 2; ++he) {
      cudaError_t e = cudaFuncSetAttribute((const void*)J->attempt[v][he],
                                           cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)bytes);
      if (e != cudaSuccess) {
        cudaGetLastError();
        J->attempt[v][0] = J->attempt[v][1] = nullptr;
        J->attempt_smem[v] = 0;
        return;
      }
    }
  };
  if (with_smem) shared_variant(1, "rs_jit_attempt_s0", "rs_jit_attempt_s1", smem_bytes(T));
  if (split_slots(T) > 0)
    shared_variant(3, "rs_jit_attempt_h0", "rs_jit_attempt_h1",
                   (size_t)split_slots(T) * kBlock * sizeof(double));
  for (int v = 0; v < kJitVariants; ++v) {
    cudaFuncAttributes fa{};
    if (J->attempt[v][0] && cudaFuncGetAttributes(&fa, (const void*)J->attempt[v][0]) == cudaSuccess)
      J->regs[v] = fa.numRegs;
    else
      cudaGetLastError();
  }
  cudaFuncAttributes fa{};
  if (J->fp64_norm[0] && cudaFuncGetAttributes(&fa, (const void*)J->fp64_norm[0]) == cudaSuccess)
    J->fp64_norm_regs = fa.numRegs;
  why->clear();
  return J;
}

// An FP64 warp instruction takes 64 cycles of its SM sub-partition, so a block's warps cost most
// where they stack on few SMs or leave a coarse last wave: 64 threads up to 2^17 cells (6,480 cells:
// 73 us per attempt at 256 threads, 40 at 64; 29,160: 70 / 66 / 54 at 256 / 128 / 64; 111,555: 199 /
// 194 / 194), 128 above (314,900 cells: 609 -> 574 us; 155,664: 300 -> 295; 615,888: 1,075 -> 1,070),
// 256 from 4 M cells on, where the last wave is nothing and the partial sums would outnumber the
// allocation-free attempt's scratch.  The strict build keeps the oracle's 256-cell partial sums.
int jit_attempt_block(int nc) {
#if RS_STRICT
  (void)nc;
  return kBlock;
#else
  return nc <= (1 << 17) ? 64 : (nc <= (1 << 22) ? 128 : kBlock);
#endif
}

// The shared part of W of a block's own threads.  (Laid out for 256 threads in blocks of 64 or 128, it
// left half to three quarters of an SM's shared memory unused: "smem" 351 -> 129 us on 76,183 cells and
// 1,331 -> 967 on 615,888, "split" 182 -> 148 and 1,063 -> 943.)
size_t jit_attempt_smem(const JitChem& J, int variant, int nc) {
  return J.attempt_smem[variant] / kBlock * jit_attempt_block(nc);
}

// Until a variant is picked, attempts of the loop keep W in registers: the fastest or within 1 % of it
// on every grid (600 s of chemistry in ms, regs / smem / regs2 / split: 76,183 cells 2.90 / 2.89 /
// 3.07 / 3.58; 133,517: 4.43 / 4.37 / 4.96 / 4.67; 211,200: 6.64 / 6.72 / 7.10 / 6.85; 615,888: 17.08 /
// 17.08 / 17.45 / 17.06).  A single attempt evaluates f(x) as well and starts alone; above 2^18 cells
// 128 registers and 16 warps per SM ("regs2") are faster there (us per call, regs / regs2: 211,200
// cells 361 / 369, 294,840: 526 / 510, 437,710: 748 / 713, 615,888: 1,006 / 969, 960,000: 1,533 / 1,483).
int jit_variant(const JitChem& J, int nc, bool reuse) {
  if (J.chosen) return J.attempt[J.variant][0] ? J.variant : 0;
  return !reuse && nc > (1 << 18) && J.attempt[2][0] ? 2 : 0;
}

// Where the attempt forms its error norm in FP64, with W in registers, whatever variant is set (the
// strict build and mechanisms beyond kPairSlots have no other norm and run the variant that is set):
// - up to one warp per SM sub-partition (152 SMs, four each), where its time is its FP64 chain (6,480
//   cells: 40 us per attempt, 45 with the float-pair norm); beyond, the pairs win (615,888 cells:
//   1,070 us with the FP64 norm, 981 with pairs, both with 128 registers);
// - at tolerances that the pairs do not resolve: the split of values below 2^-74 keeps 24 bits, which
//   is out of sight only while such an error is far below atol; outside these bounds the pairs would
//   also send cell after cell to the FP64 form, the attempt twice;
// - in place (one buffer for both states): a cell whose values leave the pairs' range reads its input
//   again, after its new state is stored.
bool jit_fp64_norm(const JitChem& J, int nc, double rtol, double atol) {
  if (!J.fp64_norm[0]) return false;
  return nc <= 152 * 128 || !(atol >= 0x1p-40 && atol <= 0x1p100 && rtol >= 0x1p-60 && rtol <= 0x1p60);
}

void jit_launch_attempt(const JitChem& J, cudaStream_t st, int nc, int nsp, const Ctl* ctl,
                        double* U0, double* U1, const double* kr, const double* em,
                        double* part, double rtol, double atol, int clamp, double* F0,
                        double* F1) {
  const int v = jit_variant(J, nc, F0 && F1);
  const bool fp64 = jit_fp64_norm(J, nc, rtol, atol) || (J.fp64_norm[0] && U0 == U1);
  cudaKernel_t k = fp64 ? J.fp64_norm[em ? 1 : 0] : J.attempt[v][em ? 1 : 0];
  const unsigned char* c = reinterpret_cast<const unsigned char*>(ctl);
  if (!F0 || !F1) F0 = F1 = nullptr;
  void* args[] = {&c, &U0, &U1, &kr, &em, &part, &nc, &nsp, &rtol, &atol, &clamp, &F0, &F1};
  const int block = jit_attempt_block(nc);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((nc + block - 1) / block);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = fp64 ? 0 : jit_attempt_smem(J, v, nc);
  cfg.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = RS_STRICT ? 0 : 1;
  cudaLaunchKernelExC(&cfg, (const void*)k, args);
}

void jit_launch_step(const JitChem& J, cudaStream_t st, int nc, int nsp, const Ctl* ctl,
                     double* U0, double* U1, const double* kr, const double* em, int clamp) {
  cudaKernel_t k = J.step[em ? 1 : 0];
  const unsigned char* c = reinterpret_cast<const unsigned char*>(ctl);
  void* args[] = {&c, &U0, &U1, &kr, &em, &nc, &nsp, &clamp};
  cudaLaunchKernel((const void*)k, dim3((nc + kBlock - 1) / kBlock), dim3(kBlock), args, 0, st);
}

void jit_launch_rcp(const JitChem& J, cudaStream_t st, const double* x, double* r, int n) {
  void* args[] = {&x, &r, &n};
  cudaLaunchKernel((const void*)J.rcp, dim3((n + 255) / 256), dim3(256), args, 0, st);
}

void jit_launch_vjp(const JitChem& J, cudaStream_t st, int nc, int nsp, const double* U,
                    const double* Uout, const double* lam, double* lam_out, const double* kr,
                    const double* em, double* ebar, double dt, int clamp, const double* kz) {
  cudaKernel_t k = kz ? J.vjpk[em ? 1 : 0] : J.vjp[em ? 1 : 0];
  void* args[] = {&nc, &nsp, &U, &Uout, &lam, &lam_out, &kr, &em, &ebar, &dt, &clamp, &kz};
  cudaLaunchKernel((const void*)k, dim3((nc + 63) / 64), dim3(64), args, 0, st);
}

void jit_launch_per_cell(const JitChem& J, cudaStream_t st, int nc, int nsp, int nblocks,
                         int threads, double* U, const double* kr, const double* em,
                         double* dtc, double* steps, unsigned long long* queue, int* status,
                         const PerCellArgs& a) {
  cudaKernel_t k = J.per_cell[em ? 1 : 0];
  PerCellArgs av = a;
  void* args[] = {&nc, &nsp, &U, &kr, &em, &dtc, &steps, &queue, &status, &av};
  cudaLaunchKernel((const void*)k, dim3(nblocks), dim3(threads), args, 0, st);
}

std::shared_ptr<WideChem> wide_chem_build(const MechTables& T, double ros_d, double ros_c32,
                                          bool per_cell, std::string* why) {
#if RS_STRICT
  *why = "the strict build walks the tables";
  return nullptr;
#else
  if (jit_chem_eligible(T) || !wide_eligible(T)) {
    *why = "mechanism outside the wide kernels' range";
    return nullptr;
  }
  const std::string src = generate_wide(T, ros_d, ros_c32, per_cell);
  Compiled cmp;
  {
    std::lock_guard<std::mutex> lk(g_mu);
    auto it = g_cache.find(src + "|wide");
    if (it != g_cache.end()) {
      cmp = it->second;
    } else {
      if (!compile_and_load(src, false, 0, &cmp, why)) return nullptr;
      g_cache[src + "|wide"] = cmp;
    }
  }
  auto Wc = std::make_shared<WideChem>();
  cudaKernel_t* k = per_cell ? &Wc->per_cell : &Wc->attempt;
  cudaError_t e = find_kernel(cmp, k, per_cell ? "rs_wide_per_cell" : "rs_wide_attempt");
  Wc->smem = wide_smem_bytes(T);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute((const void*)*k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Wc->smem);
  if (e != cudaSuccess) {
    cudaGetLastError();
    *why = std::string("wide kernels: ") + cudaGetErrorString(e);
    return nullptr;
  }
  why->clear();
  return Wc;
#endif
}
void wide_launch_attempt(const WideChem& Wc, cudaStream_t st, int nc, int nsp, const Ctl* ctl,
                         double* U0, double* U1, const double* kr, const double* em, double* part,
                         double rtol, double atol, int clamp) {
  const unsigned char* c = reinterpret_cast<const unsigned char*>(ctl);
  void* args[] = {&c, &U0, &U1, &kr, &em, &part, &nc, &nsp, &rtol, &atol, &clamp};
  cudaLaunchKernel((const void*)Wc.attempt, dim3((nc + kBlock - 1) / kBlock), dim3(kBlock), args, Wc.smem, st);
}
// One block per SM (its shared memory); fewer threads each while the cells do not fill 256 per
// SM, so that small batches still use every SM.
void wide_launch_per_cell(const WideChem& Wc, cudaStream_t st, int nsm, int nc, int nsp, double* U,
                          const double* kr, const double* em, double* dtc, double* steps,
                          unsigned long long* queue, int* status, const PerCellArgs& a) {
  const int per = (nc + nsm - 1) / nsm;
  const int thr = per >= kBlock ? kBlock : (per + 31) / 32 * 32;
  const int nb = std::min(nsm, (nc + thr - 1) / thr);
  PerCellArgs av = a;
  void* args[] = {&nc, &nsp, &U, &kr, &em, &dtc, &steps, &queue, &status, &av};
  cudaLaunchKernel((const void*)Wc.per_cell, dim3(nb), dim3(thr), args, Wc.smem, st);
}

}  // namespace rs
