// rs_jit.h -- mechanism-specialised chemistry kernels (rs_jit.cu).
//
// At rs_create the host writes the mechanism's rate products, RHS sums, exact Jacobian, the
// pivot-free LU of W = I - dt*d*J and its triangular solves out as straight-line CUDA C++
// (constant indices, constant stoichiometric coefficients) and compiles it for sm_103a with
// NVRTC.  Every work array then lives in registers (or, for W, in shared memory) and no
// thread walks an index table, which removes the table loads and the local-memory traffic of
// the table-walking kernels in rs_chem.cu.  The arithmetic follows the same association as
// those kernels, so a strict-build handle stays bit-compatible with the CPU restatement.
#pragma once
#include <cuda_runtime.h>

#include <memory>
#include <string>
#include <vector>

#include "rs_device.cuh"
#include "rs_mech.h"

namespace rs {

struct PerCellArgs;

// Variants of the global-dt attempt kernel (the autotuner picks one by timing):
//   0 "regs"   W in registers (spilled by ptxas where needed), 256 threads per SM
//   1 "smem"   W in dynamic shared memory, [slot][thread] so a warp's accesses are contiguous
//   2 "regs2"  as 0 but capped at 128 registers for 512 threads per SM
//   3 "split"  the last half of W's LU slots (at most 55) in shared memory, the rest in
//              registers, capped at 128 registers for 512 threads per SM
// in blocks of jit_attempt_block threads.
constexpr int kJitVariants = 4;
extern const char* const kJitVariantNames[kJitVariants];

struct JitChem {
  cudaKernel_t attempt[kJitVariants][2] = {};  // [variant][has emission]; null: not built
  cudaKernel_t fp64_norm[2] = {};              // the attempt of jit_fp64_norm, where the others use pairs
  int fp64_norm_regs = 0;
  cudaKernel_t per_cell[2] = {};               // [has emission]
  cudaKernel_t rcp = nullptr;                  // elementwise production reciprocal
  cudaKernel_t vjp[2] = {};                    // ROS23 step VJP [has emission]
  cudaKernel_t step[2] = {};                   // accepted step, no error estimate [has emission]
  cudaKernel_t vjpk[2] = {};                   // step VJP reading k1, z2 from the stage tape
  size_t attempt_smem[kJitVariants] = {};  // dynamic shared bytes of each attempt variant, 256 threads
  int variant = 0;      // variant used for global-dt attempts ...
  bool chosen = false;  // ... where the autotuner or the caller picked it, else jit_variant's
  double compile_ms = 0;    // NVRTC time (0 when the compiled image came from cache)
  int regs[kJitVariants] = {};  // registers per thread of each attempt variant
};

// True when the mechanism is small enough for straight-line code (all work arrays of one
// attempt fit the register file without a table walk).
bool jit_chem_eligible(const MechTables& T);

// Generate, compile (or fetch from the process-wide cache) and load the specialised kernels
// for the current device.  Returns null and sets *why when NVRTC is unavailable or fails.
std::shared_ptr<JitChem> jit_chem_build(const MechTables& T, double ros_d, double ros_c32,
                                        bool strict, std::string* why);

// The generated source (for inspection and tests).
std::string jit_chem_source(const MechTables& T, bool strict);

// NVRTC compile of generated source to an sm_103a cubin; needs no device.  With verbose the
// log carries ptxas's resource usage.  Returns false with the error text in *log.
bool jit_compile(const std::string& src, bool strict, bool verbose, std::vector<char>* cubin,
                 std::string* log, int unit = 0);  // unit: one of the source's units, 0 for all

// Threads per block of the attempt kernels over nc cells (one partial sum per block).
int jit_attempt_block(int nc);
// The variant that attempts over nc cells run: the picked one, or the grid's.  reuse: attempts of the
// adaptive loop, which keep f(x) from one to the next; false: a single attempt.
int jit_variant(const JitChem& J, int nc, bool reuse);
// Dynamic shared bytes per block of a variant over nc cells.
size_t jit_attempt_smem(const JitChem& J, int variant, int nc);
// Whether attempts run the form with the FP64 norm, whatever variant is set.
bool jit_fp64_norm(const JitChem& J, int nc, double rtol, double atol);

// Same contracts as launch_ros23_attempt / launch_chem_per_cell in rs_kernels.h.
void jit_launch_attempt(const JitChem& J, cudaStream_t st, int nc, int nsp, const Ctl* ctl,
                        double* U0, double* U1, const double* kr, const double* em,
                        double* part, double rtol, double atol, int clamp, double* F0,
                        double* F1);
// same contract as launch_ros23_step in rs_kernels.h
void jit_launch_step(const JitChem& J, cudaStream_t st, int nc, int nsp, const Ctl* ctl,
                     double* U0, double* U1, const double* kr, const double* em, int clamp);
void jit_launch_rcp(const JitChem& J, cudaStream_t st, const double* x, double* r, int n);
// same contract as launch_ros23_vjp in rs_kernels.h
void jit_launch_vjp(const JitChem& J, cudaStream_t st, int nc, int nsp, const double* U,
                    const double* Uout, const double* lam, double* lam_out, const double* kr,
                    const double* em, double* ebar, double dt, int clamp,
                    const double* kz = nullptr);
void jit_launch_per_cell(const JitChem& J, cudaStream_t st, int nc, int nsp, int nblocks,
                         int threads, double* U, const double* kr, const double* em,
                         double* dtc, double* steps, unsigned long long* queue, int* status,
                         const PerCellArgs& a);

// Straight-line forms of the table-walking attempt or per-cell kernel for mechanisms too large for
// JitChem (production build): the same bits, chosen behind the TABLE kernel kind.
struct WideChem {
  cudaKernel_t attempt = nullptr, per_cell = nullptr;
  size_t smem = 0;
};
// the one kernel asked for, or null and *why
std::shared_ptr<WideChem> wide_chem_build(const MechTables& T, double ros_d, double ros_c32,
                                          bool per_cell, std::string* why);
void wide_launch_attempt(const WideChem& W, cudaStream_t st, int nc, int nsp, const Ctl* ctl,
                         double* U0, double* U1, const double* kr, const double* em, double* part,
                         double rtol, double atol, int clamp);
void wide_launch_per_cell(const WideChem& W, cudaStream_t st, int nsm, int nc, int nsp, double* U,
                          const double* kr, const double* em, double* dtc, double* steps,
                          unsigned long long* queue, int* status, const PerCellArgs& a);

}  // namespace rs
