"""The embedded error of a transport step, whose norm is formed in float pairs, against a norm formed
in FP64: the mixed-precision step against the FP64 one (whose norm falls back to FP64 at the two small
tolerances), and the FP64 step against the strict build's.  Tolerances outside the pairs' range are
among the cases.

Bound: 1e-11 relative (the pairs' quotient 1e-13, the FP64 norm's one-step reciprocal 1e-12), plus
the norm of 2^-43 of the largest value of each tracer: the states behind the cancelling estimate
carry 47 bits and each of the four stages adds a few roundings of that size."""
import numpy as np
import pytest

from reseact.esm_gb300 import Solver, abi, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("atol", [1e-6, 1e-25, 1e-60])
@pytest.mark.parametrize("dt", [1.0, 300.0])
@pytest.mark.parametrize("grid", [(27, 14, 9), (52, 31, 13)])
def test_estimate_matches_fp64(grid, dt, atol):
    w = workloads.c2(nlon=grid[0], nlat=grid[1], nlev=grid[2], seed=0)
    u = w.u0_cellmajor().reshape(grid[0] * grid[1] * grid[2], -1)
    out = []
    for prec in (abi.RS_PREC_FP64, abi.RS_PREC_MIXED):
        s = Solver.for_workload(w, do_chemistry=False, precision=prec, atol_T=atol)
        out.append(s.single_step(abi.RS_OP_TRANSPORT, u.ravel(), 0.0, dt))
        s.close()
    ea, eb = out[0][1], out[1][1]
    ua, ub = (o[0].reshape(u.shape) for o in out)
    big = np.abs(u).max(axis=0, keepdims=True)
    floor = 2.0 ** -43 * np.sqrt(np.mean((big / (1e-4 * np.abs(u) + atol)) ** 2))
    assert np.isfinite(ea) and ea > 0.0 and abs(eb - ea) <= 1e-11 * ea + floor, (ea, eb, floor)
    assert (np.abs(ub - ua) <= 2.0 ** -40 * big).all()


@pytest.mark.parametrize("atol", [1e-6, 1e-11, 1e-25])
@pytest.mark.parametrize("dt", [1.0, 300.0])
@pytest.mark.parametrize("grid", [(27, 14, 9), (52, 31, 13)])
def test_fp64_estimate_matches_strict(grid, dt, atol):
    # FP64 states differ by a few roundings of the largest value: 2^-49 of it in place of 2^-43
    w = workloads.c2(nlon=grid[0], nlat=grid[1], nlev=grid[2], seed=0)
    u = w.u0_cellmajor().reshape(grid[0] * grid[1] * grid[2], -1)
    u[::7, 3] = 0.0
    u[::5, 4] *= 1e-30
    e = []
    for strict in (True, False):
        s = Solver.for_workload(w, strict=strict, do_chemistry=False, atol_T=atol)
        e.append(s.single_step(abi.RS_OP_TRANSPORT, u.ravel(), 0.0, dt)[1])
        s.close()
    big = np.abs(u).max(axis=0, keepdims=True)
    floor = 2.0 ** -49 * np.sqrt(np.mean((big / (1e-4 * np.abs(u) + atol)) ** 2))
    assert np.isfinite(e[0]) and e[0] > 0.0 and abs(e[1] - e[0]) <= 1e-11 * e[0] + floor, (e, floor)
