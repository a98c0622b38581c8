"""The embedded error of a mixed-precision transport step, formed in float pairs, against the FP64
transport's, and outside the pairs' range, where it is formed in FP64.

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
