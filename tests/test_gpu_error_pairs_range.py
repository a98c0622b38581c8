"""The float-pair error estimate of a chemistry attempt at the edges of its range, against the table
kernels' FP64 estimate of the same attempt (same bound as in the middle of the range: 1e-11 relative
and 2^-45 of the norm of dt f, what the cancelling FP64 sum itself loses).  Quotients above 2^64,
whose squares are beyond FP32, come from a tolerance far below the error; states and absolute
tolerances of some 1e-27 lie where a pair's low part runs out of FP32's exponents."""
import numpy as np
import pytest

from reseact.esm_gb300 import Solver, abi, workloads
from reseact.esm_gb300._lib import CHEM_KERNEL_SPECIALIZED, CHEM_KERNEL_TABLE

pytestmark = pytest.mark.gpu

GRID = dict(nlon=64, nlat=31, nlev=13)  # 25,792 cells: float pairs


def _floor(f, u, dt, rtol, atol):
    with np.errstate(over="ignore"):
        return 2.0 ** -45 * np.sqrt(np.mean((dt * f / (rtol * np.abs(u) + atol)) ** 2))


def _check(scale, dt, rtol, atol):
    w = workloads.c2(seed=0, **GRID)
    s = Solver.for_workload(w, rtol=rtol, atol_C=atol)
    u = w.u0_cellmajor() * scale
    floor = _floor(s.rhs_chem(u), u, dt, rtol, atol)
    out = []
    for kind in (CHEM_KERNEL_TABLE, CHEM_KERNEL_SPECIALIZED):
        s.set_chem_kernel(kind)
        out.append(s.single_step(abi.RS_OP_CHEMISTRY, u, 0.0, dt))
    s.close()
    (ua, ea), (ub, eb) = out
    assert np.isfinite(ea) and ea > 0.0 and abs(eb - ea) <= 1e-11 * ea + floor, (ea, eb, floor)
    assert np.abs(ub - ua).max() <= 1e-10 * np.abs(ua).max()
    return ea


@pytest.mark.parametrize("rtol,atol", [(1e-18, 1e-12), (1e-17, 1e-11)])
@pytest.mark.parametrize("dt", [60.0, 300.0])
def test_quotients_beyond_fp32_squares(rtol, atol, dt):
    assert _check(1.0, dt, rtol, atol) > 2.0 ** 64


@pytest.mark.parametrize("scale,atol", [(1e-15, 1e-24), (1e-18, 1e-27), (1e-20, 1e-29), (1e-16, 1e-35)])
@pytest.mark.parametrize("dt", [1.0, 60.0])
def test_small_states_and_tolerances(scale, atol, dt):
    _check(scale, dt, 1e-4, atol)
