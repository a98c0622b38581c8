"""The error estimate of a chemistry attempt in float pairs (large grids of the production build)
against the table kernels' FP64 estimate of the same attempt, for states and steps over many
magnitudes, and outside the pairs' range, where the estimate is formed again in FP64.

Bound: 1e-11 relative (the pairs carry ~1e-13, the FP64 norm's one-step reciprocal 1e-12), plus
what the FP64 form itself loses where the estimate is far below the tolerance: it is the
cancelling sum k1 - 2 k2 + k3 of values of the size of f, each off by up to ~250 roundings (the
RHS sums, the LU, the solves), so 2^-45 of the same norm taken of dt f."""
import numpy as np
import pytest

from reseact.esm_gb300 import Solver, abi, workloads
from reseact.esm_gb300._lib import CHEM_KERNEL_SPECIALIZED, CHEM_KERNEL_TABLE

pytestmark = pytest.mark.gpu


def _check(scale, dt, atol=1e-9):
    w = workloads.c2(nlon=64, nlat=31, nlev=13, seed=0)
    s = Solver.for_workload(w, atol_C=atol)
    u = w.u0_cellmajor() * scale
    f = s.rhs_chem(u)
    with np.errstate(over="ignore"):
        floor = 2.0 ** -45 * np.sqrt(np.mean((dt * f / (1e-4 * np.abs(u) + atol)) ** 2))
    out = []
    for kind in (CHEM_KERNEL_TABLE, CHEM_KERNEL_SPECIALIZED):
        s.set_chem_kernel(kind)
        out.append(s.single_step(abi.RS_OP_CHEMISTRY, u, 0.0, dt))
    s.close()
    (ua, ea), (ub, eb) = out
    assert np.isfinite(ea) and ea > 0.0 and abs(eb - ea) <= 1e-11 * ea + floor, (ea, eb, floor)
    assert np.abs(ub - ua).max() <= 1e-10 * np.abs(ua).max()


@pytest.mark.parametrize("scale", [1e-12, 1e-4, 1.0, 1e3])
@pytest.mark.parametrize("dt", [1e-3, 1.0, 60.0])
def test_estimate_matches_fp64(scale, dt):
    _check(scale, dt)


def test_values_beyond_the_pairs_range():
    """An absolute tolerance below the FP32 exponent range."""
    _check(1.0, 1.0, atol=1e-60)
