"""States of the mixed-precision transport carry pairs that are rounded, not truncated: over one short
step, where every limiter and flux term is far below the state, the difference from the FP64 step is
unbiased and no larger than the pairs' own roundings.

Bounds, relative to each value: the split has hi + lo = v to 2^-49; each of a step's additions (the
three stages, whose sum counts a third, u4 and the last stage) rounds a low part of at most 2^-23
once, and mostly of about 2^-24: below 2^-49.5 rms each, 2^-48 rms for all with a margin of two, and
the sum of the largest roundings, 2^-45, for every value.  Unbiased roundings of N values leave a mean
of rms / sqrt(N); 2^-51 is far above that and a quarter of the bias that truncation has."""
import numpy as np
import pytest

from reseact.esm_gb300 import Solver, abi, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("signs", [False, True])
@pytest.mark.parametrize("grid", [(27, 14, 9), (64, 31, 13)])
def test_short_step_rounds_without_bias(grid, signs):
    w = workloads.c2(nlon=grid[0], nlat=grid[1], nlev=grid[2], seed=3)
    u = w.u0_cellmajor().reshape(grid[0] * grid[1] * grid[2], -1)
    rng = np.random.default_rng(5)
    u[:, :-1] = np.abs(u[:, :-1]) * np.exp(0.5 * rng.standard_normal(u[:, :-1].shape)) + 1e-3
    if signs:  # values of either sign
        u[::3, 1] *= -1.0
    out = []
    for prec in (abi.RS_PREC_FP64, abi.RS_PREC_MIXED):
        s = Solver.for_workload(w, do_chemistry=False, precision=prec, clamp_nonneg=False)
        out.append(s.single_step(abi.RS_OP_TRANSPORT, u.ravel(), 0.0, 1e-3)[0].reshape(u.shape)[:, :-1])
        s.close()
    rel = (out[1] - out[0]) / out[0]
    assert abs(rel.mean()) <= 2.0 ** -51, rel.mean()
    assert np.sqrt(np.mean(rel ** 2)) <= 2.0 ** -48, np.sqrt(np.mean(rel ** 2))
    assert np.abs(rel).max() <= 2.0 ** -45, np.abs(rel).max()
