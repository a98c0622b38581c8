"""The FP64 transport's forms that a grid's size selects, where they are not the default: a thread per
lat / vertical line against the pencils (the same bits), on the smallest grid, odd ones and one with
open walls, in the production and the bounds-check build; and lon rows too long for shared memory,
one thread per cell, against the strict build (which equals the oracle), periodic and open.

Bound for the latter: the forms differ by the roundings of four stages of ~40 operations on values of the
size of a tracer's largest, 2^-45 of it."""
import numpy as np
import pytest

from reseact.esm_gb300 import Solver, abi, workloads

pytestmark = pytest.mark.gpu


def _work(n, walls):
    w = workloads.c2(nlon=n[0], nlat=n[1], nlev=n[2], seed=1)
    rng = np.random.default_rng(4)
    w.u0[:-1] *= np.exp(0.5 * rng.standard_normal(w.u0[:-1].shape))
    if walls == "open":
        w.grid["lon_bc"] = w.grid["lat_bc"] = abi.RS_BC_OPEN
        med = w.u0[:-1].mean(axis=(1, 2, 3))[:, None, None]
        for key, m in (("qbc_w", n[1]), ("qbc_e", n[1]), ("qbc_s", n[0]), ("qbc_n", n[0])):
            w.forcing[key] = med * np.exp(0.3 * rng.standard_normal((w.mech.ns, n[2], m)))
    return w


def _step(w, dt, shape=None, **kw):
    s = Solver.for_workload(w, do_chemistry=False, **kw)
    if shape:
        s.set_launch_shape(**shape)
    u, e = s.single_step(abi.RS_OP_TRANSPORT, w.u0_cellmajor(), 0.0, dt)
    du = s.rhs_transport(w.u0_cellmajor(), 300.0)
    s.close()
    return u, e, du


@pytest.mark.parametrize("check", [False, True])
@pytest.mark.parametrize("walls", ["closed", "open"])
@pytest.mark.parametrize("n", [(3, 3, 3), (13, 7, 5), (67, 45, 37)])
def test_lines_equal_pencils(n, walls, check):
    w = _work(n, walls)
    a, b = (_step(w, 100.0, dict(yz_line=v), check=check) for v in (0, 1))
    assert all(np.array_equal(x, y) for x, y in zip(a, b)) and np.isfinite(a[0]).all()


@pytest.mark.parametrize("walls", ["closed", "open"])
def test_rows_beyond_shared_memory(walls):
    w = _work((6000, 3, 3), walls)
    (ua, _, da), (ub, _, db) = (_step(w, 2.0, strict=strict) for strict in (True, False))
    for x, y, rows in ((ua, ub, w.nsp), (da, db, w.nsp - 1)):  # (the air mass's tendency is all cancellation)
        x, y = (v.reshape(-1, w.nsp)[:, :rows] for v in (x, y))
        assert (np.abs(y - x) <= 2.0 ** -45 * np.abs(x).max(axis=0)).all()
