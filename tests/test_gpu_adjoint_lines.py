"""The transport VJP's line kernels at the edges of their tiles against the oracle's sweep: rows and
lines shorter than the stencil's reach, one line more or less than a tile, rows that no block size
divides, periodic, mirror and open ends.  Bound: 1e-8 of the largest sensitivity, as for the whole
adjoint."""
import numpy as np
import pytest

from reseact.esm_gb300 import Solver, abi, mechanism, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,grid", [("global", (6, 5, 4)), ("global", (15, 8, 17)), ("global", (17, 33, 5)),
                                       ("global", (131, 6, 6)), ("open", (6, 6, 6)), ("open", (13, 13, 13))])
def test_transport_sweep_matches_oracle(kind, grid):
    from oracle import oracle
    oracle.build()
    rng = np.random.default_rng(7)
    nlon, nlat, nlev = grid
    if kind == "global":
        w = workloads.c2(nlon=nlon, nlat=nlat, nlev=nlev)
        mech, u, f, g, t1, dt0 = w.mech, w.u0, w.forcing_abi(), w.grid, 300.0, 15.0
    else:
        mech = mechanism.superfast()
        g, mx, my, mz, dp = workloads.regional_freestream(nlon)
        qb = np.exp(0.3 * rng.standard_normal((mech.ns, nlon, nlon)))
        dp3 = np.broadcast_to(dp[:, None, None], (nlon, nlon, nlon)).copy()
        f = abi.ForcingABI(mx=mx, my=my, mz=mz, dp=dp3, qbc_w=qb, qbc_e=qb, qbc_s=qb, qbc_n=qb)
        u = np.concatenate([np.exp(0.3 * rng.standard_normal((mech.ns, nlon, nlon, nlon))), dp3[None]])
        t1, dt0 = 0.1, 0.05
    mabi = abi.MechanismABI(mech)
    cfg = abi.make_config(g, mabi, do_chemistry=False)
    s = Solver(cfg, mabi)
    s.set_forcing(f)
    o = oracle.Oracle(cfg, f, mabi)
    u = np.ascontiguousarray(u)
    nsp = len(u)
    s.set_state(workloads.soa_to_cellmajor(u, nlon, nlat, nlev))
    s.record(True)
    _, _, _, st = s.macro_step(0.0, t1, dt0, 0.5)
    _, _, _, ost = o.record_macro_step(u.copy(), 0.0, t1, dt0, 0.5)
    assert st.naT == ost[0]
    s.record(False)
    lam = rng.standard_normal(u.shape)
    lam[:, rng.random(u.shape[1:]) < 0.3] = 0.0
    lg, _ = s.adjoint_backward(workloads.soa_to_cellmajor(lam, nlon, nlat, nlev))
    lo, _ = o.adjoint_backward(lam)
    lg = workloads.cellmajor_to_soa(lg, nsp, nlon, nlat, nlev)
    s.close()
    for a, b in zip(lg, lo):
        assert np.abs(a - b).max() <= 1e-8 * np.abs(b).max(), np.abs(a - b).max() / np.abs(b).max()
