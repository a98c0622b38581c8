"""The straight-line chemistry kernels of mechanisms too large for register-resident code
(30 species and more) against the table-walking kernels they replace: the same bits, for one
global-dt attempt and for per-cell windows with uneven step counts, with and without emissions
and the clamp, at cell counts around the block sizes."""
import numpy as np
import pytest

from reseact.esm_gb300 import Solver, abi, mechanism, workloads
from reseact.esm_gb300._lib import CHEM_KERNEL_AUTO, CHEM_KERNEL_TABLE

pytestmark = pytest.mark.gpu

MECHS = {"30x60": dict(n_species=30, n_reactions=60),
         "36x70": dict(n_species=36, n_reactions=70, seed=7),
         "44x90": dict(n_species=44, n_reactions=90, seed=3)}


def _solver(kind, mech, ncells, emission=False, **kw):
    w = workloads.c3(ncells=ncells, mech=mechanism.synthetic(**MECHS[mech]))
    if emission:
        shape = (w.mech.ns, 1, w.grid["nlat"], w.grid["nlon"])
        w.forcing["emission"] = 1e-10 * np.random.default_rng(3).random(shape)
    s = Solver.for_workload(w, **kw)
    s.set_chem_kernel(kind)
    assert s.chem_kernel()[1].get("wide") == (kind == CHEM_KERNEL_AUTO)
    return w, s


@pytest.mark.parametrize("mech", sorted(MECHS))
@pytest.mark.parametrize("ncells", [1, 255, 257, 3072])
def test_attempt_equals_table_bitwise(mech, ncells):
    out = []
    for kind in (CHEM_KERNEL_TABLE, CHEM_KERNEL_AUTO):
        w, s = _solver(kind, mech, ncells, emission=ncells == 257, chem_mode=abi.RS_CHEM_GLOBAL_DT)
        out.append([s.single_step(abi.RS_OP_CHEMISTRY, w.u0_cellmajor(), 0.0, dt) for dt in (1e-3, 2.0)])
        s.close()
    for (u0, e0), (u1, e1) in zip(*out):
        assert np.array_equal(u0, u1) and e0 == e1


@pytest.mark.parametrize("mech", sorted(MECHS))
@pytest.mark.parametrize("ncells,emission,clamp", [(1, False, True), (33, True, True),
                                                   (4096, False, False), (40960, True, True)])
def test_per_cell_window_equals_table_bitwise(mech, ncells, emission, clamp):
    out = []
    for kind in (CHEM_KERNEL_TABLE, CHEM_KERNEL_AUTO):
        # without the clamp cells can go negative and never finish: a cap on their attempts
        w, s = _solver(kind, mech, ncells, emission, clamp_nonneg=clamp, maxiters=2e4 if clamp else 60)
        s.set_state(w.u0_cellmajor())
        st = [s.macro_step(t, t + 60.0, 15.0, 1e-3, check=clamp) for t in (0.0, 60.0)]
        out.append((s.get_state(), *s.cell_steps(), [(x[0], x[3].naC, x[3].nrC) for x in st]))
        s.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
