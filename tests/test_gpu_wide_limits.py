"""The straight-line kernels at the limits of what they accept: the largest mechanism that has them
gives the table kernels' bits, one beyond says why it has none."""
import numpy as np
import pytest

from reseact.esm_gb300 import Solver, abi, mechanism, workloads
from reseact.esm_gb300._lib import CHEM_KERNEL_AUTO, CHEM_KERNEL_TABLE

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [abi.RS_CHEM_GLOBAL_DT, abi.RS_CHEM_PER_CELL])
def test_the_largest_mechanism_equals_the_table(mode):
    w = workloads.c3(ncells=1024, mech=mechanism.synthetic(n_species=64, n_reactions=90, seed=4))
    out = []
    for kind in (CHEM_KERNEL_TABLE, CHEM_KERNEL_AUTO):
        s = Solver.for_workload(w, chem_mode=mode)
        s.set_chem_kernel(kind)
        info = s.chem_kernel()[1]
        assert info["wide"] is (kind == CHEM_KERNEL_AUTO) and info["wide_why"] == ""
        if mode == abi.RS_CHEM_GLOBAL_DT:
            out.append(s.single_step(abi.RS_OP_CHEMISTRY, w.u0_cellmajor(), 0.0, 0.05))
        else:
            s.set_state(w.u0_cellmajor())
            s.macro_step(0.0, 20.0, 15.0, 1e-3)
            out.append((s.get_state(), 0.0))
        s.close()
    assert np.array_equal(out[0][0], out[1][0]) and out[0][1] == out[1][1]


def test_beyond_the_limits_the_reason_is_given():
    s = Solver.for_workload(workloads.c3(ncells=64, mech=mechanism.synthetic(n_species=64, n_reactions=100, seed=4)))
    info = s.chem_kernel()[1]
    assert info["wide"] is False and "range" in info["wide_why"]
    s.close()
