"""The tuned per-cell kernel of a mechanism too large for register-resident code: several lanes per
cell for a batch of few cells, where the last cells' latency is the window, the straight-line kernel for
larger ones.  The same bits either way."""
import numpy as np
import pytest

from reseact.esm_gb300 import Solver, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ncells,wide", [(1024, 0), (32768, 1), (1 << 20, 1)])
def test_tuned_kernel_follows_the_batch_size(ncells, wide):
    w = workloads.c3(ncells=ncells)
    t1 = 60.0 if ncells < 1 << 20 else 1.0
    res = []
    for tune in (False, True):
        s = Solver.for_workload(w)
        s.set_state(w.u0_cellmajor())
        if tune:
            c = s.autotune()["per_cell_choice"]
            assert c["wide"] == wide and (wide or c["group"] > 0), c
        s.macro_step(0.0, t1, 15.0, 1e-3)
        res.append(s.get_state())
        s.close()
    assert np.array_equal(*res)
