"""rs_ros23_attempt_noalloc with one buffer for both states: the state and the error estimate of the
call with two.  The states are the same bits; the estimates agree to the bound of the float-pair
norm, 1e-11 (in place the norm is formed in FP64).  Tolerances far below the error send the cells
beyond the pairs' range, where the FP64 form reads its input again."""
import ctypes

import numpy as np
import pytest

from reseact.esm_gb300 import Solver, abi, workloads
from reseact.esm_gb300._lib import CHEM_KERNEL_AUTO, CHEM_KERNEL_TABLE

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", [CHEM_KERNEL_AUTO, CHEM_KERNEL_TABLE])
@pytest.mark.parametrize("work,rtol,atol,dt", [("c2", 1e-4, 1e-9, 30.0), ("c2", 1e-18, 1e-12, 300.0),
                                               ("c2-small", 1e-18, 1e-12, 300.0), ("c3", 1e-4, 1e-9, 0.05)])
def test_in_place_attempt(work, rtol, atol, dt, kind):
    if work == "c3":
        w = workloads.c3(ncells=3000)
        kw = dict(chem_mode=abi.RS_CHEM_GLOBAL_DT)
    else:
        n = (64, 31, 13) if work == "c2" else (16, 9, 6)
        w, kw = workloads.c2(nlon=n[0], nlat=n[1], nlev=n[2], seed=0), {}
    s = Solver.for_workload(w, rtol=rtol, atol_C=atol, **kw)
    s.set_chem_kernel(kind)
    s.set_state(w.u0_cellmajor())
    src = torch.as_tensor(np.ascontiguousarray(w.u0).reshape(-1), device="cuda")
    res = []
    for same in (False, True):
        a = src.clone()
        b = a if same else torch.empty_like(a)
        torch.cuda.synchronize()
        e = ctypes.c_double()
        assert s.L.rs_ros23_attempt_noalloc(s.h, dt, a.data_ptr(), b.data_ptr(), ctypes.byref(e)) == abi.RS_OK
        res.append((b.cpu().numpy(), e.value))
    s.close()
    (ua, ea), (ub, eb) = res
    assert np.array_equal(ua, ub)
    assert np.isfinite(ea) and abs(eb - ea) <= 1e-11 * ea, (ea, eb)
