"""The variants of the specialised attempt kernel, on grids where they run: above one warp per SM
sub-partition (19,456 cells) in the production build, any grid in the strict build.  The same
generated arithmetic, so the same state and the same error estimate bit for bit, at cell counts that
fill neither 64- nor 128-thread blocks and on both sides of the block sizes' limit.  Where another
form runs whatever variant is set, the library says so and does not choose among one kernel's times."""
import numpy as np
import pytest

from reseact.esm_gb300 import Solver, abi, mechanism, workloads
from reseact.esm_gb300._lib import CHEM_KERNEL_SPECIALIZED

pytestmark = pytest.mark.gpu

NAMES = ("regs", "smem", "regs2", "split")
SMALL = (16, 9, 6)
LARGE = [(61, 29, 15), (73, 59, 31)]  # 26,535 and 133,517 cells


def _work(n, emission=False):
    w = workloads.c2(nlon=n[0], nlat=n[1], nlev=n[2], seed=2, steps=1)
    if emission:
        e = np.zeros((w.mech.ns, n[2], n[1], n[0]))
        e[w.mech.species.index("NO"), 0] = 1e-4 * np.exp(0.5 * np.random.default_rng(2).standard_normal((n[1], n[0])))
        w.forcing["emission"] = e
    return w


@pytest.mark.parametrize("emission", [False, True])
@pytest.mark.parametrize("n", LARGE)
def test_variants_give_the_same_bits(n, emission):
    w = _work(n, emission)
    u = w.u0_cellmajor()
    res = []
    for v in range(4):
        s = Solver.for_workload(w, do_transport=False)
        s.set_launch_shape(chem_attempt_variant=v)
        assert s.chem_kernel()[1]["runs"] == NAMES[v]
        out = [x for dt in (1e-2, 30.0) for x in s.single_step(abi.RS_OP_CHEMISTRY, u, 0.0, dt)]
        s.set_state(u)
        _, _, b, st = s.macro_step(0.0, 60.0, 15.0, 0.5)
        res.append(out + [s.get_state(), b, (st.naC, st.nrC)])
        s.close()
    for r in res[1:]:
        assert all(np.array_equal(x, y) for x, y in zip(res[0], r))


@pytest.mark.parametrize("n", LARGE)
def test_autotuned_variant_is_bitwise_neutral(n):
    w = _work(n)
    res = []
    for tune in (False, True):
        s = Solver.for_workload(w, do_transport=False)
        s.set_state(w.u0_cellmajor())
        if tune:
            rep = s.autotune()
            assert [a["runs"] for a in rep["chem_attempt"]] == list(NAMES)
            assert s.chem_kernel()[1]["variant"] == rep["chem_choice"] == s.chem_kernel()[1]["runs"]
        _, _, b, _ = s.macro_step(0.0, 60.0, 15.0, 0.5)
        res.append((s.get_state(), b))
        s.close()
    assert np.array_equal(res[0][0], res[1][0]) and res[0][1] == res[1][1]


@pytest.mark.parametrize("n,threads", list(zip(LARGE, (64, 128))))
def test_shared_memory_is_that_of_the_blocks_threads(n, threads):
    s = Solver.for_workload(_work(n), do_transport=False)
    for v, key in ((1, "smem_bytes"), (3, "split_smem_bytes")):
        s.set_launch_shape(chem_attempt_variant=v)
        info = s.chem_kernel()[1]
        assert info["runs_smem_bytes"] == info[key] * threads // 256  # smem_bytes: 256 threads
    s.close()


@pytest.mark.parametrize("n", LARGE)
def test_a_handle_starts_with_w_in_registers(n):
    s = Solver.for_workload(_work(n), do_transport=False)
    assert s.chem_kernel()[1]["runs"] == "regs"
    s.close()


@pytest.mark.parametrize("n,single", [((64, 64, 64), "regs"), ((72, 64, 64), "regs2")])
def test_single_attempts_of_large_grids(n, single):
    s = Solver.for_workload(_work(n), do_transport=False)
    info = s.chem_kernel()[1]
    assert info["runs"] == "regs" and info["runs_single"] == single
    s.set_launch_shape(chem_attempt_variant=3)  # a picked variant serves both
    info = s.chem_kernel()[1]
    assert info["runs"] == info["runs_single"] == info["variant"] == "split"
    s.close()


def test_small_grid_says_what_runs():
    w = _work(SMALL)
    s = Solver.for_workload(w)
    for v in range(4):
        s.set_launch_shape(chem_attempt_variant=v)
        info = s.chem_kernel()[1]
        assert info["variant"] == NAMES[v] and info["runs"] == "fp64_norm" and info["runs_regs"] > 0
    s.set_state(w.u0_cellmajor())
    rep = s.autotune()  # nothing to choose: the variant that was set stays
    assert {(a["runs"], a["ms"], a["regs"]) for a in rep["chem_attempt"]} == {("fp64_norm", rep["chem_attempt"][0]["ms"], info["runs_regs"])}
    assert rep["chem_choice"] == "split"
    s.close()


def test_strict_build_runs_the_variant_that_is_set():
    s = Solver.for_workload(_work(SMALL), strict=True)
    for v in range(4):
        s.set_launch_shape(chem_attempt_variant=v)
        info = s.chem_kernel()[1]
        assert info["runs"] == NAMES[v] and info["runs_regs"] == info["regs"][v]
    s.close()


@pytest.mark.parametrize("n,r", [(18, 40), (24, 50)])
def test_mechanisms_between_the_shared_memory_and_the_straight_line_limits(n, r):
    """More LU slots than fit in shared memory for 256 threads, and too many for float pairs: no smem
    variant and no form beside the variants; the others give the same bits."""
    m = mechanism.synthetic(n_species=n, n_reactions=r)
    for ncells in (1024, 20480):
        w = workloads.c3(ncells=ncells, mech=m)
        u = w.u0_cellmajor()
        res = []
        for v in (0, 2, 3):
            s = Solver.for_workload(w, chem_mode=abi.RS_CHEM_GLOBAL_DT)
            assert s.chem_kernel()[0] == CHEM_KERNEL_SPECIALIZED
            s.set_launch_shape(chem_attempt_variant=v)
            assert s.chem_kernel()[1]["runs"] == NAMES[v]
            res.append(s.single_step(abi.RS_OP_CHEMISTRY, u, 0.0, 1e-3))
            s.close()
        assert np.isfinite(res[0][0]).all() and res[0][1] > 0.0
        for a, e in res[1:]:
            assert np.array_equal(res[0][0], a) and res[0][1] == e
