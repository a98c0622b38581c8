"""Kernels that are launched programmatically behind another grid (griddepcontrol.wait) are resident
while that grid still writes.  A __restrict__ pointer promises that nobody else writes the memory
during the whole kernel, so a load through it may be formed as a non-coherent one and moved above
the wait.  Only memory written before any overlap (rate constants, emissions) may be reached that
way: read from the sources, as the reordering a compiler may choose cannot be provoked."""
import os
import re

import pytest

from reseact.esm_gb300 import abi, mechanism
from reseact.esm_gb300._lib import chem_kernel_source

CSRC = os.path.join(os.path.dirname(__file__), "..", "reseact", "esm_gb300", "csrc")
WAITS = ("griddepcontrol.wait", "await_previous()", "resolve_stage(")
# written before any overlap, or written by the kernel alone (the stage tape's slot)
SETTLED = {"kr", "em", "kzo"}


def _functions(src):
    """(parameters, body) of every device function or kernel of a source."""
    src = re.sub(r"__launch_bounds__\([^)]*\)", "", re.sub(r"//[^\n]*", "", src))
    for m in re.finditer(r"__(?:global|device)__[^;{}()]*\(", src):
        i, depth = m.end(), 1
        while depth and i < len(src):
            depth += {"(": 1, ")": -1}.get(src[i], 0)
            i += 1
        params, rest = src[m.end():i - 1], src[i:i + 8].lstrip()
        if not rest.startswith("{"):
            continue
        j = src.index("{", i)
        k, depth = j + 1, 1
        while depth and k < len(src):
            depth += {"{": 1, "}": -1}.get(src[k], 0)
            k += 1
        yield m.group(0).split()[-1].rstrip("("), params, src[j:k]


def _restricted(text):
    return set(re.findall(r"__restrict__\s+(\w+)", text)) - SETTLED


@pytest.mark.parametrize("name", sorted(f for f in os.listdir(CSRC)
                                        if f.endswith((".cu", ".cuh")) and f not in ("rs_jit.cu", "peak_probe.cu")))
def test_waiting_kernels_take_no_restricted_pointers(name):
    src = open(os.path.join(CSRC, name)).read()
    found = [f for f in _functions(src) if f[0] == "finalize_body" or any(w in f[2] for w in WAITS)]
    assert {"rs_transport.cu": 8, "rs_adv64.cuh": 5, "rs_control.cu": 3}.get(name, 0) <= len(found)
    for fn, params, body in found:
        assert not _restricted(params + body), (fn, _restricted(params + body))


def test_the_generated_attempt_takes_no_restricted_pointers():
    src = chem_kernel_source(abi.MechanismABI(mechanism.superfast()))
    found = 0
    for fn, params, body in _functions(src):
        if any(w in body for w in WAITS):
            found += 1
            assert not _restricted(params + body), (fn, _restricted(params + body))
    assert found == 1
    entry = src[src.index("#define RS_ATTEMPT("):src.index("attempt_body<HE, MODE")]
    assert not _restricted(entry.replace("\\\n", " "))
    # the controller record is read in program order
    assert "*(const int*)(ctl + OFF_DONE)" not in src[src.index("attempt_body("):src.index("per_cell_body(")]
