"""Which form the error estimate of the generated attempts takes: float pairs for mechanisms whose LU
leaves them registers, FP64 for larger ones and in the strict build."""
import pytest

from reseact.esm_gb300 import abi, mechanism
from reseact.esm_gb300._lib import chem_kernel_source


@pytest.mark.parametrize("n,r,pairs", [(0, 0, 1), (16, 30, 1), (17, 34, 0), (18, 40, 0), (28, 50, 0)])
def test_estimate_form_follows_the_lu_slots(n, r, pairs):
    m = mechanism.superfast() if n == 0 else mechanism.synthetic(n_species=n, n_reactions=r)
    assert "#define RS_PAIRS %d\n" % pairs in chem_kernel_source(abi.MechanismABI(m))
    if n == 0:
        assert "#define RS_PAIRS 0\n" in chem_kernel_source(abi.MechanismABI(m), strict=True)
