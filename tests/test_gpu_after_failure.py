"""A force evaluation whose dipole solve fails leaves side branches open (the short-range pairs add
into the force array): what follows on the context waits for them.  Forces read right after the failure
are the short-range ones, the same bits as from a call of their own; one more call adds them once more."""
import numpy as np
import pytest

from mdff20_b200.engine import FP64, MIXED, PIM_CG, PIM_CG_FUSED, Engine, MdffgpuError
from tests.golden import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [FP64, MIXED])
@pytest.mark.parametrize("solver", [PIM_CG, PIM_CG_FUSED])
def test_failing_solve(precision, solver):
    s = cases.crist192(True, extrapolate_order=0, conv_tol=1e-14)
    s.max_scf_pim_iter = 1
    e = Engine(s, precision=precision, pim_solver=solver)
    sr = Engine(s, precision=precision, pim_solver=solver)
    for x in (e, sr):
        x.gen_verletlist()
    sr.engforce_bhmftd()
    for _ in range(20):
        with pytest.raises(MdffgpuError):
            e.engforce()
        assert np.array_equal(e.forces(), sr.forces())
    e.engforce_bhmftd()
    assert np.array_equal(e.forces(), 2.0 * sr.forces())
    e.close()
    sr.close()
