"""Static dipoles on polarisable and non-polarisable types of a system without charges and without
damping: the static field reaches the polarisable ions from both types.  Every induced-dipole
solver against the oracle converged to 1e-11.  Bars: FP64 1e-8 of the largest dipole and force (the
residual measure 1e-11 times the condition of alpha^-1 - T, below 10, with room for the sums);
mixed 2e-5 of the largest dipole (that of the FP32 fields, 1e-6 of the largest field, with the same
condition; the loops stop at 1e-7) and 1e-5 rms of the forces."""
import numpy as np
import pytest

from mdff20_b200 import synth
from mdff20_b200.engine import FP64, MIXED, PIM_CG, PIM_CG_FUSED, PIM_REFERENCE, Engine
from oracle.oracle import Oracle
from tests.helpers import rel_err, rms_rel

pytestmark = pytest.mark.gpu


def _system(algo, tol):
    s = synth.silica(32, seed=4, L=13.0, rc_sr=4.0, rc_lr=5.5, skin=0.5, alpha=0.5, kmax=7, polarizable=True,
                     damping=False, conv_tol=tol, dmin=synth.PIM_DMIN)
    s.qit = [0.0, 0.0]
    s.dipit = np.array([[0.2, -0.1, 0.3], [0.4, 0.3, -0.2]])
    s.algo_pim, s.omegakO = algo, 0.8
    return s


@pytest.mark.parametrize("precision", [FP64, MIXED])
@pytest.mark.parametrize("algo,solver", [("scf", PIM_REFERENCE), ("scfkO", PIM_REFERENCE), ("scf", PIM_CG),
                                         ("scf", PIM_CG_FUSED)])
def test_static_dipoles_of_two_types(algo, solver, precision):
    o = Oracle(_system(algo, 1e-11))
    o.gen_verletlist()
    o.engforce()
    s = _system(algo, 1e-11 if precision == FP64 else 1e-7)
    mu0 = np.repeat(s.dipit, s.nionit, axis=0)
    e = Engine(s, positions=o.state()[0], precision=precision, pim_solver=solver)
    e.gen_verletlist()
    mu = e.get_dipoles()[0]
    e.engforce()
    f, u = e.forces(), e.thermo()["u_coul"]
    e.close()
    assert rel_err(mu - mu0, o.dipoles()) <= (1e-8 if precision == FP64 else 2e-5)
    assert (rel_err if precision == FP64 else rms_rel)(f, o.forces()) <= (1e-8 if precision == FP64 else 1e-5)
    assert abs(u / o.thermo()["u_coul"] - 1.0) <= (1e-8 if precision == FP64 else 1e-5)
