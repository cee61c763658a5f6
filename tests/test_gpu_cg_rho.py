"""The rho(k) that the fused CG carries along its iterates, shared out over clusters of one to eight
blocks by the number of k vectors (cg.cu): forces, energy and dipoles of the fused CG against those of
the plain CG, which sums rho(k) anew.  Both stop at a residual of 1e-11; times the condition of
alpha^-1 - T (below 10) the bar is 1e-8 of the largest value."""
import pytest

from mdff20_b200 import synth
from mdff20_b200.engine import PIM_CG, PIM_CG_FUSED, Engine
from tests.helpers import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_si", [32, 129, 260])        # one block of dipoles, just one, two
@pytest.mark.parametrize("kmax", [7, 8, 10, 13, 21])    # nk 1687, 2456, 4630, 9854, 39773
def test_fused_against_plain(n_si, kmax):
    L = max(13.0, synth.box_length(n_si, 2 * n_si, 2.2))
    s = synth.silica(n_si, seed=8, L=L, rc_sr=4.0, rc_lr=5.5, skin=0.5, alpha=0.5, kmax=kmax, polarizable=True,
                     conv_tol=1e-11, dmin=synth.PIM_DMIN)
    got = []
    for solver in (PIM_CG, PIM_CG_FUSED):
        e = Engine(s, pim_solver=solver)
        e.gen_verletlist()
        e.engforce()
        got.append((e.forces(), e.thermo()["u_coul"], e.dipole_history()[:, 0]))
        e.close()
    for a, b in zip(got[1], got[0]):
        assert rel_err(a, b) <= 1e-8
