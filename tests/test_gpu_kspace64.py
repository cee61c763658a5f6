"""FP64 k-space passes (kspace64.cu) against the oracle: every k-step instantiation, |nz|
groups past 15, degenerate k boxes, ion counts around the tiles of 8, 16 and 32 and a
triclinic cell.  Bar: the 1e-11 of the FP64 parity tests (the sums hold at most 2e6 terms,
whose rounding is below 1e-13 of the largest)."""
import numpy as np
import pytest

from mdff20_b200 import synth
from mdff20_b200.engine import Engine
from oracle.oracle import Oracle, wrapped_positions
from tests.golden import cases
from tests.helpers import rel_err

pytestmark = pytest.mark.gpu

FULL = dict(lq=1, ld=1, ldamp=0, do_forces=1, do_stress=1, do_ef=1, do_efg=1, do_dir=0, do_rec=1)
CHARGES = dict(FULL, ld=0)
DIPOLES = dict(FULL, lq=0, do_forces=0, do_stress=0)


def _system(n_si, kes, triclinic):
    s = synth.silica(n_si, seed=21, L=max(12.0, 2.5 * n_si ** (1.0 / 3.0) * 2.0), rc_sr=4.0, rc_lr=5.0, skin=0.5,
                     alpha=0.5, kmax=4, polarizable=False)
    if triclinic:
        frac = s.pos @ np.linalg.inv(s.cell)
        s.cell = s.cell.copy()
        s.cell[1, 0], s.cell[2, 1] = 1.1, -0.8
        s.pos = frac @ s.cell
    s.kES = kes
    return s


@pytest.mark.parametrize("n_si,kes,triclinic", [
    (1, (2, 3, 1), False), (2, (0, 0, 3), False), (3, (3, 0, 0), False), (5, (0, 2, 0), False),
    (11, (3, 2, 6), True), (11, (4, 3, 9), False), (21, (3, 4, 11), True), (33, (5, 5, 13), False),
    (43, (4, 4, 14), True), (43, (3, 3, 15), False), (22, (3, 2, 16), True), (10, (2, 3, 32), False),
    (130, (9, 9, 9), False),
])
def test_passes_vs_oracle(n_si, kes, triclinic):
    s = _system(n_si, kes, triclinic)
    s.pos = wrapped_positions(s)
    o, e = Oracle(s), Engine(s)
    o.gen_verletlist()
    e.gen_verletlist()
    q, mu = cases.es_inputs(s, 4)
    for flags in (FULL, CHARGES, DIPOLES):
        want = o.multipole_es(q, mu, **flags)
        got = e.multipole_es(q, mu, **flags)
        assert abs(got["u"] - want["u"]) <= 1e-11 * max(1.0, abs(want["u"])), flags
        assert rel_err(got["ef"], want["ef"]) < 1e-11, flags
        assert rel_err(got["efg"].reshape(-1, 9), want["efg"].reshape(-1, 9)) < 1e-11, flags
        assert np.abs(got["tau"] - want["tau"]).max() <= 1e-11 * max(1.0, np.abs(want["tau"]).max()), flags
        if flags["do_forces"]:
            assert rel_err(got["f"], want["f"]) < 1e-11, flags
