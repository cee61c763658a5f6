"""FP64 real-space pairs (pair.cu, pairq.cuh): in-cutoff pairs queued 32 at a time.  Fields,
forces, energy and stress of charges, dipoles and both against the oracle with rows of 0 to
about 300 listed ions, most of them outside the cut-off in some cases, and the dipoles of the
cached-factor iterations with and without ions that are not polarisable.  Bar: the 1e-11 of the
FP64 parity tests (rows of at most 300 terms; the factors' roundings are a few 1e-16)."""
import numpy as np
import pytest

from mdff20_b200 import synth
from mdff20_b200.engine import PIM_CG, Engine
from oracle.oracle import Oracle, wrapped_positions
from tests.golden import cases
from tests.helpers import rel_err

pytestmark = pytest.mark.gpu

BOTH = dict(lq=1, ld=1, ldamp=0, do_forces=1, do_stress=1, do_ef=0, do_efg=0, do_dir=1, do_rec=0)
FIELD = dict(BOTH, do_forces=0, do_stress=0, do_ef=1)
CHARGES = dict(BOTH, ld=0)
ALL = dict(BOTH, do_ef=1, do_efg=1)


@pytest.mark.parametrize("n_si,rc,skin", [(1, 1.0, 0.3), (3, 3.0, 0.0), (11, 4.0, 1.9), (33, 3.2, 2.6),
                                          (64, 6.5, 0.4), (96, 7.0, 1.0)])
@pytest.mark.parametrize("damp", [0, 1])
def test_pairs_vs_oracle(n_si, rc, skin, damp):
    s = synth.silica(n_si, seed=5, L=max(12.0, 2.6 * (3 * n_si) ** (1.0 / 3.0)), rc_sr=min(rc, 4.0), rc_lr=rc, skin=skin,
                     alpha=0.4, kmax=3, polarizable=True)
    s.pos = wrapped_positions(s)
    o, e = Oracle(s), Engine(s)
    o.gen_verletlist()
    e.gen_verletlist()
    q, mu = cases.es_inputs(s, 4)
    for base in (BOTH, FIELD, CHARGES, ALL):
        flags = dict(base, ldamp=damp)
        want, got = o.multipole_es(q, mu, **flags), e.multipole_es(q, mu, **flags)
        assert abs(got["u"] - want["u"]) <= 1e-11 * max(1.0, abs(want["u"])), flags
        if flags["do_ef"]:
            assert rel_err(got["ef"], want["ef"]) < 1e-11, flags
        if flags["do_forces"]:
            assert rel_err(got["f"], want["f"]) < 1e-11, flags
            assert np.abs(got["tau"] - want["tau"]).max() <= 1e-11 * max(1.0, np.abs(want["tau"]).max()), flags
    e.close()


@pytest.mark.parametrize("n_si,rc,skin", [(3, 3.0, 0.0), (33, 3.2, 2.6), (96, 7.0, 1.0)])
def test_cached_dipole_field_solves_the_dipoles(n_si, rc, skin):
    # the iterations run on the cached factors of the polarisable pairs; the residual
    # mu / alpha - E of their result, with E from the uncached pass (alpha_O = 1), is the one
    # they stopped at: rms over the polarisable ions below the tolerance
    tol = 1e-9
    s = synth.silica(n_si, seed=6, L=max(12.0, 2.6 * (3 * n_si) ** (1.0 / 3.0)), rc_sr=min(rc, 4.0), rc_lr=rc,
                     skin=skin, alpha=0.4, kmax=3, polarizable=True, conv_tol=tol)
    s.pos = wrapped_positions(s)
    e = Engine(s, pim_solver=PIM_CG)
    e.gen_verletlist()
    mu, _ = e.get_dipoles()
    on = np.abs(mu).max(axis=1) > 0.0
    assert on.sum() == 2 * n_si
    q = np.repeat(np.array([-1.2, 2.4]), s.nionit)
    ef = e.multipole_es(q, mu, **dict(FIELD, ldamp=1, do_rec=1))["ef"]
    assert np.sqrt(((mu - ef)[on] ** 2).sum() / on.sum()) <= 1.05 * tol
    e.close()
