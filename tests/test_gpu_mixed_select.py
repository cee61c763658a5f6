"""Which k-space passes a mixed-precision context of few ions runs: the selection by size and by
environment switches, and that a launch tuning which fails leaves it as it was.  The same passes give the same
bits, so results are compared for equality."""
import numpy as np
import pytest

from mdff20_b200 import synth
from mdff20_b200.engine import FP64, MIXED, PIM_CG, PIM_CG_FUSED, Engine, MdffgpuError
from tests.golden import cases

pytestmark = pytest.mark.gpu


def _forces(monkeypatch, precision, **env):
    with monkeypatch.context() as m:
        for k, v in env.items():
            m.setenv(k, v)
        e = Engine(cases.crist192(True, extrapolate_order=0), precision=precision, pim_solver=PIM_CG)
    e.gen_verletlist()
    e.engforce()
    f = e.forces()
    e.close()
    return f


def test_only_the_k_space_in_fp32(monkeypatch):
    f = _forces(monkeypatch, MIXED, MDFFGPU_MIXED_PARTS="rec")
    g = _forces(monkeypatch, MIXED, MDFFGPU_MIXED_PARTS="rec", MDFFGPU_RHO_TC="0", MDFFGPU_ION_TC="0")
    h = _forces(monkeypatch, FP64)
    assert np.array_equal(f, g) and not np.array_equal(f, h)


@pytest.mark.parametrize("solver", [PIM_CG, PIM_CG_FUSED])
def test_failing_tune_keeps_the_selection(solver):
    s = cases.crist192(True, extrapolate_order=0, conv_tol=1e-14)
    s.max_scf_pim_iter = 1
    e = Engine(s, precision=MIXED, pim_solver=solver)
    e.gen_verletlist()
    q = np.repeat(s.qit, s.nionit)
    mu = np.random.default_rng(1).normal(scale=0.1, size=(e.n, 3))
    flags = dict(lq=1, ld=1, do_forces=1, do_dir=1, do_rec=1)   # (a field and its gradient run in FP64)
    a = e.multipole_es(q, mu, s.alphaES, **flags)
    with pytest.raises(MdffgpuError):
        e.tune_launch(1)
    b = e.multipole_es(q, mu, s.alphaES, **flags)
    for k in ("u", "f"):
        assert np.array_equal(a[k], b[k]), k
    e.close()


# |nz| padded to 16, 32, 48 and 8, 14, 16, 32 in FP64 and FP32: few ions run in FP64 unless that is 1.05e7
# (ion, row, |nz|) more, or 5e7 in all
@pytest.mark.parametrize("n_si,kmax,fp64", [(32, 16, True), (333, 16, True), (432, 16, False), (640, 15, True),
                                            (432, 24, True), (640, 20, False), (32, 32, True), (100, 32, True), (333, 32, False),
                                            (682, 8, True), (683, 8, False)])
def test_default_by_size(n_si, kmax, fp64, monkeypatch):
    s = synth.silica(n_si, seed=3, kmax=kmax, rc_sr=4.0, rc_lr=4.0, skin=0.5, alpha=0.6, dmin=synth.PIM_DMIN)
    flags = dict(lq=1, ld=1, do_forces=1, do_rec=1)
    q, mu = np.repeat(s.qit, s.nionit), np.zeros((s.nion, 3))
    f = []
    for precision, env in ((MIXED, {}), (MIXED, dict(MDFFGPU_RHO_TC="0", MDFFGPU_ION_TC="0")), (FP64, {})):
        with monkeypatch.context() as m:
            for k, v in env.items():
                m.setenv(k, v)
            e = Engine(s, precision=precision)
        e.gen_verletlist()
        f.append(e.multipole_es(q, mu, s.alphaES, **flags)["f"])
        e.close()
    assert np.array_equal(f[0], f[2 if fp64 else 1]) and not np.array_equal(f[1], f[2])
