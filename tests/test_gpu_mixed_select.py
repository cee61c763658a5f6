"""Which k-space passes a mixed-precision context of few ions runs: the selection by environment
switches, and that a launch tuning which fails leaves it as it was.  The same passes give the same
bits, so results are compared for equality."""
import numpy as np
import pytest

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
