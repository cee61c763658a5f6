"""The FP32 k-space passes on CUDA cores: chosen by the switches for few ions, the default from 2048
to 4095 ions.  Errors against the reference's FP64 results at the bars of the mixed path (1e-5), and
recorded MD steps against kernel-by-kernel ones, with side streams and programmatic launch on
and off: no arithmetic moves between kernels, so the same bits."""
import numpy as np
import pytest

from mdff20_b200 import synth
from mdff20_b200.cellmath import wrap_positions
from mdff20_b200.engine import FP64, MIXED, PIM_CG, PIM_CG_FUSED, Engine
from tests.golden import cases
from tests.helpers import load_golden, rms_rel, tensor_rel

pytestmark = pytest.mark.gpu

FP32 = dict(MDFFGPU_RHO_TC="0", MDFFGPU_ION_TC="0")


def _engine(monkeypatch, s, env, **kw):
    with monkeypatch.context() as m:
        for k, v in env.items():
            m.setenv(k, v)
        e = Engine(s, positions=wrap_positions(s.cell, s.pos), **kw)
    e.gen_verletlist()
    e.engforce()
    return e


@pytest.mark.parametrize("name", ["silica450_pim", "silica96_rigid", "silica96_pim"])
def test_errors_small(name, monkeypatch):
    g, s = load_golden(name), cases.CASES[name]()
    s.pos = g["r_in"].reshape(-1, 3)
    e = _engine(monkeypatch, s, FP32, precision=MIXED)
    assert rms_rel(e.forces(), g["f"].reshape(-1, 3)) < 1e-5
    th = e.thermo()
    for k in ("u_coul", "u_pol", "pvir_coul"):
        assert abs(th[k] - float(g[k][0])) <= 1e-5 * max(abs(float(g[k][0])), 1e-12), k
    assert tensor_rel(th["tau_coul"], g["tau_coul"]) < 1e-5
    e.close()


def _small():
    return cases.crist192(True, extrapolate_order=2), FP32


def _default():
    s = synth.config5(cells=5)   # 3000 ions
    s.extrapolate_order = 2
    return s, {}


@pytest.mark.parametrize("system", [_small, _default])
@pytest.mark.parametrize("solver", [PIM_CG, PIM_CG_FUSED])
def test_recorded_steps_bit_identical(system, solver, monkeypatch):
    s, env = system()
    got = []
    for graph, more in ((True, {}), (False, {}), (True, dict(MDFFGPU_SIDE_STREAMS="0")),
                        (True, dict(MDFFGPU_PDL="0")), (False, dict(MDFFGPU_SIDE_STREAMS="0", MDFFGPU_PDL="0"))):
        e = _engine(monkeypatch, s, {**env, **more}, precision=MIXED, pim_solver=solver)
        e.set_graph(graph)
        got.append((e.md_steps(1, 8), *e.state()))
        e.close()
    for g in got[1:]:
        for x, y in zip(got[0], g):
            assert np.array_equal(x, y)
    ref = _engine(monkeypatch, s, {}, precision=FP64, pim_solver=solver)
    assert not np.array_equal(ref.md_steps(1, 8)[:, 3], got[0][0][:, 3])   # the passes are not the FP64 ones
    ref.close()


@pytest.mark.parametrize("system", [_small, _default])
def test_restart_continues_exactly(system, monkeypatch):
    s, env = system()
    a = _engine(monkeypatch, s, env, precision=MIXED, pim_solver=PIM_CG_FUSED)
    a.md_steps(1, 6)
    blob = a.save_state()
    b = _engine(monkeypatch, s, env, precision=MIXED, pim_solver=PIM_CG_FUSED)
    assert b.load_state(blob) == 6
    ta, tb = a.md_steps(7, 6), b.md_steps(7, 6)
    assert np.array_equal(ta, tb)
    for x, y in zip(a.state(), b.state()):
        assert np.array_equal(x, y)
    a.close()
    b.close()
