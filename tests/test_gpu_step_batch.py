"""Batches of recorded MD steps against the same steps one call at a time, where a batch
has to be undone: a list that outgrows its capacity in the middle of a run, and a run whose
positions cease to be finite (the error comes at the same step, with the records and the state
of single steps).  Also call lengths around the batch size.  The trajectories are the same
bits either way."""
import ctypes as C

import numpy as np
import pytest

from mdff20_b200 import synth
from mdff20_b200.engine import PIM_CG, Engine
from tests.golden import cases

pytestmark = pytest.mark.gpu


def _run(s, nsteps, graph, calls=None, **kw):
    e = Engine(s, **kw)
    e.set_graph(graph)
    e.gen_verletlist()
    e.engforce()
    th = np.full((nsteps, 12), -1.0)
    rc, first = 0, 1
    for k in calls or [nsteps]:
        rc = e.L.mdffgpu_md_steps(e.h, first, k, th[first - 1:].ctypes.data_as(C.POINTER(C.c_double)))
        first += k
        if rc:
            break
    st = e.state()
    builds = e.thermo()["nlist_builds"]
    e.close()
    return rc, th, st, builds


def _same(a, b):
    assert a[0] == b[0] and a[3] == b[3]
    np.testing.assert_array_equal(a[1], b[1])
    for x, y in zip(a[2], b[2]):
        np.testing.assert_array_equal(x, y)


def _collapse():
    """1728 atoms in a corner of a large box, moving inwards: the first list's capacity follows
    from that packing and is outgrown on the way."""
    s = synth.lj_fcc(ncell=3, rc=3.5, skin=0.3, dt=0.005)
    g = np.stack(np.meshgrid(*[np.arange(12.0)] * 3, indexing="ij"), -1).reshape(-1, 3)
    rng = np.random.default_rng(2)
    s.pos = (g - 5.5) * 1.3 + 0.01 * rng.standard_normal(g.shape)
    s.vel = -0.6 * s.pos
    s.cell, s.nionit = np.eye(3) * 40.0, [len(g)]
    return s


def test_list_outgrown_in_a_batch():
    from scipy.spatial import cKDTree
    s = _collapse()
    cut = s.cutshortrange + s.skindiff
    most = lambda p: max(len(x) for x in cKDTree(p).query_ball_point(p, cut))  # noqa: E731
    a = _run(s, 90, True)
    assert a[0] == 0 and most(a[2][0]) > most(s.pos) * 5 / 4 + 64   # past the capacity grown at the first build
    _same(a, _run(s, 90, True, [1] * 90))
    # kernel by kernel the build count of the outgrown step's record already holds the second build
    b = _run(s, 90, False)
    np.testing.assert_array_equal(a[1][:, :9], b[1][:, :9])
    np.testing.assert_array_equal(a[2][0], b[2][0])


def test_not_finite_in_a_batch():
    s = synth.lj_fcc(ncell=4, dt=0.12)
    a, b = _run(s, 64, True), _run(s, 64, True, [1] * 64)
    done = int((a[1][:, 0] != -1.0).sum())
    assert a[0] == 5 and 1 < done < 63 and (done + 1) % 16 != 1
    _same(a, b)


@pytest.mark.parametrize("pim", [False, True])
def test_call_lengths(pim):
    s = cases.crist192(True, extrapolate_order=2, conv_tol=1e-8) if pim else synth.lj_fcc(ncell=4, skin=0.02)
    kw = dict(pim_solver=PIM_CG) if pim else {}
    n = 40
    a = _run(s, n, True, **kw)
    for calls in ([1, 2, 15, 16, 6], [17, 23], [33, 7]):
        _same(a, _run(s, n, True, calls, **kw))
    _same(a, _run(s, n, False, **kw))
