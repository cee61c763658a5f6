"""List build and CSR half lists where their parts can go wrong: more ions than one bitmap
window of the CSR fill (65536), a triclinic cell scanned as one cell with the list radius
next to half the cell width, ions on box faces and pairs at exactly the list radius, and a
caller buffer that is too short.  Lists are whole numbers: equality."""
import ctypes as C

import numpy as np
import pytest

from mdff20_b200 import synth
from mdff20_b200.engine import Engine, MdffgpuError
from oracle.oracle import Oracle, wrapped_positions
from tests.golden import cases

pytestmark = pytest.mark.gpu


def _half_csr(n, i, j):
    """Unique unordered pairs as CSR rows under the parity rule (src/verlet.c:82-83)."""
    a = np.concatenate([i, j]).astype(np.int64)
    b = np.concatenate([j, i]).astype(np.int64)
    keep = ((a > b) & ((a + b) % 2 == 0)) | ((a < b) & ((a + b) % 2 != 0))
    a, b = a[keep], b[keep]
    order = np.lexsort((b, a))
    return np.concatenate([[0], np.cumsum(np.bincount(a, minlength=n))]), b[order]


def test_csr_past_one_window():
    from scipy.spatial import cKDTree
    s = synth.lj_fcc(ncell=26, seed=5)
    rng = np.random.default_rng(1)
    L = s.cell[0, 0]
    s.pos = np.mod(s.pos + 0.05 * rng.standard_normal(s.pos.shape), L)
    assert s.nion > 65536
    e = Engine(s)
    e.gen_verletlist()
    pairs = cKDTree(s.pos, boxsize=L).query_pairs(s.cutshortrange + s.skindiff, output_type="ndarray")
    point, lst = _half_csr(s.nion, pairs[:, 0], pairs[:, 1])
    got = e.verletlist(0)
    assert np.array_equal(got[0], point) and np.array_equal(got[1], lst)


def _triclinic():
    s = cases.silica96(False)
    frac = s.pos @ np.linalg.inv(s.cell)
    s.cell = s.cell.copy()
    s.cell[1, 0], s.cell[2, 0], s.cell[2, 1] = 1.3, -0.7, 0.9
    s.pos = frac @ s.cell
    s.cutlongrange = 0.499 * float(s.cell[0, 0]) - 1.2
    return s


def _lattice():
    # spacing exactly 1, list radii exactly 3 and 4 (pairs on the sphere), ions on the faces
    s = synth.lj_fcc(ncell=3, rho=0.5)
    g = np.stack(np.meshgrid(*[np.arange(12.0)] * 3, indexing="ij"), -1).reshape(-1, 3) - 6.0
    s.cell, s.pos, s.vel, s.nionit = np.eye(3) * 12.0, g, None, [len(g)]
    s.cutshortrange, s.cutlongrange, s.skindiff = 2.5, 3.5, 0.5
    return s


@pytest.mark.parametrize("make", [_triclinic, _lattice])
def test_lists_vs_oracle(make):
    s = make()
    s.pos = wrapped_positions(s)
    o, e = Oracle(s), Engine(s)
    o.gen_verletlist()
    e.gen_verletlist()
    for which in (0, 1):
        a, b = o.verletlist(which), e.verletlist(which)
        assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1]), which


def test_short_buffer_is_refused_and_filled():
    s = cases.silica96(False)
    e = Engine(s)
    e.gen_verletlist()
    point, lst = e.verletlist(1)
    ip = lambda a: a.ctypes.data_as(C.POINTER(C.c_int))  # noqa: E731
    buf, pt, cnt = np.full(len(lst), -1, np.int32), np.zeros(s.nion + 1, np.int32), C.c_int(0)
    cap = len(lst) - 7
    with pytest.raises(MdffgpuError):
        e._check(e.L.mdffgpu_get_verletlist(e.h, 1, ip(pt), ip(buf), cap, C.byref(cnt)))
    assert cnt.value == len(lst) and np.array_equal(pt, point)
    assert np.array_equal(buf[:cap], lst[:cap]) and (buf[cap:] == -1).all()
