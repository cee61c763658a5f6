"""Lists of ions that all share one cell (triclinic boxes, boxes below three list radii): one and two
ions per warp (from 3000 ions), counts that leave a warp half used, pairs at exactly the list radius.
Whole numbers: equality with the oracle's lists."""
import numpy as np
import pytest

from mdff20_b200 import synth
from mdff20_b200.engine import Engine
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


def _check(s):
    o, e = Oracle(s, wrap=False), Engine(s, positions=s.pos)
    o.gen_verletlist()
    e.gen_verletlist()
    for which in (0, 1):
        a, b = o.verletlist(which), e.verletlist(which)
        assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
    e.close()


@pytest.mark.parametrize("tri", [False, True])
@pytest.mark.parametrize("n", [1, 2, 33, 2999, 3000, 3001, 4097])
def test_sizes(n, tri):
    s = synth.lj_fcc(ncell=3)
    L = max(6.0, (n / 0.4) ** (1.0 / 3.0))
    A = np.eye(3) * L
    if tri:
        A[1, 0], A[2, 0], A[2, 1] = 0.1 * L, -0.07 * L, 0.08 * L
    s.cell, s.vel, s.nionit = A, None, [n]
    s.pos = (np.random.default_rng(n).random((n, 3)) * 3.0 - 1.0) @ A
    s.cutshortrange, s.cutlongrange, s.skindiff = 2.0, (2.5 if tri else 0.35 * L), 0.3
    _check(s)


def test_pairs_on_the_sphere():
    g = np.stack(np.meshgrid(*[np.arange(15.0)] * 3, indexing="ij"), -1).reshape(-1, 3) - 7.0
    s = synth.lj_fcc(ncell=3)
    s.cell, s.pos, s.vel, s.nionit = np.eye(3) * 15.0, g, None, [len(g)]
    s.cutshortrange, s.cutlongrange, s.skindiff = 2.5, 5.5, 0.5   # radii exactly 3 and 6, 3375 ions
    _check(s)
