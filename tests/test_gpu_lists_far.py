"""Lists of ions whose coordinates lie many boxes away from those of others: the difference of two
fractional coordinates then rounds visibly, and the pair set is that of the reference's FP64
operations, rounding included (the FP32 decision of the list build starts from wrapped coordinates,
which do not show it).  Whole numbers: equality with the oracle's lists of the same coordinates."""
import numpy as np
import pytest

from mdff20_b200 import synth
from mdff20_b200.engine import Engine
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ncell,rc", [(7, 3.0), (7, 4.5)])   # three or more cells per direction, one cell
@pytest.mark.parametrize("power", [0, 20, 40])
def test_far_ions(ncell, rc, power):
    s = synth.lj_fcc(ncell=ncell, rc=rc)
    rng = np.random.default_rng(3)
    s.pos = s.pos + 0.1 * rng.standard_normal(s.pos.shape)
    if power:
        s.pos[::2, 0] += 2.0 ** power * s.cell[0, 0]
    o, e = Oracle(s, wrap=False), Engine(s, positions=s.pos)
    o.gen_verletlist()
    e.gen_verletlist()
    for which in (0, 1):
        a, b = o.verletlist(which), e.verletlist(which)
        assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
    e.close()
