"""multipole_es calls of different flags one after another on one context (its arrays are kept between
calls) against the same calls on fresh contexts: the same bits."""
import numpy as np
import pytest

from mdff20_b200.engine import Engine
from tests.golden import cases

pytestmark = pytest.mark.gpu


def test_calls_in_a_row():
    s = cases.silica96(True)
    rng = np.random.default_rng(2)
    args = [(rng.normal(size=s.nion), rng.normal(size=(s.nion, 3))) for _ in range(2)]
    e = Engine(s)
    e.gen_verletlist()
    for k, flags in enumerate(cases.ES_FLAG_SETS + cases.ES_FLAG_SETS[::-1]):
        fl = dict(zip(cases.ES_FLAG_NAMES, flags))
        q, mu = args[k % 2]
        new = Engine(s)
        new.gen_verletlist()
        a, b = e.multipole_es(q, mu, s.alphaES, **fl), new.multipole_es(q, mu, s.alphaES, **fl)
        new.close()
        for key in a:
            assert np.array_equal(a[key], b[key]), (fl, key)
    e.close()
