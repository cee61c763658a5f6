"""Contexts and histograms are created and destroyed in one thread while another records MD steps:
neither call may wait for, or fail on, a stream that is being recorded.  The recorded steps give the
same bits as without company."""
import threading

import numpy as np
import pytest

from mdff20_b200 import synth
from mdff20_b200.engine import Engine
from mdff20_b200.rdf import RDF

pytestmark = pytest.mark.gpu


def _system():
    return synth.lj_fcc(4, seed=5)


def _run(e, reps):
    out = []
    for k in range(reps):
        e.set_graph(False)   # drops the recording
        e.set_graph(True)
        e.md_steps(2 * k, 2)
        out.append(e.state()[0].copy())
    return np.array(out)


@pytest.mark.parametrize("what", ["rdf", "engine"])
def test_create_while_recording(what):
    s = _system()
    ref, e = Engine(s), Engine(s)
    want = _run(ref, 200)
    stop, errors = threading.Event(), []

    def create():
        try:
            while not stop.is_set():
                if what == "rdf":
                    RDF([s.nion], 3.0).close()
                else:
                    Engine(s).close()
        except BaseException as x:
            errors.append(x)

    t = threading.Thread(target=create)
    t.start()
    try:
        got = _run(e, 200)
    finally:
        stop.set()
        t.join()
    if errors:
        raise errors[0]
    np.testing.assert_array_equal(got, want)
    ref.close()
    e.close()
