"""A call of mdffgpu_md_steps_host that fails before its last step leaves the caller's output
arrays as they were, also where they are the arrays of its input: the steps run in batches of 16,
and the state of a batch that is undone is not handed out.  Values are compared for equality."""
import ctypes as C

import numpy as np
import pytest

from mdff20_b200 import synth
from mdff20_b200.engine import Engine

pytestmark = pytest.mark.gpu


def _engine():
    e = Engine(synth.lj_fcc(ncell=4, dt=0.12))   # leaves the finite numbers after some steps
    e.gen_verletlist()
    e.engforce()
    return e


def _ptrs(arrs):
    return (C.POINTER(C.c_double) * len(arrs))(*[a.ctypes.data_as(C.POINTER(C.c_double)) for a in arrs])


@pytest.mark.parametrize("same", [False, True])
def test_failing_call_leaves_the_outputs(same):
    e = _engine()
    th = np.full((64, 12), -1.0)
    e.L.mdffgpu_md_steps(e.h, 1, 64, th.ctypes.data_as(C.POINTER(C.c_double)))
    done = int((th[:, 0] != -1.0).sum())
    e.close()
    nsteps = done // 16 * 16 + 16   # the failing step lies in the last batch, not at its end
    assert 1 < done < nsteps - 1
    e = _engine()
    inp = [np.empty(e.n) for _ in range(9)]
    e.state_soa(*inp)
    del inp[6:]
    out = inp + [np.full(e.n, -7.0) for _ in range(3)] if same else [np.full(e.n, -7.0) for _ in range(9)]
    before = [a.copy() for a in out]
    rec = np.full((nsteps, 12), -1.0)
    rc = e.L.mdffgpu_md_steps_host(e.h, 1, nsteps, _ptrs(inp), rec.ctypes.data_as(C.POINTER(C.c_double)),
                                   _ptrs(out))
    assert rc == 5 and np.array_equal(rec[:done], th[:done]) and (rec[done:] == -1.0).all()
    for a, b in zip(out, before):
        assert np.array_equal(a, b)
    e.close()


@pytest.mark.parametrize("nsteps", [1, 15, 16, 17, 33])
def test_outputs_are_the_state(nsteps):
    s = synth.lj_fcc(ncell=4)
    e = Engine(s)
    e.gen_verletlist()
    e.engforce()
    out = [np.empty(e.n) for _ in range(9)]
    e.md_steps_host(1, nsteps, None, out)
    for k, x in enumerate(e.state()):
        assert np.array_equal(np.stack(out[3 * k:3 * k + 3], 1), x)
    e.close()
