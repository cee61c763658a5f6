"""Several fit plans over the same contexts: each holds its own recorded evaluations, theta, targets
and results, so plans with other configurations, scales and targets give, in any order and after one
of them is gone, what the host-driven batch gives for theirs.  Bars: the dipoles start from those of the
evaluation before and stop at a residual of 1e-11, times the condition of alpha^-1 - T (below 10)
1e-10 in the dipoles, which is at most 1e-8 of a force difference of 5 % and of the loss; the
gradient's adjoint solve stops at a relative residual no larger, 1e-7 with the cancellation in its
sums."""
import ctypes as C

import numpy as np
import pytest

from mdff20_b200 import fit
from mdff20_b200.engine import PIM_CG, Engine, FitPlan
from mdff20_b200.cellmath import wrap_positions

pytestmark = pytest.mark.gpu


def _batch(engines, targets, scale, theta):
    n = len(engines)
    ctx = (C.c_void_p * n)(*[e.h.value for e in engines])
    dp = C.POINTER(C.c_double)
    tg = [np.ascontiguousarray(t) for t in targets]
    res = np.zeros(1 + fit.NPARAM)
    rc = engines[0].L.mdffgpu_fit_batch(ctx, n, fit.SI_TYPE, fit.O_TYPE, theta.ctypes.data_as(dp),
                                        (dp * n)(*[t.ctypes.data_as(dp) for t in tg]), C.c_double(scale), 1,
                                        res.ctypes.data_as(dp))
    assert rc == 0
    return res[0], res[1:]


def _close(a, b):
    assert abs(a[0] - b[0]) <= 1e-8 * abs(b[0])
    assert np.max(np.abs(a[1] - b[1]) / np.maximum(np.abs(b[1]), 1e-30)) < 1e-7


def test_plans_in_turn():
    systems = fit.config4(sizes=[96, 192, 96] + [96] * 10, conv_tol=1e-11)
    th0 = fit.theta_of(systems[0])
    th1 = fit.perturbed_theta(th0, seed=2, frac=0.01)
    ta = fit.target_forces(systems, fit.perturbed_theta(th0, seed=9))
    tb = fit.target_forces(systems, fit.perturbed_theta(th0, seed=10, frac=0.02))
    es = [Engine(s, positions=wrap_positions(s.cell, s.pos), pim_solver=PIM_CG) for s in systems]
    for e in es:
        e.gen_verletlist()
    sets = [(slice(0, 13), ta, 0.01), (slice(1, 3), tb, 0.5), (slice(0, 2), ta, 2.0)]
    ref = [[_batch(es[k], t[k], w, th) for th in (th0, th1)] for k, t, w in sets]
    plans = [FitPlan(es[k], fit.SI_TYPE, fit.O_TYPE, t[k], w) for k, t, w in sets]
    for th, which in ((th0, 0), (th1, 1), (th0, 0)):
        for p, r in zip(plans, ref):
            _close(p.eval(th), r[which])
    _close(plans[1].eval(th1), ref[1][1])
    # a single evaluation with other targets leaves the plans'
    es[1].force_match(fit.SI_TYPE, fit.O_TYPE, ta[1], 1.0)
    _close(plans[1].eval(th1), ref[1][1])
    plans[0].close()
    _close(plans[2].eval(th0), ref[2][0])
    new = FitPlan(es[0:2], fit.SI_TYPE, fit.O_TYPE, tb[0:2], 0.25)
    _close(new.eval(th1), _batch(es[0:2], tb[0:2], 0.25, th1))
    _close(plans[1].eval(th0), ref[1][0])
    for p in plans[1:] + [new]:
        p.close()
    for e in es:
        e.close()
