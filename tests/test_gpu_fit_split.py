"""A recorded batch of many configurations, whose FP64 k-space passes are split for half of the SMs
(fit.cu, capture_fit), against the sum of single evaluations, split for all of them.  The
regrouped sums differ by rounding only: FP64 to the bars of the three-configuration test
(1e-12, 1e-10); mixed, FP32 sums of at most 1e4 terms, whose rounding grows to about
sqrt(1e4) 6e-8 = 6e-6 of the largest term, to 1e-4 of loss and gradient."""
import numpy as np
import pytest

from mdff20_b200 import fit
from mdff20_b200.engine import MIXED

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,nconf", [(0, 5), (0, 14), (MIXED, 5), (MIXED, 14), (MIXED, 30)])
def test_many_configurations_are_the_sum_of_single_evaluations(precision, nconf):
    systems = fit.config4(sizes=[96, 192, 288][:1 + nconf % 3] * nconf)[:nconf]
    th0 = fit.theta_of(systems[0])
    targets = fit.target_forces(systems, fit.perturbed_theta(th0, seed=9))
    b = fit.ForceMatchBatch(systems, targets, precision=precision)
    loss, grad = b.loss_grad(th0)
    sq, gs = 0.0, np.zeros(fit.NPARAM)
    for e, t in zip(b.engines, targets):
        e.fit_set_params(fit.SI_TYPE, fit.O_TYPE, th0)
        a, g = e.force_match(fit.SI_TYPE, fit.O_TYPE, t, b.scale)
        sq += a
        gs += g
    lt, gt = (1e-12, 1e-10) if precision == 0 else (1e-4, 1e-4)
    assert abs(loss - 0.5 * b.scale * sq) <= lt * loss
    assert np.max(np.abs(grad - gs) / np.maximum(np.abs(gs), 1e-30)) < gt
    b.close()
