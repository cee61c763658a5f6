"""The FP32 ion pass leaves the slices of A p to the cluster's update (cg.cu, comb_ap): dipoles of
mixed precision, with the CUDA-core and the tensor-core ion pass at counts of polarisable ions
around a block of 512, against FP64 ones.  Bar 2e-5 of the largest dipole: the FP32 fields hold
1e-6 of the largest field (the bar of the mixed force tests), times the condition of alpha^-1 - T
of these systems, below 10."""
import numpy as np
import pytest

from mdff20_b200 import synth
from mdff20_b200.engine import MIXED, PIM_CG, PIM_CG_FUSED, Engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_si", [33, 256, 257])
@pytest.mark.parametrize("solver", [PIM_CG, PIM_CG_FUSED])
@pytest.mark.parametrize("tc", ["0", "1"])
def test_mixed_dipoles_vs_fp64(n_si, solver, tc, monkeypatch):
    monkeypatch.setenv("MDFFGPU_RHO_TC", "0")
    monkeypatch.setenv("MDFFGPU_ION_TC", tc)
    L = max(13.0, 2.6 * (3 * n_si) ** (1.0 / 3.0))
    s = synth.silica(n_si, seed=8, L=L, rc_sr=4.0, rc_lr=5.5, skin=0.5, alpha=0.5, kmax=7, polarizable=True,
                     conv_tol=1e-8)
    mu = []
    for precision in (0, MIXED):
        e = Engine(s, precision=precision, pim_solver=solver)
        e.gen_verletlist()
        mu.append(e.get_dipoles()[0])
        e.close()
    assert np.abs(mu[1] - mu[0]).max() <= 2e-5 * np.abs(mu[0]).max()
