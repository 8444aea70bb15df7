"""Photonuclear at energies whose product with the cross-section's scale would
overflow although the cross-section does not: finite where the oracle is."""
import numpy as np
import pytest
import torch

import oracle
from noa_gb300 import dcs
from noa_gb300.elements import ELEMENTS, MUON_MASS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,bound", [("fp64", 1e-8), ("fp32c", 1e-6)])
@pytest.mark.parametrize("lo,hi", [(200, 250), (250, 299)])
def test_photonuclear(cuda_device, precision, bound, lo, hi):
    g = np.random.default_rng(21)
    K = 10.0 ** g.uniform(lo, hi, 3000)
    q = K * 10.0 ** g.uniform(-2.5, -0.01, K.size)
    exp = oracle.dcs(2, K, q, ELEMENTS[1], MUON_MASS)
    got = dcs.map(2, torch.from_numpy(K).cuda(), torch.from_numpy(q).cuda(), ELEMENTS[1], MUON_MASS,
                  precision).cpu().numpy()
    assert np.isfinite(exp).all() and (exp > 0).sum() > 1000
    assert np.array_equal(got == 0, exp == 0) and (np.abs(got - exp) <= bound * exp).all()
