"""Ionisation's recoil integrals where the lowest nodes are closed (recoil
energies below 0.62 I) and the rest of a CTA's first step is open: the step
leaves the work queue just short of a batch, and the next step's nodes are added
to it.  Energies in one width of CTA each: one an SM, two, and more."""
import numpy as np
import pytest
import torch

import oracle
from noa_gb300 import dcs
from noa_gb300.elements import ELEMENTS, MUON_MASS
from tests.parity import assert_fp64_parity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("z,xlow", [(11, 5e-9), (82, 1e-8), (82, 2e-8), (82, 4e-8)])
@pytest.mark.parametrize("min_points", [300, 480, 508, 512, 1536])
def test_low_cut(cuda_device, z, xlow, min_points):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for n in (sms, 2 * sms, 2 * sms + 1, 700):
        K = np.geomspace(11., 100., n)
        tk = torch.from_numpy(K).cuda()
        for moment in (0, 1):
            got = dcs.recoil_integral("ionisation", moment, torch.full_like(tk, -7.0), tk, xlow, ELEMENTS[z], MUON_MASS,
                                      min_points).cpu().numpy()
            exp = oracle.recoil_integral(3, moment, K, xlow, ELEMENTS[z], MUON_MASS, min_points)
            assert_fp64_parity(got, exp, f"n={n} moment={moment}")
