"""Energy-loss integrals and soft scattering at the numbers of energies where
the CTA's width changes, with node counts around its batches (192, 320)."""
import numpy as np
import pytest
import torch

from noa_gb300 import dcs
from tests.parity import PROCESSES

pytestmark = pytest.mark.gpu


def widths():
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return sms, sms + 1, 2 * sms, 2 * sms + 1


@pytest.mark.parametrize("min_points", [192, 193, 318, 319, 508, 513, 1536])
@pytest.mark.parametrize("process", range(4), ids=PROCESSES)
def test_energies(cuda_device, process, min_points):
    K = torch.from_numpy(10.0 ** np.random.default_rng(6).uniform(-3, 6, 900)).cuda()
    whole = dcs.recoil_integral(process, 1, torch.zeros_like(K), K, min_points=min_points)
    for n in widths():
        got = dcs.recoil_integral(process, 1, torch.zeros_like(K[:n]), K[:n], min_points=min_points)
        # compilations of one sum of positive terms in one order: a few ulp a term
        assert torch.allclose(got, whole[:n], rtol=1e-12, atol=0.0), n


def test_soft_scattering(cuda_device):
    K = torch.from_numpy(10.0 ** np.random.default_rng(7).uniform(-3, 6, 900)).cuda()
    whole = dcs.soft_scattering(torch.zeros_like(K), K)
    for n in widths():
        assert torch.allclose(dcs.soft_scattering(torch.zeros_like(K[:n]), K[:n]), whole[:n], rtol=1e-12, atol=0.0), n
