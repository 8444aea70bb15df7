"""Transverse transport coefficients with a lane a pole (few energies) and with
one thread an energy (many): the same IEEE operations in the same order, so the
same bits, for one cut-off and for one an energy, the smallest (the asymptotic
form) among them."""
import numpy as np
import pytest
import torch

from noa_gb300 import dcs
from noa_gb300.elements import ELEMENTS, MUON_MASS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("z", [1, 82])
def test_same_bits(cuda_device, z):
    limit = 64 * torch.cuda.get_device_properties(0).multi_processor_count
    n = limit + 5000
    g = np.random.default_rng(9)
    K = torch.from_numpy(10.0 ** g.uniform(-3, 6, n)).cuda()
    mu = torch.from_numpy(10.0 ** g.uniform(-30, 0, n)).cuda()
    fCM, screen, fspin, inv = (torch.zeros((n, *s), dtype=torch.float64, device="cuda") for s in ((2,), (9,), (), ()))
    dcs.coulomb_data(fCM, screen, fspin, inv, K, ELEMENTS[z], MUON_MASS)
    for cut in (mu, mu[:1]):
        whole = torch.zeros((n, 2), dtype=torch.float64, device="cuda")
        dcs.coulomb_transport(whole, screen, fspin, cut)
        for m in (1, 7, 9, 1001, limit, limit + 1):
            got = torch.full((m + 8, 2), -7.0, dtype=torch.float64, device="cuda")
            dcs.coulomb_transport(got[:m], screen[:m], fspin[:m], cut[:m])
            assert torch.equal(got[:m].view(torch.int64), whole[:m].view(torch.int64)), m
            assert bool((got[m:] == -7.0).all())
