"""hard_scattering gives an energy 1, 4, 8, 16 or 32 lanes by the number of
elements and energies: every group size against the CPU oracle, at element
counts that fill a group's elements, spill into a second round and exceed the
lanes, and at energy counts that leave a warp's last groups empty."""
import numpy as np
import pytest
import torch

import oracle
from noa_gb300 import dcs
from noa_gb300.elements import BATCH_Z, ELEMENTS, MUON_MASS

pytestmark = pytest.mark.gpu


def inputs(nel, n):
    K = 10.0 ** np.random.default_rng(nel * 1000 + n).uniform(-3, 6, n)
    rows = [oracle.coulomb_data(K, ELEMENTS[BATCH_Z[i % len(BATCH_Z)]], MUON_MASS) for i in range(nel)]
    fCM, screen, fspin, invlambda = (np.ascontiguousarray(np.stack([r[j] for r in rows])) for j in range(4))
    G = np.ascontiguousarray(np.stack([oracle.coulomb_transport(r[1], r[2], 1.0) for r in rows]))
    return G, fCM, screen, invlambda, fspin


# (32, 1): the smallest; 1 element: 4 lanes, then 1 beyond 77824 energies; 2: 8, 4, 1; 3 - 5: 16 (9 - 15 terms);
# 6 - 10: 32; 11 and 35: more elements than a group holds at once
CASES = [(1, 1), (1, 33), (1, 77_825), (2, 1), (2, 31), (2, 40_001), (3, 7), (4, 50), (5, 19_457), (6, 9), (10, 65),
         (10, 9_729), (10, 80_001), (11, 17), (35, 5)]


@pytest.mark.parametrize("nel,n", CASES)
def test_groups(cuda_device, nel, n):
    G, fCM, screen, invlambda, fspin = inputs(nel, n)
    t = [torch.from_numpy(a).cuda() for a in (G, fCM, screen, invlambda, fspin)]
    mu0, lb = (torch.full((n,), -7.0, dtype=torch.float64, device="cuda") for _ in range(2))
    dcs.hard_scattering(mu0, lb, *t)
    exp = oracle.hard_scattering(G, fCM, screen, invlambda, fspin)
    for got, e in ((mu0.cpu().numpy(), exp[0]), (lb.cpu().numpy(), exp[1])):
        # the same IEEE operations but for the last bit of CUDA's log, which the cancelling
        # pole terms can amplify to 1e-8 in a few energies
        rel = np.abs(got - e) / np.where(e != 0, np.abs(e), 1.0)
        assert rel.max() <= 1e-7
        assert np.median(rel) <= 1e-15


def test_groups_agree_bit_for_bit(cuda_device):
    """An energy's result does not depend on how many lanes share it."""
    arrays = inputs(3, 60_000)
    t = [torch.from_numpy(a).cuda() for a in arrays]
    ref = [torch.zeros(60_000, dtype=torch.float64, device="cuda") for _ in range(2)]
    dcs.hard_scattering(*ref, *t)
    for n in (100, 19_000, 38_000):
        part = [torch.from_numpy(np.ascontiguousarray(a[:, :n])).cuda() for a in arrays]
        got = [torch.zeros(n, dtype=torch.float64, device="cuda") for _ in range(2)]
        dcs.hard_scattering(*got, *part)
        for g, r in zip(got, ref):
            assert torch.equal(g.view(torch.int64), r[:n].view(torch.int64))
