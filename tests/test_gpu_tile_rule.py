"""The sizes at which the launch shape changes: a call's tile and grid follow
its number of pairs (energies), which must not show in the results."""
import numpy as np
import pytest
import torch

from noa_gb300 import dcs
from noa_gb300.elements import ELEMENTS
from noa_gb300.workload import kinetic_recoil
from tests.parity import PROCESSES

pytestmark = pytest.mark.gpu

# 152 SMs x resident CTAs (5, 7) x tiles of 8 .. 256 pairs, and the smallest calls
SIZES = [1, 2, 7, 8, 9, 127, 129, 6079, 6080, 6081, 8511, 8513, 97_280, 97_281, 194_559, 194_561, 272_383, 272_385,
         389_121, 544_769]


@pytest.mark.parametrize("precision", ["fp64", "fp32c"])
@pytest.mark.parametrize("process", range(4), ids=PROCESSES)
def test_pairs(cuda_device, process, precision):
    K, q = (torch.from_numpy(a).cuda() for a in kinetic_recoil(max(SIZES) + 1000, offset=5 << 20))
    whole = dcs.map(process, K, q, ELEMENTS[26], precision=precision)
    for n in SIZES:
        for start in (0, 999):
            got = torch.full((n + 2,), -7.0, dtype=torch.float64, device="cuda")
            dcs.vmap(process, got[1:n + 1], K[start:start + n], q[start:start + n], ELEMENTS[26], precision=precision)
            # a pair's result depends on the pair only, and nothing else is written
            assert torch.equal(got[1:n + 1].view(torch.int64), whole[start:start + n].view(torch.int64)), n
            assert float(got[0]) == -7.0 and float(got[n + 1]) == -7.0


@pytest.mark.parametrize("min_points", [1, 60, 180, 1536])
@pytest.mark.parametrize("process", range(4), ids=PROCESSES)
def test_energies(cuda_device, process, min_points):
    n_max = 6100 if min_points < 1000 else 310
    K = torch.from_numpy(10.0 ** np.random.default_rng(4).uniform(-3, 6, n_max)).cuda()
    whole = dcs.recoil_integral(process, 0, torch.zeros_like(K), K, min_points=min_points)
    for n in (1, 2, 151, 152, 153, 305, 3041, 6080, 6081):
        if n <= n_max:
            got = dcs.recoil_integral(process, 0, torch.zeros_like(K[:n]), K[:n], min_points=min_points)
            # the wide and the narrow CTA are two compilations of one sum
            assert torch.allclose(got, whole[:n], rtol=1e-12, atol=0.0), n


def test_soft_scattering(cuda_device):
    K = torch.from_numpy(10.0 ** np.random.default_rng(5).uniform(-3, 6, 25_000)).cuda()
    whole = dcs.soft_scattering(torch.zeros_like(K), K)
    for n in (1, 151, 152, 153, 6080, 6081, 24_319, 24_321):
        got = dcs.soft_scattering(torch.zeros_like(K[:n]), K[:n])
        assert torch.allclose(got, whole[:n], rtol=1e-12, atol=0.0), n
