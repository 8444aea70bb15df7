"""FP32C bremsstrahlung and ionisation at the edges of the map kernel's tiles,
and pair production where its float intermediates leave the float range (the
FP64 redo answers there): the form's bound, 1e-6, against the FP64 kernels.
Pair production's float-float step in batches of every length, forced by a
tolerance that most float estimates miss; the estimate bounds the error, so the
tolerance is the bound."""
import numpy as np
import pytest
import torch

from noa_gb300 import _lib, dcs
from noa_gb300.elements import ELEMENTS, MUON_MASS
from noa_gb300.workload import kinetic_recoil
from tests.parity import PROCESSES

pytestmark = pytest.mark.gpu


def check(got, exp, bound=1e-6):
    assert torch.equal(got == 0, exp == 0)
    nz = exp != 0
    assert bool(((got[nz] - exp[nz]).abs() <= bound * exp[nz].abs()).all())


@pytest.mark.parametrize("process", [0, 3], ids=[PROCESSES[0], PROCESSES[3]])
@pytest.mark.parametrize("per_cta,extra", [(0, 1), (0, 33), (0, 257), (32, -1), (32, 1), (257, 3), (1024, 1)])
def test_map_tiles(cuda_device, process, per_cta, extra):
    n = 4 * torch.cuda.get_device_properties(0).multi_processor_count * per_cta + extra
    K, q = (torch.from_numpy(a).cuda() for a in kinetic_recoil(n))
    out = torch.full((n + 512,), -7.0, dtype=torch.float64, device="cuda")
    dcs.vmap(process, out[:n], K, q, ELEMENTS[1], MUON_MASS, "fp32c")
    check(out[:n], dcs.map(process, K, q, ELEMENTS[1], MUON_MASS))
    assert bool((out[n:] == -7.0).all())


@pytest.mark.parametrize("z", [1, 82])
def test_pair_production_beyond_float(cuda_device, z):
    g = np.random.default_rng(12)
    K = 10.0 ** g.uniform(15, 40, 20_000)
    q = K * 10.0 ** g.uniform(-20, 0, K.size)
    K, q = torch.from_numpy(K).cuda(), torch.from_numpy(q).cuda()
    got, exp = (dcs.map(1, K, q, ELEMENTS[z], MUON_MASS, p) for p in ("fp32c", "fp64"))
    check(got, exp)


@pytest.mark.parametrize("n", [1, 31, 33, 255, 257, 513, 5000, 400_003])
def test_float_float_batches(cuda_device, n):
    K, q = (torch.from_numpy(a).cuda() for a in kinetic_recoil(n))
    out = torch.full((n + 512,), -7.0, dtype=torch.float64, device="cuda")
    _lib.check(_lib.load().noa_dcs_cuda_vmap_fp32c(1, out.data_ptr(), K.data_ptr(), q.data_ptr(), n,
                                                   _lib.element_struct(ELEMENTS[26]), MUON_MASS, 2e-7, None))
    check(out[:n], dcs.map(1, K, q, ELEMENTS[26], MUON_MASS), 2e-7)
    assert bool((out[n:] == -7.0).all())
