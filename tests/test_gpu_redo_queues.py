"""FP32C with every pair rejected (a tolerance no estimate meets, or NaN
energies): the redo and third queues are then fed a whole step at a time, and
the results are those of the FP64 bodies."""
import numpy as np
import pytest
import torch

from noa_gb300 import _lib, dcs
from noa_gb300.batched import BatchPlan
from noa_gb300.elements import BATCH_Z, ELEMENTS, MUON_MASS
from noa_gb300.workload import kinetic_recoil
from tests.parity import PROCESSES

pytestmark = pytest.mark.gpu


def open_pairs(n):
    """Pairs that are open in every process, or nearly all."""
    g = np.random.default_rng(8)
    K = 10.0 ** g.uniform(1.5, 5, n)
    return K, K * g.uniform(0.01, 0.5, n)


def fp32c(process, K, q, element, tolerance):
    out = torch.full_like(K, -7.0)
    _lib.check(_lib.load().noa_dcs_cuda_vmap_fp32c(process, out.data_ptr(), K.data_ptr(), q.data_ptr(), K.numel(),
                                                   _lib.element_struct(element), MUON_MASS, tolerance, None))
    return out


@pytest.mark.parametrize("n", [31, 33, 300, 5000, 1_000_003])
@pytest.mark.parametrize("process", range(4), ids=PROCESSES)
def test_all_rejected(cuda_device, process, n):
    K, q = (torch.from_numpy(a).cuda() for a in open_pairs(n))
    got = fp32c(process, K, q, ELEMENTS[26], 1e-30)
    exp = dcs.map(process, K, q, ELEMENTS[26])
    torch.cuda.synchronize()
    # the same FP64 bodies, compiled in another kernel (bremsstrahlung: the
    # reference's form); ill-conditioned pair-production pairs move by 1e-11
    assert torch.allclose(got, exp, rtol=1e-9, atol=0.0)


@pytest.mark.parametrize("threads,items", [(128, 1), (128, 8), (256, 4)])
@pytest.mark.parametrize("process", range(4), ids=PROCESSES)
def test_all_rejected_batched(cuda_device, process, threads, items):
    counts = [700, 1, 4096, 0, 33_333]
    K, q = (torch.from_numpy(a).cuda() for a in open_pairs(sum(counts)))
    els = [ELEMENTS[z] for z in BATCH_Z[:5]]
    got = torch.full_like(K, -7.0)
    with BatchPlan(process, els, counts, precision="fp32c", tolerance=1e-30) as plan:
        plan.set_tile(threads, items, 2)
        plan.execute(got, K, q)
        torch.cuda.synchronize()
    exp = torch.cat([dcs.map(process, k, r, el) for k, r, el in zip(K.split(counts), q.split(counts), els)])
    assert torch.allclose(got, exp, rtol=1e-9, atol=0.0)


@pytest.mark.parametrize("process", range(4), ids=PROCESSES)
def test_all_nan(cuda_device, process):
    K, q = (torch.from_numpy(a).cuda() for a in kinetic_recoil(100_000))
    K[:] = float("nan")
    got, exp = (dcs.map(process, K, q, ELEMENTS[26], precision=p) for p in ("fp32c", "fp64"))
    assert torch.equal(torch.isnan(got), torch.isnan(exp))
    assert torch.equal(got[~torch.isnan(got)], exp[~torch.isnan(exp)])
