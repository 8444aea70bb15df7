"""The surrogate's fallback list around its tiles' and queues' sizes, with no
trusted cell and a tolerance that no estimate meets: every open pair passes
the redo queues, and the results are those of the FP64 bodies."""
import numpy as np
import pytest
import torch

from noa_gb300 import dcs
from noa_gb300.elements import BATCH_Z, ELEMENTS, MUON_MASS
from noa_gb300.surrogate import GRID, Surrogate, init_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts", [[1], [31, 0, 2], [0, 256], [255, 33, 7000], [200_001, 1, 99_999]], ids=str)
@pytest.mark.parametrize("process", [1, 2], ids=["pair_production", "photonuclear"])
def test_all_rejected(cuda_device, process, counts):
    g = np.random.default_rng(9)
    n = sum(counts)
    K = 10.0 ** g.uniform(1.5, 5, n)
    K, q = (torch.from_numpy(a).cuda() for a in (K, K * g.uniform(0.003, 0.999, n)))
    s = Surrogate(process)
    s.set_params(init_params(0), np.array([0, 0, 0, 0, 1, 1, 1, 1, 0, 1], dtype=np.float32))
    got, stats = s.infer(K, q, counts, tolerance=1e-30, trust=np.zeros((len(BATCH_Z), *GRID), dtype=np.uint8))
    at = np.concatenate([[0], np.cumsum(counts)])
    exp = torch.cat([dcs.map(process, K[a:b].clone(), q[a:b].clone(), ELEMENTS[z], MUON_MASS)
                     for z, a, b in zip(BATCH_Z, at[:-1], at[1:])])
    torch.cuda.synchronize()
    assert stats["network"] == 0 and stats["fallback"] >= int((exp != 0).sum())
    # the same FP64 bodies, compiled in another kernel: ill-conditioned
    # pair-production pairs move by 1e-11
    assert torch.equal(got == 0, exp == 0)
    assert torch.allclose(got, exp, rtol=1e-9, atol=0.0)


@pytest.mark.parametrize("n", [1, 127, 128, 129, 513, 5000])
@pytest.mark.parametrize("process", [1, 2], ids=["pair_production", "photonuclear"])
def test_network_tiles(cuda_device, process, n):
    """Every cell trusted: a pair's value does not depend on the tiles around
    it, nor on where its list ends."""
    g = np.random.default_rng(10)
    K = 10.0 ** g.uniform(1.5, 5, 20_000)
    K, q = (torch.from_numpy(a).cuda() for a in (K, K * g.uniform(0.003, 0.999, K.size)))
    s = Surrogate(process)
    s.set_params(init_params(3), np.array([0, 0, 0, 0, 0.1, 0.1, 1, 1, 0, 1], dtype=np.float32))
    ones = np.ones((len(BATCH_Z), *GRID), dtype=np.uint8)
    every, stats = s.infer(K, q, [K.numel()], trust=ones)
    some, few = s.infer(K[:n].clone(), q[:n].clone(), [n], trust=ones)
    assert stats["status"] == few["status"] == 0 and stats["network"] > 0.9 * K.numel()
    assert torch.equal(some, every[:n])
