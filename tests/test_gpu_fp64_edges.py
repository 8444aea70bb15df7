"""The FP64 kernels where their lean and their IEEE-ordered forms meet, and on
inputs of unusual size: pairs around K / q = 1 + 2^-11 .. 1 + 2^-9 (the edge
rule on high words), pair production's argmin around 1 - 2^-10, photonuclear
windows about to close, and every combination of zeros, infinities, NaN, tiny,
huge and negative energies, against the CPU oracle."""
import numpy as np
import pytest
import torch

import oracle
from noa_gb300 import dcs
from noa_gb300.elements import ELEMENTS, MUON_MASS, TAU_MASS
from tests.parity import PROCESSES, assert_conditioned, conditioning, same_or_both_nan

pytestmark = pytest.mark.gpu


def evaluate(process, K, q, element, mass):
    tk, tq = torch.from_numpy(K).cuda(), torch.from_numpy(q).cuda()
    return dcs.map(process, tk, tq, element, mass).cpu().numpy()


def near_edges(mass):
    rng = np.random.default_rng(11)
    n = 20_000
    K = 10.0 ** rng.uniform(-3, 6, n)
    gap = 2.0 ** rng.uniform(-14, -7, n)
    q = np.concatenate([K / (1 + gap), K[: n // 4] / (1 + 2.0 ** -10), K[n // 4: n // 2] / (1 + 2.0 ** -11)])
    Ks = [K, K[: n // 2]]
    # pair production: argmin -> 1 as q -> 4 me
    q4 = 4 * 0.510998910e-3 * (1 + 10.0 ** rng.uniform(-9, -1, n))
    # photonuclear: the window closes as Q2min, which grows with q / (E - q), meets Q2max
    K3 = 10.0 ** rng.uniform(0, 3, n)
    q3 = K3 + mass - mass * mass / (2 * 0.931494) * (1 + 10.0 ** rng.uniform(-5, 0, n)) * rng.choice([1, 1.5], n)
    return np.concatenate(Ks + [K, K3]), np.concatenate([q, q4, q3])


@pytest.mark.parametrize("process", range(4), ids=PROCESSES)
@pytest.mark.parametrize("z,mass", [(1, MUON_MASS), (11, TAU_MASS), (82, MUON_MASS)])
def test_edges(cuda_device, process, z, mass):
    K, q = near_edges(mass)
    el = ELEMENTS[z]
    got, exp = evaluate(process, K, q, el, mass), oracle.dcs(process, K, q, el, mass)
    assert np.array_equal(got == 0, exp == 0)
    assert_conditioned(got, exp, conditioning(process, K, q, el, mass, exp), PROCESSES[process])


@pytest.mark.parametrize("process", range(4), ids=PROCESSES)
def test_unusual_inputs(cuda_device, process):
    v = np.array([0.0, -0.0, -1.0, 5e-324, 1e-300, 1e-30, 1e-20, 1e-3, 0.2, 1.0, 1.5, 30.0, 1e3, 1e6, 1e20, 1e28, 1e29,
                  1e40, 1e100, np.inf, -np.inf, np.nan])
    K, q = (a.ravel().copy() for a in np.meshgrid(v, v))
    el = ELEMENTS[11]
    got, exp = evaluate(process, K, q, el, MUON_MASS), oracle.dcs(process, K, q, el, MUON_MASS)
    fin = np.isfinite(exp)
    bad = np.flatnonzero((np.isfinite(got) != fin) | ((got == 0) != (exp == 0)))
    assert bad.size == 0, [(K[i], q[i], got[i], exp[i]) for i in bad[:8]]
    assert same_or_both_nan(got[~fin], exp[~fin])
    m = fin & (exp != 0)
    assert np.all(np.abs(got[m] - exp[m]) <= 1e-8 * np.abs(exp[m]))
