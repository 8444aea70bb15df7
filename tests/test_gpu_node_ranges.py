"""Pair production and photonuclear on both sides of the ranges in which their
nodes are evaluated in fixed point (beta, argmin and xi; the window's ends and
width, the element's shadowing exponent), against the CPU oracle with the
per-point bar of the parity tests."""
import numpy as np
import pytest
import torch

import oracle
from noa_gb300 import dcs
from noa_gb300.elements import ELEMENTS, MUON_MASS, TAU_MASS, AtomicElement
from tests.parity import PROCESSES, assert_conditioned, conditioning

pytestmark = pytest.mark.gpu

ME, M = 0.510998910e-3, 0.931494


def check(process, K, q, element, mass):
    got = dcs.map(process, torch.from_numpy(K).cuda(), torch.from_numpy(q).cuda(), element, mass).cpu().numpy()
    exp = oracle.dcs(process, K, q, element, mass)
    assert np.array_equal(got == 0, exp == 0)
    assert (exp != 0).any()
    assert_conditioned(got, exp, conditioning(process, K, q, element, mass, exp), PROCESSES[process])


def near(rng, centre, n=1500):
    return centre * 2.0 ** rng.uniform(-1.5, 1.5, n)


@pytest.mark.parametrize("mass", [MUON_MASS, TAU_MASS, 4 * ME], ids=["muon", "tau", "light"])
@pytest.mark.parametrize("name", ["argmin", "beta", "xi", "scale"])
def test_pair_production(cuda_device, name, mass):
    rng = np.random.default_rng(5)
    if name == "argmin":   # about 4 me / q = 2^-50
        q = near(rng, 4 * ME * 2.0 ** 50)
        K = q * 10.0 ** rng.uniform(0.01, 2, q.size)
    elif name == "beta":   # 1 .. 2^50: q / K -> 1
        K = 10.0 ** rng.uniform(1, 6, 3000)
        q = K * (1 - 2.0 ** -rng.uniform(1, 12, K.size))
    elif name == "xi":     # xf argmin = (m / me)^2 beta / 2 * argmin about 2^-85
        K = near(rng, 1e14)
        q = near(rng, 2.0 ** -85 * K ** 2 / (ME * (mass / ME) ** 2))
        q = np.maximum(q, 8 * ME)
    else:                  # beta's powers of two
        K = 10.0 ** rng.uniform(0, 4, 3000)
        beta = 2.0 ** rng.integers(-3, 8, K.size) * (1 + rng.uniform(-1e-9, 1e-9, K.size))
        q = (K + mass) * (np.sqrt(beta * beta + 2 * beta) - beta)
    check(1, K, q, ELEMENTS[11], mass)


@pytest.mark.parametrize("element", [ELEMENTS[1], ELEMENTS[82], AtomicElement(A=1e8, I=1e-7, Z=90)],
                         ids=["H", "Pb", "heavy"])
@pytest.mark.parametrize("name", ["upper", "lower", "width"])
def test_photonuclear(cuda_device, name, element):
    rng = np.random.default_rng(6)
    mass = MUON_MASS
    if name == "upper":    # Q2max = 2 M q about 2^41
        q = near(rng, 2.0 ** 41 / (2 * M))
        K = q * 10.0 ** rng.uniform(0.01, 2.6, q.size)
    elif name == "lower":  # Q2min = m^2 y^2 / (1 - y) about 2^-26, for a mass that reaches it
        mass = 0.02
        q = 10.0 ** rng.uniform(0, 4, 3000)
        K = q / near(rng, 2.0 ** -13 / mass, q.size)
    else:                  # a window of a factor 1.05 .. 16, which the tau reaches below the edge q = E - m
        mass = TAU_MASS
        K = 10.0 ** rng.uniform(0.5, 5, 3000)
        factor = 2.0 ** rng.uniform(0.02, 4, K.size)
        q = K + mass - (K + mass) * factor * mass * mass / (2 * M * (K + mass) + factor * mass * mass)
    check(2, K, q, element, mass)
