"""Bremsstrahlung with nu = q / E rounded to nearest, as in the reference: 1 - nu
amplifies nu's last bit towards q = E, so a quotient of 1.5 ulp shows there as
ten times the rounding of everything else.  Against the formula in long double on
the rounded E and nu."""
import numpy as np
import pytest
import torch

from noa_gb300 import dcs
from noa_gb300.elements import ELEMENTS, MUON_MASS, TAU_MASS

pytestmark = pytest.mark.gpu

LD = np.longdouble
ME = 0.510998910e-3


@pytest.mark.parametrize("z,mass", [(1, MUON_MASS), (11, MUON_MASS), (82, TAU_MASS)])
@pytest.mark.parametrize("low", [1e-3, 1e-2, 1e-1])
def test_rounded_nu(cuda_device, z, mass, low):
    el = ELEMENTS[z]
    rng = np.random.default_rng(12)
    K = 10.0 ** rng.uniform(0.5, 6, 20_000)
    E = K + mass
    q = E * (1 - low * 10.0 ** rng.uniform(0.1, 0.9, K.size))
    got = dcs.map("bremsstrahlung", torch.from_numpy(K).cuda(), torch.from_numpy(q).cuda(), el, mass).cpu().numpy()

    nu = (q / E).astype(LD)
    m, me, sqrte = LD(mass), LD(ME), LD(1.648721271)
    BZn = LD(202.4 if z == 1 else 182.7 * float(z) ** (-1. / 3.))
    BZe = LD(446. if z == 1 else 1429. * float(z) ** (-2. / 3.))
    Dn = LD(1.54 * el.A ** 0.27)
    rem = LD(5.63588e-13) * me / m
    delta = m * m / 2 / E.astype(LD) * nu / (1 - nu)
    phi_n = np.maximum(np.log(BZn * (m + delta * (Dn * sqrte - 2)) / (Dn * (me + delta * sqrte * BZn))), 0)
    phi_e = np.log(BZe * m / ((1 + delta * (m / (me * me * sqrte))) * (me + delta * sqrte * BZe)))
    phi_e = np.where(q < E / (1 + 0.5 * mass * mass / (ME * E)), np.maximum(phi_e, 0), 0)
    s = z * phi_n + phi_e
    exp = LD(7.297182e-7) * rem * rem * z * s * (LD(4) / 3 * (1 / nu - 1) + nu) * LD(1e3) * LD(6.02214076e23) / LD(el.A)

    # After nu: up to 12 roundings of half an ulp in each logarithm's argument
    # (delta 5, the linear forms and their constants 5, quotient 2), absolute in
    # the logarithm, and its own ulp; a dozen in the product of the rest.
    u = LD(2.0 ** -53)
    k = s > 0
    bar = 12 * u * (z + 1 + s) / np.where(k, s, 1) + 12 * u
    assert np.array_equal(got[~k] == 0, np.ones((~k).sum(), bool))
    err = np.abs(got[k] - exp[k]) / exp[k]
    worst = int(np.argmax(err / bar[k]))
    assert np.all(err <= bar[k]), (float(err[worst]), float(bar[k][worst]))
