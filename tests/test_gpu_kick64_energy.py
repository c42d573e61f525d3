"""The FP64 kick's energy where the kick is as large as the momentum.

tau' = w e' and x = x_lab + x' w with w = -z_lab / pz' (coord_transform.py:46-54)
leave the new longitudinal momentum, and with it the energy e' = 1/beta + delta',
to be read back from the outputs: pz' = rho e' with rho = -z_lab / tau', so
e'^2 (1 - rho^2) = px'^2 + py'^2 + (m c / p_ref)^2.  The kernel forms delta' as an
increment; both have to agree whatever the field.  rho carries some 12 roundings
of 2^-53, e' gamma'^2 times that: 1.2e-14 at gamma' = 3, taken twice.
"""
import numpy as np
import pytest

from conftest import has_gpu
from oracle import sc_oracle

pytestmark = pytest.mark.gpu

if not has_gpu():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import torch  # noqa: E402

from ocelot_gb300 import SpaceCharge  # noqa: E402

DEV = torch.device("cuda", 0)


def strong_kick(n=6000):
    """A millimetre of 0.6 MeV electrons whose own field changes their momenta by tens of per cent."""
    rp, q = sc_oracle.gaussian_beam(n, 21, charge=0.5e-9)
    for row, sigma in ((0, 1e-3), (1, 1e-3), (2, 1e-3), (3, 1e-3), (4, 1e-3), (5, 1e-3)):
        rp[row] *= sigma / np.std(rp[row])
    return rp, q, 0.0006, 0.1, (24, 24, 31)


def energy_mismatch(rp, out, energy):
    """max |e' of delta' / e' of the other outputs - 1| (gamma' < 3, pz' of some size), and the largest change of delta."""
    L = np.longdouble
    x, xq, y, yq, tau, d = rp.astype(L)
    gamma = L(energy) / L(sc_oracle.m_e_GeV)
    mu2 = 1 / (gamma * gamma - 1)
    ib = np.sqrt(1 + mu2)
    e = ib + d
    pz = np.sqrt(e * e - mu2 - xq * xq - yq * yq)
    o = out.astype(L)
    rho = pz * tau / (e * o[4])
    en = np.sqrt((o[1] ** 2 + o[3] ** 2 + mu2) / (1 - rho * rho))
    ok = (en * en < 9 * mu2) & (np.abs(rho) > 0.2) & (np.abs(tau) > 1e-5)
    assert ok.sum() > len(tau) // 2
    return float(np.max(np.abs((ib + o[5]) / en - 1)[ok])), float(np.max(np.abs(o[5] - d)[ok]))


def test_energy_follows_from_the_momenta():
    rp, q, energy, dz, mesh = strong_kick()
    d = torch.from_numpy(rp).to(DEV)
    sc = SpaceCharge(nmesh_xyz=mesh, precision="fp64", device=DEV)
    sc.apply_device(d, torch.from_numpy(q).to(DEV), energy, dz)
    sc.check()
    mismatch, change = energy_mismatch(rp, d.cpu().numpy(), energy)
    assert change > 0.3
    assert mismatch < 2.5e-14
