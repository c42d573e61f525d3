"""The mesh extent and the FP64 kick at the edges of their tiles and branches.

The extent lists up to 16 candidates per block for the last block and lets a
block with more evaluate its own; the FP64 kick recomputes grid coordinates
near the edge of the sampled range with the reference's operations.  Checked
against the oracle: NGP cells exactly, rparticles at the plain form's 1e-10
per row (relative, in norm).
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
MESH = [33, 20, 48]


def _beam(kind, n):
    rp, q = sc_oracle.gaussian_beam(n, 5 + n % 97, charge=250e-12)
    if kind == "lattice":  # many particles share each extreme coordinate
        for row, levels in ((0, 11), (2, 7), (4, 23)):
            lim = np.abs(rp[row]).max()
            rp[row] = np.round(rp[row] / lim * levels) * (lim / levels)
        rp[1] = rp[3] = 0.0
        q = q * (1.0 + 0.3 * np.sin(np.arange(n)))
    elif kind == "tilted":  # a large mean angle: the rotated coordinates cancel
        rp[1] += 0.05
        rp[3] -= 0.02
        rp[4] *= 10.0
    elif kind == "mirrored":  # a symmetric beam: extremes at whole grid coordinates
        m = n // 2
        rp[:, m:2 * m] = rp[:, :m]
        for row in (0, 2, 4):
            rp[row, m:2 * m] *= -1.0
        rp[1] = rp[3] = 0.0
        rp[5] = 0.0
    return rp, q


@pytest.mark.parametrize("kind,n", [("gauss", 4), ("gauss", 511), ("gauss", 1025), ("gauss", 70_001),
                                    ("lattice", 3000), ("lattice", 50_001), ("tilted", 20_000), ("mirrored", 20_000)])
def test_cells_and_fp64_kick_match_the_oracle(kind, n):
    rp, q = _beam(kind, n)
    ref, rec = rp.copy(), {}
    sc_oracle.sc_apply(ref, q, 0.130, 0.1, MESH, record=rec)
    for precision in ("fp64", "fp32"):
        d = torch.from_numpy(rp).to(DEV)
        sc = SpaceCharge(nmesh_xyz=MESH, precision=precision, device=DEV)
        sc.apply_device(d, torch.from_numpy(q).to(DEV), 0.130, 0.1)
        sc.check()
        keys = sc.engine().region("keys")[:n].cpu().numpy().astype(np.int64)
        if kind != "mirrored":  # there cells are decided by the last bit of the frame (a mean of ~0)
            assert np.array_equal(keys, rec["keys"]), precision
        if precision == "fp64" and kind != "mirrored":
            out = d.cpu().numpy()
            assert max(np.linalg.norm(out[r] - ref[r]) / np.linalg.norm(ref[r]) for r in range(6)) < 1e-10
        assert torch.isfinite(d).all()
