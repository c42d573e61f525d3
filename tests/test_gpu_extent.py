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


@pytest.mark.parametrize("shift", [None, -0.4, 0.45])
@pytest.mark.parametrize("mesh", [(256, 6, 5), (7, 250, 9), (6, 5, 200), (16, 96, 130), (33, 33, 33)])
def test_fp64_gather_over_mesh_shapes(mesh, shift):
    """The kick itself (output - input), with the mesh moved so that particles
    leave the sampled range at one end.  Either side's fields carry up to 1e-9 of
    cancellation noise from the integrated Green's function (against extended
    precision), so 5e-9 of the kick."""
    from ocelot_gb300.sc import Engine
    n = 5000
    rp, q = sc_oracle.gaussian_beam(n, sum(mesh), charge=1e-9)
    rp[:, 7] = rp[:, 8] = 0.0
    ref = rp.copy()
    sc_oracle.sc_apply(ref, q, 0.0065, 0.1, mesh, mesh_scale=None if shift is None else 1.0, mesh_shift=shift)
    d = torch.from_numpy(rp).to(DEV)
    eng = Engine(mesh, "fp64", DEV)
    eng.kick(d, torch.from_numpy(q).to(DEV), n, 0.0065, 0.1, *(() if shift is None else (1.0, shift)))
    eng.check_status()
    out = d.cpu().numpy()
    for r in (1, 3, 5):
        k = ref[r] - rp[r]
        assert np.linalg.norm(out[r] - rp[r] - k) < 5e-9 * np.linalg.norm(k), r


def _off_axis_beam(n=20_000, x0=0.1875, h=2.0 ** -23, cells=32, energy=0.130):
    """A beam ``x0 / h`` = 1.6 million cells off the axis whose x lie on cell faces
    or one last place (2^-55) below, and move by half that place on the way to
    the lab: the last bit of the reference's operations decides their cells."""
    rng = np.random.default_rng(11)
    half = n // 2
    gam = energy / sc_oracle.m_e_GeV
    beta = np.sqrt(1 - gam ** -2)
    rp = np.zeros((6, n))
    k = rng.integers(1, cells, half)
    k[0] = 0
    tau = 1e-5 * (1 + rng.random(half))
    drift = 2.0 ** -56 / (beta * tau) * (1 + 8e-7 * (rng.random(half) - 0.5))
    drift[rng.random(half) < 0.8] = 0.0  # few enough that the mean stays on a whole cell
    drift[k == 0] = 0.0
    for s, sl in ((1, slice(0, half)), (-1, slice(half, n))):  # mirrored about the middle
        rp[0, sl] = x0 + s * (k - cells // 2) * h
        rp[1, sl] = s * drift
        rp[4, sl] = tau
    rp[0, half:][drift != 0] -= 2.0 ** -55
    rp[2] = 1e-4 * rng.standard_normal(n)
    return rp, np.full(n, 2.0 ** -52), (cells + 3, 20, 24), energy


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_cells_of_an_off_axis_beam_on_faces(precision):
    """Far off the axis the last place of a coordinate is many 1e-12 of a cell."""
    rp, q, mesh, energy = _off_axis_beam()
    rec = {}
    sc_oracle.sc_apply(rp.copy(), q, energy, 1e-6, mesh, record=rec)
    d = torch.from_numpy(rp).to(DEV)
    sc = SpaceCharge(nmesh_xyz=mesh, precision=precision, device=DEV)
    sc.apply_device(d, torch.from_numpy(q).to(DEV), energy, 1e-6)
    sc.check()
    keys = sc.engine().region("keys")[:rp.shape[1]].cpu().numpy().astype(np.int64)
    assert np.array_equal(keys, rec["keys"])


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_mirrored_beam_up_to_the_tie_of_its_mesh(precision, monkeypatch):
    """A beam symmetric about the axis has a mean of ~0 and extremes at whole grid
    coordinates: rounding decides on which of two cells the mesh starts, and on which
    side of a face the extremes lie.  Against the oracle on the device's choice of
    these, the cells have to be the oracle's (within 1e-11 of a face either side's)
    and the FP64 kick as near as for any other beam."""
    n = 20_000
    rp, q = _beam("mirrored", n)
    rec = {}
    sc_oracle.sc_apply(rp.copy(), q, 0.130, 0.1, MESH, record=rec)
    d = torch.from_numpy(rp).to(DEV)
    sc = SpaceCharge(nmesh_xyz=MESH, precision=precision, device=DEV)
    sc.apply_device(d, torch.from_numpy(q).to(DEV), 0.130, 0.1)
    sc.check()
    keys = sc.engine().region("keys")[:n].cpu().numpy().astype(np.int64)
    cells = np.stack([keys // (MESH[1] * MESH[2]), keys // MESH[2] % MESH[1], keys % MESH[2]], axis=1)
    start = np.rint(np.median(cells - np.floor(rec["X"]) - 1, axis=0))
    assert np.abs(start).max() <= 1
    X = rec["X"] + start
    side = cells - np.floor(X) - 1
    assert np.abs(side).max() <= 1
    assert (np.abs(X - np.rint(X))[side != 0] < 1e-11).all()
    assert (side == 0).all(axis=1).mean() > 0.99
    if precision == "fp64":
        geometry = sc_oracle.mesh_geometry
        monkeypatch.setattr(sc_oracle, "mesh_geometry", lambda *a, **k: (geometry(*a, **k)[0] + start, rec["steps"]))
        monkeypatch.setattr(sc_oracle, "ngp_keys", lambda *a: keys)
        ref = rp.copy()
        sc_oracle.sc_apply(ref, q, 0.130, 0.1, MESH)
        out = d.cpu().numpy()
        assert max(np.linalg.norm(out[r] - ref[r]) / np.linalg.norm(ref[r]) for r in range(6)) < 1e-10
        for r in (1, 3, 5):
            k = ref[r] - rp[r]
            assert np.linalg.norm(out[r] - ref[r]) < 5e-9 * np.linalg.norm(k), r
