"""Transforms at every line length of the two-step form (64, 96, 128, 192 and
256 points) on meshes that fill half of the padded length, leave one cell or
many unused, and mix lengths with the Stockham ones: the potential within 1e-12
(FP64) and 1e-6 (FP32) relative in norm of the oracle's, whose FFTs are numpy's
on 2N - 1 points."""
import numpy as np
import pytest

from conftest import has_gpu
from oracle import sc_oracle

pytestmark = pytest.mark.gpu

if not has_gpu():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from ocelot_gb300 import SpaceCharge  # noqa: E402

MESHES = [([32, 48, 64], (64, 96, 128)), ([64, 32, 48], (128, 64, 96)),
                                         ([96, 128, 20], (192, 256, 48)), ([17, 96, 128], (48, 192, 256)),
                                         ([33, 49, 65], (96, 128, 192)), ([30, 100, 97], (64, 256, 256)),
                                         ([128, 9, 33], (256, 24, 96))]


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("fp32", 1e-6)])
@pytest.mark.parametrize("mesh,padded", MESHES)
def test_potential_at_two_step_lengths(mesh, padded, precision, tol):
    sc = SpaceCharge(nmesh_xyz=mesh, precision=precision)
    assert sc.engine().fft_shape() == padded
    q = np.random.default_rng(sum(mesh)).random(mesh) * 1e-15
    steps = (3e-6, 4e-6, 2e-5)
    ref = sc_oracle.potential(q, steps)
    phi = sc.potential(q, steps)
    assert np.linalg.norm(phi - ref) / np.linalg.norm(ref) < tol


@pytest.mark.parametrize("mesh,padded", MESHES)
def test_fp64_potential_scales_by_powers_of_two(mesh, padded):
    """A line's exponent is the only place where its magnitude enters the FP64
    transforms, so scaling the charge by a power of two scales every bit of the
    potential; charges over many decades, an empty grid and one bad value."""
    sc = SpaceCharge(nmesh_xyz=mesh, precision="fp64")
    g = np.random.default_rng(sum(mesh) + 1)
    q = g.random(mesh) * 10.0 ** (-20 * g.random(mesh)) * 1e-12
    q[g.random(mesh) < 0.5] = 0
    steps = (1e-5, 2e-5, 4e-5)
    p = np.asarray(sc.potential(q, steps))
    assert np.isfinite(p).all() and p.any()
    for k in (-500, 600):
        assert np.array_equal(np.asarray(sc.potential(np.ldexp(q, k), steps)), np.ldexp(p, k))
    assert not np.asarray(sc.potential(np.zeros(mesh), steps)).any()
    for bad in (np.nan, np.inf):
        q[1, 2, 3] = bad
        assert not np.isfinite(np.asarray(sc.potential(q, steps))).any()


@pytest.mark.parametrize("mesh", [[32, 48, 64], [96, 128, 20], [24, 20, 12]])
def test_fp64_potential_at_the_edge_of_the_exponent_range(mesh):
    """Denormal charges, and denormal potentials, are rounded to whole units of 2^-1074
    and not dropped.  Cells of metres keep the spectrum's values near the charges' own
    2^-1040, which have 34 bits left, and the potentials' below 2^-1029 at 45: 2^-28 of the same
    charges in range (numpy's transforms: 5e-13)."""
    sc = SpaceCharge(nmesh_xyz=mesh, precision="fp64")

    def change(q, steps):
        p, ref = np.asarray(sc.potential(q, steps)), np.asarray(sc.potential(np.ldexp(q, 1000), steps))
        return np.linalg.norm(np.ldexp(p, 1000) - ref) / np.linalg.norm(ref), np.abs(p).max()

    off, _ = change(np.ldexp(np.random.default_rng(3).random(mesh), -1040), (1.0, 2.0, 4.0))
    assert off < 2.0 ** -28
    off, top = change(np.ldexp(np.random.default_rng(4).random(mesh), -1015), (2.0 ** 60, 2.0 ** 60, 2.0 ** 61))
    assert 0 < top < 2.0 ** -1022
    assert off < 2.0 ** -28
