"""The Green's function kept for an unchanged mesh step, after a call that stopped.

A kick whose particles lie outside its mesh stops after the mesh is known and before
(or while) the Green's function for it is made; the next call with the same step has
to make it.  Compared bit for bit with an engine that has seen no error.
"""
import numpy as np
import pytest

from conftest import has_gpu
from oracle import sc_oracle

pytestmark = pytest.mark.gpu

if not has_gpu():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import torch  # noqa: E402

from ocelot_gb300.sc import Engine  # noqa: E402

DEV = torch.device("cuda", 0)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_a_stopped_kick_leaves_no_green_function_behind(precision):
    mesh, n, energy = (128, 120, 126), 5000, 0.130  # long enough to make that the kick stops first
    rp, q = sc_oracle.gaussian_beam(n, 17, charge=250e-12)
    q = torch.from_numpy(q).to(DEV)

    def kick(eng, shift, size=1.0):
        d = torch.from_numpy(rp * size).to(DEV)
        eng.kick(d, q, n, energy, 0.1, 1.0, shift)
        eng.check_status()
        return d.cpu().numpy()

    want = kick(Engine(mesh, precision, DEV), 0.25)
    eng = Engine(mesh, precision, DEV)
    kick(eng, 0.25, 1.5)  # a Green's function of other steps is in place
    with pytest.raises(ValueError, match="outside the mesh"):
        kick(eng, 60.0)
    assert np.array_equal(kick(eng, 0.25), want)
