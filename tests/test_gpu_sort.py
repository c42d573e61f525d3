"""The radix sort at the edges of its tilings (256, 1024 and 4096 keys a block, from
64k and 512k keys on), as a permutation and with the charges of a deposit."""
import numpy as np
import pytest

from conftest import has_gpu
from oracle import sc_oracle

pytestmark = pytest.mark.gpu

if not has_gpu():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import torch  # noqa: E402

from ocelot_gb300 import SpaceCharge  # noqa: E402
from ocelot_gb300.sorting import stable_sort_keys  # noqa: E402

DEV = torch.device("cuda", 0)


@pytest.mark.parametrize("n", [255, 65_536, 65_537, 524_288, 524_289, 614_401])
@pytest.mark.parametrize("bits,spread", [(9, None), (18, None), (18, 40.0), (22, 3.0)])
def test_sort_at_the_tilings_edges(n, bits, spread):
    rng = np.random.default_rng(n + bits)
    k = rng.integers(0, 1 << bits, n) if spread is None else \
        np.clip(rng.normal((1 << bits) / 2, spread, n), 0, (1 << bits) - 1).astype(np.int64)
    sk, perm = stable_sort_keys(torch.from_numpy(k.astype(np.int32)).to(DEV), bits)
    order = np.argsort(k, kind="stable")
    assert np.array_equal(perm.cpu().numpy(), order)
    assert np.array_equal(sk.cpu().numpy(), k[order])


@pytest.mark.parametrize("n,mesh", [(100_001, (24, 20, 64)), (600_001, (63, 63, 63)), (700_000, (100, 80, 70))])
def test_fp64_deposit_is_bincount(n, mesh):
    """Two and three radix passes, charges of different size."""
    rp, q = sc_oracle.gaussian_beam(n, 3, charge=1e-9)
    q = q * (1.0 + 0.5 * np.sin(np.arange(n)))
    sc = SpaceCharge(nmesh_xyz=mesh, precision="fp64", device=DEV)
    sc.apply_device(torch.from_numpy(rp).to(DEV), torch.from_numpy(q).to(DEV), 0.130, 0.1)
    sc.check()
    keys = sc.engine().region("keys")[:n].cpu().numpy().astype(np.int64)
    grid = sc.engine().region("qgrid").cpu().numpy().reshape(-1)
    assert np.array_equal(grid, np.bincount(keys, q, int(np.prod(mesh))))
