"""The PME charge spread and the gather by columns of the stencil (need a B200):
neither depends on an atom's place in its warp."""
import numpy as np
import pytest
import torch

import nbk
import pme as opme
from test_pme import PME_ENERGY_TOL, PME_VIRIAL_TOL

pytestmark = pytest.mark.gpu


# Sites far apart, each with atoms within one or two grid cells and some at the
# ends of the box, site by site and dealt round the sites; one atom to 1,500, so
# that the last warp of the gather is partly filled, and more than begin the large
# form of the spread. The grid's integers are the
# same, so energy, virial and each atom's force are equal bit for bit; energy and
# virial hold the bounds of the PME tests.
@pytest.mark.parametrize("order", [4, 6, 8])
@pytest.mark.parametrize("n,K", [(1, (8, 8, 8)), (2, (16, 18, 20)), (3, (16, 18, 20)), (31, (8, 9, 10)),
                                 (33, (32, 30, 36)), (1500, (64, 60, 72)), (60001, (64, 60, 72))])
def test_pme_does_not_depend_on_the_atoms_order(order, n, K):
    rng = np.random.default_rng(100 * order + n)
    sites = rng.random((max(n // 3, 1), 3))
    sites[::7] = rng.choice([0.0, 0.999], (len(sites[::7]), 3))
    at = np.sort(rng.integers(0, len(sites), n))
    atoms = np.zeros((n, 4), np.float32)
    atoms[:, :3] = (sites[at] + rng.random((n, 3)) * 1.5 / np.array(K)) % 1.0
    atoms[:, :3] -= atoms[:, :3] >= 1.0
    atoms[:, 3] = rng.normal(size=n) * 5.0
    atoms[n // 2, 3] = 0.0
    L = np.diag([30.0, 31.0, 33.0])
    rank = np.arange(n) - np.searchsorted(at, at)      # the atom's number in its site
    deal = np.lexsort((at, rank))
    got = []
    for idx in (np.arange(n), deal):
        p = nbk.Pme(K, order, 0.3)
        f = torch.zeros((n, 3), device="cuda")
        p.compute(torch.from_numpy(np.ascontiguousarray(atoms[idx])).cuda(), n, L, f)
        E, W = p.energy_virial()
        back = np.empty((n, 3), np.float32)
        back[idx] = f.cpu().numpy()
        got.append((E, np.asarray(W), back))
        p.close()
    assert got[0][0] == got[1][0]
    assert np.array_equal(got[0][1], got[1][1])
    assert np.array_equal(got[0][2], got[1][2])
    Eo, Wo, _ = opme.pme(atoms, L, K, order, 0.3)
    assert abs(got[0][0] - Eo) <= PME_ENERGY_TOL * abs(Eo)
    assert np.abs(got[0][1] - Wo).max() <= PME_VIRIAL_TOL * np.abs(Wo).max()
