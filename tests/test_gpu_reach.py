"""Evaluations whose cutoff reaches beyond the pairlist distance the handle was
created with (needs a B200): slow forces, energy and virial against a sum over all
pairs of the minimum images in 64 bits; the gradient, which takes the handle's
own cutoff, likewise."""
import dataclasses

import numpy as np
import pytest

import nbk
from helpers import (ALL, ENERGY_TOL, FORCE_RMS_TOL, PARAMS, VIRIAL_TOL, GpuRun, real_slots, rms_rel,
                     water_box)

pytestmark = pytest.mark.gpu

CS = 0.3


def _all_pairs(p, beta, rc, reach, w):
    """Slow forces, energy and virial per unit of the library's, and the gradient
    of sum w.S + CS E in positions and charges, by atom."""
    import torch
    slot = p.slotOfAtom
    start = p.patches[:, 2]
    patch = np.searchsorted(start, slot, side="right") - 1
    x = torch.tensor(p.xyzq[slot, :3].astype(np.float64) + p.patchCenter[patch], requires_grad=True)
    q = torch.tensor(p.xyzq[slot, 3].astype(np.float64), requires_grad=True)
    w = torch.tensor(w[slot].astype(np.float64))
    L = torch.tensor(np.diag(p.lattice).astype(np.float64))
    i, j = np.triu_indices(len(slot), 1)
    xn = x.detach().numpy()
    d = xn[j] - xn[i]
    image = torch.tensor(np.rint(d / L.numpy()))
    near = ((d - (image * L).numpy()) ** 2).sum(1) < reach * reach
    excl = set(map(tuple, np.sort(p.system.arrays()["fullExcl"], axis=1)))
    n = len(slot)
    keys = np.array([a * n + b for a, b in excl])
    near &= ~np.isin(i.astype(np.int64) * n + j, keys)
    i, j, image = torch.tensor(i[near]), torch.tensor(j[near]), image[torch.tensor(near)]
    d = x[j] - x[i] - image * L
    s = (d * d).sum(1)
    r = s.sqrt()
    phi = (3.0 - s / rc ** 2) / (2.0 * rc) - torch.erf(beta * r) / r
    E = (q[i] * q[j] * phi).sum()
    S, = torch.autograd.grad(-E, x, create_graph=True)
    gX, gQ = torch.autograd.grad((w * S).sum() + CS * E, (x, q), retain_graph=True)
    g, = torch.autograd.grad(E, d, retain_graph=True)         # dE/dd per pair
    W = -(g.T @ d)
    return [t.detach().numpy() for t in (S, E, W, gX, gQ)]


# Tables up to 10.5 A: in shared memory, and at the larger coefficients in global
# memory or, for the force factor, none; and a coefficient so small that erf(x) is
# about x over the whole range.
@pytest.mark.parametrize("beta,switch", [(0.2579, 7.5), (0.2579, 9.0), (0.6, 7.5), (1.2, 7.5), (0.02, 7.5)])
def test_cutoff_beyond_the_handles_pairlist_distance(beta, switch):
    import torch
    rc, pl, reach = 9.0, 10.5, 13.0
    p = nbk.Packed(water_box(seed=3, nwater=700, box=28.0))
    params = dataclasses.replace(PARAMS, ewaldcof=beta, cutoff=rc, switchdist=switch, pairlistdist=pl)
    run = GpuRun(p, params)
    n, v, lib = p.atomStorageSize, p.v, nbk.dev_lib()
    xyzq = torch.from_numpy(p.xyzq.copy()).cuda()
    import ctypes as C
    assert lib.nbk_build_tile_lists(run.nb._h, v.numPatches, n, v.maxTileListLen, v.lata, v.latb, v.latc,
                                    C.cast(v.patches, C.c_void_p), xyzq.data_ptr(), 1, 13.5 * 13.5,
                                    None) == 0
    for flags in (ALL | nbk.NBK_PAIRLIST, nbk.NBK_SLOW, ALL):
        assert lib.nbk_nonbonded_force(run.nb._h, n, flags, v.lata, v.latb, v.latc, xyzq.data_ptr(), 1,
                                       reach * reach, None, run.dS.data_ptr(), None, None,
                                       run.dX.data_ptr(), None) == 0
        torch.cuda.synchronize()
        S = run.dX[3:].T.cpu().numpy().astype(np.float64) / nbk.FORCE_FIXED_SCALE
        if flags == nbk.NBK_SLOW:
            first = S
    ve = run.nb.virial_energy(ALL)
    rng = np.random.default_rng(8)
    w = np.zeros((n, 4), np.float32)
    w[:, :3] = rng.standard_normal((n, 3))
    dw, zero = torch.from_numpy(w).cuda(), torch.zeros((n, 4), device="cuda")
    g = torch.zeros((n, 4), device="cuda")
    dim = p.system.lj_table()[0]
    gab = torch.zeros(2 * dim * dim, dtype=torch.float64, device="cuda")
    run.nb.adjoint(zero, dw, 0.0, 0.0, CS, g, gab)
    g = g.cpu().numpy().astype(np.float64)
    So, Eo, Wo, _, _ = _all_pairs(p, beta, rc, reach, w[:, :3])
    _, _, _, gX, gQ = _all_pairs(p, beta, rc, rc, w[:, :3])
    slot = p.slotOfAtom
    err = dict(first=rms_rel(first[slot], So), slow=rms_rel(S[slot], So),
               energy=abs(ve.energySlow - Eo) / abs(Eo),
               virial=rms_rel(np.array(ve.virialSlow).reshape(3, 3), Wo),
               gX=rms_rel(g[slot, :3], gX), gQ=rms_rel(g[slot, 3], gQ))
    print(beta, switch, " ".join(f"{k}={e:.2e}" for k, e in err.items()))
    for k in ("first", "slow", "gX", "gQ"):
        assert err[k] <= FORCE_RMS_TOL, err
    assert err["energy"] <= ENERGY_TOL and err["virial"] <= VIRIAL_TOL, err
