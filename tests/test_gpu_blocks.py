"""The block-order kernels' dispatch (needs a B200): the slow force factor from
its table and from the erfc form, the adjoint's table in shared and in global
memory, lists split by the rule on their number, and the patch sort with equal
coordinates."""
import dataclasses

import numpy as np
import pytest

import nbk
import oracle
from helpers import (ALL, ENERGY_TOL, FORCE_RMS_TOL, PARAMS, VIRIAL_TOL, GpuRun, mixed_box, real_slots,
                     rel, rms_rel, split_rule, water_box, wider_lj)

pytestmark = pytest.mark.gpu


def _step(p, params, flags):
    run = GpuRun(p, params)
    run.build()
    run.eval(flags | nbk.NBK_PAIRLIST)
    return run, run.eval(flags)


# A table has (pairlistdist^2 + 2) / step rows, the step falling with beta^2: 94
# rows at the first parameters (eight copies), six at the second, one copy at the
# third, and more than the table may have (1,024, at beta pairlistdist of about 12)
# at the last two, which take the erfc form. Tolerance: that of every force test
# against FP64.
@pytest.mark.parametrize("beta,cutoff,switch,pl,rows", [
    (0.2579, 12.0, 10.0, 13.5, 94), (0.02, 9.0, 7.0, 10.5, 6), (0.6, 9.0, 9.0, 10.5, 451),
    (0.6, 12.0, 10.0, 13.5, 739), (1.0, 12.0, 10.0, 13.5, 0), (1.2, 12.0, 10.0, 16.0, 0)])
def test_slow_force_table_and_erfc_form(beta, cutoff, switch, pl, rows):
    assert len(nbk.force_table(beta, cutoff, pl)[0]) == rows
    params = dataclasses.replace(PARAMS, ewaldcof=beta, cutoff=cutoff, switchdist=switch,
                                 pairlistdist=pl)
    p = nbk.Packed(mixed_box(seed=5, natoms=6200), patch_dim=pl)
    _, (F, S, _, _) = _step(p, params, nbk.NBK_SLOW)
    Fo, So, _ = oracle.Oracle(p, params).forces(1)
    real = real_slots(p)
    assert rms_rel(F[real], Fo[real]) < FORCE_RMS_TOL
    assert rms_rel(S[real], So[real]) < FORCE_RMS_TOL


# 1, 2 or 4 work items per list by the rule on their number: every sum is the
# one of unsplit lists, bit for bit (the force and the precise kernel), and of the
# other splits.
@pytest.mark.parametrize("make,split", [(lambda: water_box(seed=3, nwater=900, box=30.0), 4),
                                        (lambda: mixed_box(seed=4, natoms=9001), 4),
                                        (lambda: mixed_box(seed=4, natoms=24000), 2),
                                        (lambda: mixed_box(seed=4, natoms=50003), 1)])
def test_split_lists_give_the_sums_of_whole_lists(make, split):
    p = nbk.Packed(make())
    assert split_rule(p) == split
    run, (_, _, res, X) = _step(p, PARAMS, ALL)
    assert run.nb.tuning(ALL)["warps_per_list"] == split
    for other in {1, 2, 4} - {split}:
        run.nb.set_tuning(ALL, 4, other)
        _, _, one, X1 = run.eval(ALL)
        assert np.array_equal(X, X1)
        for k in res:
            assert np.array_equal(res[k], one[k]), k


# The adjoint's slow table: eight copies in shared memory; one copy at the small
# steps of a large beta; global memory when not even one fits (more than 768
# rows). Also without the slow term. Tolerance: FP32 pair terms, as the forces.
@pytest.mark.parametrize("beta,pl,slow,copies", [(0.2579, 13.5, True, 8), (1.0, 13.5, True, 1),
                                                 (1.0, 16.0, True, 0), (0.2579, 13.5, False, 8)])
def test_adjoint_table_placement(beta, pl, slow, copies):
    import torch
    rows = len(nbk.slow_table(beta, PARAMS.cutoff, pl)[0])  # 32 bytes each in FP32, in 24 KB
    assert copies == next((c for c in (8, 4, 2, 1) if rows * 32 * c <= 24 * 1024), 0)
    params = dataclasses.replace(PARAMS, ewaldcof=beta, pairlistdist=pl)
    sy = mixed_box(seed=6, natoms=6200)
    p = nbk.Packed(sy, patch_dim=pl)
    n, dim = p.atomStorageSize, sy.lj_table()[0]
    run, _ = _step(p, params, ALL if slow else nbk.NBK_ENERGY)
    rng = np.random.default_rng(8)
    w = [np.zeros((n, 4), np.float32) for _ in range(2)]
    for a in w:
        a[:, :3] = rng.standard_normal((n, 3))
    dev = [torch.from_numpy(a).cuda() for a in w]
    g = torch.zeros((n, 4), device="cuda")
    gab = torch.zeros(2 * dim * dim, dtype=torch.float64, device="cuda")
    run.nb.adjoint(dev[0], dev[1], 0.1, 0.2, 0.3 if slow else 0.0, g, gab, slow=slow)
    torch.cuda.synchronize()
    wS = w[1][:, :3] if slow else np.zeros((n, 3))
    _, gX, gQ, gA, gB = oracle.Oracle(p, params).adjoint(
        w[0][:, :3].astype(np.float64), wS.astype(np.float64), 0.1, 0.2, 0.3 if slow else 0.0)
    real = real_slots(p)
    got = g.cpu().numpy().astype(np.float64)
    assert rms_rel(got[real, :3], gX[real]) < FORCE_RMS_TOL
    assert rms_rel(got[real, 3], gQ[real]) < FORCE_RMS_TOL
    ab = gab.cpu().numpy()
    assert rms_rel(ab[:dim * dim], gA.reshape(-1)) < FORCE_RMS_TOL
    assert rms_rel(ab[dim * dim:], gB.reshape(-1)) < FORCE_RMS_TOL


# The LJ table in shared memory beside the slow table's copies: from 62 types on
# fewer copies, and with many rows (the second coefficient) no table where one copy
# costs a block. Types that no atom has change nothing but the form: with the
# short table every bit stays; the erfc form holds the tolerance of every test.
@pytest.mark.parametrize("beta,exact", [(0.2579, True), (0.6, False)])
@pytest.mark.parametrize("types", [61, 62, 70, 80, 110])
def test_wide_lj_tables(beta, exact, types):
    params = dataclasses.replace(PARAMS, ewaldcof=beta)
    p = nbk.Packed(mixed_box(seed=5, natoms=6200))
    flags = ALL | nbk.NBK_CORRECTIONS
    _, (F, S, res, X) = _step(p, params, flags)
    run = GpuRun(p, params)
    run.nb = nbk.Nonbonded(params, wider_lj(p.system.lj_table(), types))
    run.nb.setup(p)
    run.build()
    run.eval(flags | nbk.NBK_PAIRLIST)
    F1, S1, res1, X1 = run.eval(flags)
    if exact:
        assert np.array_equal(X, X1)
        for k in res:
            assert np.array_equal(res[k], res1[k]), k
    assert rms_rel(F1, F) < FORCE_RMS_TOL and rms_rel(S1, S) < FORCE_RMS_TOL
    # the launch shapes and the flags change no bit, whatever the form
    for shape in ((4, 1), (5, 2), (6, 4)):
        run.nb.set_tuning(flags, *shape)
        assert np.array_equal(run.eval(flags)[3], X1)
    assert np.array_equal(run.eval(nbk.NBK_SLOW | nbk.NBK_CORRECTIONS)[3], X1)


# The precise kernel's table: eight, four copies or one in shared memory (40 KB), or
# in global memory. Energies, slow virial and pair count as in every parity test.
@pytest.mark.parametrize("beta,cutoff,pl,copies", [(0.2579, 12.0, 13.5, 8), (0.34, 10.0, 11.5, 4),
                                                   (0.45, 9.0, 10.5, 1), (0.6, 12.0, 13.5, 1),
                                                   (1.0, 12.0, 16.0, 0)])
def test_precise_table_placement(beta, cutoff, pl, copies):
    rows = nbk.slow_table(beta, cutoff, pl)[0].shape[0]
    assert copies == next((c for c in (8, 4, 1) if rows * 48 * c <= 40 * 1024), 0)
    params = dataclasses.replace(PARAMS, ewaldcof=beta, cutoff=cutoff, switchdist=cutoff - 1.0,
                                 pairlistdist=pl)
    p = nbk.Packed(mixed_box(seed=5, natoms=6200), patch_dim=pl)
    run, (_, _, res, _) = _step(p, params, ALL)
    _, _, ro = oracle.Oracle(p, params).forces(1)
    for k in ("energyElec", "energySlow"):
        assert rel(res[k], ro[k]) <= ENERGY_TOL, k
    assert rms_rel(res["virialSlow"], ro["virialSlow"]) <= VIRIAL_TOL
    assert run.nb.pair_count() == ro["pairs"]


def _bisect(pos, ids):
    """The patch sort on the host: parts split at block boundaries, ordered by
    (coordinate on the longest axis, id)."""
    order = list(range(len(ids)))

    def split_point(b, e):
        for W in (32, 16, 8):
            if b // W < (e - 1) // W:
                s = ((b + e + W) // (2 * W)) * W
                s += W if s <= b else 0
                s -= W if s >= e else 0
                return s if b < s < e else -1
        return -1

    def part(b, e):
        s = split_point(b, e)
        if s < 0:
            return
        x = pos[order[b:e]]
        ext = x.max(0) - x.min(0)
        axis = 1 if ext[1] > ext[0] else 0
        axis = 2 if ext[2] > ext[axis] else axis
        order[b:e] = sorted(order[b:e], key=lambda a: (pos[a, axis], ids[a]))
        part(b, s)
        part(s, e)

    part(0, len(ids))
    return np.array(order)


@pytest.mark.parametrize("grid", [0.0, 0.5, 4.0])  # 0: as generated; else coordinates on a grid (ties)
def test_patch_sort_order_with_equal_coordinates(grid):
    import torch
    s = mixed_box(seed=9, natoms=5003)
    p = nbk.Packed(s)
    L = nbk.ResidentLayout(s, p, shuffle_seed=3)
    pos = L.pos.T.copy()
    if grid:
        pos = np.round(pos / grid) * grid
        for k, axis in enumerate("xyz"):
            L.dev[axis] = torch.from_numpy(np.ascontiguousarray(pos[:, k])).cuda()
    order = torch.zeros(len(L.ids), dtype=torch.int32, device="cuda")
    L.sort_patch_atoms(order)
    got = order.cpu().numpy()
    for q in range(L.numPatches):
        b, k = L.records[q, 1], L.records[q, 3]
        assert np.array_equal(got[b:b + k], _bisect(pos[b:b + k], L.ids[b:b + k])), q


# Whatever the coordinates and ids hold (a blown-up integration, NaN or infinities
# among them), the order of a patch is a permutation of its atoms; patches without
# such atoms keep their order, and signed zeros are equal.
@pytest.mark.parametrize("bad", ["one nan", "all nan", "inf", "same ids", "zeros"])
def test_patch_sort_orders_any_input(bad):
    import torch
    s = mixed_box(seed=9, natoms=5003)
    L = nbk.ResidentLayout(s, nbk.Packed(s), shuffle_seed=3)
    pos, ids = L.pos.T.copy(), L.ids.copy()
    hit = range(0, L.numPatches, 2)
    rng = np.random.default_rng(1)
    for q in hit:
        b, k = L.records[q, 1], L.records[q, 3]
        part = pos[b:b + k]
        if bad == "one nan":
            part[k // 2] = np.nan
        elif bad == "all nan":
            part[:] = np.nan
        elif bad == "inf":
            part[rng.random(part.shape) < 0.3] = np.inf
            part[rng.random(part.shape) < 0.3] = -np.inf
            part[rng.random(part.shape) < 0.1] = np.nan
        elif bad == "same ids":
            ids[b:b + k] = 7
            part[:] = np.round(part / 4.0) * 4.0
        else:
            part[:] = rng.choice([0.0, -0.0, 1.0], part.shape)
    for k, axis in enumerate("xyz"):
        L.dev[axis] = torch.from_numpy(np.ascontiguousarray(pos[:, k])).cuda()
    L.dev["id"] = torch.from_numpy(ids).cuda()
    order = torch.zeros(len(ids), dtype=torch.int32, device="cuda")
    L.sort_patch_atoms(order)
    got = order.cpu().numpy()
    for q in range(L.numPatches):
        b, k = L.records[q, 1], L.records[q, 3]
        assert np.array_equal(np.sort(got[b:b + k]), np.arange(k)), q
        if q not in hit or bad == "zeros":
            assert np.array_equal(got[b:b + k], _bisect(pos[b:b + k], ids[b:b + k])), q
