"""The calls that a user's program makes on the B200 nonbonded path, as timed cases.

A molecular-dynamics engine calls this library once or twice per time step, so
the cases are its steps: fast forces alone (the inner steps of multiple time
stepping), fast and slow forces (the ordinary step), forces with energies and
virial (output and pressure-control steps), the pairlist rebuild every ten or
so steps, the GPU-resident step after atom migration, many replicas in one
call, the gradient of a loss on forces and energies, and the long-range PME
part. The listed systems are the ones the benchmark and the tests use: water
boxes of 2,700 and 9,000 atoms, mixed systems (chains and water) of 24,000,
92,224 and 1,066,628 atoms, and 64 replicas of 2,000 to 40,000 atoms.

The topology of a system (charges, types, exclusions, patches) is generated
once per process and shared, as a program keeps it for a whole run; the seed
moves every atom by N(0, 0.05 A) before the tile lists are built, and by
another N(0, 0.02 A) between the build and a steady step, as time steps do.
"""
import collections
import copy
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "namd-3.0_b200"))
import nbk  # noqa: E402

COULOMB = 332.0636
DEVICE = "cuda:0"
BENCH_BOX = (108.0, 108.0, 78.0)   # of the 92,224-atom system; other systems are cubes
FLAGS = {"f": 0, "v": nbk.NBK_VIRIAL, "e": nbk.NBK_ENERGY, "s": nbk.NBK_SLOW,
         "c": nbk.NBK_CORRECTIONS}
# the record of energies and virials, by quantity
RECORD = {"virial": slice(0, 9), "virial_slow": slice(9, 18), "vdw": slice(18, 19),
          "elec": slice(19, 20), "slow": slice(20, 21), "rest": slice(21, 31)}


def _case(name, kind, system, natoms, flags, **more):
    c = {"name": name, "kind": kind, "system": system, "natoms": natoms, "flags": flags,
         "cutoff": 12.0, "switchdist": 10.0, "ewaldcof": 0.2579}
    c.update(more)
    return c


def listed():
    """flags: f fast forces, s slow forces, e energies, v virials, c the
    corrections of excluded and 1-4 pairs."""
    return [
        # the smallest box whose patches do not meet themselves: a step of a
        # few microseconds of arithmetic, where launches and latency count
        _case("water2700 fs", "step", "water", 2700, "fsc"),
        # the plain water box, called as an engine that keeps its atoms on the
        # host does: page-locked positions in, page-locked forces and energies out
        _case("water9000 evs host", "step", "water", 9000, "fevsc", host=True),
        # the benchmark's system: an inner step of multiple time stepping
        _case("mixed92224 f", "step", "mixed", 92224, "f"),
        # the ordinary step
        _case("mixed92224 fs", "step", "mixed", 92224, "fsc"),
        # the benchmark's step: everything, no corrections
        _case("mixed92224 evs", "step", "mixed", 92224, "fevs"),
        # the step that rebuilds and refines the tile lists
        _case("mixed92224 rebuild evs", "rebuild", "mixed", 92224, "fevs"),
        # GPU-resident integrator, after atoms changed patches: sort, types,
        # positions, lists, forces, force arrays in the integrator's order
        _case("mixed92224 migrate fs", "migrate", "mixed", 92224, "fs"),
        # the large system of the precision study
        _case("mixed1066628 evs", "step", "mixed", 1066628, "fevsc"),
        # 64 independent replicas, log-uniform in size, one call
        _case("batch64 evs", "batch", "mixed", 2000, "fevs", most=40000, replicas=64),
        # gradient of a loss on forces and energies: positions, charges, LJ table
        _case("mixed24000 adjoint", "adjoint", "mixed", 24000, "fs"),
        # long-range part of the benchmark's system: forces, order 4, 1 A grid
        _case("pme92224 o4", "pme", "mixed", 92224, "f", order=4, spacing=1.0),
        # and of the large system, with energy and virial read back
        _case("pme1066628 o4 ev", "pme", "mixed", 1066628, "fev", order=4, spacing=1.0),
    ]


def draw(rng):
    kind = rng.choice(["step"] * 6 + ["rebuild", "rebuild", "migrate", "batch", "adjoint", "pme", "pme"])
    most = {"step": 400000, "rebuild": 400000, "migrate": 300000, "batch": 5000, "adjoint": 60000,
            "pme": 400000}[kind]
    least = 2000 if kind == "batch" else 3000
    n = int(math.exp(rng.uniform(math.log(least), math.log(most))))
    system = "mixed" if kind in ("batch", "adjoint", "pme") else rng.choice(["water", "mixed", "mixed"])
    if system == "water":
        n -= n % 3
    flags = {"step": ["f", "fs", "fsc", "fsc", "fev", "fvs", "fevs", "fevsc"],
             "rebuild": ["f", "fsc", "fevs", "fevsc"], "migrate": ["f", "fs"],
             "batch": ["f", "fs", "fevs", "fevsc"], "adjoint": ["f", "fs", "fs"],
             "pme": ["f", "fev"]}[kind]
    c = _case("", kind, system, n, rng.choice(flags))
    del c["name"]
    c["cutoff"] = rng.choice([12.0, 12.0, 12.0, 10.0, 9.0])
    # a program that truncates plainly passes switchdist = cutoff
    c["switchdist"] = c["cutoff"] - 2.0 if rng.random() < 0.85 else c["cutoff"]
    c["ewaldcof"] = {12.0: 0.2579, 10.0: 0.312, 9.0: 0.348}[c["cutoff"]]
    if kind == "step":
        c["host"] = rng.random() < 0.25
    if kind == "batch":
        c["most"] = int(n * math.exp(rng.uniform(0.3, 3.0)))
        c["replicas"] = rng.randint(3, 32)
    if kind == "pme":
        c["order"] = rng.choice([4, 4, 6, 8])
        c["spacing"] = {4: 1.0, 6: 1.5, 8: 2.0}[c["order"]]
    return c


# ---------------------------------------------------------------------------
# what a program keeps for a whole run
# ---------------------------------------------------------------------------
Topology = collections.namedtuple("Topology", "systems packed params lj arrays layout")
_topologies = collections.OrderedDict()   # the two last used


def _params(case):
    return nbk.NonbondedParams(cutoff=case["cutoff"], switchdist=case["switchdist"],
                               pairlistdist=case["cutoff"] + 1.5, ewaldcof=case["ewaldcof"])


def _sizes(case):
    rng = np.random.default_rng(1203)
    lo, hi = math.log(case["natoms"]), math.log(case["most"])
    return np.exp(rng.uniform(lo, hi, case["replicas"])).astype(int)


def _topology(case):
    key = tuple(case.get(k) for k in ("kind", "system", "natoms", "most", "replicas", "cutoff",
                                      "switchdist", "ewaldcof"))
    if key in _topologies:
        _topologies.move_to_end(key)
        return _topologies[key]
    params = _params(case)
    water = case["system"] == "water"
    kind = nbk.NBK_SYS_WATER if water else nbk.NBK_SYS_MIXED

    def make(seed, n):
        box = BENCH_BOX if n == 92224 else None
        frac = 0.0 if water else (0.25 if n > 1000000 else 0.3)
        return nbk.System(kind, seed, int(n), frac, box=box)

    if case["kind"] == "batch":
        systems = [make(5000 + r, n) for r, n in enumerate(_sizes(case))]
        packed = nbk.Packed.many(systems, patch_dim=params.pairlistdist)
    else:
        systems = [make(2, case["natoms"])]
        packed = nbk.Packed(systems[0], patch_dim=params.pairlistdist)
    layout = None
    if case["kind"] == "migrate":
        layout = nbk.ResidentLayout(systems[0], packed, shuffle_seed=5)
    t = Topology(systems, packed, params, systems[0].lj_table(), [s.arrays() for s in systems], layout)
    _topologies[key] = t
    while len(_topologies) > 2:
        _topologies.popitem(last=False)
    return t


def _flags(case):
    f = 0
    for letter in case["flags"]:
        f |= FLAGS[letter]
    return f


def _record():
    ve = torch.zeros(31, dtype=torch.float64, device=DEVICE)
    return ve, {k: ve[s] for k, s in RECORD.items()}


def _noise(generator, n, sigma):
    return torch.randn((n, 3), generator=generator, device=DEVICE, dtype=torch.float64) * sigma


def _moved(packed, xyzq, natoms, generator, sigma):
    """xyzq with every atom moved; a patch's padding slots repeat its last atom."""
    at = torch.from_numpy(packed.atomIndex.copy()).to(DEVICE).long()
    out = xyzq.clone()
    out[:, :3] = (out[:, :3].double() + _noise(generator, natoms, sigma)[at]).float()
    return out


def _fft_size(length):
    k = max(8, int(math.ceil(length)))
    while True:
        m = k
        for f in (2, 3, 5):
            while m % f == 0:
                m //= f
        if m == 1:
            return k
        k += 1


def prepare(case, seed):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(seed)
    if case["kind"] == "pme":
        return _prepare_pme(case, g)
    t = _topology(case)
    p = t.packed
    n = p.atomStorageSize
    natoms = int(p.atomIndex.max()) + 1
    flags = _flags(case)
    st = torch.cuda.current_stream().cuda_stream
    nb = nbk.Nonbonded(t.params, t.lj, 0)
    nb.setup(p, stream=st)
    if case["kind"] == "batch":
        nb.set_replicas(p, stream=st)
    slow = "s" in case["flags"]
    s = {"case": case, "nb": nb, "packed": p, "flags": flags, "topology": t, "slow": slow,
         "natoms": natoms, "stream": st,
         "F": torch.zeros((n, 4), device=DEVICE), "S": torch.zeros((n, 4), device=DEVICE) if slow else None}
    s["wants_ve"] = bool(flags & (nbk.NBK_ENERGY | nbk.NBK_VIRIAL))
    if case["kind"] == "migrate":
        return _prepare_migrate(case, s, g)
    built = _moved(p, torch.from_numpy(p.xyzq.copy()).to(DEVICE), natoms, g, 0.05)
    s["built"] = built
    nb.build_tile_lists(p, xyzq=built, stream=st)
    nb.force(p, flags | nbk.NBK_PAIRLIST, xyzq=built, d_forces=s["F"], d_forcesSlow=s["S"], stream=st)
    s["x"] = _moved(p, built, natoms, g, 0.02)
    if case["kind"] == "batch":
        s["ve"] = torch.zeros((p.numReplicas, 31), dtype=torch.float64, device=DEVICE)
        s["record"] = {k: s["ve"][:, sl] for k, sl in RECORD.items()}
    else:
        s["ve"], s["record"] = _record()
    if case.get("host"):
        s["hx"] = s["x"].cpu().pin_memory().numpy()
        s["hF"] = torch.zeros((n, 4)).pin_memory()
        s["hS"] = torch.zeros((n, 4)).pin_memory() if slow else None
        s["hve"] = torch.zeros(31, dtype=torch.float64).pin_memory()
        s["hrecord"] = {k: s["hve"][sl] for k, sl in RECORD.items()}
    if case["kind"] == "adjoint":
        nb.force(p, flags, xyzq=s["x"], d_forces=s["F"], d_forcesSlow=s["S"], stream=st)
        dim = t.lj[0]
        for k in ("wF", "wS"):
            w = torch.zeros((n, 4), device=DEVICE)
            w[:, :3] = torch.randn((n, 3), generator=g, device=DEVICE)
            s[k] = w
        s["grad"] = torch.zeros((n, 4), device=DEVICE)
        s["gab"] = torch.zeros(2 * dim * dim, dtype=torch.float64, device=DEVICE)
        s["mask"] = np.zeros(dim, dtype=np.int32)
        s["mask"][:dim - 2] = 1   # the chains' types; the water model is not fitted
    torch.cuda.synchronize()
    return s


def _prepare_migrate(case, s, g):
    t = s["topology"]
    layout = copy.copy(t.layout)
    n = s["natoms"]
    d = dict(layout.dev)
    noise = _noise(g, n, 0.05)
    for k, axis in enumerate("xyz"):
        d[axis] = d[axis] + noise[:, k]
    layout.dev = d
    s["layout"] = layout
    s["nb"].set_exclusions_by_atom(layout.excl_by_atom)
    s["order"] = torch.zeros(n, dtype=torch.int32, device=DEVICE)
    s["status"] = torch.zeros(1, dtype=torch.int32, device=DEVICE)
    s["x"] = torch.zeros((t.packed.atomStorageSize, 4), device=DEVICE)
    s["bonded"] = torch.randn((3, n), generator=g, device=DEVICE, dtype=torch.float64)
    s["normal"], s["nbond"], s["slow_force"] = (
        torch.zeros((3, n), dtype=torch.float64, device=DEVICE) for _ in range(3))
    torch.cuda.synchronize()
    return s


def _prepare_pme(case, g):
    t = _topology(case)
    a = t.arrays[0]
    n = len(a["charge"])
    box = np.asarray(a["box"], dtype=np.float64)
    K = [_fft_size(b / case["spacing"]) for b in box]
    pos = torch.from_numpy(a["pos"]).to(DEVICE) + _noise(g, n, 0.05)
    q = torch.from_numpy(a["charge"].astype(np.float32)).to(DEVICE)
    atoms = torch.zeros((n, 4), device=DEVICE)
    st = torch.cuda.current_stream().cuda_stream
    # the atoms in patch order, as an engine hands them over
    order = torch.from_numpy(np.argsort(t.packed.slotOfAtom)).to(DEVICE)
    xyz = [pos[order, d].contiguous() for d in range(3)]
    nbk.Pme.atoms_from_positions(*xyz, q[order].contiguous(), math.sqrt(COULOMB),
                                 np.concatenate([np.diag(box).reshape(-1), np.zeros(3)]), atoms, stream=st)
    torch.cuda.synchronize()
    flags = _flags(case)
    return {"case": case, "pme": nbk.Pme(K, case["order"], case["ewaldcof"], 0), "atoms": atoms, "n": n,
            "lattice": np.diag(box), "K": K, "force": torch.zeros((n, 3), device=DEVICE), "flags": flags,
            "stream": st}


# ---------------------------------------------------------------------------
def run(s):
    return _RUN[s["case"]["kind"]](s)


def _run_step(s):
    nb, p, st, flags = s["nb"], s["packed"], s["stream"], s["flags"]
    if "hx" in s:
        nb.force(p, flags, xyzq=s["hx"], d_forces=s["F"], d_forcesSlow=s["S"], h_forces=s["hF"],
                 h_forcesSlow=s["hS"], stream=st)
        out = {"F": s["hF"], "S": s["hS"]}
        if s["wants_ve"]:
            nb.virial_energy_to(s["hve"].data_ptr(), False, stream=st)
            out["record"] = s["hrecord"]
        return out
    nb.force(p, flags, xyzq=s["x"], d_forces=s["F"], d_forcesSlow=s["S"], stream=st)
    out = {"F": s["F"], "S": s["S"]}
    if s["wants_ve"]:
        nb.virial_energy_to(s["ve"].data_ptr(), True, stream=st)
        out["record"] = s["record"]
    return out


def _run_rebuild(s):
    nb, p, st = s["nb"], s["packed"], s["stream"]
    nb.build_tile_lists(p, xyzq=s["x"], stream=st)
    nb.force(p, s["flags"] | nbk.NBK_PAIRLIST, xyzq=s["x"], d_forces=s["F"], d_forcesSlow=s["S"], stream=st)
    out = {"F": s["F"], "S": s["S"]}
    if s["wants_ve"]:
        nb.virial_energy_to(s["ve"].data_ptr(), True, stream=st)
        out["record"] = s["record"]
    return out


def _run_migrate(s):
    nb, p, st, layout = s["nb"], s["packed"], s["stream"], s["layout"]
    layout.sort_patch_atoms(s["order"], status=s["status"], stream=st)
    nb.update_vdw_types_excl_device(layout, s["order"], status=s["status"], stream=st)
    layout.set_compute_positions(s["order"], s["x"], stream=st)
    nb.build_tile_lists(p, xyzq=s["x"], stream=st)
    nb.force(p, s["flags"] | nbk.NBK_PAIRLIST, xyzq=s["x"], stream=st)
    nb.accumulate_forces_to_soa(layout, s["order"], 2 if s["slow"] else 1, s["normal"], s["nbond"],
                                s["slow_force"], f_bond=s["bonded"], stream=st)
    return {"order": s["order"], "normal": s["normal"], "nbond": s["nbond"],
            "slow": s["slow_force"] if s["slow"] else None}


def _run_batch(s):
    nb, st = s["nb"], s["stream"]
    nb.force(s["packed"], s["flags"], xyzq=s["x"], d_forces=s["F"], d_forcesSlow=s["S"], stream=st)
    out = {"F": s["F"], "S": s["S"]}
    if s["wants_ve"]:
        nb.virial_energy_batch_to(s["ve"].data_ptr(), True, stream=st)
        out["record"] = s["record"]
    return out


def _run_adjoint(s):
    s["nb"].adjoint(s["wF"], s["wS"], 0.1, 0.1, 0.1, s["grad"], s["gab"], type_mask=s["mask"],
                    slow=s["slow"], stream=s["stream"])
    return {"grad": s["grad"], "gab": s["gab"]}


def _run_pme(s):
    p, st = s["pme"], s["stream"]
    p.compute(s["atoms"], s["n"], s["lattice"], s["force"], s["flags"], stream=st)
    if s["flags"]:
        energy, virial = p.energy_virial(st)
        return {"force": s["force"], "energy": energy, "virial": virial}
    return {"force": s["force"]}


_RUN = {"step": _run_step, "rebuild": _run_rebuild, "migrate": _run_migrate, "batch": _run_batch,
        "adjoint": _run_adjoint, "pme": _run_pme}


# ---------------------------------------------------------------------------
def work(case):
    """Bytes: positions, charges and types read once, forces written once.
    Operations: per pair within the cutoff (0.1 atoms/A^3) 40 for the fast
    force, 90 with the slow one, 65 more (64-bit) for energies and virials,
    250 for the gradient; PME: order^3 points spread and gathered, and two
    transforms of 2.5 K log2 K each."""
    n = int(_sizes(case).sum()) if case["kind"] == "batch" else case["natoms"]
    if case["kind"] == "pme":
        side = n / 0.1 / case["spacing"] ** 3
        return {"bytes": 28.0 * n, "flops": n * case["order"] ** 3 * 9.0 + 5.0 * side * math.log2(side)}
    pairs = 0.5 * n * 0.1 * 4.0 / 3.0 * math.pi * case["cutoff"] ** 3
    slow = "s" in case["flags"]
    per = 90.0 if slow else 40.0
    if "e" in case["flags"] or ("v" in case["flags"] and slow):
        per += 65.0
    nbytes = n * (20.0 + 16.0 * (1 + slow))
    if case["kind"] == "adjoint":
        per, nbytes = 250.0, n * (20.0 + 16.0 * (1 + slow) + 16.0)
    if case["kind"] == "migrate":
        nbytes += n * (36.0 + 24.0 + 48.0)
    return {"bytes": nbytes, "flops": pairs * per}


def tolerance(case):
    """About four times what the FP32 pair forces and the FP32 transform show
    against 64 bits (2e-6 of the slow forces of water, 1e-6 elsewhere); the
    largest single difference is that of a short pair's force rounding."""
    if case["kind"] == "pme":
        return {"rel": 1e-5, "max": 2e-4}
    return {"rel": 1e-5, "max": 2e-4}


# ---------------------------------------------------------------------------
# the same quantities in 64 bits
# ---------------------------------------------------------------------------
def _pair_chunks(p, x, r2max, chunk=24_000_000):
    """Chunks (i slot, j slot, d = x_j - x_i, compute) of the pairs of the
    computes within the cutoff: every atom of patch 1 with every atom of patch
    2, self computes once per pair, full exclusions left out."""
    dev = x.device
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
    patches, comp = t(p.patches).long(), t(p.computes_patch).long()
    off = t(p.computes_offset).double()
    lat = t(np.ascontiguousarray(p.replicaLattice)).double()[t(p.replicaOfCompute).long()]
    shift = (off[:, :, None] * lat).sum(1)
    most = int(patches[:, 0].max())
    lanes = torch.arange(most, device=dev)
    idx, em = t(p.atomIndex).long(), t(p.exclIndexMaxDiff).long()
    bits = t(p.exclusionBits.view(np.int32)).long() & 0xFFFFFFFF
    step = max(1, chunk // (most * most))
    for c0 in range(0, len(comp), step):
        c = torch.arange(c0, min(len(comp), c0 + step), device=dev)
        p1, p2 = comp[c, 0], comp[c, 1]
        si, sj = (patches[q, 2][:, None] + lanes for q in (p1, p2))
        vi, vj = (lanes < patches[q, 0][:, None] for q in (p1, p2))
        top = len(x) - 1
        xi = x[si.clamp(max=top)] + shift[c][:, None]
        xj = x[sj.clamp(max=top)]
        r2 = torch.zeros((len(c), most, most), dtype=torch.float64, device=dev)
        for k in range(3):
            r2 += (xj[:, None, :, k] - xi[:, :, None, k]) ** 2
        own = (p1 == p2) & (off[c] == 0).all(1)
        ok = (r2 < r2max) & vi[:, :, None] & vj[:, None, :]
        ok &= ~own[:, None, None] | (lanes[None, :] > lanes[:, None])[None]
        b, u, w = ok.nonzero(as_tuple=True)
        del r2, ok
        i, j = si[b, u], sj[b, w]
        diff = idx[j] - idx[i]
        near = diff.abs() <= em[i, 1]
        bit = (diff + em[i, 0]).clamp(min=0, max=32 * len(bits) - 1)
        out = near & ((bits[bit >> 5] >> (bit & 31)) & 1).bool()
        b, i, j = b[~out], i[~out], j[~out]
        yield i, j, x[j] - x[i] - shift[c][b], c[b]


def _terms(case, s, qq, A, B):
    """Energies and (dE/dr)/r of LJ, fast and slow electrostatics at s = r^2."""
    rc, rs, beta = case["cutoff"], case["switchdist"], case["ewaldcof"]
    rc2, rs2 = rc * rc, rs * rs
    r = s.sqrt()
    i6 = s ** -3
    w, dw = (A * i6 - B) * i6, (-6.0 * A * i6 + 3.0 * B) * i6 / s        # d/ds
    if rs < rc:
        c1 = (rc2 - rs2) ** -3
        t = s.clamp(min=rs2)
        sw = c1 * (rc2 - t) ** 2 * (rc2 + 2.0 * t - 3.0 * rs2)
        dsw = torch.where(s > rs2, 6.0 * c1 * (rc2 - t) * (rs2 - t), torch.zeros_like(s))
        w, dw = w * sw, dw * sw + w * dsw
    h = (3.0 - s / rc2) / (2.0 * rc)
    erf = torch.erf(beta * r)
    gauss = 2.0 * beta / math.sqrt(math.pi) * torch.exp(-beta * beta * s)
    e = {"vdw": w, "elec": qq * (1.0 / r - h), "slow": qq * (h - erf / r)}
    fast = 2.0 * dw + qq * (rc ** -3 - r ** -3)
    slow = qq * (-(rc ** -3) - (gauss - erf / r) / s)
    return e, fast, slow


def _lj(t, dev):
    dim = t.lj[0]
    return [torch.from_numpy(np.concatenate([s.lj_table()[k] for s in t.systems])).to(dev)
            .reshape(len(t.systems), dim * dim) for k in (1, 2, 3, 4)]


def _add_forces(out, i, j, g, d):
    f = g[:, None] * d
    out.index_add_(0, i, f)
    out.index_add_(0, j, -f)


def _exact_forces(case, t, x, q):
    """Fast and slow forces per slot, and the record per replica."""
    p = t.packed
    dev, n = x.device, len(x)
    tabs = _lj(t, dev)
    dim = t.lj[0]
    types = torch.from_numpy(p.vdwTypes.copy()).to(dev).long()
    rep_of = torch.from_numpy(p.replicaOfCompute.copy()).to(dev).long()
    F, S = (torch.zeros((n, 3), dtype=torch.float64, device=dev) for _ in range(2))
    ve = torch.zeros((max(p.numReplicas, 1), 31), dtype=torch.float64, device=dev)

    def record(rep, e, fast, slow, d):
        dd = (d[:, :, None] * d[:, None, :]).reshape(-1, 9)
        ve[:, 0:9].index_add_(0, rep, -fast[:, None] * dd)
        ve[:, 9:18].index_add_(0, rep, -slow[:, None] * dd)
        for k, name in enumerate(("vdw", "elec", "slow")):
            ve[:, 18 + k].index_add_(0, rep, e[name])

    for i, j, d, c in _pair_chunks(p, x, case["cutoff"] ** 2):
        rep = rep_of[c]
        ty = types[i] * dim + types[j]
        e, fast, slow = _terms(case, (d * d).sum(1), q[i] * q[j], tabs[0][rep, ty], tabs[1][rep, ty])
        _add_forces(F, i, j, fast, d)
        _add_forces(S, i, j, slow, d)
        record(rep, e, fast, slow, d)
    if "c" in case["flags"]:
        rc, beta = case["cutoff"], case["ewaldcof"]
        slot_rep = torch.from_numpy(np.repeat(np.arange(max(p.numReplicas, 1)),
                                              np.diff(p.replicaSlotStart))).to(dev)
        lat = torch.from_numpy(np.ascontiguousarray(p.replicaLattice)).to(dev).double()
        for tuples, mod in ((p.modified, True), (p.excluded, False)):
            if not len(tuples) or (not mod and "s" not in case["flags"]):
                continue
            i, j = (torch.from_numpy(tuples[k].copy()).to(dev).long() for k in ("i", "j"))
            rep = slot_rep[i]
            off = torch.from_numpy(tuples["off"].copy()).to(dev).double()
            d = x[j] - x[i] - (off[:, :, None] * lat[rep]).sum(1)
            s = (d * d).sum(1)
            keep = s < rc * rc
            i, j, d, s, rep = i[keep], j[keep], d[keep], s[keep], rep[keep]
            qq, zero = q[i] * q[j], torch.zeros_like(s)
            r = s.sqrt()
            if mod:
                q14 = (1.0 - t.params.scale14) * qq
                ty = types[i] * dim + types[j]
                e, fast, _ = _terms(case, s, -q14, tabs[2][rep, ty] - tabs[0][rep, ty],
                                    tabs[3][rep, ty] - tabs[1][rep, ty])
                e["slow"] = -q14 * (3.0 - s / rc ** 2) / (2.0 * rc)
                slow = q14 / rc ** 3
            else:
                erf = torch.erf(beta * r)
                gauss = 2.0 * beta / math.sqrt(math.pi) * torch.exp(-beta * beta * s)
                e = {"vdw": zero, "elec": zero, "slow": -qq * erf / r}
                fast, slow = zero, qq * (erf / r - gauss) / s
            _add_forces(F, i, j, fast, d)
            _add_forces(S, i, j, slow, d)
            record(rep, e, fast, slow, d)
    if "e" not in case["flags"]:
        ve[:, 18:21] = 0
    if "v" not in case["flags"]:
        ve[:, 0:18] = 0
    if "s" not in case["flags"]:
        ve[:, 9:18] = 0
        ve[:, 20] = 0
    return F, S, ve


def _float4(f):
    return torch.cat([f, torch.zeros_like(f[:, :1])], 1)


def exact(case, seed):
    s = prepare(case, seed)
    if case["kind"] == "pme":
        return _exact_pme(s)
    t, p = s["topology"], s["packed"]
    if case["kind"] == "migrate":
        return _exact_migrate(s)
    x, q = s["x"][:, :3].double(), s["x"][:, 3].double()
    if case["kind"] == "adjoint":
        return _exact_adjoint(s, x, q)
    F, S, ve = _exact_forces(case, t, x, q)
    out = {"F": _float4(F), "S": _float4(S) if s["slow"] else None}
    if s["wants_ve"]:
        ve = ve if case["kind"] == "batch" else ve[0]
        out["record"] = {k: ve[..., sl] for k, sl in RECORD.items()}
    return out


def _exact_migrate(s):
    """Forces do not depend on the order of the atoms within a patch: they are
    formed in the host's slot order and handed back in buffer order."""
    t, p, layout = s["topology"], s["packed"], s["layout"]
    ids = torch.from_numpy(layout.ids).to(DEVICE).long()
    pos = torch.empty((s["natoms"], 3), dtype=torch.float64, device=DEVICE)
    pos[ids] = torch.stack([layout.dev[k] for k in "xyz"], 1)
    centre = torch.from_numpy(p.patchCenter.copy()).to(DEVICE)
    atom = torch.from_numpy(p.atomIndex.copy()).to(DEVICE).long()
    start = torch.from_numpy(p.patches[:, 2].copy()).to(DEVICE).long()
    patch = torch.searchsorted(start, torch.arange(len(atom), device=DEVICE), right=True) - 1
    x = pos[atom] - centre[patch]
    q = torch.from_numpy(p.xyzq[:, 3].copy()).to(DEVICE).double()
    F, S, _ = _exact_forces(s["case"], t, x, q)
    slot = torch.from_numpy(p.slotOfAtom.copy()).to(DEVICE).long()[ids]
    return {"order": None, "normal": s["bonded"], "nbond": F[slot].T.contiguous(),
            "slow": S[slot].T.contiguous() if s["slow"] else None}


def _exact_adjoint(s, x, q):
    case, t, p = s["case"], s["topology"], s["packed"]
    dim = t.lj[0]
    types = torch.from_numpy(p.vdwTypes.copy()).to(DEVICE).long()
    mask = torch.from_numpy(s["mask"]).to(DEVICE).bool()
    A, B = (a[0].clone().requires_grad_(True) for a in _lj(t, DEVICE)[:2])
    x, q = x.clone().requires_grad_(True), q.clone().requires_grad_(True)
    wF, wS = s["wF"][:, :3].double(), s["wS"][:, :3].double()
    shifted = [(i, j, d.detach() - (x[j] - x[i]).detach())
               for i, j, d, _ in _pair_chunks(p, x.detach(), case["cutoff"] ** 2, chunk=6_000_000)]
    for i, j, sh in shifted:
        d = x[j] - x[i] + sh
        ty = types[i] * dim + types[j]
        fit = (mask[types[i]] | mask[types[j]])
        a = torch.where(fit, A[ty], A.detach()[ty])
        b = torch.where(fit, B[ty], B.detach()[ty])
        e, fast, slow = _terms(case, (d * d).sum(1), q[i] * q[j], a, b)
        loss = (fast * ((wF[i] - wF[j]) * d).sum(1)).sum() + 0.1 * (e["vdw"].sum() + e["elec"].sum())
        if s["slow"]:
            loss = loss + (slow * ((wS[i] - wS[j]) * d).sum(1)).sum() + 0.1 * e["slow"].sum()
        loss.backward()
    return {"grad": torch.cat([x.grad, q.grad[:, None]], 1), "gab": torch.cat([A.grad, B.grad])}


def _spline(w, order):
    """B-spline weights on the points cell + k, k = 0..order-1 (Essmann et al. 1995)."""
    th = [1.0 - w, w]
    for m in range(3, order + 1):
        up = [None] * m
        up[m - 1] = w * th[m - 2] / (m - 1)
        for k in range(1, m - 1):
            up[k] = ((w + (m - 1 - k)) * th[k - 1] + (k + 1 - w) * th[k]) / (m - 1)
        up[0] = (1.0 - w) * th[0] / (m - 1)
        th = up
    return torch.stack(th, 1)


def _exact_pme(s):
    """Smooth PME on the given fractional atoms. A grid coordinate K u is formed
    in 32 bits, as the fractional coordinates come; all that follows is 64-bit."""
    K, order, beta = s["K"], s["case"]["order"], s["case"]["ewaldcof"]
    atoms, L = s["atoms"], np.asarray(s["lattice"])
    vol, R = float(np.linalg.det(L)), np.linalg.inv(L).T
    q = atoms[:, 3].double()
    cell, th, dth = [], [], []
    for d in range(3):
        f = atoms[:, d] * float(K[d])
        c = f.long()
        w = (f - c.float()).double()
        cell.append((c[:, None] + torch.arange(order, device=DEVICE)) % K[d])
        th.append(_spline(w, order))
        low = _spline(w, order - 1)
        z = torch.zeros_like(low[:, :1])
        dth.append(torch.cat([z, low], 1) - torch.cat([low, z], 1))
    grid = torch.zeros(K[0] * K[1] * K[2], dtype=torch.float64, device=DEVICE)

    def at():
        for c in range(order):
            for b in range(order):
                for a in range(order):
                    yield a, b, c, (cell[2][:, c] * K[1] + cell[1][:, b]) * K[0] + cell[0][:, a]

    for a, b, c, where in at():
        grid.index_add_(0, where, q * th[0][:, a] * th[1][:, b] * th[2][:, c])
    hat = torch.fft.rfftn(grid.reshape(K[2], K[1], K[0]))
    k = [torch.arange(n, device=DEVICE, dtype=torch.float64) for n in (K[0] // 2 + 1, K[1], K[2])]
    sg = [k[0]] + [torch.where(k[d] <= K[d] // 2, k[d], k[d] - K[d]) for d in (1, 2)]
    m = [(R[0, d] * sg[0])[None, None, :] + (R[1, d] * sg[1])[None, :, None] + (R[2, d] * sg[2])[:, None, None]
         for d in range(3)]
    msq = m[0] ** 2 + m[1] ** 2 + m[2] ** 2
    msq[0, 0, 0] = 1.0
    mod = []
    for d in range(3):
        w0 = _spline(torch.zeros(1, dtype=torch.float64, device=DEVICE), order)[0]
        arg = 2.0 * math.pi / K[d] * k[d][:, None] * torch.arange(order, device=DEVICE)
        mod.append(1.0 / ((arg.cos() @ w0) ** 2 + (arg.sin() @ w0) ** 2))
    pe = (math.pi / beta) ** 2
    C = torch.exp(-pe * msq) / (math.pi * vol * msq) * mod[0][None, None, :] * mod[1][None, :, None] * mod[2][:, None, None]
    C[0, 0, 0] = 0.0
    weight = torch.full_like(k[0], 2.0)
    weight[0] = 1.0
    if K[0] % 2 == 0:
        weight[K[0] // 2] = 1.0
    fac = weight * (hat.real ** 2 + hat.imag ** 2) * C
    energy = 0.5 * float(fac.sum())
    virial = np.zeros((3, 3))
    for a in range(3):
        for b in range(3):
            v = 2.0 * (pe + 1.0 / msq) * m[a] * m[b] - (1.0 if a == b else 0.0)
            virial[a, b] = -0.5 * float((fac * v).sum())
    phi = (torch.fft.irfftn(hat * C, s=(K[2], K[1], K[0])) * float(K[0] * K[1] * K[2])).reshape(-1)
    f = torch.zeros((len(q), 3), dtype=torch.float64, device=DEVICE)
    for a, b, c, where in at():
        g = phi[where]
        f[:, 0] += dth[0][:, a] * th[1][:, b] * th[2][:, c] * g
        f[:, 1] += th[0][:, a] * dth[1][:, b] * th[2][:, c] * g
        f[:, 2] += th[0][:, a] * th[1][:, b] * dth[2][:, c] * g
    scale = torch.tensor(K, dtype=torch.float64, device=DEVICE)
    force = -q[:, None] * ((f * scale) @ torch.from_numpy(R).to(DEVICE))
    if s["flags"]:
        return {"force": force, "energy": energy, "virial": virial}
    return {"force": force}
