"""What a user of this framework has it do, as calls through the public entry
points of cassandra_gb300: single energies and trial batches, the adjoint,
batched CBMC Widom insertion, and NVT, NPT and grand-canonical chains, in both
precisions.  Sizes are those of the tests, the golden systems and the benchmark.

A state is an opened context with its box loaded and its energies computed, as
a host program holds it between calls; a pass of a chain goes on from the state
that the last one left, with the next seed.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import cassandra_gb300 as cg
from cassandra_gb300 import abi, workloads
from cassandra_gb300.system import CHARGE_FACTOR, KBOLTZ, PI, TWOPI, BoxSpec, ForceField, MoleculeSet, System

ENERGY = [n for n, _ in abi.CassEnergy._fields_]
SIGMA, RHO = 3.73, 0.6  # the benchmark's LJ fluid: sigma and reduced density


def listed():
    return [
        # a host that keeps its own CBMC loop: one stage of 12 trial positions of a
        # three-atom fragment against a 500-atom box, one call per stage
        {"name": "trials_lj500", "kind": "trials", "n": 500, "trials": 12, "fp64": True},
        # the start energy of a small LJ box (the reference's NIST check has 30 to 800 atoms)
        {"name": "energy_lj800", "kind": "energy_lj", "n": 800, "fp64": True},
        # the start energy of 750 SPC/E waters with Ewald (the reference's NIST check)
        {"name": "energy_water750", "kind": "energy_water", "n": 750, "tol": 1e-5, "fp64": True},
        # energy and adjoint of the benchmark's 4096 waters at new coordinates: one
        # configuration of a parameter fit or of a fluctuation-formula run
        {"name": "gradient_water4096", "kind": "gradient", "n": 4096, "tol": 1e-6},
        # a first look at a frame: few insertions into one small box
        {"name": "widom_1box", "kind": "widom", "boxes": 1, "nmin": 300, "nmax": 300, "insertions": 250, "fp64": False},
        # the benchmark's batch: butane into 64 uneven boxes, 10^6 insertions in all
        {"name": "widom_64box", "kind": "widom", "boxes": 64, "nmin": 200, "nmax": 4000, "insertions": 15625,
         "fp64": False},
        # the plain-FP64 path on 16 of such boxes
        {"name": "widom_fp64", "kind": "widom", "boxes": 16, "nmin": 200, "nmax": 4000, "insertions": 1000, "fp64": True},
        # charged insertions: water into 256 waters with Ewald
        {"name": "widom_water", "kind": "widom_water", "n": 256, "insertions": 3000, "fp64": False},
        # one NVT chain of 500 LJ spheres, ten sweeps of translations (an equilibration block)
        {"name": "nvt_lj500", "kind": "nvt_lj", "chains": 1, "n": 500, "sweeps": 10, "fp64": False},
        # one NVT chain of 256 waters with Ewald, translations and rotations, in FP64
        {"name": "nvt_water256_fp64", "kind": "nvt_water", "chains": 1, "n": 256, "sweeps": 2, "fp64": True},
        # grand-canonical butane in 16 half-filled boxes over a range of chemical potentials
        {"name": "gcmc_butane16", "kind": "gcmc", "boxes": 16, "n": 200, "steps": 1000, "fp64": False},
        # NPT of the benchmark's 4096 waters: a quarter of a sweep and a volume move
        {"name": "npt_water4096", "kind": "npt", "n": 4096, "tol": 1e-6, "moves": 1024},
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["trials", "energy_lj", "energy_water", "gradient", "widom", "widom", "widom_water", "nvt_lj",
                       "nvt_water", "gcmc"])
    fp64 = rng.random() < 0.5
    if kind == "trials":
        return {"kind": kind, "n": log_int(100, 4000), "trials": rng.randint(1, 32), "fp64": fp64}
    if kind == "energy_lj":
        return {"kind": kind, "n": log_int(30, 4000), "fp64": fp64}
    if kind == "energy_water":
        return {"kind": kind, "n": log_int(100, 2000), "tol": 1e-5, "fp64": fp64}
    if kind == "gradient":
        return {"kind": kind, "n": log_int(64, 4000), "tol": rng.choice([1e-5, 1e-6])}
    if kind == "widom":
        boxes = log_int(1, 16 if fp64 else 48)
        lo = log_int(200, 1500)
        return {"kind": kind, "boxes": boxes, "nmin": lo, "nmax": rng.randint(lo, 4000),
                "insertions": log_int(64, 1000 if fp64 else 12000), "fp64": fp64}
    if kind == "widom_water":
        return {"kind": kind, "n": log_int(100, 500), "insertions": log_int(64, 1500 if fp64 else 3000), "fp64": fp64}
    if kind == "nvt_lj":
        return {"kind": kind, "chains": log_int(1, 64 if fp64 else 304), "n": log_int(100, 800), "sweeps": rng.randint(1, 4), "fp64": fp64}
    if kind == "nvt_water":
        return {"kind": kind, "chains": log_int(1, 16 if fp64 else 96), "n": log_int(64, 300), "sweeps": 1, "fp64": fp64}
    return {"kind": "gcmc", "boxes": log_int(1, 32), "n": log_int(50, 250), "steps": log_int(50, 500 if not fp64 else 100),
            "fp64": fp64}


# -- boxes ----------------------------------------------------------------------

def lj_positions(sizes, lengths, min_dist, rng):
    """Random sequential addition in every box at once, in rounds: sizes[b] points of
    [-L/2, L/2)^3 at least min_dist apart.  A cell is too small for two of them."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    want, length = (torch.tensor(np.asarray(v), device=dev) for v in (sizes, lengths))
    nc = (length * (1.7321 / min_dist)).long() + 1
    base = torch.cumsum(nc ** 3, 0) - nc ** 3
    taken = torch.full((int((nc ** 3).sum()),), -1, dtype=torch.int64, device=dev)
    off = torch.cartesian_prod(*[torch.arange(-2, 3, device=dev)] * 3)
    off = off[off.any(1)]
    pos, box = torch.zeros((0, 3), dtype=torch.float64, device=dev), torch.zeros(0, dtype=torch.int64, device=dev)

    def clash(p, bx, grid, at, before):  # a point of `at` within min_dist (with `before`: an earlier one of the same list)
        L, n = length[bx], nc[bx]
        c = torch.minimum(((p / L[:, None] + 0.5) * n[:, None]).long(), n[:, None] - 1)
        hit = torch.zeros(len(p), dtype=torch.bool, device=dev)
        for o in off if before else torch.cat([off, off[:1] * 0]):
            w = torch.remainder(c + o, n[:, None])
            j = grid[base[bx] + (w[:, 0] * n + w[:, 1]) * n + w[:, 2]]
            d = p - at[j.clamp(min=0)] if len(at) else p + 9e9
            d = d - L[:, None] * torch.round(d / L[:, None])
            near = (j >= 0) & ((d * d).sum(1) < min_dist ** 2)
            hit |= near & (j < torch.arange(len(p), device=dev)) if before else near
        return hit

    def cell(p, bx):
        L, n = length[bx, None], nc[bx, None]
        c = torch.minimum(((p / L + 0.5) * n).long(), n - 1)
        return base[bx] + (c[:, 0] * n[:, 0] + c[:, 1]) * n[:, 0] + c[:, 2]

    for _ in range(1000):
        left = want - torch.bincount(box, minlength=len(want))
        if not bool((left > 0).any()):
            order = torch.argsort(box, stable=True)
            return [v.cpu().numpy() for v in torch.split(pos[order], [int(w) for w in want])]
        bx = torch.repeat_interleave(torch.arange(len(want), device=dev), torch.where(left > 0, left + 16, 0 * left))
        p = torch.tensor(rng.random((len(bx), 3)) - 0.5, device=dev) * length[bx, None]
        ok = ~clash(p, bx, taken, pos, False)
        p, bx = p[ok], bx[ok]
        here, first = np.unique(cell(p, bx).cpu().numpy(), return_index=True)  # one of a cell's points, the first
        p, bx = (v[torch.tensor(np.sort(first), device=dev)] for v in (p, bx))
        new = torch.full_like(taken, -1)
        new[cell(p, bx)] = torch.arange(len(p), device=dev)
        ok = ~clash(p, bx, new, p, True)
        p, bx = p[ok], bx[ok]
        start = torch.cumsum(torch.bincount(bx, minlength=len(want)), 0) - torch.bincount(bx, minlength=len(want))
        ok = torch.arange(len(p), device=dev) - start[bx] < left[bx]  # no more than the box still wants
        p, bx = p[ok], bx[ok]
        taken[cell(p, bx)] = len(pos) + torch.arange(len(p), device=dev)
        pos, box = torch.cat([pos, p]), torch.cat([box, bx])
    raise RuntimeError("could not place all spheres")


def rotations(n, rng):
    q = rng.normal(size=(n, 4))
    a, b, c, d = (q / np.linalg.norm(q, axis=1, keepdims=True)).T
    return np.stack([a * a + b * b - c * c - d * d, 2 * (b * c - a * d), 2 * (b * d + a * c),
                     2 * (b * c + a * d), a * a - b * b + c * c - d * d, 2 * (c * d - a * b),
                     2 * (b * d - a * c), 2 * (c * d + a * b), a * a - b * b - c * c + d * d], -1).reshape(n, 3, 3)


def on_lattice(base, mass, n, length, min_dist, rng):
    """n rigid copies of `base` on a cubic lattice, orientations drawn anew until no two
    neighbours come closer than min_dist; [n, atoms, 3]."""
    side = int(math.ceil(n ** (1.0 / 3.0) - 1e-9))
    base = base - (base * mass[:, None]).sum(0) / mass.sum()
    site = np.arange(n)
    ijk = np.stack([site // (side * side), site // side % side, site % side], -1)
    com = (ijk + 0.5) * (length / side) - 0.5 * length
    xyz = com[:, None] + base @ rotations(n, rng).transpose(0, 2, 1)
    off = [o for o in np.ndindex(3, 3, 3) if o > (1, 1, 1)]
    for _ in range(200):
        bad = np.zeros(n, dtype=bool)
        for o in off:
            j3 = (ijk + np.array(o) - 1) % side
            j = (j3[:, 0] * side + j3[:, 1]) * side + j3[:, 2]
            i = np.flatnonzero((j < n) & (j != site))
            d = xyz[i][:, :, None] - xyz[j[i]][:, None]
            d -= length * np.round(d / length)
            bad[i[((d ** 2).sum(-1) < min_dist ** 2).any((1, 2))]] = True
        if not bad.any():
            break
        xyz[bad] = com[bad][:, None] + base @ rotations(int(bad.sum()), rng).transpose(0, 2, 1)
    return xyz


def water_spec(c):
    n = c["n"]
    length = 19.7 * (n / 256.0) ** (1.0 / 3.0) if c["kind"] not in ("gradient", "npt") else 49.7 * (n / 4096.0) ** (1.0 / 3.0)
    rcut = min(12.0 if c["kind"] in ("gradient", "npt") else 9.8, 0.49 * length)
    return BoxSpec(length=(length,) * 3, rcut_vdw=rcut, rcut_coul=rcut, rcut_cbmc=min(6.5, rcut), rcut_low=0.85,
                   charge_style=abi.CHARGE_COUL, charge_sum_style=abi.QQ_EWALD, ewald_tol=c.get("tol", 1e-5),
                   temperature=298.0)


def system_of(c, seed):
    """(System without molecules, im, is, ibox, xyz): the boxes of a case and where their molecules stand."""
    rng = np.random.default_rng(seed)
    kind = c["kind"]
    if kind in ("energy_water", "gradient", "widom_water", "nvt_water", "npt"):
        sp, nb, n = workloads.water_species(), c.get("chains", 1), c["n"]
        boxes = [water_spec(c)] * nb
        mass = np.array([a.mass for a in sp.atoms])
        xyz = [on_lattice(sp.libraries[0][0], mass, n, boxes[0].length[0], 1.5, rng) for _ in range(nb)]
        im, is_ = np.arange(1, n * nb + 1), np.ones(n * nb)
        species, most = [sp], [n * nb + (1 if kind == "widom_water" else 0)]
    elif kind == "gcmc":
        sp, nb, n = workloads.butane_species(300.0, 1000, seed), c["boxes"], c["n"]
        boxes = [BoxSpec(length=(40.0,) * 3, rcut_vdw=14.0, rcut_cbmc=6.5, rcut_low=1.0, temperature=300.0)] * nb
        th = math.radians(114.0)  # the all-trans chain
        a = np.array([0.5 * th, -0.5 * th, 0.5 * th]) + 0.5 * PI - 0.5 * th
        step = 1.54 * np.stack([np.cos(a - a.mean()), np.sin(a - a.mean()), 0 * a], -1)
        base = np.concatenate([np.zeros((1, 3)), np.cumsum(step, 0)])
        mass = np.array([a.mass for a in sp.atoms])
        xyz = [on_lattice(base, mass, n, 40.0, 2.5, rng) for _ in range(nb)]
        im, is_ = np.arange(1, n * nb + 1), np.ones(n * nb)
        species, most = [sp], [(2 * n + 200) * nb]
    else:
        sp = workloads.lj_sphere_species()
        lj = {"rcut": 14.0, "low": 1.0, "length": lambda n: 35.0 * (n / 500.0) ** (1.0 / 3.0)}
        if kind in ("widom", "trials"):
            lj = {"rcut": 14.0, "low": 2.0, "length": lambda n: (n / RHO) ** (1.0 / 3.0) * SIGMA}
        sizes = rng.integers(c["nmin"], c["nmax"] + 1, c["boxes"]) if kind == "widom" else [c["n"]] * c.get("chains", 1)
        lengths = [lj["length"](int(n)) for n in sizes]
        xyz = [x[:, None] for x in lj_positions(sizes, lengths, 0.8 * SIGMA, rng)]
        boxes = [BoxSpec(length=(v,) * 3, rcut_vdw=min(lj["rcut"], 0.5 * v), rcut_cbmc=6.5, rcut_low=lj["low"],
                         temperature=150.0) for v in lengths]
        total = sum(len(x) for x in xyz)
        im, is_ = np.arange(1, total + 1), np.ones(total)
        species, most = [sp], [total]
        if kind in ("widom", "trials"):
            species, most = [sp, workloads.butane_species(150.0, 1000, seed + 1)], [total, 1]
    ibox = np.repeat(np.arange(1, len(boxes) + 1), [len(x) for x in xyz])
    s = System(species, boxes, MoleculeSet(), ForceField(species), most)
    return s, im, is_, ibox, np.concatenate([x.ravel() for x in xyz])


def trial_positions(c, s, seed):
    """[trials, 3, 3]: the first fragment of butane at random centres and orientations."""
    rng = np.random.default_rng([seed, 1])
    lib = s.species[1].libraries[0]
    f = lib[rng.integers(0, len(lib), c["trials"])]
    f = f - f.mean(1, keepdims=True)
    cen = (rng.random((c["trials"], 1, 3)) - 0.5) * s.boxes[0].length[0]
    return f @ rotations(c["trials"], rng).transpose(0, 2, 1) + cen


def prepare(case, seed):
    c = case
    s, im, is_, ibox, xyz = system_of(c, seed)
    fp64 = c["kind"] == "gradient" or c.get("fp64", False)
    ctx = cg.open_system(s, precision=abi.PREC_FP64 if fp64 else abi.PREC_MIXED)
    ctx.set_molecules(im, is_, ibox, xyz)
    st = {"case": c, "ctx": ctx, "seed": seed, "pass": 0, "boxes": list(range(1, len(s.boxes) + 1)),
          "mol": (im.astype(np.int32), is_.astype(np.int32), ibox.astype(np.int32), xyz)}
    if c["kind"] == "trials":
        st["xyz"] = trial_positions(c, s, seed)
        return st
    if c["kind"] not in ("energy_lj", "energy_water", "gradient"):
        for b in st["boxes"]:
            ctx.system_total_energy(b)
    ns = len(s.species)
    st["disp"], st["rot"] = [[0.8] * ns] * len(s.boxes), [[0.4] * ns] * len(s.boxes)
    if c["kind"] == "npt":
        st["length"] = s.boxes[0].length[0]
    if c["kind"] == "gcmc":
        st["mu"] = list(np.linspace(-30.0, -20.0, len(s.boxes)))
    return st


def energy_row(e):
    return [e[n] for n in ENERGY]


def chain_outputs(st, res):
    """Energies and counters per chain, and where the molecules of a single NVT or NPT chain stand."""
    out = {"energy": np.array([energy_row(r["energy"]) for r in res]),
           "counts": np.array([[v for k, v in r.items() if k.startswith("n_")] for r in res], dtype=np.int64)}
    if len(res) == 1 and st["case"]["kind"] != "gcmc":
        im, is_ = st["mol"][0], st["mol"][1]
        out["xyz"] = np.concatenate([st["ctx"].get_molecule(int(m), int(s)) for m, s in zip(im, is_)])
    return out


def run(state):
    st = state
    c, ctx = st["case"], st["ctx"]
    kind, seed = c["kind"], st["seed"] * 1000 + st["pass"]
    st["pass"] += 1
    if kind == "trials":
        e, ov = ctx.cbmc_trial_energies(1, 2, [2, 1, 3], st["xyz"])
        return {"e": e, "overlap": ov}
    if kind in ("energy_lj", "energy_water"):
        e, ov = ctx.system_total_energy(1)
        return {"energy": np.array(energy_row(e)), "overlap": ov}
    if kind == "gradient":  # a new configuration comes in, energy and derivatives go out
        ctx.set_molecules(*st["mol"])
        e, g, de, ds, dq = ctx.system_gradient(1, 3 * c["n"])
        return {"energy": np.array(energy_row(e)), "dr": g, "deps": de, "dsig": ds, "dq": dq}
    if kind in ("widom", "widom_water"):
        water, small = kind == "widom_water", c["insertions"] * c.get("boxes", 1) <= 100000
        # every insertion's record where there are few, as an analysis of the distribution reads it
        r = ctx.widom_insert(1 if water else 2, st["boxes"], c["insertions"], 12, 12, seed=seed, trace=small)
        r, tr = r if small else (r, None)
        out = {"sum": np.array([x["widom_sum"] for x in r]), "prefactor": np.array([x["prefactor"] for x in r]),
               "counts": np.array([[x["n_insertions"], x["n_overlaps"], x["n_trials"]] for x in r], dtype=np.int64)}
        if small:
            out.update({k: tr[k] for k in ("widom_var", "ln_pbias", "e_inter", "selected_trial", "overlap")})
        return out
    if kind in ("nvt_lj", "nvt_water"):
        res, st["disp"], st["rot"] = ctx.mc_sweeps(st["boxes"], c["sweeps"], st["disp"], st["rot"], seed=seed,
                                                   prob_translate=1.0 if kind == "nvt_lj" else 0.5)
        return chain_outputs(st, res)
    if kind == "npt":
        res, st["disp"], st["rot"] = ctx.mc_sweeps([1], 1, st["disp"], st["rot"], seed=seed, prob_translate=0.5,
                                                   steps_per_sweep=c["moves"])
        e, ov = ctx.volume_scale(1, st["length"] * (1.001 if st["pass"] % 2 else 1.0))
        return chain_outputs(st, res) | {"scaled": np.array(energy_row(e)), "overlap": ov}
    res = ctx.gcmc(st["boxes"], c["steps"], 1, st["mu"], [[1.0]] * c["boxes"], [[0.5]] * c["boxes"], seed=seed)
    where = ctx.molecule_boxes(1)
    xyz = np.zeros((len(where), 4, 3))
    for m in np.flatnonzero(where):
        xyz[m] = ctx.get_molecule(int(m) + 1, 1)
    return chain_outputs(st, res) | {"boxes": where, "xyz": xyz}


# -- what a pass cannot do without -------------------------------------------------

def in_sphere(rho, r):
    return rho * 4.0 / 3.0 * math.pi * r ** 3


def n_kvectors(b):
    p = -math.log(b.ewald_tol)
    h = 2.0 * p / b.rcut_coul
    return 0.5 * 4.0 / 3.0 * math.pi * (h * b.length[0] / (2.0 * math.pi)) ** 3


def work(case):
    """Atoms and results once each; 15 operations for a distance and 8 for a Lennard-Jones
    pair within its cutoff (about 40 for a charged one), 8 for a k-vector and atom."""
    c, kind = case, case["kind"]
    water = kind in ("energy_water", "gradient", "widom_water", "nvt_water", "npt")
    if water:
        b = water_spec(c)
        n = 3 * c["n"]
        rho, nk = n / b.volume, n_kvectors(b)
        near = in_sphere(rho, b.rcut_coul)
        sys_flops = n * near / 2 * 60.0 + nk * n * 8.0
        sys_bytes = 32.0 * n + 8 * 14
        if kind == "energy_water":
            return {"bytes": sys_bytes, "flops": sys_flops}
        if kind == "gradient":
            return {"bytes": sys_bytes + 24.0 * n, "flops": 2 * n * near / 2 * 60.0 + 3 * nk * n * 8.0}
        if kind == "widom_water":
            per = 3 * near * 60.0 + 12 * 3 * in_sphere(rho, b.rcut_cbmc) * 23.0 * 0.25 + nk * 30.0
            return {"bytes": sys_bytes + 48.0 * c["insertions"], "flops": c["insertions"] * per}
        moves = c["moves"] if kind == "npt" else c["n"] * c["sweeps"] * c["chains"]
        per = 2 * 3 * near * 60.0 + nk * 40.0  # old and new pair sums, one set of phases
        w = {"bytes": 24.0 * n * c.get("chains", 1) + moves * nk * 16.0, "flops": moves * per}
        return {"bytes": w["bytes"] + sys_bytes, "flops": w["flops"] + sys_flops} if kind == "npt" else w
    rho = RHO / SIGMA ** 3
    if kind == "trials":
        return {"bytes": 32.0 * c["n"] + 80.0 * c["trials"], "flops": c["trials"] * 3 * in_sphere(rho, 6.5) * 23.0}
    if kind == "gcmc":
        rho = 4 * c["n"] / 40.0 ** 3
        moves = c["steps"] * c["boxes"]
        per = 0.4 * 2 * 4 * in_sphere(rho, 14.0) * 23.0 + 0.6 * (4 * in_sphere(rho, 14.0) + 48 * in_sphere(rho, 6.5)) * 23.0
        return {"bytes": 96.0 * c["n"] * c["boxes"], "flops": moves * per}
    if kind == "widom":
        n, box = 0.5 * (c["nmin"] + c["nmax"]), (0.5 * (c["nmin"] + c["nmax"]) / rho) ** (1.0 / 3.0)
        per = (4 * in_sphere(rho, min(14.0, 0.5 * box)) + 29 * in_sphere(rho, 6.5)) * 23.0
        return {"bytes": c["boxes"] * (16.0 * n + 33.0 * c["insertions"]), "flops": c["boxes"] * c["insertions"] * per}
    rho = 500 / 35.0 ** 3
    near = in_sphere(rho, min(14.0, 0.5 * (c["n"] / rho) ** (1.0 / 3.0)))
    if kind == "energy_lj":
        return {"bytes": 32.0 * c["n"], "flops": c["n"] * near / 2 * 23.0}
    moves = c["n"] * c["sweeps"] * c["chains"]
    return {"bytes": 24.0 * c["n"] * c["chains"], "flops": moves * 2 * near * 23.0}


# -- the same numbers from plain torch in 64 bits ------------------------------------

def exact(case, seed):
    """Energies, trial energies and the adjoint; the chains and the Widom insertions are
    sequences of random decisions and have no such value."""
    if case["kind"] not in ("trials", "energy_lj", "energy_water", "gradient"):
        return None
    s, _, _, _, xyz = system_of(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    f64 = {"dtype": torch.float64, "device": dev}
    b, ff = s.boxes[0], s.ff
    length = b.length[0]

    def fold(d):
        return torch.where(d > 0.5 * length, d - length, torch.where(d < -0.5 * length, d + length, d))

    if case["kind"] == "trials":
        x, t = torch.tensor(xyz.reshape(-1, 3), **f64), torch.tensor(trial_positions(case, s, seed), **f64)
        d = fold(t[:, :, None] - x)
        r2 = (d * d).sum(-1)
        k = [s.species[1].type_index[a - 1] - 1 for a in (2, 1, 3)]
        eps, sig = (torch.tensor(v[k, 0], **f64)[None, :, None] for v in (ff.eps, ff.sig))
        s6 = (sig * sig / r2) ** 3
        e = torch.where(r2 <= b.rcut_cbmc ** 2, 4.0 * eps * (s6 * s6 - s6), 0.0 * r2).sum((1, 2))
        ov = (r2 < b.rcut_low ** 2).any(2).any(1)
        return {"e": torch.where(ov, 0.0 * e, e).cpu().numpy(), "overlap": ov.cpu().numpy()}

    sp = s.species[0]
    na, n = sp.natoms, len(xyz) // 3
    x = torch.tensor(xyz.reshape(-1, 3), **f64).requires_grad_(True)
    eps, sig = (torch.tensor(v, **f64).requires_grad_(True) for v in (ff.eps, ff.sig))
    qs = torch.tensor([a.charge for a in sp.atoms], **f64).requires_grad_(True)
    ty = torch.tensor([t - 1 for t in sp.type_index], device=dev)
    atom = torch.arange(n, device=dev) % na
    rc = max(b.rcut_vdw, b.rcut_coul)
    pi, pj = [], []
    with torch.no_grad():  # the pairs within the cutoff, j > i
        for i0 in range(0, n, 2048):
            d = fold(x[i0:i0 + 2048, None] - x)
            i, j = torch.nonzero((d * d).sum(-1) <= rc * rc * (1 + 1e-9), as_tuple=True)
            keep = j > i + i0
            pi.append(i[keep] + i0)
            pj.append(j[keep])
    pi, pj = torch.cat(pi), torch.cat(pj)
    inter = torch.div(pi, na, rounding_mode="floor") != torch.div(pj, na, rounding_mode="floor")
    e = {k: torch.zeros((), **f64) for k in ENERGY}
    alpha = math.sqrt(-math.log(b.ewald_tol)) / b.rcut_coul if na > 1 else 0.0

    def pairs(i, j, intra):
        d = x[i] - x[j]
        d = d if intra else fold(d)
        r2 = (d * d).sum(-1)
        ti, tj = ty[atom[i]], ty[atom[j]]
        if not intra:
            s6 = (sig[ti, tj] ** 2 / r2) ** 3
            e["inter_vdw"] = e["inter_vdw"] + torch.where(r2 <= b.rcut_vdw ** 2, 4 * eps[ti, tj] * (s6 * s6 - s6), 0 * r2).sum()
        if na > 1:  # Abramowitz and Stegun 7.1.26, the erfc that the energy is defined with
            r = torch.sqrt(r2)
            t = 1.0 / (1.0 + 0.3275911 * alpha * r)
            f = t * (0.254829592 + t * (-0.284496736 + t * (1.421413741 + t * (-1.453152027 + t * 1.061405429)))) * \
                torch.exp(-(alpha * r) ** 2)
            v = CHARGE_FACTOR * qs[atom[i]] * qs[atom[j]] / r * (f - 1.0 if intra else f)
            e["inter_q"] = e["inter_q"] + torch.where(r2 <= b.rcut_coul ** 2, v, 0 * v).sum()

    pairs(pi[inter], pj[inter], False)
    if na > 1:
        pairs(pi[~inter], pj[~inter], True)
    nb = torch.bincount(ty, minlength=ff.ntypes).double() * (n // na)
    e["lrc"] = 2 * PI / b.volume * (nb[:, None] * nb * 4 * eps * (sig ** 12 / (9 * b.rcut_vdw ** 9) -
                                                                  sig ** 6 / (3 * b.rcut_vdw ** 3))).sum()
    grad = case["kind"] == "gradient"
    if na > 1:
        e["self"] = -CHARGE_FACTOR * alpha / 1.7724538509 * (qs * qs).sum() * (n // na)
        hcut = -2.0 * math.log(b.ewald_tol) / b.rcut_coul
        m = int(hcut * length / TWOPI) + 1
        k = torch.cartesian_prod(torch.arange(-m, m + 1, device=dev), torch.arange(-m, m + 1, device=dev),
                                 torch.arange(0, m + 1, device=dev)).flip(-1).double()
        h = TWOPI * k / length
        h2 = (h * h).sum(-1)
        keep = (h2 < hcut * hcut) & (h2 > 0)
        h, h2, k = h[keep], h2[keep], k[keep]
        cn = (1.0 + (k[:, 0] != 0).double()) * TWOPI / b.volume * torch.exp(-h2 / (4 * alpha * alpha)) / h2
        for a in range(0, len(h), 1024):
            ph = h[a:a + 1024] @ x.T
            q = qs[atom]
            er = CHARGE_FACTOR * (cn[a:a + 1024] * (((torch.cos(ph) * q).sum(1)) ** 2 + ((torch.sin(ph) * q).sum(1)) ** 2)).sum()
            if grad:
                er.backward()
            e["reciprocal"] = e["reciprocal"] + er.detach()
    e["inter"] = e["inter_vdw"] + e["inter_q"] + e["lrc"] + e["self"] + e["reciprocal"]
    e["total"] = e["inter"] + 0.0
    row = np.array([float(e[k].detach()) for k in ENERGY])
    if not grad:
        return {"energy": row, "overlap": False}
    (e["inter_vdw"] + e["inter_q"] + e["lrc"] + e["self"]).backward()

    def pair_entries(g):  # the derivative of a symmetric pair parameter, in both of its entries
        return (g + g.T - torch.diag(torch.diag(g))).cpu().numpy()

    return {"energy": row, "dr": x.grad.cpu().numpy(), "deps": pair_entries(eps.grad), "dsig": pair_entries(sig.grad),
            "dq": qs.grad.cpu().numpy()}
