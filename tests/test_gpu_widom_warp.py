"""The warp-wide neighbour queries of the mixed Widom kernel where their branches
change: boxes whose stencils span the box (cell rows, folded), boxes that use the
voxel lists for the CBMC radius only or for both radii, an uneven and a
non-cubic box (empty and long lists), and insertion counts around a warp.  Each
insertion against the FP64 oracle: the same status and selected trial, energies
within 2e-5 of the sum of |pair energies| -- the rounding of FP32 coordinates
(1e-6 A) on steep pairs."""
import numpy as np
import pytest

import cassandra_gb300 as cg
from cassandra_gb300 import abi, workloads
from cassandra_gb300.system import BoxSpec, ForceField, MoleculeSet, System
from oracle import oracle

pytestmark = pytest.mark.gpu


def _system(boxes):
    """boxes: (number of spheres, edges, filled fraction of the x edge)."""
    rng = np.random.default_rng(5)
    solvent, solute = workloads.lj_sphere_species(), workloads.butane_species(150.0, 200, 8)
    ms, specs, loc = MoleculeSet(), [], 1
    for b, (n, edges, part) in enumerate(boxes):
        edges = np.asarray(edges, dtype=float)
        side = max(edges)
        spots = workloads.lj_fluid_box(int(n * side ** 3 / (np.prod(edges) * part)) + 1, side, 2.984, rng)
        # a shorter edge leaves out the last 1.1 A, so that no two images come within rcut_low
        keep = (np.abs(spots) <= np.where(edges < side, 0.5 * edges - 1.1, 0.5 * side)).all(1) & (spots[:, 0] < (part - 0.5) * edges[0])
        for p in spots[keep][:n]:
            ms.add(loc, 1, b + 1, p[None])
            loc += 1
        specs.append(BoxSpec(length=tuple(edges), rcut_vdw=min(14.0, 0.5 * min(edges)), rcut_cbmc=6.5, rcut_low=2.0,
                             temperature=150.0))
    return System([solvent, solute], specs, ms, ForceField([solvent, solute]), [loc - 1, 1])


@pytest.mark.parametrize("n_ins", [1, 31, 33, 700])
@pytest.mark.parametrize("boxes", [
    [(180, (20.0, 20.0, 20.0), 1.0)],                                  # three cells a side: rows, folded
    [(300, (29.6, 29.6, 29.6), 1.0), (1, (40.0, 40.0, 40.0), 1.0)],    # lists for the CBMC radius; one atom
    [(1300, (48.3, 48.3, 48.3), 1.0)],                                 # lists for both radii
    [(500, (60.0, 50.0, 50.0), 0.4), (700, (30.0, 45.0, 52.0), 1.0)],  # uneven; not cubic
])
def test_widom_warp_queries(boxes, n_ins):
    s = _system(boxes)
    ids = list(range(1, len(boxes) + 1))
    with oracle.open_system(s) as o, cg.open_system(s, precision=abi.PREC_MIXED) as m:
        for b in ids:
            o.system_total_energy(b)
            m.system_total_energy(b)
        ro, to = o.widom_insert(2, ids, n_ins, 12, 12, seed=77, trace=True)
        rm, tm = m.widom_insert(2, ids, n_ins, 12, 12, seed=77, trace=True)
        again, ta = m.widom_insert(2, ids, n_ins, 12, 12, seed=77, trace=True)
    assert again == rm and ta.tobytes() == tm.tobytes()
    assert np.array_equal(to["overlap"], tm["overlap"])
    assert np.array_equal(to["selected_trial"], tm["selected_trial"])
    ok = to["overlap"] == 0
    assert (np.abs(tm["e_inter"] - to["e_inter"])[ok] <= 2e-5 * to["e_inter_abs"][ok] + 1e-7).all()
    assert [r["n_overlaps"] for r in rm] == [r["n_overlaps"] for r in ro]


@pytest.mark.parametrize("n_ins", [1, 33, 400])
@pytest.mark.parametrize("boxes", [
    [(180, (20.0, 20.0, 20.0), 1.0), (0, (30.0, 30.0, 30.0), 1.0)],    # cutoff of half the edge: two images listed; no atoms
    [(1300, (48.3, 48.3, 48.3), 1.0), (1, (40.0, 40.0, 40.0), 1.0)],
    [(500, (60.0, 50.0, 50.0), 0.4), (700, (30.0, 45.0, 52.0), 1.0)],
])
def test_widom_warp_queries_fp64(boxes, n_ins):
    """The FP64 kernel: equal decisions, energies to the rounding of FP64 sums."""
    s = _system(boxes)
    ids = list(range(1, len(boxes) + 1))
    with oracle.open_system(s) as o, cg.open_system(s, precision=abi.PREC_FP64) as g:
        for b in ids:
            o.system_total_energy(b)
            g.system_total_energy(b)
        ro, to = o.widom_insert(2, ids, n_ins, 12, 7, seed=78, trace=True)
        rg, tg = g.widom_insert(2, ids, n_ins, 12, 7, seed=78, trace=True)
        again, ta = g.widom_insert(2, ids, n_ins, 12, 7, seed=78, trace=True)
    assert again == rg and ta.tobytes() == tg.tobytes()
    assert np.array_equal(to["overlap"], tg["overlap"])
    assert np.array_equal(to["selected_trial"], tg["selected_trial"])
    ok = to["overlap"] == 0
    assert np.allclose(tg["widom_var"][ok], to["widom_var"][ok], rtol=1e-8, atol=0)
    assert (np.abs(tg["e_inter"] - to["e_inter"])[ok] <= 1e-11 * to["e_inter_abs"][ok] + 1e-9).all()
    assert np.allclose(tg["e_inter_abs"][ok], to["e_inter_abs"][ok], rtol=1e-11)
