"""Widom insertions on the routes and at the edges where the kernels' branches change."""
import numpy as np
import pytest

import cassandra_gb300 as cg
from cassandra_gb300 import abi, workloads
from cassandra_gb300.system import Atom, BoxSpec, ForceField, MoleculeSet, Species, System
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("l_coul_cbmc", [False, True])
def test_energy_table_counts_the_charges(l_coul_cbmc):
    """Estimate_MoleculePair_Energy adds the table's Coulomb entry whatever L_Coul_CBMC says.
    The mixed kernel against the oracle: a pair at a bin's edge may fall into the neighbouring
    bin in FP32, everything else agrees."""
    s = workloads.water_nvt_system(nboxes=1, nmol=64, length=12.4, rcut=6.0)
    s.species[0].l_coul_cbmc = l_coul_cbmc
    s.max_molecules = [65]
    with oracle.open_system(s) as o, cg.open_system(s, precision=abi.PREC_MIXED) as m:
        for c in (o, m):
            c.system_total_energy(1)
            c.set_cbmc_options(energy_table_res=1000)
        to = o.widom_insert(1, [1], 600, 12, 12, seed=3, trace=True)[1]
        tm = m.widom_insert(1, [1], 600, 12, 12, seed=3, trace=True)[1]
    both = (to["overlap"] == 0) & (tm["overlap"] == 0)
    assert (to["overlap"] == tm["overlap"]).mean() > 0.99 and both.sum() > 50
    assert (to["selected_trial"] == tm["selected_trial"])[both].mean() > 0.99
    # FP32 sums are within 1e-5 of the terms; the odd pair of the neighbouring bin stays out of the median
    first = np.abs(tm["e_first_trial_sum"] / np.where(both, to["e_first_trial_sum"], 1.0) - 1.0)[both]
    assert np.median(first) < 1e-4


def _rod_system(length=9.6, sites=12, spacing=2.5):
    """Spheres in a small box and a rigid rod that reaches past the neighbouring images."""
    ball = Species(atoms=[Atom("B", 20.0, 0.0, ("LJ", 60.0, 1.6))], scale_vdw=(0, 0, 0, 0), scale_qq=(0, 0, 0, 0),
                   fragments=[[1]], libraries=[np.zeros((1, 1, 3))])
    site = np.zeros((sites, 3))
    site[:, 0] = spacing * np.arange(sites)
    rod = Species(atoms=[Atom("R", 15.0, 0.0, ("LJ", 40.0, 1.4)) for _ in range(sites)], scale_vdw=(0, 0, 0, 0),
                  scale_qq=(0, 0, 0, 0), fragments=[list(range(1, sites + 1))], libraries=[site[None]])
    ms = MoleculeSet()
    for k, p in enumerate(workloads.lj_fluid_box(12, length, 2.0, np.random.default_rng(4))):
        ms.add(k + 1, 1, 1, p[None])
    box = BoxSpec(length=(length,) * 3, rcut_vdw=4.0, rcut_cbmc=3.0, rcut_low=0.7, temperature=200.0)
    return System([ball, rod], [box], ms, ForceField([ball, rod]), [12, 1])


@pytest.mark.parametrize("prec", [abi.PREC_FP64])
def test_atoms_beyond_the_neighbouring_images(prec):
    """A test molecule longer than the box: Minimum_Image_Separation moves a separation by one
    box edge at most, so its far atoms see no box atom, or an image that is not the nearest."""
    s = _rod_system()
    with oracle.open_system(s) as o, cg.open_system(s, precision=prec) as g:
        o.system_total_energy(1)
        g.system_total_energy(1)
        to = o.widom_insert(2, [1], 400, 12, 12, seed=8, trace=True)[1]
        tg = g.widom_insert(2, [1], 400, 12, 12, seed=8, trace=True)[1]
    assert np.array_equal(to["overlap"], tg["overlap"])
    assert np.array_equal(to["selected_trial"], tg["selected_trial"])
    ok = to["overlap"] == 0
    assert ok.sum() > 50
    tol = 1e-11 if prec == abi.PREC_FP64 else 2e-5  # sums of FP64 terms; FP32 coordinates of a few ulps of 2 box edges
    assert (np.abs(tg["e_inter"] - to["e_inter"])[ok] <= tol * to["e_inter_abs"][ok] + 1e-7).all()


def test_far_atoms_in_the_mixed_kernels_rows():
    """The same box with the mixed kernel, whose stencils span it: equal decisions.  (Its FP32
    coordinates of two box edges are too coarse for energies of pairs this steep.)"""
    s = _rod_system()
    with oracle.open_system(s) as o, cg.open_system(s, precision=abi.PREC_MIXED) as m:
        o.system_total_energy(1)
        m.system_total_energy(1)
        to = o.widom_insert(2, [1], 400, 12, 12, seed=8, trace=True)[1]
        tm = m.widom_insert(2, [1], 400, 12, 12, seed=8, trace=True)[1]
    assert np.array_equal(to["overlap"], tm["overlap"])
    assert (to["selected_trial"] == tm["selected_trial"]).mean() >= 0.995


def _alone_and_together(s, prec, is_, n_ins, pick, band=1.0, **opts):
    """Records of box `pick` from a call for it alone and from one for all boxes."""
    ids = list(range(1, len(s.boxes) + 1))
    with cg.open_system(s, precision=prec) as g:
        for b in ids:
            g.system_total_energy(b)
        if opts:
            g.set_cbmc_options(**opts)
        g.set_widom_band(band)
        g.set_widom_autotune(False)
        one, t1 = g.widom_insert(is_, [pick], n_ins, 12, 12, seed=5, trace=True)
        every, ta = g.widom_insert(is_, ids, n_ins, 12, 12, seed=5, trace=True)
    return one[0], t1[0], every[pick - 1], ta[pick - 1]


@pytest.mark.parametrize("prec", [abi.PREC_FP64, abi.PREC_MIXED])
@pytest.mark.parametrize("sizes", [[250] * 40, [1000, 300, 600] * 10])
def test_an_insertion_does_not_depend_on_the_other_boxes(prec, sizes):
    """One insertion per warp in the call for one box, 16 and more in that for all of them."""
    s = workloads.widom_batch_system(nboxes=len(sizes), sizes=sizes, seed=6, nconfig=100)
    one, t1, among, ta = _alone_and_together(s, prec, 2, 2400, 1)
    assert t1.tobytes() == ta.tobytes()
    assert one == among


@pytest.mark.parametrize("opts", [{"energy_table_res": 1000}, {"sector_overlap": True, "rmin_u_max": 300.0},
                                  {"energy_table_res": 1000, "sector_overlap": True, "rmin_u_max": 300.0}])
def test_cbmc_options_in_the_mixed_kernel(opts):
    """The options' queries on the neighbour lists, per insertion: FP32 may put a pair into the
    neighbouring bin of the table or across an r_min, everything else is the oracle's."""
    s = workloads.widom_batch_system(nboxes=2, sizes=[1300, 220], seed=3, nconfig=100)
    with oracle.open_system(s) as o, cg.open_system(s, precision=abi.PREC_MIXED) as m:
        for c in (o, m):
            for b in (1, 2):
                c.system_total_energy(b)
            c.set_cbmc_options(**opts)
        to = o.widom_insert(2, [1, 2], 300, 12, 12, seed=21, trace=True)[1]
        tm = m.widom_insert(2, [1, 2], 300, 12, 12, seed=21, trace=True)[1]
        alone = m.widom_insert(2, [2], 300, 12, 12, seed=21, trace=True)[1]
    assert (to["overlap"] == tm["overlap"]).mean() > 0.98
    assert (to["selected_trial"] == tm["selected_trial"]).mean() > 0.95
    both = (to["overlap"] == 0) & (tm["overlap"] == 0)
    near = np.abs(tm["e_inter"] - to["e_inter"]) <= 2e-5 * to["e_inter_abs"] + 1e-7
    assert near[both].mean() > 0.9 and both.sum() > 100
    assert alone[0].tobytes() == tm[1].tobytes()


def _spheres(edges, n, rng, jitter=0.3):
    """n spheres on a jittered lattice of the box."""
    edges = np.asarray(edges, dtype=float)
    step = (np.prod(edges) / n) ** (1.0 / 3.0)
    sides = np.maximum(1, np.ceil(edges / step - 1e-9)).astype(int)
    grid = np.array(np.meshgrid(*[np.arange(k) for k in sides], indexing="ij")).reshape(3, -1).T
    grid = grid[np.sort(rng.choice(len(grid), min(n, len(grid)), replace=False))]
    return ((grid + 0.5) / sides - 0.5) * edges + rng.uniform(-jitter, jitter, (len(grid), 3))


def _sphere_system(boxes, rcut=14.0, seed=2):
    """boxes: (edges, spheres); butane as the test molecule."""
    rng = np.random.default_rng(seed)
    ball, but = workloads.lj_sphere_species(), workloads.butane_species(150.0, 200, 8)
    ms, specs, k = MoleculeSet(), [], 1
    for b, (edges, n) in enumerate(boxes):
        for p in _spheres(edges, n, rng):
            ms.add(k, 1, b + 1, p[None])
            k += 1
        specs.append(BoxSpec(length=tuple(edges), rcut_vdw=min(rcut, 0.5 * min(edges)), rcut_cbmc=6.5, rcut_low=2.0,
                             temperature=150.0))
    return System([ball, but], specs, ms, ForceField([ball, but]), [k - 1, 1])


def _against_the_oracle(s, prec, n_ins, n_ref, is_=2, seed=31):
    """The first n_ref insertions of every box against the oracle's, the rest unseen."""
    ids = list(range(1, len(s.boxes) + 1))
    with oracle.open_system(s) as o, cg.open_system(s, precision=prec) as g:
        for b in ids:
            g.system_total_energy(b)
            o.system_total_energy(b)
        to = o.widom_insert(is_, ids, n_ref, 12, 12, seed=seed, trace=True)[1]
        tg = g.widom_insert(is_, ids, n_ins, 12, 12, seed=seed, trace=True)[1][:, :n_ref]
    assert np.array_equal(to["overlap"], tg["overlap"])
    same = to["selected_trial"] == tg["selected_trial"]
    assert same.all() if prec == abi.PREC_FP64 else same.mean() >= 0.99  # FP32 weights at a boundary
    ok = (to["overlap"] == 0) & same
    assert ok.sum() >= 0.1 * ok.size
    tol = 1e-11 if prec == abi.PREC_FP64 else 2e-5
    far = np.abs(tg["e_inter"] - to["e_inter"]) > tol * to["e_inter_abs"] + 1e-7
    assert far[ok].mean() <= (0.0 if prec == abi.PREC_FP64 else 0.01)  # another dihedral trial


@pytest.mark.parametrize("prec", [abi.PREC_FP64, abi.PREC_MIXED])
@pytest.mark.parametrize("boxes", [
    [((24.0, 60.0, 50.0), 900)],                         # two full radii span x and no other edge
    [((28.5, 28.5, 28.5), 300), ((13.5, 30.0, 13.2), 60)],  # just above two radii; two CBMC radii just fit
    [((12.4, 12.4, 40.0), 80), ((9.0, 9.0, 9.0), 9)],    # the CBMC radius spans too
])
def test_boxes_of_about_two_radii(prec, boxes):
    _against_the_oracle(_sphere_system(boxes), prec, 300, 300)


@pytest.mark.parametrize("prec", [abi.PREC_FP64, abi.PREC_MIXED])
@pytest.mark.parametrize("boxes", [
    [((400.0, 400.0, 400.0), 500), ((300.0, 60.0, 90.0), 40)],  # voxels wider than a fraction of the radius
    [((1000.0, 1000.0, 30.0), 300), ((60.0, 60.0, 60.0), 1)],
])
def test_dilute_boxes(prec, boxes):
    _against_the_oracle(_sphere_system(boxes), prec, 400, 400)


@pytest.mark.parametrize("prec", [abi.PREC_FP64, abi.PREC_MIXED])
@pytest.mark.parametrize("n", [8000, 14000])
def test_large_boxes(prec, n):
    """A box that leaves room for fewer warps, and one that stays in global memory."""
    edge = (n / 0.6) ** (1.0 / 3.0) * 3.73
    _against_the_oracle(_sphere_system([((edge,) * 3, n)]), prec, 30, 30)


def test_more_than_2_to_the_17_atoms():
    """The mixed kernel on lists against the FP64 one on cells."""
    n = 135000
    edge = (n / 0.6) ** (1.0 / 3.0) * 3.73
    s = _sphere_system([((edge,) * 3, n)])
    t = []
    for prec in (abi.PREC_FP64, abi.PREC_MIXED):
        with cg.open_system(s, precision=prec) as g:
            g.system_total_energy(1)
            t.append(g.widom_insert(2, [1], 50000 if prec == abi.PREC_MIXED else 500, 12, 12, seed=3, trace=True)[1][0, :500])
    assert np.array_equal(t[0]["overlap"], t[1]["overlap"])
    same = t[0]["selected_trial"] == t[1]["selected_trial"]
    ok = (t[0]["overlap"] == 0) & same
    assert same.mean() >= 0.99 and ok.sum() > 50
    far = np.abs(t[1]["e_inter"] - t[0]["e_inter"]) > 5e-5 * t[0]["e_inter_abs"] + 1e-7  # coordinates of 230 A in FP32
    assert far[ok].mean() <= 0.01


@pytest.mark.parametrize("prec", [abi.PREC_FP64, abi.PREC_MIXED])
@pytest.mark.parametrize("edges, n", [((30.0, 34.0, 32.0), 380), ((20.0, 19.0, 21.0), 90), ((45.0, 45.0, 45.0), 1000)])
def test_full_warps(prec, edges, n):
    """A call of 32 insertions per warp: the records of the oracle, and the bits of a short call."""
    s = _sphere_system([(edges, n)])
    n_ins = 130000 if prec == abi.PREC_MIXED else 60000
    _against_the_oracle(s, prec, n_ins, 300)
    with cg.open_system(s, precision=prec) as g:
        g.system_total_energy(1)
        few = g.widom_insert(2, [1], 2500, 12, 12, seed=4, trace=True)[1][0]
        many = g.widom_insert(2, [1], n_ins, 12, 12, seed=4, trace=True)[1][0][:2500]
    assert few.tobytes() == many.tobytes()


def test_full_warps_of_charged_insertions():
    """Charges with a Coulomb cutoff other than the vdW one, in a box that has lists for both
    radii: the charged band notes and terms of the lists."""
    s = workloads.water_nvt_system(nboxes=1, nmol=1100, length=33.0, rcut=9.0)
    s.boxes[0].rcut_vdw = 8.2
    s.max_molecules = [1101]
    _against_the_oracle(s, abi.PREC_MIXED, 2000, 250, is_=1)
    with cg.open_system(s, precision=abi.PREC_MIXED) as g:
        g.system_total_energy(1)
        few = g.widom_insert(1, [1], 1500, 12, 12, seed=4, trace=True)[1][0]
        assert g.stats()["widom_fixups"] > 10
        g.set_widom_band(30.0)
        wide = g.widom_insert(1, [1], 1500, 12, 12, seed=4, trace=True)[1][0]
        assert g.stats()["widom_fixups"] > 500
    ok = few["overlap"] == 0
    assert np.array_equal(few["overlap"], wide["overlap"])
    assert (np.abs(few["e_inter"] - wide["e_inter"])[ok] <= 1e-6 * few["e_inter_abs"][ok] + 1e-7).all()


def test_band_notes_do_not_depend_on_the_other_boxes():
    """Bands so wide that a full warp meets more pairs in them than it had room for."""
    s = workloads.widom_batch_system(nboxes=30, sizes=[1000, 300, 600] * 10, seed=6, nconfig=100)
    one, t1, among, ta = _alone_and_together(s, abi.PREC_MIXED, 2, 4000, 1, band=60.0)
    assert t1.tobytes() == ta.tobytes()
    assert one == among


def test_batches_of_more_lists_than_fit():
    """40 boxes of 20,000 atoms need more than 4 GB of lists: worked off in pieces, every box as alone."""
    edge = (20000 / 0.6) ** (1.0 / 3.0) * 3.73
    spots = _spheres((edge,) * 3, 20000, np.random.default_rng(1))
    ball, but = workloads.lj_sphere_species(), workloads.butane_species(150.0, 200, 8)
    nb = 40
    box = BoxSpec(length=(edge,) * 3, rcut_vdw=14.0, rcut_cbmc=6.5, rcut_low=2.0, temperature=150.0)
    s = System([ball, but], [box] * nb, MoleculeSet(), ForceField([ball, but]), [nb * len(spots), 1])
    n_ins = 22000
    with cg.open_system(s, precision=abi.PREC_MIXED) as g:
        g.set_molecules(np.arange(1, nb * len(spots) + 1), np.ones(nb * len(spots)), np.repeat(np.arange(1, nb + 1), len(spots)),
                        np.tile(spots.ravel(), nb))
        for b in range(1, nb + 1):
            g.system_total_energy(b)
        every, ta = g.widom_insert(2, list(range(1, nb + 1)), n_ins, 4, 4, seed=5, trace=True)
        for b in (1, 21, nb):
            one, t1 = g.widom_insert(2, [b], n_ins, 4, 4, seed=5, trace=True)
            assert t1[0].tobytes() == ta[b - 1].tobytes()
            assert one[0] == every[b - 1]


@pytest.mark.parametrize("prec", [abi.PREC_FP64, abi.PREC_MIXED])
def test_a_box_without_lists_beside_others(prec):
    """The last box is too small for lists (a radius reaches beyond the neighbouring images): the
    others keep theirs, and every box its own bits."""
    s = _sphere_system([((40.0, 40.0, 40.0), 700), ((9.0, 9.0, 9.0), 9), ((30.0, 50.0, 30.0), 500)])
    _against_the_oracle(s, prec, 300, 300)
    for pick in (1, 2, 3):
        one, t1, among, ta = _alone_and_together(s, prec, 2, 300, pick)
        assert t1.tobytes() == ta.tobytes()
        assert one == among
