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
