"""Ewald boxes whose three edges differ: the phase tables have another length in each
dimension.  A long x edge gives k-vector rows of more than 64 vectors (cut into pieces)
and more powers than the move and insertion kernels' tables hold; a long z edge the
long way of the other dimension.  Against the FP64 oracle."""
import numpy as np
import pytest

import cassandra_gb300 as cg
from cassandra_gb300 import abi, workloads
from cassandra_gb300.system import BoxSpec, ForceField, MoleculeSet, System
from oracle import oracle
from test_gpu_grad import FD_TOL, H_REL, _oracle_energy

pytestmark = pytest.mark.gpu

BOXES = {"uneven": ((14.0, 18.0, 23.0), 6.5), "long_x": ((112.0, 13.0, 12.4), 6.0), "long_z": ((12.6, 13.4, 90.0), 6.0)}


def _system(name, nmax=40):
    edges, rcut = BOXES[name]
    rng = np.random.default_rng(12)
    sp = workloads.water_species()
    base = sp.libraries[0][0] - np.average(sp.libraries[0][0], axis=0, weights=[15.999, 1.008, 1.008])
    sites = [[(i + 0.5) / n * L - 0.5 * L for i in range(n)] for L in edges for n in [int(L // 4.1)]]
    spots = np.array(np.meshgrid(*sites, indexing="ij")).reshape(3, -1).T
    spots = spots[np.sort(rng.choice(len(spots), min(nmax, len(spots)), replace=False))]
    ms = MoleculeSet()
    for k, p in enumerate(spots):
        ms.add(k + 1, 1, 1, base @ workloads.random_rotation(rng).T + p)
    box = BoxSpec(length=edges, rcut_vdw=rcut, rcut_coul=rcut, rcut_cbmc=5.0, rcut_low=0.85,
                  charge_style=abi.CHARGE_COUL, charge_sum_style=abi.QQ_EWALD, ewald_tol=1e-5, temperature=298.0)
    return System([sp], [box], ms, ForceField([sp]), [len(spots) + 1])


@pytest.mark.parametrize("name", list(BOXES))
def test_energy_and_gradient(name):
    s = _system(name)
    n = 3 * len(s.molecules.im)
    with oracle.open_system(s) as o, cg.open_system(s, precision=abi.PREC_FP64) as g:
        eo, eg = o.system_total_energy(1)[0], g.system_total_energy(1)[0]
        _, grad, _, _, dq = g.system_gradient(1, n)
    scale = sum(abs(eo[k]) for k in ("inter_vdw", "inter_q", "reciprocal", "self"))
    for k in eo:
        assert abs(eg[k] - eo[k]) <= 1e-10 * scale, k
    top = np.abs(grad).max()
    for k in (0, 7, 21, n // 3 - 1):  # molecules
        for d in range(3):
            e = []
            for sign in (1, -1):
                xyz = [x.copy() for x in s.molecules.xyz]
                h = H_REL * max(1.0, abs(xyz[k][1, d]))
                xyz[k][1, d] += sign * h
                e.append(_oracle_energy(s, xyz))
            assert abs((e[0] - e[1]) / (2 * h) - grad[3 * k + 1, d]) <= FD_TOL * top, (k, d)


@pytest.mark.parametrize("name", list(BOXES))
def test_moves(name):
    s = _system(name)
    out = []
    for open_ctx in (oracle.open_system, lambda x: cg.open_system(x, precision=abi.PREC_FP64)):
        with open_ctx(s) as c:
            c.system_total_energy(1)
            r = c.mc_sweeps([1], 4, [[0.6]], [[0.5]], seed=3, prob_translate=0.5)
            out.append((r, np.concatenate([c.get_molecule(m, 1) for m in s.molecules.im])))
    (ro, do, to), xo = out[0]
    (rg, dg, tg), xg = out[1]
    assert {k: v for k, v in ro[0].items() if k.startswith("n_")} == {k: v for k, v in rg[0].items() if k.startswith("n_")}
    scale = sum(abs(ro[0]["energy"][k]) for k in ("inter_vdw", "inter_q", "reciprocal", "self"))
    for k in ("total", "inter_vdw", "inter_q", "reciprocal"):
        assert abs(ro[0]["energy"][k] - rg[0]["energy"][k]) <= 1e-9 * scale, k
    assert np.abs(xo - xg).max() <= 1e-8


@pytest.mark.parametrize("prec", [abi.PREC_FP64, abi.PREC_MIXED])
@pytest.mark.parametrize("name", list(BOXES))
def test_insertions(name, prec):
    s = _system(name)
    with oracle.open_system(s) as o, cg.open_system(s, precision=prec) as g:
        o.system_total_energy(1)
        g.system_total_energy(1)
        to = o.widom_insert(1, [1], 200, 12, 12, seed=9, trace=True)[1]
        tg = g.widom_insert(1, [1], 200, 12, 12, seed=9, trace=True)[1]
        # sum of |terms| of the reciprocal part: its FP32 phases in a mixed context
        recip = abs(o.system_total_energy(1)[0]["reciprocal"])
    assert np.array_equal(to["overlap"], tg["overlap"])
    same = to["selected_trial"] == tg["selected_trial"]
    assert same.all() if prec == abi.PREC_FP64 else same.mean() >= 0.99  # FP32 weights at a boundary
    ok = (to["overlap"] == 0) & same
    assert ok.sum() > 100
    tol = 1e-10 if prec == abi.PREC_FP64 else 2e-5
    assert (np.abs(tg["e_inter"] - to["e_inter"])[ok] <= tol * (to["e_inter_abs"][ok] + recip) + 1e-7).all()
