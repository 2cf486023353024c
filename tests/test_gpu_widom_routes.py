"""Widom insertions on the routes and at the edges where the kernels' branches change."""
import numpy as np
import pytest

import cassandra_gb300 as cg
from cassandra_gb300 import abi, workloads
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
