"""CTAs per chain of cass_mc_sweeps: every size that the automatic choice takes can be asked
for, is reported, and makes the same decisions."""
import numpy as np
import pytest

import cassandra_gb300 as cg
import mc_helpers
from cassandra_gb300 import abi

pytestmark = pytest.mark.gpu


def _chain(ctas):
    s = mc_helpers.water_small()
    with cg.open_system(s, precision=abi.PREC_FP64) as g:
        g.system_total_energy(1)
        g.set_mc_cluster(ctas)
        r = g.mc_sweeps([1], 3, [[0.5]], [[0.5]], seed=6, prob_translate=0.5)[0][0]
        return r, mc_helpers.positions(g, s), g.stats()["gcmc_cluster"]


def test_cluster_sizes_make_the_same_chain():
    one, x1, used = _chain(1)
    assert used == 1
    for ctas in (3, 8, 16):
        r, x, used = _chain(ctas)
        assert used == ctas
        assert {k: v for k, v in r.items() if k.startswith("n_")} == {k: v for k, v in one.items() if k.startswith("n_")}
        assert abs(r["energy"]["total"] - one["energy"]["total"]) <= 1e-10 * abs(one["energy"]["self"])
        assert np.abs(x - x1).max() <= 1e-9
    assert _chain(0)[2] == 16  # the automatic choice for one Ewald box


def test_other_cluster_sizes_are_refused():
    s = mc_helpers.water_small()
    with cg.open_system(s, precision=abi.PREC_FP64) as g:
        for ctas in (-1, 9, 15, 17):
            with pytest.raises(abi.CassError):
                g.set_mc_cluster(ctas)
