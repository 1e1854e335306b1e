"""Launch shape of full-list ensembles: members that nobody tuned take the register
budget by the atoms of the whole ensemble, and follow their run alone bit for bit
whichever shape that run takes. A shape shows in the launches: members of one shape
share a force launch."""
import numpy as np
import pytest

import mdb

from test_gpu_cp import replica

pytestmark = pytest.mark.gpu


def plain_launches(ens, first):
    n0 = ens.launches
    ens.run(9, first_step=first, max_samples=0)  # no rebuild among steps 20k .. 20k + 8
    return ens.launches - n0


@pytest.mark.parametrize("N,count,budget", [(4, 3, 0), (4, 5, 2), (8, 7, 0), (8, 9, 2)])
def test_budget_by_total_atoms(N, count, budget):
    pairs = [replica(20, 0.84, 1.44, N, "mixed") for _ in range(count)]  # 32,000 atoms each
    (extra, spare) = replica(5, 0.84, 1.44, N, "mixed")
    ens = mdb.Ensemble([p[0] for p in pairs] + [extra])
    counts = {}
    for k, variant in enumerate((budget, 2 - budget)):
        extra.tune("force_variant", variant)
        counts[variant] = plain_launches(ens, 20 * k)
        ens.run(11, first_step=20 * k + 9, max_samples=0)
    # the tuned member of the same shape joins the others' launch
    assert counts[budget] < counts[2 - budget], counts
    a, b = pairs[0]
    for k in range(2):
        b.run(20, first_step=20 * k, max_samples=0)
    a.update_single_atoms()
    b.update_single_atoms()
    for p, q in zip(a.atoms(), b.atoms()):
        assert np.array_equal(p, q)
    ens.close()
    for s in [m for p in pairs for m in p] + [extra, spare]:
        s.close()
