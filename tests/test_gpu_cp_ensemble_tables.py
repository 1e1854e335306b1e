"""An ensemble whose member tables and block maps are uploaded again and again (a
member's setting changes between runs): every run sees the new tables, so untouched
full-list members follow their run alone bit for bit."""
import numpy as np
import pytest

import mdb

from test_gpu_cp import replica

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,check", [(4, 0.0), (8, 0.0), (4, 0.15)])
def test_tables_before_the_first_step(N, check):
    # some thousand blocks per map: uploads large enough to take longer than a call
    groups = [replica(20, 0.84, 1.44, N, "mixed") for _ in range(2)]
    members = [m for g in groups for m in g]
    alone = members.pop()
    extra, spare = replica(5, 0.84, 1.44, N, "mixed")
    for m in members + [alone, extra]:
        if check:
            m.set_rebuild_check(check)
    ens = mdb.Ensemble(members + [extra])
    for k in range(24):
        extra.tune("force_variant", 2 * (k % 2))
        ens.run(3, first_step=3 * k, max_samples=0)
        alone.run(3, first_step=3 * k, max_samples=0)
        alone.update_single_atoms()
        want = alone.atoms()
        for m in members:
            m.update_single_atoms()
            for p, q in zip(m.atoms(), want):
                assert np.array_equal(p, q), k
    ens.close()
    for s in members + [alone, extra, spare]:
        s.close()
