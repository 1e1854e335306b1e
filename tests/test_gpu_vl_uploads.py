"""Tables and lists uploaded right before the work that reads them: every evaluation
sees the last upload, however often they change."""
import numpy as np
import pytest

import mdb
from conftest import EAM_FILE

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_eam_tables_change_between_evaluations(precision):
    tab = mdb.read_funcfl(EAM_FILE)
    other = dict(tab, **{k: 0.5 * tab[k] for k in ("frho_spline", "rhor_spline", "z2r_spline")})
    hp = mdb.host_params(nx=6, ny=6, nz=6, eam=tab, rho=4.0 / 3.615 ** 3, temp=1600.0)
    x, v, t = mdb.create_fcc(hp)
    x = x + np.random.default_rng(1).uniform(-0.2, 0.2, x.shape)
    x = np.mod(x, [hp.xprd, hp.yprd, hp.zprd])
    hp.from_file = 1
    want = []
    for e in (tab, other):
        s = mdb.system_from_host(hp, len(t), eam=e, precision=precision)
        s.set_atoms(x, v, t)
        s.setup()
        s.synchronize()
        s.compute_force()
        want.append(s.atoms()[2])
    assert not np.array_equal(*want)
    for k in range(20):
        s.set_eam((tab, other)[k % 2])
        s.compute_force()
        assert np.array_equal(s.atoms()[2], want[k % 2]), k


def test_caller_lists_change_between_evaluations():
    x, v, t, num, nb = mdb.stub_system(3000, "rand", 76, nreps=2)
    s, _, _ = mdb.stub_context(x, v, t, num, nb)
    lists, want = [(num, nb), (num // 2, nb)], []
    for n, rows in lists:
        s.set_neighbor_list(n, rows)
        s.synchronize()
        s.compute_force()
        want.append(s.atoms()[2])
    assert not np.array_equal(*want)
    for k in range(20):
        s.set_neighbor_list(*lists[k % 2])
        s.compute_force()
        assert np.array_equal(s.atoms()[2], want[k % 2]), k
