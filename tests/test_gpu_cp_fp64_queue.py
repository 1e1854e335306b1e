"""Edges of the FP64 cluster-pair kernel's queues of pairs: rows with more pairs
inside the cutoff than a queue holds, and ragged last clusters. Full lists bit
for bit the oracle's, half lists (atomics) to 1e-12 of the force scale."""
import numpy as np
import pytest

import mdb
import oracle as O

pytestmark = pytest.mark.gpu


def melted(drop=0, steps=33, **kw):
    """Positions, velocities and types after some oracle steps, without the last
    `drop` atoms."""
    o = O.Oracle(**kw)
    o.lattice()
    o.setup()
    o.run(steps)
    x, v, _, t = o.atoms()
    n = len(t) - drop
    return x[:n].copy(), v[:n].copy(), t[:n].copy()


@pytest.mark.parametrize("N", [4, 8])
@pytest.mark.parametrize("half", [0, 1])
@pytest.mark.parametrize("cut", [2.5, 3.8])
def test_cluster_rows_longer_than_the_queue(cut, half, N):
    kw = dict(nx=6, ny=7, nz=6, cutforce=cut)
    x, v, t = melted(drop=2, **kw)
    hp = mdb.host_params(**kw)
    mdb.create_fcc(hp)
    common = dict(xprd=hp.xprd, yprd=hp.yprd, zprd=hp.zprd, cutforce=hp.cutforce,
                  cutneigh=hp.cutneigh, dt=hp.dt, dtforce=hp.dtforce, mass=hp.mass,
                  ntypes=hp.ntypes)
    s = mdb.ClusterSystem(natoms=len(t), cluster_n=N, half_neigh=half, **common)
    s.set_atoms(x, v, t)
    s.setup()
    o = O.OracleCP(x, v, t, M=4, N=N, half=half, natoms=len(t), **common)
    o.setup()
    o.force()
    ok = np.concatenate([np.arange(4) < k for k in o.iclusters()[0]])
    f, fo = s.slots()[2][:len(ok)][ok], o.slots()[2][:len(ok)][ok]
    if half:
        rms = np.sqrt(np.mean(np.sum(fo * fo, axis=1)))
        assert np.abs(f - fo).max() <= 1e-12 * rms
    else:
        assert np.array_equal(f, fo)
    s.compute_force(energy=True)
    assert s.thermo()["PE"] == pytest.approx(o.thermo()["PE"], rel=1e-10)
