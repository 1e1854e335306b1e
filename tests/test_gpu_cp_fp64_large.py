"""FP64 cluster pairs with half lists on both sides of the size where the kernel
changes: forces and energies of full lists (bit-exact with the reference's order in
small systems) up to FP64 summation order."""
import numpy as np
import pytest

import mdb

from test_gpu_cp_cpw import C5_TYPES

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,N,types", [(55, 4, None), (58, 4, None), (58, 4, C5_TYPES),
                                       (65, 8, None), (65, 8, C5_TYPES), (81, 8, None)])
def test_half_lists_match_full_lists(n, N, types):
    extra = dict(types=types, cutforce=2.5 * max(types[1])) if types else {}
    hp = mdb.host_params(nx=n, ny=n - 1, nz=n, **extra)
    x, v, t = mdb.create_fcc(hp)
    x = np.mod(x + np.random.default_rng(n).uniform(-0.03, 0.03, x.shape),
               [hp.xprd, hp.yprd, hp.zprd])
    pt = dict(epsilon_per_type=types[0], sigma_per_type=types[1]) if types else {}
    out = []
    for half in (0, 1):
        s = mdb.ClusterSystem(xprd=hp.xprd, yprd=hp.yprd, zprd=hp.zprd, cutforce=hp.cutforce,
                              cutneigh=hp.cutneigh, dt=hp.dt, dtforce=hp.dtforce,
                              ntypes=hp.ntypes, natoms=len(t), cluster_n=N, half_neigh=half,
                              precision="fp64", **pt)
        s.set_atoms(x, v, t)
        s.setup()
        s.compute_force(energy=True)
        ok = np.concatenate([np.arange(4) < k for k in s.iclusters()[0]])
        xs, _, f, _ = s.slots()
        out.append((xs[:len(ok)][ok], f[:len(ok)][ok], s.thermo()["PE"]))
        s.close()
    (xf, ff, pf), (xh, fh, ph) = out
    assert np.array_equal(xf, xh)
    rms = np.sqrt(np.mean(np.sum(ff * ff, axis=1)))
    # sums of some 60 terms of up to 100 times the rms force, in another order
    assert np.abs(ff - fh).max() <= 1e-12 * rms
    assert ph == pytest.approx(pf, rel=1e-12)
