"""Edges of the tiled Verlet lists and of the FP64 kernels that share an atom: row
lengths around multiples of a tile's 8 entries, list capacities that are no
multiple of it (grown or not), runs of more than 32 candidates, and atom counts
that leave the last block partly empty. Everything is bit for bit the oracle's
(half-list forces: 1e-12 of the force scale, atomics)."""
import numpy as np
import pytest

import mdb
import oracle as O
from conftest import EAM_FILE

pytestmark = pytest.mark.gpu


def melted(drop=0, steps=33, **kw):
    """Box, positions, velocities and types after some oracle steps, without the
    last `drop` atoms."""
    o = O.Oracle(**kw)
    o.lattice()
    o.setup()
    o.run(steps)
    x, v, _, t = o.atoms()
    n = len(t) - drop
    return x[:n].copy(), v[:n].copy(), t[:n].copy()


def both(x, v, t, hp, precision="fp64", eam=None, okw=None, **over):
    hp.from_file = 1
    s = mdb.system_from_host(hp, len(t), eam=eam, precision=precision, **over)
    s.set_atoms(x, v, t)
    s.setup()
    o = O.Oracle(from_file=1, xprd=hp.xprd, yprd=hp.yprd, zprd=hp.zprd, **(okw or {}))
    o.set_atoms(x, v, t)
    o.setup()
    o.force()
    return s, o


def assert_same_rows(s, o):
    n, rows = s.neighbor_list()
    n2, rows2 = o.neighbor_list()
    assert np.array_equal(n, n2)
    for i in range(len(n)):
        assert np.array_equal(rows[i, :n[i]], rows2[i, :n[i]]), i
    return n


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("half", [0, 1])
@pytest.mark.parametrize("maxneighs", [8, 77, 79, 80, 81, 100])
def test_rows_and_capacities(maxneighs, half, precision):
    kw = dict(nx=7, ny=6, nz=5, half_neigh=half)
    x, v, t = melted(drop=3, **kw)
    hp = mdb.host_params(**kw)
    mdb.create_fcc(hp)
    s, o = both(x, v, t, hp, precision, maxneighs=maxneighs, okw=dict(half_neigh=half))
    n = assert_same_rows(s, o)
    assert len(set(n % 8)) == 8  # rows end at every place of a tile
    f, fo = s.atoms()[2], o.atoms()[2]
    rms = np.sqrt(np.mean(np.sum(fo * fo, axis=1)))
    if precision == "fp64" and not half:
        assert np.array_equal(f, fo)
    else:
        assert np.sqrt(np.mean(np.sum((f - fo) ** 2, axis=1))) <= (
            1e-12 if precision == "fp64" else 1e-5) * rms


@pytest.mark.parametrize("half", [0, 1])
def test_long_runs_of_candidates(half):
    # three times the density: runs of bins hold 35 atoms, rows more than 200 entries
    kw = dict(nx=7, ny=8, nz=9, half_neigh=half, rho=2.5, temp=0.1)
    x, v, t = melted(steps=1, **kw)
    hp = mdb.host_params(**kw)
    mdb.create_fcc(hp)
    s, o = both(x, v, t, hp, okw=dict(half_neigh=half))
    n = assert_same_rows(s, o)
    assert n.max() > (100 if half else 200)
    f, fo = s.atoms()[2], o.atoms()[2]
    if half:
        assert np.abs(f - fo).max() <= 1e-12 * np.abs(fo).max()
    else:
        assert np.array_equal(f, fo)


@pytest.mark.parametrize("drop", [0, 1, 15])
def test_eam_fp64_partly_filled_blocks(drop):
    tab = mdb.read_funcfl(EAM_FILE)
    hp = mdb.host_params(nx=5, ny=6, nz=5, eam=tab, rho=4.0 / 3.615 ** 3, temp=1600.0)
    x, v, t = mdb.create_fcc(hp)
    x = x + np.random.default_rng(drop).uniform(-0.2, 0.2, x.shape)
    x = np.mod(x, [hp.xprd, hp.yprd, hp.zprd])
    n = len(t) - drop
    s, o = both(x[:n], v[:n], t[:n], hp, eam=tab,
                okw=dict(eam_file=EAM_FILE, force_field=1))
    assert_same_rows(s, o)
    assert np.array_equal(s.atoms()[2], o.atoms()[2])
    assert np.array_equal(s.eam_fp()[:n], o.eam_fp()[:n])
    s.compute_force(energy=True)
    assert s.thermo()["PE"] == pytest.approx(o.thermo()["PE"], rel=1e-10)
