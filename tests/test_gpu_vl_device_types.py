"""Atom types in device memory at the Verlet-list atom boundary: any address is
taken, bad types are refused before the context's atoms change."""
import numpy as np
import pytest
import torch

import mdb

pytestmark = pytest.mark.gpu


def liquid(n, **kw):
    hp = mdb.host_params(nx=n, ny=n, nz=n)
    x, v, t = mdb.create_fcc(hp)
    hp.from_file = 1
    return mdb.system_from_host(hp, len(t), **kw), x, v, t


def on_device(x, v):
    return [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (x, v)]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("offset", [0, 1, 2, 3])
def test_types_at_any_address(offset, precision):
    a, x, v, t = liquid(5, precision=precision)
    b, _, _, _ = liquid(5, precision=precision)
    a.set_atoms(x, v, t)
    dx, dv = on_device(x, v)
    raw = torch.zeros(4 * len(t) + 4, dtype=torch.uint8, device="cuda")
    raw[offset:offset + 4 * len(t)] = torch.from_numpy(t.astype(np.int32).view(np.uint8)).cuda()
    torch.cuda.synchronize()
    b.set_atoms_ptr(len(t), dx.data_ptr(), dv.data_ptr(), raw.data_ptr() + offset)
    a.setup()
    b.setup()
    for p, q in zip(a.atoms(), b.atoms()):
        assert np.array_equal(p, q)


@pytest.mark.parametrize("bad", [-1, 8])
def test_refused_types_leave_the_atoms(bad):
    a, x, v, t = liquid(4)
    a.set_atoms(x, v, t)
    a.setup()
    before = a.atoms()
    _, x2, v2, t2 = liquid(6)  # more atoms than the context has room for
    dx, dv = on_device(x2, v2)
    t2 = t2.copy()
    t2[len(t2) // 2] = bad
    dt = torch.from_numpy(t2.astype(np.int32)).cuda()
    torch.cuda.synchronize()
    with pytest.raises(mdb.MdbError):
        a.set_atoms_ptr(len(t2), dx.data_ptr(), dv.data_ptr(), dt.data_ptr())
    a.nlocal = len(t)
    for p, q in zip(before, a.atoms()):
        assert np.array_equal(p, q)
    # the next call goes through
    dt[len(t2) // 2] = 0
    torch.cuda.synchronize()
    a.set_atoms_ptr(len(t2), dx.data_ptr(), dv.data_ptr(), dt.data_ptr())
    assert np.array_equal(a.atoms()[0], x2)
