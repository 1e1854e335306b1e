"""The mixed cluster-pair kernel's launch shape by size: on both sides of its limits,
alone and in an ensemble, the forces and energies of one i-cluster per warp up to FP32
summation order."""
import pytest

import mdb

from test_gpu_cp import replica
from test_gpu_cp_cpw import C5_TYPES, forces
from test_gpu_cp_pairs import SUM_ORDER, rel, system, valid_forces

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,N,half,types", [
    (16, 4, 1, None), (17, 4, 1, None), (25, 4, 1, None), (26, 4, 1, None),
    (17, 8, 1, None), (26, 4, 0, None), (26, 8, 0, None), (17, 4, 1, C5_TYPES),
    # eight i-clusters per warp: several types, more than 2^20 atoms
    (65, 4, 1, C5_TYPES), (65, 4, 0, C5_TYPES),
])
def test_default_shape(n, N, half, types):
    s, _ = system(n, N, half, types=types, steps=20 if n > 30 else 60)
    s.compute_force(energy=True)
    f, e = valid_forces(s), s.thermo()["PE"]
    f1, e1 = forces(s, 1)
    r, m = rel(f, f1)
    assert r <= SUM_ORDER and m <= 20 * SUM_ORDER, (r, m)
    assert e == pytest.approx(e1, rel=1e-6)
    s.close()


@pytest.mark.parametrize("N", [4, 8])
def test_half_list_ensemble_across_sizes(N):
    """Untuned half-list members of 500, 13,500 and 19,652 atoms all take the shape of a
    large system; alone they run one and two (4x4) or four i-clusters per warp."""
    pairs = [replica(n, 0.8442, 1.44, N, "mixed", half=1) for n in (5, 15, 17)]
    ens = mdb.Ensemble([p[0] for p in pairs])
    got = ens.run(30, max_samples=8)
    for k, (a, b) in enumerate(pairs):
        f = valid_forces(a)
        pe = a.thermo()["PE"]
        a.compute_force(energy=True)  # the same state and lists, the member's own launch
        r, m = rel(f, valid_forces(a))
        assert r <= SUM_ORDER and m <= 20 * SUM_ORDER, (k, r, m)
        assert got[k][-1]["PE"] == pytest.approx(a.thermo()["PE"], rel=1e-6)
        assert pe == pytest.approx(a.thermo()["PE"], rel=1e-6)
        want = b.run(30, max_samples=8)
        # separate mixed runs, one per summation order
        assert got[k][-1]["T"] == pytest.approx(want[-1]["T"], rel=1e-3)
    ens.close()
    for p in pairs:
        for s in p:
            s.close()
