"""Potential energies of ensemble members: the samples of an ensemble run and the
members' own thermo() between runs, in any order. A member alone and the batched
launch of its group may write different numbers of energy partials (launch
shapes by size), so each reduction has to sum its own."""
import numpy as np
import pytest

import mdb

from test_gpu_cp import replica

pytestmark = pytest.mark.gpu

TYPES = ([0.5, 1.5, 0.8, 1.2], [0.8, 1.2, 1.0, 0.9])


def fresh_pe(member, twin):
    """PE of the member's present state, evaluated by the twin from a new build."""
    member.update_single_atoms()
    twin.set_atoms(*member.atoms())
    twin.update_atoms_pbc()
    twin.setup()
    return twin.thermo()["PE"]


# FP32 pair energies of one state, other lists and another summation order: each
# rounds to a few 2^-24 of its value, whose sum of absolute values is a few |PE|
PE_REL = 1e-5


@pytest.mark.parametrize("batched", [1, 0])
@pytest.mark.parametrize("half", [0, 1])
@pytest.mark.parametrize("N,types", [(4, None), (8, None), (4, TYPES)])
def test_member_energies_between_runs(N, types, half, batched):
    pairs = [replica(n, rho, T, N, "mixed", half=half, types=types)
             for n, rho, T in [(7, 0.84, 1.44), (8, 0.80, 1.0)]]
    members = [p[0] for p in pairs]
    ens = mdb.Ensemble(members, batched=batched)

    def same(values):
        for (a, b), pe in zip(pairs, values):
            assert pe == pytest.approx(fresh_pe(a, b), rel=PE_REL)

    # the members' own energies first, then runs with and without samples
    ens.run(20, max_samples=0)
    same([m.thermo()["PE"] for m in members])
    got = ens.run(20, first_step=20, max_samples=8)
    assert [s["step"] for s in got[0]] == [30, 40]
    same([g[-1]["PE"] for g in got])
    same([m.thermo()["PE"] for m in members])
    # an energy evaluation by the member itself, then a sample of the kept graph
    for m in members:
        m.compute_force(energy=True)
    same([m.thermo()["PE"] for m in members])
    got = ens.run(10, first_step=40, max_samples=8)
    same([g[-1]["PE"] for g in got])
    same([m.thermo()["PE"] for m in members])
    # the last step is no sample: the energy of the state the run left
    ens.run(15, first_step=50, max_samples=8)
    same([m.thermo()["PE"] for m in members])
    ens.close()
    for a, b in pairs:
        a.close()
        b.close()
