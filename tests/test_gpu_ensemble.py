"""An ensemble of independent realisations in one context
(hst_gpu_create_batch): every kernel of the substep covers all members in one
launch; each member must evolve exactly as it does alone in its own
context."""
import numpy as np
import pytest
import torch

from homogenenousshearturbulence_b200 import hst
from tests.gpu_util import c1_deck, rel_l2, seeded_field, traced

pytestmark = pytest.mark.gpu

CASES = {
    "default": dict(),
    "exact_s2_edges": dict(exact_shift=True, s2_amplitude=0.5, s2_period=0.7),  # nzd = 3 nz: ghost-row transforms
    "mixed": dict(precision="mixed", exact_shift=True),
    "tall": dict(nx=15, nz=16, ny=512, exact_shift=True),  # slabs of 16 rows
    # 3655 columns a member: three members together have enough for a narrower solver group than one
    "more_columns": dict(nx=42, nz=42),
    "hard_damping": dict(damp_kpar=3.0, damp_kperp=2.0, damp_hard=True, s2_amplitude=0.4, s2_period=0.5),
}


@pytest.mark.parametrize("case", sorted(CASES))
def test_ensemble_members_match_single_contexts(case):
    """Three members with their own seeds, 5 time steps in one ensemble
    context against three single contexts: every member the same bits (the
    same operations on the same data), the CFL number the largest of the
    members'."""
    deck = c1_deck(**CASES[case])
    fields = [seeded_field(deck, seed=s, k0=4.0, energy=0.1) for s in (1, 2, 3)]
    ens = hst.Solver(deck, members=3)
    assert hst.lib().hst_gpu_members(ens._h) == 3
    ens.time = 0.0
    for m, V in enumerate(fields):
        ens.select(m)
        ens.set_velocity(V)
    singles = []
    for V in fields:
        s = hst.Solver(deck)
        s.time = 0.0
        s.set_velocity(V)
        singles.append(s)
    for _ in range(5):
        ens.timestep(deck["deltat"])
        for s in singles:
            s.timestep(deck["deltat"])
    assert ens.cfl == max(s.cfl for s in singles)
    for m, s in enumerate(singles):
        ens.select(m)
        a, b = ens.velocity(), s.velocity()
        assert np.array_equal(a, b), (case, m, rel_l2(a, b))
        s.close()
    ens.close()


def blocks_of_a_step(s, tmp_path):
    """{kernel: the blocks of its launch} of one time step"""
    return {name: int(np.prod(e["args"]["grid"])) for e in traced(s, 1, tmp_path) if e.get("cat") == "kernel"
            for name in ("k_shift", "k_solve_half") if name in e["name"]}


@pytest.mark.parametrize("members,nx,ny,nz", [(8, 31, 64, 32), (12, 15, 32, 16), (8, 63, 128, 64), (1, 31, 64, 32)])
def test_ensemble_solves_run_on_all_blocks(members, nx, ny, nz, tmp_path):
    """The implicit solves cover an ensemble's columns with as many blocks as
    the shift, which has the same warps and needs no factor scratch: the
    scratch holds the columns of every member, not of one."""
    deck = c1_deck(nx=nx, ny=ny, nz=nz, exact_shift=True)
    s = hst.Solver(deck, members=members)
    s.time = 0.0
    s.timesteps(1)
    s.sync()
    got = blocks_of_a_step(s, tmp_path)
    assert got["k_shift"] > 0 and got["k_solve_half"] == got["k_shift"], got
    s.close()


def test_a_context_holds_what_it_says():
    """hst_gpu_device_bytes and the rounding of some twenty-five allocations to 2 MiB (12 MB here) are all that a
    context takes: the solves' factors lie in the product buffer (a scratch of their own took 34 MB more)"""
    deck = c1_deck(nx=63, nz=64, ny=256, exact_shift=True)
    s = hst.Solver(deck)  # loads the kernels
    s.timesteps(1)
    s.sync()
    s.close()
    free = torch.cuda.mem_get_info()[0]
    s = hst.Solver(deck)
    took = free - torch.cuda.mem_get_info()[0]
    s.close()
    said = hst.device_bytes(**{k: deck[k] for k in ("nx", "ny", "nz", "alfa0", "beta0", "ly")})
    assert said <= took + (2 << 20) and took <= said + (28 << 20), (said, took)


def test_a_refused_ensemble_gives_its_memory_back():
    """more members than the device holds: the creation is refused half way, and what it had allocated is free again"""
    hst.Solver(c1_deck(), members=2).close()
    free = torch.cuda.mem_get_info()[0]
    deck = c1_deck()
    members = int(1.1 * free / hst.device_bytes(**{k: deck[k] for k in ("nx", "ny", "nz", "alfa0", "beta0", "ly")}))
    with pytest.raises(hst.HstError) as e:
        hst.Solver(deck, members=min(members, 4096))
    assert e.value.code == hst.ENOMEM
    assert torch.cuda.mem_get_info()[0] >= free - (64 << 20)


def test_ensemble_refuses_bad_members():
    deck = c1_deck()
    ens = hst.Solver(deck, members=2)
    with pytest.raises(hst.HstError) as e:
        ens.select(2)
    assert e.value.code == hst.EARG
    with pytest.raises(hst.HstError):
        ens.autotune(deck["deltat"], 1)
    ens.close()
