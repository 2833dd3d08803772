"""The solve stage's forms against the oracle: 512 rows, whose tables lie in
shared memory, and 1024 and 2048 rows, whose tables have no room there beside
the lines and are read through L1 (k_shift, k_solve_half, and k_dy_sums of the
statistics)."""
import numpy as np
import pytest

from homogenenousshearturbulence_b200 import hst
from tests.gpu_util import c1_deck, make_pair, rel_l2, run_pair, seeded_field

pytestmark = pytest.mark.gpu

CASES = {
    # 512 rows: slabs of 16 rows
    "exact": dict(nx=15, nz=16, ny=512, exact_shift=True),
    "default_s2": dict(nx=15, nz=16, ny=512, s2_amplitude=0.5, s2_period=0.7),
    "exact_mixed": dict(nx=31, nz=32, ny=512, exact_shift=True, precision="mixed"),  # 2 nxd = nzd = 96
    "hard_damping": dict(nx=15, nz=16, ny=512, damp_kpar=3.0, damp_kperp=2.0, damp_hard=True, exact_shift=True),
}


@pytest.mark.parametrize("case", sorted(CASES))
def test_solve_stage_of_512_rows(case):
    """3 time steps of a 512-row deck within the precision's bound of the oracle."""
    deck = c1_deck(**CASES[case])
    V0 = seeded_field(deck, seed=6, k0=4.0, energy=0.1)
    s, o = make_pair(deck, V0)
    Vg, Vo = run_pair(s, o, deck["deltat"], 3)
    tol = 1e-5 if deck.get("precision") == "mixed" else 1e-12
    assert rel_l2(Vg, Vo) <= tol
    s.close()


@pytest.mark.parametrize("ny", [1024, 2048])
@pytest.mark.parametrize("ystretch", [0.0, 0.8])
def test_solve_stage_with_tables_through_l1(ny, ystretch):
    """1 time step and the statistics of a tall deck; the lines' conditioning, and with it the rounding, grows with the
    square of the rows (2e-13 at 512)"""
    deck = c1_deck(nx=5, nz=4, ny=ny, exact_shift=True, deltat=0.0005, ystretch=ystretch)
    V0 = seeded_field(deck, seed=6, k0=3.0, energy=0.1)
    s, o = make_pair(deck, V0)
    Vg, Vo = run_pair(s, o, deck["deltat"], 1)
    assert rel_l2(Vg, Vo) <= 1e-12 * (ny / 512) ** 2
    for c in range(3):  # the same field in both
        o.field(c)[...] = Vg[c]
    sums, exz = s.outstats_sums()
    want, exz_o = o.outstats_sums()
    got = np.array([sums[k] for k in hst.Solver.SUM_NAMES])
    assert np.abs(got - want).max() <= 1e-11 * np.abs(want).max()
    assert np.abs(exz - exz_o).max() <= 1e-12 * exz_o.max()
    s.close()
