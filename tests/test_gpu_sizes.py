"""The substep's kernels at the sizes where they can go wrong: every compiled
x and z transform length with the most retained modes it takes and with few,
row counts that leave short tiles and uneven slabs, and the two forms of the
right-hand sides, each against the oracle (or the other form).  Tolerances:
1e-12 relative L2 in FP64 and 1e-5 in mixed precision, the bounds the substep
is held to everywhere; a few 1e-15 and 1e-8 are what these sizes show.
"""
import ctypes as ct

import numpy as np
import pytest
import torch

import oracle
from homogenenousshearturbulence_b200 import hst
from tests.gpu_util import c1_deck, make_pair, rel_l2, run_pair, seeded_field, traced

pytestmark = pytest.mark.gpu

TOL = {"fp64": 1e-12, "mixed": 1e-5}


def against_oracle(deck, steps=1, k0=4.0, seed=5):
    V0 = seeded_field(deck, seed=seed, k0=k0, energy=0.1)
    s, o = make_pair(deck, V0)
    Vg, Vo = run_pair(s, o, deck["deltat"], steps)
    prec = deck.get("precision", "fp64")
    err, cfl, cfl_o = rel_l2(Vg, Vo), s.cfl, oracle.lib().ora_get_cfl(o.h)
    s.close()
    assert err <= TOL[prec], err
    assert abs(cfl - cfl_o) <= (1e-12 if prec == "fp64" else 1e-5) * cfl_o


def most_modes(N):
    """the largest nx whose 2 nxd is N (nx + 1 <= (N + 1) / 3)"""
    nx = (N - 2) // 3
    return nx if hst.padded_sizes(nx, 8)[0] * 2 == N else nx - 1


@pytest.mark.parametrize("N", [12, 24, 32, 48, 64, 96, 128, 192, 256, 512, 768, 1024])
@pytest.mark.parametrize("few", [False, True])
def test_x_lengths(N, few):
    """the x stage at N points, S2 active (the ghost rows' own transforms): the most modes and the fewest"""
    against_oracle(c1_deck(nx=N // 4 if few else most_modes(N), nz=16, ny=12, s2_amplitude=0.5, s2_period=0.7, time=0.1))


@pytest.mark.parametrize("N", [96, 192, 384, 768])
def test_x_lengths_mixed(N):
    against_oracle(c1_deck(nx=N // 4 + 1, nz=32, ny=32, s2_amplitude=0.5, s2_period=0.7, time=0.1, precision="mixed"))


def xprod_ms(nx):
    s = hst.Solver(c1_deck(nx=nx, ny=64, nz=40))
    s.timesteps(2)
    s.set_profiling(True)
    times = []
    for _ in range(5):
        s.reset_kernel_times()
        s.timesteps(5)
        times.append(s.kernel_times()["xprod"][0])
    s.close()
    return min(times)


def test_short_x_lengths_are_known_to_the_compiler():
    """the x stage at 48 points against 96, whose plan has half the exchanges: 1.7 times its time, 2.4 with the indices
    of the 48 points computed at run time"""
    assert hst.padded_sizes(15, 40)[0] == 24 and hst.padded_sizes(31, 40)[0] == 48
    assert xprod_ms(15) <= 2.05 * xprod_ms(31)


@pytest.mark.parametrize("N", [12, 24, 48, 64, 96, 128, 192, 256, 384, 512, 768, 1024])
@pytest.mark.parametrize("ny", [12, 34])
def test_z_lengths(N, ny):
    """the z transforms at N points on rows that leave a short last y tile; nz = N / 3 (ghost-row transforms) where N
    allows it"""
    nz = N // 3
    assert hst.padded_sizes(15, nz)[1] == N
    against_oracle(c1_deck(nx=15, nz=nz, ny=ny, s2_amplitude=0.5, s2_period=0.7, time=0.1))


@pytest.mark.parametrize("N", [96, 192, 384, 768])
def test_z_lengths_mixed(N):
    against_oracle(c1_deck(nx=31, nz=N // 4, ny=32, precision="mixed", exact_shift=True))


@pytest.mark.parametrize("ny", [8, 10, 18, 30, 34, 62, 94, 150, 258, 514])
@pytest.mark.parametrize("exact", [False, True])
def test_rows(ny, exact):
    """rows that no group of lanes divides and that are not a multiple of the 32-row tiles: slabs of two lengths, a
    short last tile; a stretched grid on every third"""
    against_oracle(c1_deck(nx=9, nz=8, ny=ny, exact_shift=exact, s2_amplitude=0.3, s2_period=0.7,
                           ystretch=0.8 if ny % 3 == 0 else 0.0))


@pytest.mark.parametrize("columns", [(7, 4), (63, 64)])
def test_lanes_follow_the_columns(columns):
    """128 rows: few columns (wide solver groups) and many (narrow ones)"""
    nx, nz = columns
    against_oracle(c1_deck(nx=nx, nz=nz, ny=128, exact_shift=True))


def solve_us(nx, ny, nz):
    """microseconds of hst_gpu_linsolve on (nx + 1)(2 nz + 1) columns of ny rows (the least of five means of ten)"""
    s = hst.Solver(c1_deck(nx=nx, ny=ny, nz=nz, linear=True))
    stream, best = torch.cuda.ExternalStream(s.stream), np.inf
    for _ in range(5):
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        a.record(stream)
        for _ in range(10):
            assert hst.lib().hst_gpu_linsolve(s._h, ct.c_double(1000.0), ct.c_double(0.0)) == 0
        b.record(stream)
        s.sync()
        best = min(best, a.elapsed_time(b) * 100.0)
    s.close()
    return best


@pytest.mark.parametrize("ny", [256, 512])
def test_few_columns_take_no_longer_than_more(ny):
    """136 columns, a warp or two an SM, against 1281 of the same rows: the blocks' own start (the tables into shared
    memory) must not outweigh the solves.  1.0 is what these sizes show; 2.2 and 2.5 with the tables copied one
    load at a time."""
    assert solve_us(7, ny, 8) <= 1.5 * solve_us(20, ny, 30)


@pytest.mark.parametrize("columns", [((60, 60), (63, 75)), ((42, 42), (50, 50))])
def test_a_last_round_of_columns_is_spread(columns):
    """64 rows: 7381 and 9664 columns, 3655 and 5151, of which the larger just exceed what is resident at once: the
    time must not double for the rest (1.0 and 1.3 is what these sizes show; 1.9 with that rest on a few SMs)"""
    few, more = (solve_us(nx, 64, nz) for nx, nz in columns)
    assert more <= 1.65 * few


@pytest.mark.parametrize("nx,ny,nz,lanes", [(50, 256, 50, 16), (63, 64, 75, 8), (100, 96, 100, 8), (20, 512, 60, 32)])
def test_rounds_of_columns_are_alike(monkeypatch, nx, ny, nz, lanes, tmp_path):
    """columns above one round: the shift's and the solves' blocks have the warps that fill every round (0.9 of the
    places and more; 0.5 to 0.8 with as many warps as fit)"""
    monkeypatch.setenv("HST_LINE_LANES", str(lanes))
    s = hst.Solver(c1_deck(nx=nx, ny=ny, nz=nz, exact_shift=True, linear=True))
    s.timesteps(1)
    s.sync()
    columns, seen = (nx + 1) * (2 * nz + 1), set()
    for e in traced(s, 1, tmp_path):
        for name in ("k_shift", "k_solve_half"):
            if e.get("cat") == "kernel" and name in e["name"]:
                places = e["args"]["grid"][0] * e["args"]["block"][0] // lanes
                assert columns >= 0.9 * places * -(-columns // places), (name, places)
                seen.add(name)
    s.close()
    assert len(seen) == 2


@pytest.mark.parametrize("lanes", [None, "2", "4", "8", "16", "32"])
@pytest.mark.parametrize("ny", [64, 1024, 2048])
def test_lanes_asked_for(monkeypatch, ny, lanes):
    """every width that HST_LINE_LANES can ask for: from about 910 rows two lanes have no room, from about 1820 four,
    and the context then keeps its own width; the steps and every kind of line solve run either way"""
    if lanes:
        monkeypatch.setenv("HST_LINE_LANES", lanes)
    deck = c1_deck(nx=3, nz=2, ny=ny, exact_shift=True, deltat=0.0005)
    V0 = seeded_field(deck, seed=2, k0=3.0)
    s, o = make_pair(deck, V0)
    Vg, Vo = run_pair(s, o, deck["deltat"], 1)
    # the tall lines are ill-conditioned in proportion to ny^2 (2e-13 at 512 rows)
    assert rel_l2(Vg, Vo) <= 1e-12 * max(1.0, (ny / 512) ** 2)
    shift = s.shear_shifts(0.37)
    for c in range(3):
        o.field(c)[...] = Vg[c]
    for kind in (hst.KIND_D2V, hst.KIND_ETA, hst.KIND_POISSON, hst.KIND_D0, hst.KIND_DY):
        s.upload(hst.RHS1, np.zeros(s.shape, np.complex128))
        s.line_solve(kind, 123.4, hst.V2, hst.RHS1, shift=shift)
        o.field(5)[...] = 0.0
        o.line_solve(kind, 123.4, 1, 5, shift=shift)
        assert rel_l2(s.download(hst.RHS1), o.field(5)) <= 1e-11 * max(1.0, (ny / 512) ** 2), kind
    s.close()


@pytest.mark.parametrize("ny", [1024, 2048])
def test_autotune_leaves_out_what_has_no_room(ny):
    """tall lines: four lanes have no room at 2048 rows, and the others are tried"""
    deck = c1_deck(nx=3, nz=2, ny=ny)
    V0 = seeded_field(deck, seed=2, k0=3.0)
    s = hst.Solver(deck)
    s.time = 0.0
    s.set_velocity(V0)
    before = s.velocity()
    report = s.autotune(deck["deltat"], steps=1)
    assert [f"P={P}:" in report for P in (32, 16, 8, 4)] == [True, True, True, ny == 1024], report
    assert np.array_equal(s.velocity(), before)
    s.timestep(deck["deltat"])
    s.close()


@pytest.mark.parametrize("ny,exact,linear", [(34, False, False), (34, True, False), (150, False, False), (64, True, True),
                                             (30, False, True)])
def test_streamed_right_hand_sides_equal_row_by_row(monkeypatch, ny, exact, linear):
    """the streamed right-hand sides against the row-by-row ones (HST_RHS_TILED=0, read at every step): the two sum
    the products in another order, so they differ by rounding only (1e-13)"""
    deck = c1_deck(nx=15, nz=16, ny=ny, exact_shift=exact, linear=linear, damp_kpar=3.0, damp_kperp=2.0, damp_rate=0.5,
                   damp_edge=0.3, s2_amplitude=0.3, s2_period=0.7, time=0.2)
    V0 = seeded_field(deck, seed=4)
    out = []
    for env in (None, "0"):
        if env is not None:
            monkeypatch.setenv("HST_RHS_TILED", env)
        s = hst.Solver(deck)
        s.time = deck["time"]
        s.set_velocity(V0)
        for _ in range(2):
            s.timestep(deck["deltat"])
        out.append(np.concatenate([s.velocity(), s.download(hst.OLD1)[None], s.download(hst.OLD2)[None]]))
        s.close()
    for a, b in zip(*out):
        assert rel_l2(a, b) <= 1e-13


@pytest.mark.parametrize("over", [dict(), dict(damp_hard=True, damp_kpar=2.0, damp_kperp=2.0, s2_amplitude=0.5, s2_period=0.7)])
def test_the_first_steps_allocate_nothing(over, tmp_path):
    """every buffer of a step, the pinned copies of a turning damping table among them, is there once the context is"""
    s = hst.Solver(c1_deck(exact_shift=True, **over))
    s.time = 0.1
    calls = [e["name"] for e in traced(s, 2, tmp_path) if e.get("cat") == "cuda_runtime"]
    s.close()
    assert any("Launch" in c for c in calls)
    assert not [c for c in calls if "Malloc" in c or "HostAlloc" in c], calls


@pytest.mark.parametrize("change", ["tables", "autotune"])
def test_queued_steps_keep_their_tables(change):
    """new tables (and the trial tables of autotuning) take effect after the steps that are still queued: the same bits
    as when the caller waits for those steps first"""
    deck = c1_deck(nx=31, nz=32, ny=64, exact_shift=True)
    other = hst.Solver(dict(deck, ystretch=0.8))
    out = []
    for wait in (True, False):
        s = hst.Solver(deck)
        s.time = 0.0
        s.set_velocity(seeded_field(deck, seed=3))
        s.timesteps(200)
        if wait:
            s.sync()
        if change == "tables":
            s.set_tables(der=other.der, y=other.y, dyl=other.dyl)
        else:
            s.autotune(deck["deltat"], steps=1)
        out.append(s.velocity())
        s.close()
    other.close()
    assert np.array_equal(*out)


def test_a_replaced_grid_is_not_taken_as_uniform():
    """a caller that replaces der, y and dyl of a uniform deck by a stretched grid's gets the stretched deck's result
    (the node phases must follow the y table, not the deck), in both forms of the shift"""
    for exact in (False, True):
        deck = c1_deck(nx=7, nz=8, ny=32, exact_shift=exact, ystretch=0.8)
        V0 = seeded_field(deck, seed=3)
        a = hst.Solver(deck)
        b = hst.Solver(dict(deck, ystretch=0.0))
        b.set_tables(der=a.der, y=a.y, dyl=a.dyl)
        for s in (a, b):
            s.time = 0.0
            s.set_velocity(V0)
            s.timestep(deck["deltat"])
        assert rel_l2(b.velocity(), a.velocity()) <= 1e-14
        a.close()
        b.close()


@pytest.mark.parametrize("ny", [10, 34, 64, 150])
def test_outstats_rows(ny):
    """the statistics and the column energies on uneven slabs against the oracle (1e-12: sums of one sign, and the
    stresses' cancelling ones scaled by the variances)"""
    deck = c1_deck(nx=9, nz=8, ny=ny, s2_amplitude=0.3, s2_period=0.7, time=0.1)
    s, o = make_pair(deck, seeded_field(deck, seed=6))
    sums, exz = s.outstats_sums()
    want, exz_o = o.outstats_sums()
    got = np.array([sums[k] for k in hst.Solver.SUM_NAMES])
    assert np.abs(got - want).max() <= 1e-12 * np.abs(want).max()
    assert np.abs(exz - exz_o).max() <= 1e-12 * exz_o.max()
    s.close()


@pytest.mark.parametrize("ny", [10, 30, 150, 258])
def test_line_solve_rows(ny):
    """every kind of line solve on uneven slabs against the oracle"""
    deck = c1_deck(nx=5, nz=4, ny=ny, ystretch=0.5 if ny == 150 else 0.0)
    s, o = make_pair(deck, seeded_field(deck, seed=8))
    rng = np.random.default_rng(ny)
    f = rng.standard_normal(s.shape) + 1j * rng.standard_normal(s.shape)
    shift = s.shear_shifts(0.37)
    s.upload(hst.V2, f)
    s.fill_ghosts(hst.V2, *shift)
    f = s.download(hst.V2)
    for kind, lam in ((hst.KIND_D2V, 2.5e4), (hst.KIND_ETA, 3.0e3), (hst.KIND_POISSON, 0.0), (hst.KIND_D0, 0.0),
                      (hst.KIND_DY, 0.0)):
        s.upload(hst.RHS1, np.zeros(s.shape, np.complex128))
        s.line_solve(kind, lam, hst.V2, hst.RHS1, shift=shift)
        o.field(1)[...] = f
        o.field(5)[...] = 0.0
        o.line_solve(kind, lam, 1, 5, shift=shift)
        assert rel_l2(s.download(hst.RHS1), o.field(5)) <= 1e-11, kind
    s.close()
