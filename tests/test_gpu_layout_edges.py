"""Edges of the kernels' register and shared-memory layouts, bit for bit against the oracle."""
import numpy as np
import pytest

from bubbleensemble_implicitextension_b200 import workloads as W
from tests.helpers import assert_bitwise, ragged_ensemble, run_gpu

pytestmark = pytest.mark.gpu

KEYS = ["state", "uacc", "iuacc", "n_accepted", "n_rejected", "n_bicg_iter", "n_rhs", "status"]


@pytest.mark.parametrize("rec", [0, 1])
@pytest.mark.parametrize("n,bw", [(7, 3), (9, 4), (33, 3), (66, 4), (97, 5)])
def test_banded_operator_around_its_register_diagonals(n, bw, rec, gpu, oracle_lib):
    """2 bw + 1 diagonals below, at and above the eight kept in registers, and a band of every column."""
    ens = W.ring_ensemble(n_systems=3, n_units=n, band_width=bw)
    ens.max_steps_per_period = 300
    got = run_gpu(ens, n_periods=1, reset_at=-1, bicg_recurrence=rec)
    want = oracle_lib.run(ens, n_periods=1, reset_at=-1, bicg_variant=rec)
    assert_bitwise(got, want, KEYS)


def _bounded(ens, budget=250):
    ens.max_steps_per_period = budget
    return ens


@pytest.mark.parametrize("rec", [0, 1])
def test_own_matrices_at_the_edges_of_the_work_splits(rec, gpu, oracle_lib):
    """Pairs of rows and column groups of one warp (N <= 32, in runs of 8, 16 and 32 columns), quads of rows with
    every remainder of N mod 4 on two and on four warps."""
    ens = _bounded(ragged_ensemble([1, 2, 3, 8, 9, 15, 16, 17, 31, 32, 33, 35, 63, 64, 65, 66, 67, 126, 128], seed=5))
    got = run_gpu(ens, n_periods=1, reset_at=-1, bicg_recurrence=rec)
    want = oracle_lib.run(ens, n_periods=1, reset_at=-1, bicg_variant=rec)
    assert_bitwise(got, want, KEYS)


@pytest.mark.parametrize("rec", [0, 1])
@pytest.mark.parametrize("factored", [False, True])
@pytest.mark.parametrize("n", [7, 16, 17, 31, 34, 63, 65, 99, 127])
def test_shared_matrices_at_the_edges_of_the_work_splits(n, factored, rec, gpu, oracle_lib):
    """One matrix for the launch, symmetric with unit factors or not, at odd sizes of every class."""
    ens = _bounded(W.c3_ensemble(n_systems=3, n_units=n, n_periods=1, cube_um=400.0 * (n / 32) ** (1 / 3),
                                 factored=factored), 120)
    got = run_gpu(ens, n_periods=1, reset_at=-1, bicg_recurrence=rec, shared_matrices=True)
    want = oracle_lib.run(ens, n_periods=1, reset_at=-1, bicg_variant=rec, shared_assoc=factored or n > 32)
    assert_bitwise(got, want, KEYS)


@pytest.mark.parametrize("rec", [0, 1])
def test_step_budget_inside_an_event_and_two_frequencies(rec, gpu, oracle_lib):
    """The dual-frequency drive of the uneven clouds (both elementary-function paths) with a small step budget."""
    ens = _bounded(W.c2_ensemble(n_systems=24, seed=8, n_periods=2, reset_at=1), 200)
    got = run_gpu(ens, bicg_recurrence=rec)
    want = oracle_lib.run(ens, n_periods=2, reset_at=1, bicg_variant=rec)
    assert_bitwise(got, want, KEYS)


@pytest.mark.parametrize("rec", [0, 1])
def test_one_warp_systems(rec, gpu, oracle_lib):
    """Systems of up to 32 units on one warp each (few systems run on teams of four by default), own matrices and
    one shared symmetric matrix."""
    ens = _bounded(ragged_ensemble([1, 2, 7, 8, 9, 15, 16, 17, 24, 31, 32], seed=6))
    got = run_gpu(ens, n_periods=1, reset_at=-1, bicg_recurrence=rec, warps_per_system=1)
    want = oracle_lib.run(ens, n_periods=1, reset_at=-1, bicg_variant=rec)
    assert_bitwise(got, want, KEYS)
    for n in (9, 32):
        ens = _bounded(W.c1_ensemble(n_pa=2, n_f=2, n_units=n, factored=True))
        got = run_gpu(ens, n_periods=1, reset_at=-1, bicg_recurrence=rec, warps_per_system=1)
        want = oracle_lib.run(ens, n_periods=1, reset_at=-1, bicg_variant=rec, shared_assoc=True)
        assert_bitwise(got, want, KEYS)


@pytest.mark.parametrize("rec", [0, 1])
@pytest.mark.parametrize("banded", [False, True])
@pytest.mark.parametrize("n,systems", [(66, 301), (35, 597)])
def test_more_systems_than_eight_warps_an_sm_hold(n, systems, banded, rec, gpu, oracle_lib):
    """The kernels compiled for sixteen warps an SM: shared symmetric matrix and banded storage, two and four warps."""
    ens = (W.ring_ensemble(n_systems=systems, n_units=n, band_width=2) if banded
           else W.c3_ensemble(n_systems=systems, n_units=n, n_periods=1))
    ens = _bounded(ens, 12)
    got = run_gpu(ens, n_periods=1, reset_at=-1, bicg_recurrence=rec)
    want = oracle_lib.run(ens, n_periods=1, reset_at=-1, bicg_variant=rec)
    assert_bitwise(got, want, KEYS)


@pytest.mark.parametrize("systems", [4, 200, 700])
def test_unit_factors_need_a_shared_matrix(systems, gpu):
    """Coupling factors other than 1 with a matrix per system are refused whichever one-warp kernel or team the
    number of systems selects."""
    from bubbleensemble_implicitextension_b200 import solver as S
    ens = W.c1_ensemble(n_pa=systems, n_f=1, n_units=8)
    ps = ens.make_solver()
    try:
        ps.set_array(S.ListOfVariables.CouplingRowScale, np.full(ens.total_units, 2.0))
        ps.SynchroniseFromHostToDevice(S.ListOfVariables.All)
        with pytest.raises(S.BesError, match="CouplingRowScale"):
            ps.solve_periods(1, -1)
    finally:
        ps.close()


@pytest.mark.parametrize("n,bw,systems", [(20, 2, 4), (50, 1, 4), (128, 1, 320), (128, 9, 4), (32, 9, 4)])
def test_unit_factors_are_refused_with_banded_storage(n, bw, systems, gpu):
    """Narrow and wide bands on one, two and four warps, and the kernel of many systems."""
    from bubbleensemble_implicitextension_b200 import solver as S
    ens = W.ring_ensemble(n_systems=systems, n_units=n, band_width=bw)
    ps = ens.make_solver()
    try:
        ps.set_array(S.ListOfVariables.CouplingColumnScale, np.full(ens.total_units, 2.0))
        ps.SynchroniseFromHostToDevice(S.ListOfVariables.All)
        with pytest.raises(S.BesError, match="CouplingColumnScale"):
            ps.solve_periods(1, -1)
    finally:
        ps.close()


@pytest.mark.parametrize("wps", [0, 1])
def test_autotuner_leaves_the_kernel_of_small_systems_to_the_rule(wps, gpu):
    """A capped run is no measure of teams against one warp a system: only warps per CTA are tuned there (teams: 4
    and 8 warps; one warp: 1, 2 and 4)."""
    from bubbleensemble_implicitextension_b200 import solver as S
    ens = _bounded(W.c1_ensemble(n_pa=2, n_f=2, n_units=32, factored=True), 50)
    ps = ens.make_solver()
    try:
        ps.SolverOption(S.ListOfSolverOptions.WarpsPerSystem, wps)
        ps.SynchroniseFromHostToDevice(S.ListOfVariables.All)
        tuned = ps.autotune(n_periods=1, step_cap=20)
        assert tuned["warps_per_system"][0] == wps
        assert tuned["candidates"] == (3 if wps else 2)
    finally:
        ps.close()
