"""The one-warp kernels of systems of up to 32 units (own matrices with the column share in shared or in tensor
memory, one shared symmetric matrix) bit for bit against the oracle, at the numbers of systems that select them:
fewer systems than SMs run on teams of four warps by default."""
import numpy as np
import pytest

from bubbleensemble_implicitextension_b200 import workloads as W
from tests.helpers import assert_bitwise, ragged_ensemble, run_gpu

pytestmark = pytest.mark.gpu

KEYS = ["state", "uacc", "iuacc", "n_accepted", "n_rejected", "n_bicg_iter", "n_rhs", "status"]


def _check(ens, budget, rec, oracle_lib, shared=False, **options):
    ens.max_steps_per_period = budget
    got = run_gpu(ens, n_periods=1, reset_at=-1, bicg_recurrence=rec, **options)
    want = oracle_lib.run(ens, n_periods=1, reset_at=-1, bicg_variant=rec, shared_assoc=shared)
    assert_bitwise(got, want, KEYS)


@pytest.mark.parametrize("rec", [0, 1])
def test_32_units_own_matrices_few_systems(rec, gpu, oracle_lib):
    """Column share in tensor memory, no guards on N."""
    _check(ragged_ensemble([32] * 5, seed=3), 250, rec, oracle_lib, warps_per_system=1)


@pytest.mark.parametrize("rec", [0, 1])
@pytest.mark.parametrize("systems", [160, 600])
def test_32_units_own_matrices(systems, rec, gpu, oracle_lib):
    """Tensor memory up to four systems an SM, shared memory beyond."""
    _check(ragged_ensemble([32] * systems, seed=4), 25, rec, oracle_lib)


@pytest.mark.parametrize("rec", [0, 1])
@pytest.mark.parametrize("systems", [160, 600])
def test_mixed_units_own_matrices(systems, rec, gpu, oracle_lib):
    sizes = [1, 2, 7, 8, 9, 15, 16, 17, 24, 31, 32]
    _check(ragged_ensemble([sizes[k % len(sizes)] for k in range(systems)], seed=5), 25, rec, oracle_lib)


@pytest.mark.parametrize("rec", [0, 1])
def test_mixed_units_beside_larger_systems(rec, gpu, oracle_lib):
    """The column share stays in shared memory where systems of more than one warp run beside them."""
    sizes = [3, 8, 17, 32, 33, 70]
    _check(ragged_ensemble([sizes[k % len(sizes)] for k in range(160)], seed=6), 12, rec, oracle_lib)


@pytest.mark.parametrize("rec", [0, 1])
@pytest.mark.parametrize("n,systems", [(32, 160), (32, 310), (31, 310), (17, 310), (9, 310), (2, 310)])
def test_one_shared_symmetric_matrix(n, systems, rec, gpu, oracle_lib):
    ens = W.c1_ensemble(n_pa=systems, n_f=1, n_units=n, factored=True, f_range=(60.0, 60.0))
    _check(ens, 25, rec, oracle_lib, shared=True)


@pytest.mark.parametrize("rec", [0, 1])
@pytest.mark.parametrize("wps,shapes", [(1, (1, 2, 4)), (0, (4, 8))])
@pytest.mark.parametrize("factored", [False, True])
def test_warps_per_block_of_one_warp_systems_and_teams(factored, wps, shapes, rec, gpu):
    """Shapes that differ: one to four one-warp systems a CTA, one and two teams a CTA."""
    ens = W.c1_ensemble(factored=factored).subset(list(range(0, 256, 37)))
    ens.max_steps_per_period = 250
    runs = [run_gpu(ens, n_periods=1, reset_at=-1, warps_per_system=wps, warps_per_block=wpb, bicg_recurrence=rec)
            for wpb in shapes]
    for other in runs[1:]:
        assert_bitwise(other, runs[0], KEYS)
