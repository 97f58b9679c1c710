"""Edges of the kernels' register and shared-memory layouts, bit for bit against the oracle."""
import numpy as np
import pytest

from bubbleensemble_implicitextension_b200 import workloads as W
from tests.helpers import assert_bitwise, run_gpu

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
