"""stream_kernel with one correlation: compiled for one block per SM where a
pass has no more steps than the GPU has SMs, otherwise not.

Tolerance: as for every pass, 1e-4 of the FP64 oracle.
"""
import numpy as np
import pytest

from oracle import oracle_ffi as of
from tests import helpers as H

RTOL = 1e-4


@pytest.mark.gpu
@pytest.mark.parametrize("n_cb", [2, 160])
@pytest.mark.parametrize("n_dir", [3, 4, 5, 8, 10, 16])
def test_pass_matches_fp64_oracle(built, n_dir, n_cb):
    """A step per channel block and more: 2 blocks are far fewer steps than
    SMs, 160 more than any B200 has."""
    obs = H.small_observation(n_stations=11, n_directions=n_dir, n_channels=2 * n_cb, n_cb=n_cb,
                              n_times=2, seed=53, n_sources=2)
    prob = H.problem_from_observation(obs, 1, 1)
    sol0 = H.perturbed_start(obs, prob, scale=0.1)
    ref = of.perform_iteration(prob, sol0, precision=64)
    got = H.make_solver(prob).PerformIteration(H.solve_data_from_problem(prob), sol0)
    err = np.abs(got - ref) / np.maximum(np.abs(ref), 1e-12)
    assert np.nanmax(err) < RTOL, np.nanmax(err)
