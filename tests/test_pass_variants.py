"""The pipelined pass over the lane layouts it chooses from: directions per
lane and lanes per run change at 5, 10, 20 and 48 directions (two
correlations) and at 3, 6, 12 and 24 (four), and a solve of more than 64
iterations takes several launches.

Tolerance: a pass sums fewer than 1e3 FP32 products per element in chains of
at most 1e2 (eps 6e-8 each, against terms of the same sign in the denominator):
1e-5 at worst before the division; 1e-4 is the parity contract of a pass and
of a solve.
"""
import numpy as np
import pytest

from oracle import oracle_ffi as of
from tests import helpers as H

pytestmark = pytest.mark.gpu

RTOL = 1e-4


@pytest.mark.parametrize("ncorr,npol,n_dir,n_stations", [
    (2, 2, 1, 62), (2, 2, 5, 23), (2, 2, 6, 23), (2, 2, 10, 27), (2, 2, 11, 9),
    (2, 2, 20, 20), (2, 2, 21, 23), (2, 2, 40, 13), (2, 2, 48, 9),
    (2, 1, 1, 9), (2, 1, 5, 62), (2, 1, 7, 23), (2, 1, 20, 9), (2, 1, 24, 21),
    (4, 2, 1, 23), (4, 2, 3, 62), (4, 2, 4, 9), (4, 2, 7, 23), (4, 2, 13, 13),
    (4, 2, 24, 9), (4, 1, 5, 23), (4, 1, 24, 9)])
def test_pass_matches_fp64_oracle(built, ncorr, npol, n_dir, n_stations):
    obs = H.small_observation(n_stations=n_stations, n_directions=n_dir, n_channels=7,
                              n_cb=2, n_times=3, seed=31)
    prob = H.problem_from_observation(obs, ncorr, npol, leakage=0.05)
    sol0 = H.perturbed_start(obs, prob)
    ref = of.perform_iteration(prob, sol0, precision=64)
    got = H.make_solver(prob).PerformIteration(H.solve_data_from_problem(prob), sol0)
    err = np.abs(got - ref) / np.maximum(np.abs(ref), 1e-12)
    assert np.nanmax(err) < RTOL, np.nanmax(err)


@pytest.mark.parametrize("iterations", [1, 2, 64, 65, 130])
def test_solve_of_several_launches(built, iterations):
    obs = H.small_observation(n_stations=10, n_directions=2, n_channels=6, n_cb=2,
                              n_times=2, seed=17)
    prob = H.problem_from_observation(obs)
    sol0 = H.perturbed_start(obs, prob, scale=0.05)
    st = of.settings(max_iterations=iterations, accuracy=1e-30, detect_stalling=False)
    ref = sol0.copy()
    r, mags = of.solve(prob, ref, st, precision=64, n_threads=2)
    solver = H.make_solver(prob, max_iterations=iterations, accuracy=1e-30,
                           detect_stalling=False)
    got = sol0.copy()
    res = solver.Solve(H.solve_data_from_problem(prob), got, 0.0)
    assert res.iterations == r.iterations
    assert len(res.step_magnitudes) == len(mags)
    assert H.max_rel_diff(got, ref) < RTOL
