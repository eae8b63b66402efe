"""The pipelined pass at the sizes where its layout changes: the wide variant
for 13 to 20 directions, and tiles whose sums are staged in the ring stage of
their last row, up to the largest array that fits.

Tolerance: as for every pass, 1e-4 of the FP64 oracle.
"""
import numpy as np
import pytest

from oracle import oracle_ffi as of
from tests import helpers as H

RTOL = 1e-4


@pytest.mark.gpu
@pytest.mark.parametrize("powers", [0, 1])
@pytest.mark.parametrize("npol,n_dir,n_st", [
    (2, 20, 140), (2, 16, 256), (2, 16, 295), (2, 13, 374), (2, 20, 229), (2, 21, 219),
    (2, 5, 400), (2, 5, 512), (2, 4, 600), (1, 5, 900), (2, 40, 95), (2, 48, 72), (1, 16, 512), (1, 16, 576), (1, 20, 468), (1, 36, 223)])
def test_pass_and_solve(built, npol, n_dir, n_st, powers):
    from dp3_b200 import ddsolve
    n_cb, n_it = 2, 3
    obs = H.small_observation(n_stations=n_st, n_directions=n_dir, n_channels=3, n_cb=n_cb,
                              n_times=1, seed=n_st, n_sources=1)
    prob = H.problem_from_observation(obs, 2, npol)
    sol0 = H.perturbed_start(obs, prob, scale=0.1)
    st = ddsolve.default_settings()
    st.max_iterations, st.accuracy, st.detect_stalling = n_it, 1e-30, 0
    assert ddsolve.describe_layout(n_st, n_dir, 2, npol).pipelined
    ctx = ddsolve.Context(n_st, [1] * n_dir, n_cb, 2, npol)
    ctx.set_settings(st)
    ctx.set_plan_tuning(model_powers=powers)
    for cb in range(n_cb):
        ctx.set_channel_block_regular(cb, 1, obs.cfg.n_baselines, obs.cfg.cb_channels[cb],
                                      prob["data"][cb], prob["model"][cb], obs.antenna1,
                                      obs.antenna2)
    got = ctx.perform_iteration(sol0)
    ref = of.perform_iteration(prob, sol0, precision=64)
    err = np.abs(got - ref) / np.maximum(np.abs(ref), 1e-12)
    assert np.nanmax(err) < RTOL, np.nanmax(err)
    sol, want = sol0.copy(), sol0.copy()
    ctx.solve(sol)
    # one launch of pipe_kernel beside the three that prepare it
    assert ctx.last_launch_count() <= 4
    ctx.close()
    of.solve(prob, want, of.settings(max_iterations=n_it, accuracy=1e-30, detect_stalling=False),
             precision=64)
    assert H.max_rel_diff(sol, want) < RTOL
