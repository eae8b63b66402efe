"""Paths of the pipelined pass that its other tests do not take: model powers
precomputed or summed in the row loop on every lane layout, a pass that is
begun and given up because the solve has stopped, chains of passes over several
launches.

Tolerance: a pass and a solve within 1e-4 of the FP64 oracle; runs of the same
sums in the same order give the same bits.
"""
import numpy as np
import pytest

from oracle import oracle_ffi as of
from tests import helpers as H

pytestmark = pytest.mark.gpu

RTOL = 1e-4


def _context(prob, obs, **settings):
    from dp3_b200 import ddsolve
    st = ddsolve.default_settings()
    for k, v in settings.items():
        setattr(st, k, v)
    cfg = obs.cfg
    ctx = ddsolve.Context(cfg.n_stations, list(cfg.nspd), cfg.n_channel_blocks,
                          prob["n_correlations"], prob["n_pol"])
    ctx.set_settings(st)
    for cb, n_ch in enumerate(cfg.cb_channels):
        ctx.set_channel_block_regular(cb, cfg.n_times, cfg.n_baselines, n_ch, prob["data"][cb],
                                      prob["model"][cb], obs.antenna1, obs.antenna2)
    return ctx


@pytest.mark.parametrize("powers", [0, 1])
@pytest.mark.parametrize("ncorr,npol,n_dir,n_st", [
    (2, 2, 1, 62), (2, 2, 5, 23), (2, 2, 6, 23), (2, 2, 10, 27), (2, 2, 20, 20), (2, 2, 23, 23),
    (2, 2, 48, 9), (2, 1, 1, 9), (2, 1, 7, 23), (2, 1, 19, 9), (2, 1, 24, 21), (2, 1, 41, 13),
    (4, 2, 1, 23), (4, 2, 3, 30), (4, 2, 5, 9), (4, 2, 12, 23), (4, 2, 24, 9), (4, 1, 2, 23),
    (4, 1, 6, 23), (4, 1, 11, 13), (4, 1, 23, 9)])
def test_model_powers(built, ncorr, npol, n_dir, n_st, powers):
    from dp3_b200 import ddsolve
    assert ddsolve.describe_layout(n_st, n_dir, ncorr, npol).pipelined
    obs = H.small_observation(n_stations=n_st, n_directions=n_dir, n_channels=7, n_cb=2,
                              n_times=3, seed=37)
    prob = H.problem_from_observation(obs, ncorr, npol, leakage=0.05)
    sol0 = H.perturbed_start(obs, prob)
    ref = of.perform_iteration(prob, sol0, precision=64)
    ctx = _context(prob, obs)
    ctx.set_plan_tuning(use_pipe=1, model_powers=powers)
    got = ctx.perform_iteration(sol0)
    ctx.close()
    err = np.abs(got - ref) / np.maximum(np.abs(ref), 1e-12)
    assert np.nanmax(err) < RTOL, np.nanmax(err)


def test_solve_stops_on_a_pass_already_begun(built):
    """The step falls from more than twice the accuracy to below it in one
    iteration: the next pass has begun when the verdict comes. It changes
    nothing, and the next solve on the context finds everything in order."""
    obs = H.small_observation(n_stations=12, n_directions=1, n_channels=6, n_cb=2,
                              n_times=2, seed=17)
    prob = H.problem_from_observation(obs)
    sol0 = H.perturbed_start(obs, prob, scale=0.3)
    kw = dict(max_iterations=14, detect_stalling=False, step_size=0.6)
    _, mags = of.solve(prob, sol0.copy(), of.settings(accuracy=1e-30, **kw), precision=64,
                       n_threads=2)
    k = 2
    accuracy = 1.1 * mags[k]
    assert mags[:k].min() > 2.2 * accuracy
    ref = sol0.copy()
    r, ref_mags = of.solve(prob, ref, of.settings(accuracy=accuracy, **kw), precision=64,
                           n_threads=2)
    assert r.iterations == k + 1 and r.has_converged
    ctx = _context(prob, obs, accuracy=accuracy, **kw)
    sols = []
    for _ in range(3):
        got, got_mags = sol0.copy(), np.zeros(14)
        res = ctx.solve(got, got_mags)
        assert res.iterations == r.iterations and res.has_converged
        np.testing.assert_allclose(got_mags[:k + 1], ref_mags[:k + 1], rtol=1e-3)
        assert not got_mags[k + 1:].any()
        assert H.max_rel_diff(got, ref) < RTOL
        sols.append(got)
    ctx.close()
    np.testing.assert_array_equal(sols[1], sols[0])
    np.testing.assert_array_equal(sols[2], sols[0])


@pytest.mark.parametrize("device", [False, True])
@pytest.mark.parametrize("n_passes", [1, 64, 65, 130])
def test_chain_of_several_launches(built, n_passes, device):
    """Passes chained on the device are the passes one by one, bit for bit."""
    import torch
    obs = H.small_observation(n_stations=12, n_directions=1, n_channels=6, n_cb=2,
                              n_times=2, seed=19)
    prob = H.problem_from_observation(obs)
    ctx = _context(prob, obs)
    sol0 = H.perturbed_start(obs, prob, scale=0.1)
    want, sol = [], sol0
    for _ in range(n_passes):
        sol = ctx.perform_iteration(sol)
        want.append(sol)
    start = torch.from_numpy(sol0).cuda() if device else sol0
    got = ctx.perform_iterations(start, n_passes)
    if device:
        got = got.cpu().numpy()
    ctx.close()
    assert np.isfinite(want[-1]).all()
    np.testing.assert_array_equal(got, np.stack(want))
