"""The control step of the pipelined solve: the CTA that runs it replaces the
non-finite solutions of a pass and decides on every interval of a batch, with
all of its warps, once every CTA has finalised the pass.

Tolerance: 1e-4, the parity contract of a solve (after phase referencing; the
replaced solutions, means of amplitudes of solved ones, as they are).
"""
import numpy as np
import pytest

from oracle import oracle_ffi as of
from tests import helpers as H

RTOL_SOLVE = 1e-4


def _flag_antenna(prob, antenna, blocks):
    """Zeroes an antenna's visibilities in some channel blocks: its denominator
    is zero there and its solutions are replaced after every pass."""
    for cb in blocks:
        ap = prob["antenna_pairs"][cb]
        bad = (ap[:, 0] == antenna) | (ap[:, 1] == antenna)
        prob["data"][cb][bad] = 0
        prob["model"][cb][:, bad] = 0


@pytest.mark.gpu
@pytest.mark.parametrize("n_dir,n_st,n_intervals", [(2, 9, 1), (2, 9, 5), (21, 30, 3)])
def test_non_finite_blocks_of_every_interval(built, n_dir, n_st, n_intervals):
    """One interval and batches, each interval with an antenna of its own
    flagged in its last channel block (11 and 7 consumer warps)."""
    from dp3_b200 import ddsolve
    n_it, n_cb = 12, 3
    probs, refs, its = [], [], []
    for g in range(n_intervals):
        obs = H.small_observation(n_stations=n_st, n_directions=n_dir, n_channels=6, n_cb=n_cb,
                                  n_times=2, seed=40 + g, n_sources=2)
        prob = H.problem_from_observation(obs)
        _flag_antenna(prob, 1 + g, [n_cb - 1])
        ref = H.unit_solutions(prob)
        r, _ = of.solve(prob, ref, of.settings(max_iterations=n_it, accuracy=1e-30,
                                               detect_stalling=False), precision=64, n_threads=2)
        probs.append(prob)
        refs.append(ref)
        its.append(r.iterations)
    st = ddsolve.default_settings()
    st.max_iterations, st.accuracy, st.detect_stalling = n_it, 1e-30, 0
    ctx = ddsolve.Context(n_st, [1] * n_dir, n_intervals * n_cb, 2, 2)
    ctx.set_settings(st)
    if n_intervals > 1:
        ctx.set_intervals([g * n_cb for g in range(n_intervals + 1)])
    for g, prob in enumerate(probs):
        for cb in range(n_cb):
            ctx.set_channel_block(g * n_cb + cb, prob["data"][cb], prob["model"][cb],
                                  prob["antenna_pairs"][cb], prob["solution_map"][cb])
    sol = np.ones((n_intervals * n_cb,) + refs[0].shape[1:], np.complex128)
    res = ctx.solve_batch(sol) if n_intervals > 1 else [ctx.solve(sol)]
    ctx.close()
    for g, ref in enumerate(refs):
        got = sol[g * n_cb:(g + 1) * n_cb]
        assert res[g].iterations == its[g]
        np.testing.assert_allclose(got[-1, 1 + g], ref[-1, 1 + g], rtol=RTOL_SOLVE)
        ok = np.arange(n_st) != 1 + g
        assert H.max_rel_diff(got[:, ok], ref[:, ok]) < RTOL_SOLVE


@pytest.mark.gpu
@pytest.mark.parametrize("n_dir,n_intervals,max_iterations", [(2, 1, 70), (2, 3, 5), (21, 1, 5)])
def test_wait_limit_ends_the_solve(built, n_dir, n_intervals, max_iterations):
    """A grid barrier that is never complete: the solve ends with an error
    within the limit of its waits, the launches queued behind it do nothing,
    and the next solve on the context is what it was before (the same bits:
    every sum has a fixed order)."""
    from dp3_b200 import ddsolve
    n_cb = 2
    obs = H.small_observation(n_stations=12, n_directions=n_dir, n_channels=4, n_cb=n_cb,
                              n_times=2, seed=3, n_sources=2)
    st = ddsolve.default_settings()
    st.max_iterations, st.accuracy, st.detect_stalling = max_iterations, 1e-30, 0
    ctx = ddsolve.Context(12, [1] * n_dir, n_intervals * n_cb, 2, 2)
    ctx.set_settings(st)
    if n_intervals > 1:
        ctx.set_intervals([g * n_cb for g in range(n_intervals + 1)])
    for cb in range(n_intervals * n_cb):
        ctx.set_channel_block_regular(cb, 2, obs.cfg.n_baselines, obs.cfg.cb_channels[cb % n_cb],
                                      obs.data[cb % n_cb], obs.model[cb % n_cb], obs.antenna1,
                                      obs.antenna2)
    solve = ctx.solve_batch if n_intervals > 1 else ctx.solve
    before = np.ones((n_intervals * n_cb, 12, n_dir, 2), np.complex128)
    solve(before)
    assert ddsolve.lib().ddsolve_check_wait_limit(ctx._h, 20) == 5
    after = np.ones_like(before)
    solve(after)
    ctx.close()
    np.testing.assert_array_equal(after, before)


@pytest.mark.gpu
def test_launches_stop_with_the_solve(built):
    """However many iterations are allowed, a solve that stops early has queued
    at most one launch in vain (of 64 iterations each, for a small array)."""
    obs = H.small_observation(n_stations=10, n_directions=2, n_channels=6, n_cb=2,
                              n_times=2, seed=17)
    prob = H.problem_from_observation(obs)
    solver = H.make_solver(prob, max_iterations=6400, accuracy=1e-2, detect_stalling=False)
    sol = H.unit_solutions(prob)
    res = solver.Solve(H.solve_data_from_problem(prob), sol, 0.0)
    assert res.iterations <= 64
    assert solver._ctx.last_launch_count() <= 2 + 3, solver._ctx.last_launch_count()


@pytest.mark.gpu
def test_launches_are_bounded_in_time(built):
    """Launches of many passes over a large interval would hold the GPU from
    other contexts: 40 passes over 266 MB take two launches."""
    from dp3_b200 import ddsolve
    n_st, n_dir, n_cb, n_t, n_ch = 62, 10, 10, 10, 8
    a1, a2 = (x.astype(np.uint32) for x in np.triu_indices(n_st, 1))
    rng = np.random.default_rng(0)
    model = rng.standard_normal((n_dir, n_t * len(a1) * n_ch, 2, 2), dtype=np.float32)
    data = model.sum(0)
    st = ddsolve.default_settings()
    st.max_iterations, st.accuracy, st.detect_stalling = 40, 1e-30, 0
    ctx = ddsolve.Context(n_st, [1] * n_dir, n_cb, 2, 2)
    ctx.set_settings(st)
    for cb in range(n_cb):
        ctx.set_channel_block_regular(cb, n_t, len(a1), n_ch, data, model, a1, a2)
    sol = np.full((n_cb, n_st, n_dir, 2), 1.1 + 0.1j)
    assert ctx.solve(sol).iterations == 41  # the cap, not converged
    assert 2 + 2 <= ctx.last_launch_count() <= 2 + 3
    ctx.close()
    # every block holds the same data (its rows split over other CTAs)
    assert np.isfinite(sol).all() and H.max_rel_diff(sol[:1], sol[-1:]) < RTOL_SOLVE
