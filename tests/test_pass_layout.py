"""The packed layout and the kernel chosen for a context's dimensions (CPU)."""
import pytest

# Most stations with 1, 2, ... directions for which a ring of two bulk-copy
# stages fits, by correlations and solution polarizations.
STATIONS = {
    (2, 2): (
        2862, 1860, 1330, 842, 672, 543, 441, 328, 269, 219, 176, 130, 374, 350,
        329, 295, 279, 264, 251, 229, 219, 209, 200, 185, 178, 170, 164, 153, 147,
        142, 137, 129, 124, 120, 116, 110, 106, 103, 100, 95, 92, 89, 86, 82, 80,
        77, 75, 72),
    (2, 1): (
        4999, 2419, 2262, 1754, 1217, 995, 743, 616, 550, 388, 336, 265, 727, 682,
        610, 576, 571, 496, 492, 468, 430, 411, 380, 365, 361, 326, 323, 311, 291,
        281, 264, 255, 252, 233, 230, 223, 211, 204, 194, 188, 186, 174, 172, 166,
        159, 154, 147, 143),
    (4, 2): (
        2588, 1550, 1001, 555),
    (4, 1): (
        4999, 2016, 1702, 1157),
}


@pytest.mark.parametrize("n_corr,n_pol", [(4, 4), (1, 1)])
@pytest.mark.parametrize("n_st,n_dir", [(2, 1), (62, 4), (62, 10), (512, 5)])
def test_tiles_of_the_other_kernels(built, n_corr, n_pol, n_st, n_dir):
    """Full-Jones solutions and one correlation have no pipelined kernel; their
    tiles do not follow its width."""
    from dp3_b200 import ddsolve
    layout = ddsolve.describe_layout(n_st, n_dir, n_corr, n_pol)
    assert not layout.pipelined and layout.tile_runs == 224


def test_describe_layout_checks_the_dimensions(built):
    from dp3_b200 import ddsolve
    with pytest.raises(RuntimeError, match="invalid"):
        ddsolve.describe_layout(1, 4, 2, 2)
    with pytest.raises(RuntimeError, match="unsupported"):
        ddsolve.describe_layout(10, 4, 1, 2)


@pytest.mark.parametrize("n_corr,n_pol,n_dir", [
    (nc, np_, d + 1) for (nc, np_), limits in STATIONS.items() for d in range(len(limits))])
def test_arrays_that_the_pipelined_pass_takes(built, n_corr, n_pol, n_dir):
    """Up to these sizes the pass runs on pipe_kernel (beyond, it is
    stream_kernel with a launch per step of an iteration, 1.5 times as slow and
    more)."""
    from dp3_b200 import ddsolve
    limit = STATIONS[n_corr, n_pol][n_dir - 1]
    for n_st in (2, 62, limit // 2, limit * 3 // 4, limit - 1, limit):
        layout = ddsolve.describe_layout(min(n_st, limit), n_dir, n_corr, n_pol)
        assert layout.pipelined and layout.stages >= 2, n_st
        assert layout.lanes_per_run * layout.directions_per_lane >= n_dir
