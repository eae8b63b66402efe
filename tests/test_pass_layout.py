"""The packed layout and the kernel chosen for a context's dimensions (CPU)."""
import pytest


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
