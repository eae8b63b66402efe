"""How the solver library is put together (CPU)."""
import os


def test_pass_variants_are_compiled_apart():
    """Every source file to an object of its own, none optimised in parts (the
    parts depend on what else the file holds): the code of ddsolve.cu's kernels
    does not change with the variants of pipe_kernel."""
    from dp3_b200 import build
    sources = build.solver_sources()
    names = [os.path.basename(s) for s in sources]
    assert "ddsolve.cu" in names and len(names) > 1
    for src in sources:
        text = open(src).read()
        # only the files of the variants name them
        assert ('"pipe_entries.cuh"' in text) == (os.path.basename(src) != "ddsolve.cu"), src
        command = build.solver_command(src, "out.o")
        assert not any("split-compile" in c for c in command) and "-c" in command
