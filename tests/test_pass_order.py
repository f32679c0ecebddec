"""A later material's pass reads what the grid update and the re-binning ahead wrote only after pass_acquire
(pass_begin in mpm_kernels_binned.cuh): it starts without a wait of its own, so a line its SM held from before would be
an older one."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mpm_cuda_b200", "csrc")


@pytest.mark.parametrize("source,function", [("mpm_kernels_binned.cuh", "chunk_loop"),
                                             ("mpm_kernels_runs.cuh", "run_chunks")])
def test_nothing_is_read_ahead_of_the_acquire(source, function):
    with open(os.path.join(CSRC, source)) as f:
        body = f.read().split(f" void {function}(const")[1]
    head, found, _ = body[body.index("{"):].partition("pass_acquire(A)")
    assert found
    code = re.sub(r"//[^\n]*", "", head)
    assert not re.search(r"ChunkList\s+\w+\(A\)|A\.(n_chunks|chunks|cursor|scenes|grid_vel|epoch)\b|pb\.", code)
