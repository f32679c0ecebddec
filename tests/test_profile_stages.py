"""mpm_profile_stages times the launches that mpm_step makes and advances the state as it does."""
import numpy as np
import pytest

from mpm_cuda_b200 import _lib as L
from mpm_cuda_b200.sim import Simulation

from test_material_passes import three_materials
from test_stream_order import engine_functions


def test_deterministic_stages_come_from_the_substep():
    """The deterministic branch launches nothing of its own: what it times is what enqueue_det_substep runs."""
    body = engine_functions()["profile_stages"]
    branch = body[body.index("} else if (deterministic()) {"):]
    branch = branch[:branch.index("} else {")]
    assert "<<<" not in branch and "cudaLaunchKernelEx" not in branch
    assert "enqueue_grid_update();" in branch and "enqueue_det_p2g(true" in branch
    substep = engine_functions()["enqueue_det_substep"]
    assert "enqueue_grid_update();" in substep and "enqueue_det_p2g(true" in substep


@pytest.mark.gpu
@pytest.mark.parametrize("d", [3, 2])
def test_deterministic_state_is_that_of_the_substeps(gpu, d):
    sc = three_materials(d, (4.0, 3.0, 5.0), 41)
    with Simulation([sc], p2g_mode=L.P2G_DETERMINISTIC) as a, Simulation([sc], p2g_mode=L.P2G_DETERMINISTIC) as b:
        stages = a.profile_stages(5)
        b.step(5)
        assert len(stages) == 3 and all(s > 0 for s in stages)
        x, y = a.get_state(0), b.get_state(0)
        for q in ("x", "v", "C", "F", "aux"):
            assert np.array_equal(x[q], y[q]), q
        a.step(3)
        b.step(3)
        assert np.array_equal(a.positions(0), b.positions(0))
