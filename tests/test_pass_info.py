"""mpm_get_pass_info: what a handle's fused passes are, on either kind of grid."""
import numpy as np
import pytest

from mpm_cuda_b200 import _lib as L
from mpm_cuda_b200 import scenes as S
from mpm_cuda_b200.sim import Simulation

from test_material_passes import three_materials


def test_null_handle():
    assert L.load().mpm_get_pass_info(None, None, None) == L.ERR_INVALID


@pytest.mark.gpu
@pytest.mark.parametrize("config,pool,sums", [(0, 0, 0), (12, 0, 0), (20, 0, 0), (24, 0, 1), (31, 0, 1), (34, 0, 0),
                                              (0, 512, 0), (12, 512, 1), (13, 512, 1), (20, 512, 1), (16, 512, 0)])
def test_run_sums_on_either_grid(gpu, config, pool, sums):
    """The configurations that sum runs are others on a paged grid than on a dense one (sums_runs); a fused launch per
    material present."""
    sc = three_materials(3, (2.0, 2.0, 2.0), 3)
    with Simulation([sc], kernel_config=config, grid_pool_blocks=pool) as sim:
        assert sim.pass_info() == (bool(sums), 3)
        sim.step(2)
        assert sim.pass_info() == (bool(sums), 3)
    with Simulation([S.c0_jello2d()], kernel_config=config, grid_pool_blocks=pool) as sim:
        assert sim.pass_info() == (bool(sums), 1)
