"""The passes of a scene's materials run into one another (pass_begin and pass_end in mpm_kernels_binned.cuh): what
follows the last of them has to find all of them finished."""
import numpy as np
import pytest

from mpm_cuda_b200 import _lib as L
from mpm_cuda_b200 import scenes as S
from mpm_cuda_b200.sim import Scene, Simulation

from helpers import compare, group_from_arrays, oracle_for


def three_materials(d, radii, seed):
    h = 1.0 / 32
    groups = []
    for k, (mat, r) in enumerate(zip((S.jello(), S.snow(), S.water()), radii)):
        center = np.full(d, 0.5)
        center[0] += (k - 1) * 2 * h
        x, v, C, F, aux = S.perturbed_blob(d, mat, n_grid=32, h=h, ppc=8, radius_cells=r, seed=seed + k, center=center)
        groups.append(group_from_arrays(mat, h, 8, x, v, C, F, aux))
    return Scene(dim=d, n=(32,) * d, h=h, dt=1e-4, groups=groups, bc_type=L.BC_SLIP, bc_lo=3, bc_hi=3)


@pytest.mark.gpu
@pytest.mark.parametrize("d,radii", [(3, (6.0, 1.0, 3.0)), (3, (1.0, 6.0, 6.0)), (2, (6.0, 6.0, 1.0))])
@pytest.mark.parametrize("config", [0, 25, 30])
def test_three_materials(gpu, d, radii, config):
    """Overlapping blobs of uneven sizes, re-binned every third substep.  Twelve substeps may gather six times the
    rounding that the two of one step may: x 5e-6, v and C 3e-4, F and aux 2e-5, times 6."""
    sc = three_materials(d, radii, 300)
    orc = oracle_for(sc)
    assert orc.step(12) == 0
    for graph in (True, False):
        with Simulation([sc], kernel_config=config, rebin_interval=3, use_graph=graph) as sim:
            sim.step(12)
            assert sim.device_errors() == 0
            compare(sim.get_state(0), orc.state(), {"x": 3e-5, "v": 1.8e-3, "C": 1.8e-3, "F": 1.2e-4, "aux": 1.2e-4})
