"""Launches of their own for the small chunks of a state that has sprayed (wants_split_small in mpm_config.cuh)."""
import numpy as np
import pytest

from mpm_cuda_b200 import _lib as L
from mpm_cuda_b200 import scenes as S
from mpm_cuda_b200.sim import Scene, Simulation

from helpers import compare, group_from_arrays, oracle_for

TOL = {"x": 5e-6, "v": 3e-4, "C": 3e-4, "F": 2e-5, "aux": 2e-5}  # two substeps of mixed groups


def scene_at(groups, h):
    return Scene(dim=3, n=(32,) * 3, h=h, dt=1e-4, bc_type=L.BC_SLIP, bc_lo=3, bc_hi=3,
                 groups=[group_from_arrays(m, h, 8, *a) for m, a in groups])


@pytest.mark.gpu
@pytest.mark.parametrize("config,pool", [(25, 0), (28, 0), (31, 0), (20, 512)])
def test_sprayed_and_gathered_again(gpu, config, pool):
    """A dense block of jello and snow, the same particles strewn over the grid with one full block among them, then
    dense again: every stretch of two substeps from a state that was set matches the oracle, before and after the
    launches change (the counters are read at the end of a step, so the third and fourth substep differ)."""
    h, rng = 1.0 / 32, np.random.default_rng(17)
    dense, spray = [], []
    for k, mat in enumerate((S.jello(), S.snow())):
        center = np.array([0.4 + 0.15 * k, 0.5, 0.5])
        x, v, C, F, aux = S.perturbed_blob(3, mat, n_grid=32, h=h, ppc=8, radius_cells=4.5, seed=70 + k, center=center)
        dense.append((mat, (x, v, C, F, aux)))
        xs = h * (4 + 24 * rng.random(x.shape))
        xs[:300] = h * (np.array([8.0, 12.0, 16.0]) + 0.6 + 3 * rng.random((300, 3)))
        spray.append((mat, (xs, 0.1 * v, 0 * C, F, aux)))
    cat = lambda g, q: np.concatenate([a[q] for _, a in g])
    with Simulation([scene_at(dense, h)], kernel_config=config, grid_pool_blocks=pool) as sim:
        for state in (dense, spray, dense):
            for _ in range(3):
                sim.set_state(0, x=cat(state, 0), v=cat(state, 1), C_=cat(state, 2), F=cat(state, 3), aux=cat(state, 4))
                orc = oracle_for(scene_at(state, h))
                assert orc.step(2) == 0
                sim.step(1)
                sim.step(1)
                assert sim.device_errors() == 0
                compare(sim.get_state(0), orc.state(), TOL)
