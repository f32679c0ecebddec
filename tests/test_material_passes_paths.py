"""Passes of several materials that run into one another (pass_begin, pass_end) on the paths beside the dense single
scene: what a later pass reads -- page table, scene table with the dt chosen on the device, velocities of the grid update
-- has to be this substep's, and what follows has to find every pass finished, the small chunks' launches among them."""
import numpy as np
import pytest

from mpm_cuda_b200 import _lib as L
from mpm_cuda_b200 import scenes as S
from mpm_cuda_b200.sim import Scene, Simulation

from helpers import compare, oracle_for
from test_material_passes import three_materials

# twelve substeps may gather six times the rounding that the two of one step may (x 5e-6, v and C 3e-4, F and aux 2e-5)
TOL = {"x": 3e-5, "v": 1.8e-3, "C": 1.8e-3, "F": 1.2e-4, "aux": 1.2e-4}
RADII = ((6.0, 1.0, 3.0), (1.0, 6.0, 6.0), (4.0, 4.0, 4.0))


@pytest.mark.gpu
@pytest.mark.parametrize("config", [4, 12, 20])
def test_paged(gpu, config):
    sc = three_materials(3, RADII[0], 310)
    orc = oracle_for(sc)
    assert orc.step(12) == 0
    with Simulation([sc], kernel_config=config, rebin_interval=3, grid_pool_blocks=512) as sim:
        sim.step(12)
        assert sim.device_errors() == 0
        compare(sim.get_state(0), orc.state(), TOL)


@pytest.mark.gpu
@pytest.mark.parametrize("pool", [0, 2048])
@pytest.mark.parametrize("d", [3, 2])
def test_batch(gpu, d, pool):
    scs = [three_materials(d, r, 320 + 10 * k) for k, r in enumerate(RADII)]
    orcs = [oracle_for(sc) for sc in scs]
    for orc in orcs:
        assert orc.step(12) == 0
    for config in (0, 13) if pool else (0, 25, 30):
        with Simulation(scs, kernel_config=config, rebin_interval=3, grid_pool_blocks=pool) as sim:
            sim.step(12)
            assert sim.device_errors() == 0
            for k, orc in enumerate(orcs):
                compare(sim.get_state(k), orc.state(), TOL)


@pytest.mark.gpu
@pytest.mark.parametrize("config", [0, 26])
def test_adaptive(gpu, config):
    """The oracle takes the dt sequence that the device chose, read between substeps."""
    sc = three_materials(3, RADII[2], 330)
    sc.dt = 2e-3
    with Simulation([sc], kernel_config=config, rebin_interval=3, adaptive_dt=True, cfl=0.05) as sim:
        dts = []
        for _ in range(12):
            dts.append(sim.scene_time(0)[1])
            sim.step(1)
        assert sim.device_errors() == 0
        got = sim.get_state(0)
    assert len(set(dts)) > 1 and max(dts) < 1e-4
    orc = oracle_for(sc)
    for dt in dts:
        orc.grid.dt = dt
        assert orc.step(1) == 0
    compare(got, orc.state(), TOL)
