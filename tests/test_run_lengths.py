"""Run sums over a chunk whose runs have lengths on both sides of what the ordering tells apart (run_chunks:
1 to 15 particles, 16 and more together), with particles that have left the chunk's window among them: a run lost,
summed twice or put on another's place shows in the grid's mass."""
import numpy as np
import pytest

from mpm_cuda_b200 import _lib as L
from mpm_cuda_b200 import scenes as S
from mpm_cuda_b200.sim import Scene, Simulation

from helpers import compare, group_from_arrays, oracle_for

H, DT, STEPS = 1.0 / 32, 1e-4, 12
LENGTHS = (1, 2, 15, 16, 17, 40, 3, 14)


def one_block_scene(drifters, repeat):
    """One group per run, of its own density, at rest on the bases (8, y, z) of the block [8, 12)^3, and `drifters`
    groups of one particle each at (11, y, z) that move 0.4 cells a substep away from the others."""
    rng = np.random.default_rng(61)
    groups = []
    for k, n in enumerate(LENGTHS):
        n *= repeat
        base = np.array([8, 8 + k % 4, 8 + 2 * (k // 4)])
        x = (base + 0.6 + 0.8 * rng.random((n, 3))) * H
        groups.append((S.jello(rho=1000.0 * (1 + k)), x, np.zeros((n, 3))))
    for k in range(drifters):
        base = np.array([11, 8 + k % 4, 8 + k // 4])
        groups.append((S.jello(rho=700.0 * (1 + k)), (base + 0.6 + 0.3 * rng.random((1, 3))) * H,
                       np.array([[0.4 * H / DT, 0.0, 0.0]])))
    out = []
    for mat, x, v in groups:
        n = len(x)
        C = 0.1 * rng.standard_normal((n, 3, 3)) if not v.any() else np.zeros((n, 3, 3))
        g = group_from_arrays(mat, H, 8, x, v, C, np.tile(np.eye(3), (n, 1, 1)), np.ones(n))
        g.aux = None  # jello: 1
        out.append(g)
    return Scene(dim=3, n=(32,) * 3, h=H, dt=DT, groups=out, gravity=(0.0, 0.0, 0.0), bc_type=L.BC_SLIP, bc_lo=3,
                 bc_hi=3)


@pytest.mark.gpu
@pytest.mark.parametrize("pool,configs", [(0, (24, 25, 26, 27, 28, 29, 30, 31)), (512, (12, 13, 20))])
@pytest.mark.parametrize("drifters,repeat", [(0, 1), (12, 1), (12, 3)])
def test_mixed_lengths(gpu, pool, configs, drifters, repeat):
    """The last grid update's mass: a sum of up to 324 terms, n u = 2e-5 of a node's mass; the drifters' weights follow
    positions off by 12 (u x + 5 u v dt) = 1e-6, 3e-5 cells, 1e-4 of their mass.  The lightest run is a fiftieth of the
    heaviest node.  States: the tolerances of the same motion in test_run_sums.py, but for C, which is 0 for the
    drifters and carries 4 / h times the rounding of their speed."""
    sc = one_block_scene(drifters, repeat)
    orc = oracle_for(sc)
    assert orc.step(STEPS) == 0
    want = np.asarray(orc.grid_mass()).ravel()
    for k in configs:
        with Simulation([sc], kernel_config=k, grid_pool_blocks=pool, rebin_interval=64) as sim:
            sim.step(STEPS)
            assert sim.device_errors() == 0
            assert sim.pass_info()[0]
            assert (sim.bin_stats()[0] > 0) == (drifters > 0)
            mass, _ = sim.get_grid(0)
            compare(sim.get_state(0), orc.state(), {"x": 2e-5, "v": 2e-3, "F": 1e-4, "aux": 1e-4},
                    fields=("x", "v", "F", "aux"))
        assert np.all(np.abs(mass - want) <= 2e-4 * want + 2e-5 * want.max()), k
