"""The fused kernel that sums the particles sharing a stencil base before it
reduces them into the grid (mpm_kernels_runs.cuh), against the FP64 oracle."""
import numpy as np
import pytest

from mpm_cuda_b200 import _lib as L
from mpm_cuda_b200 import scenes as S
from mpm_cuda_b200.sim import Scene, Simulation

from helpers import compare, group_from_arrays, oracle_for

# launch configurations with run sums: one, two and three particles per thread, 128 and 256 threads
CONFIGS = (24, 25, 27, 30, 31)


def one_cell_scene(d, n, seed):
    """n particles whose stencils all start at one node, the last node of a grid block along x."""
    rng = np.random.default_rng(seed)
    h = 1.0 / 32
    base = np.array([15, 12, 13][:d])
    x = (base + 0.5 + rng.random((n, d))) * h
    v = np.array([0.4, -0.6, 0.3][:d]) + 0.1 * rng.standard_normal((n, d))
    C = rng.standard_normal((n, d, d))
    F = np.eye(d) + 0.03 * rng.standard_normal((n, d, d))
    g = group_from_arrays(S.jello(), h, 8, x, v, C, F, np.ones(n))
    g.aux = None  # jello: 1
    return Scene(dim=d, n=(32,) * d, h=h, dt=1e-4, groups=[g], bc_type=L.BC_SLIP, bc_lo=3, bc_hi=3)


@pytest.mark.gpu
@pytest.mark.parametrize("d", [3, 2])
@pytest.mark.parametrize("n", [1, 31, 33, 128, 129, 700])
def test_runs_of_one_base(gpu, d, n):
    """One run per chunk, from a single particle to several full chunks.  A sequential FP32 sum of n terms is off by at
    most n u: 4.2e-5 at 700 for mass and for momentum, so v by 8.4e-5 at most; C = 4/h sum w v d turns that into up to
    4/h 8.4e-5 |v| = 1e-2, 5e-3 of its largest entry (about 3)."""
    sc = one_cell_scene(d, n, 5 + n)
    orc = oracle_for(sc)
    assert orc.step(2) == 0
    for k in CONFIGS:
        with Simulation([sc], kernel_config=k) as sim:
            sim.step(2)
            assert sim.device_errors() == 0
            compare(sim.get_state(0), orc.state(), {"x": 2e-6, "v": 1e-4, "C": 5e-3, "F": 1e-5, "aux": 1e-5})


@pytest.mark.gpu
@pytest.mark.parametrize("d,name", [(3, "jello"), (3, "snow"), (2, "jello")])
def test_particles_outside_the_window_are_runs_of_their_own(gpu, d, name):
    """Particles that leave their chunk's window between re-binnings (0.4 cells per substep, no re-binning) scatter as
    single records; tolerances of the same motion with the direct scatter."""
    h, dt = 1.0 / 32, 1e-4
    mat = {"jello": S.jello(), "snow": S.snow()}[name]
    x, v, C, F, aux = S.perturbed_blob(d, mat, n_grid=32, h=h, ppc=2, radius_cells=5.0, seed=91, center=np.full(d, 0.5))
    v[:] = np.array([1.2, -0.8, 0.6][:d]) * (0.4 * h / dt / 1.2)
    sc = Scene(dim=d, n=(32,) * d, h=h, dt=dt, bc_type=L.BC_SLIP, bc_lo=3, bc_hi=3,
               groups=[group_from_arrays(mat, h, 2, x, v, 0 * C, F, aux)])
    orc = oracle_for(sc)
    assert orc.step(12) == 0
    for k in CONFIGS:
        with Simulation([sc], kernel_config=k, rebin_interval=32) as sim:
            sim.step(12)
            compare(sim.get_state(0), orc.state(), {"x": 2e-5, "v": 2e-3, "C": 5e-3, "F": 1e-4, "aux": 1e-4})
            assert sim.bin_stats()[0] > 0


@pytest.mark.gpu
@pytest.mark.parametrize("n", [33, 257])
def test_paged_grid(gpu, n):
    """The cell-major 128-thread configurations of a paged grid sum runs: one long run, and particles that leave their
    window (tolerances of the two tests above)."""
    sc = one_cell_scene(3, n, 3 + n)
    h, dt = sc.h, 1e-4
    x, v, C, F, aux = S.perturbed_blob(3, S.jello(), n_grid=32, h=h, ppc=2, radius_cells=5.0, seed=92, center=np.full(3, 0.5))
    v[:] = np.array([1.2, -0.8, 0.6]) * (0.4 * h / dt / 1.2)
    fast = Scene(dim=3, n=(32,) * 3, h=h, dt=dt, bc_type=L.BC_SLIP, bc_lo=3, bc_hi=3,
                 groups=[group_from_arrays(S.jello(), h, 2, x, v, 0 * C, F, aux)])
    orc, orc_fast = oracle_for(sc), oracle_for(fast)
    assert orc.step(2) == 0 and orc_fast.step(12) == 0
    for k in (12, 13, 20):
        with Simulation([sc], kernel_config=k, grid_pool_blocks=512) as sim:
            sim.step(2)
            compare(sim.get_state(0), orc.state(), {"x": 2e-6, "v": 1e-4, "C": 5e-3, "F": 1e-5, "aux": 1e-5})
        with Simulation([fast], kernel_config=k, grid_pool_blocks=512, rebin_interval=32) as sim:
            sim.step(12)
            compare(sim.get_state(0), orc_fast.state(), {"x": 2e-5, "v": 2e-3, "C": 5e-3, "F": 1e-4, "aux": 1e-4})
            assert sim.bin_stats()[0] > 0
