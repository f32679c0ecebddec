"""The deterministic P2G's counting sort (mpm_kernels_det.cuh): long and short runs, against the FP64 oracle and
against itself."""
import numpy as np
import pytest

from mpm_cuda_b200 import _lib as L
from mpm_cuda_b200 import scenes as S
from mpm_cuda_b200.sim import Scene, Simulation

from helpers import compare, group_from_arrays, oracle_for


@pytest.mark.gpu
@pytest.mark.parametrize("d", [3, 2])
@pytest.mark.parametrize("n_cell,n_spread", [(1, 0), (257, 0), (33, 300), (700, 2000)])
def test_long_and_short_runs(gpu, d, n_cell, n_spread):
    """n_cell particles of one base node (the last of a grid block) interleaved in creation order with n_spread strewn
    over the domain.  Bitwise the same on every run.  A sequential FP32 sum of n terms is off by at most n u: at 700
    4.2e-5 for mass and for momentum, so v by 8.4e-5 at most; C = 4/h sum w v d turns that into up to
    4/h 8.4e-5 |v| = 1e-2, 5e-3 of its largest entry (about 3)."""
    rng = np.random.default_rng(n_cell + n_spread)
    h, n = 1.0 / 32, n_cell + n_spread
    x = h * (4 + 24 * rng.random((n, d)))
    at = rng.permutation(n)[:n_cell]
    x[at] = (np.array([15, 12, 13][:d]) + 0.5 + rng.random((n_cell, d))) * h
    v = np.array([0.4, -0.6, 0.3][:d]) + 0.1 * rng.standard_normal((n, d))
    C = rng.standard_normal((n, d, d))
    F = np.eye(d) + 0.03 * rng.standard_normal((n, d, d))
    g = group_from_arrays(S.jello(), h, 8, x, v, C, F, np.ones(n))
    g.aux = None  # jello: 1
    sc = Scene(dim=d, n=(32,) * d, h=h, dt=1e-4, groups=[g], bc_type=L.BC_SLIP, bc_lo=3, bc_hi=3)
    orc = oracle_for(sc)
    assert orc.step(2) == 0
    runs = []
    for _ in range(3):
        with Simulation([sc], p2g_mode=L.P2G_DETERMINISTIC) as sim:
            sim.step(2)
            assert sim.device_errors() == 0
            runs.append(sim.get_state(0))
    compare(runs[0], orc.state(), {"x": 2e-6, "v": 1e-4, "C": 5e-3, "F": 1e-5, "aux": 1e-5})
    for r in runs[1:]:
        for q in ("x", "v", "C", "F", "aux"):
            assert np.array_equal(r[q], runs[0][q])
