"""Nodes whose mass lies below the normal numbers' range (a stencil weight of 1e-25 of a light particle) count as empty
in every P2G path, with mass_eps = 0 too: their reciprocal is infinite."""
import numpy as np
import pytest

from mpm_cuda_b200 import _lib as L
from mpm_cuda_b200.sim import MaterialParams, Scene, Simulation

from helpers import TOL_STEP, compare, group_from_arrays, oracle_for

SIDE, H = 32, 1.0 / 32


def light_particles(d):
    """Particles 5 cells apart, 1 to 3 ulps beside a cell's middle along the first d - 1 axes: their last node there has
    a weight near 1e-25 (3D) and 1e-12 (2D), and their masses put its mass at 1e-38 and below."""
    k = np.arange(1, 4)
    ulp = np.spacing(np.float32(10.5)) * k
    at = np.stack(np.meshgrid(*[[5.5 + 5 * i for i in range(3)]] * d, indexing="ij"), -1).reshape(-1, d)
    at[:, 0] += 5.0
    x = np.float32(at)
    for a in range(d - 1):
        x[:, a] = np.float32(10.5) + np.float32(ulp)[np.arange(len(x)) % 3] + np.float32(at[:, a] - 10.5)
    x[:, d - 1] += np.float32(0.21)
    n = len(x)
    mass = 1e-14 if d == 3 else 1e-27
    rho = mass * 8 / H ** d
    mat = MaterialParams(type=L.JELLO, E=100.0 * rho, nu=0.3, rho=rho)
    v = np.tile(np.float32([0.7, -0.4, 0.3][:d]), (n, 1))
    eye = np.tile(np.eye(d), (n, 1, 1))
    g = group_from_arrays(mat, H, 8, x.astype(np.float64) * H, v, 0 * eye, eye, np.ones(n))
    return Scene(dim=d, n=(SIDE,) * d, h=H, dt=1e-4, groups=[g], gravity=(0.0, -9.8, 0.0)[:d], bc_type=L.BC_SLIP, bc_lo=3,
                 bc_hi=3, mass_eps=0.0)


@pytest.mark.parametrize("d", [3, 2])
def test_the_scene_has_such_nodes(d):
    orc = oracle_for(light_particles(d))
    assert orc.step(1) == 0
    m = np.asarray(orc.grid_mass()).ravel()
    assert np.any((m > 1e-44) & (m < 2e-39))


@pytest.mark.gpu
@pytest.mark.parametrize("d", [3, 2])
@pytest.mark.parametrize("kw", [dict(p2g_mode=L.P2G_DETERMINISTIC), dict(p2g_mode=L.P2G_DIRECT), dict(kernel_config=4),
                                dict(kernel_config=25)])
def test_one_substep(gpu, d, kw):
    """The nodes left out carry at most 1e-24 (3D) and 1e-11 (2D) of a particle's mass: the tolerances of one substep.
    (C is 4 / h = 128 times the rounding of the speeds here, 0 in the oracle.)"""
    sc = light_particles(d)
    orc = oracle_for(sc)
    assert orc.step(1) == 0
    with Simulation([sc], **kw) as sim:
        assert sim.step_status(1) == L.OK
        compare(sim.get_state(0), orc.state(), TOL_STEP, fields=("x", "v", "F", "aux"))
