"""When the small chunks of a state get launches of their own, and that they do: on 2D, batched and adaptive runs beside
the dense and paged 3D ones, and for a state that is loaded into a fresh handle."""
import ctypes as C

import numpy as np
import pytest

from mpm_cuda_b200 import _lib as L
from mpm_cuda_b200 import scenes as S
from mpm_cuda_b200.sim import Scene, Simulation

from helpers import compare, group_from_arrays, oracle_for

TOL = {"x": 5e-6, "v": 3e-4, "C": 3e-4, "F": 2e-5, "aux": 2e-5}  # two substeps of mixed groups


SIDE = {3: 32, 2: 128}  # nodes: enough blocks for the particles to spray over


def states(d, seed):
    """The groups of a scene, dense and strewn over the grid with one full block among them."""
    h, rng = 1.0 / SIDE[d], np.random.default_rng(seed)
    dense, spray = [], []
    for k, mat in enumerate((S.jello(), S.snow())):
        center = np.array([0.4 + 0.15 * k, 0.5, 0.5])[:d]
        x, v, B, F, aux = S.perturbed_blob(d, mat, n_grid=SIDE[d], h=h, ppc=8 if d == 3 else 24,
                                           radius_cells=4.5 if d == 3 else 6.0, seed=seed + k, center=center)
        dense.append((mat, (x, v, B, F, aux)))
        xs = h * (4 + (SIDE[d] - 8) * rng.random(x.shape))
        xs[:300] = h * (np.array([8.0, 12.0, 16.0])[:d] + 0.6 + 3 * rng.random((300, d)))
        spray.append((mat, (xs, 0.1 * v, 0 * B, F, aux)))
    return dense, spray


def scene_at(groups, d):
    h = 1.0 / SIDE[d]
    return Scene(dim=d, n=(SIDE[d],) * d, h=h, dt=1e-4, bc_type=L.BC_SLIP, bc_lo=3, bc_hi=3,
                 groups=[group_from_arrays(m, h, 8, *a) for m, a in groups])


def load(sim, k, groups):
    cat = lambda q: np.concatenate([a[q] for _, a in groups])  # noqa: E731
    sim.set_state(k, x=cat(0), v=cat(1), C_=cat(2), F=cat(3), aux=cat(4))


@pytest.mark.gpu
@pytest.mark.parametrize("d,config,pool,scenes,adaptive", [(3, 25, 0, 1, False), (3, 20, 512, 1, False),
                                                           (2, 31, 0, 1, False), (3, 27, 0, 2, False),
                                                           (3, 28, 0, 1, True), (3, 20, 1024, 2, False)])
def test_off_on_off(gpu, d, config, pool, scenes, adaptive):
    """Dense, sprayed, dense again: one launch per material, two, one; two substeps from a state that was set match the
    oracle in each stretch.  (With cfl 1 the adaptive bound stays above dt.)"""
    both = [states(d, 90 + 10 * k) for k in range(scenes)]
    with Simulation([scene_at(b[0], d) for b in both], kernel_config=config, grid_pool_blocks=pool,
                    adaptive_dt=adaptive, cfl=1.0) as sim:
        for which, launches in ((0, 2), (1, 4), (0, 2)):
            for _ in range(3):
                for k, b in enumerate(both):
                    load(sim, k, b[which])
                sim.step(1)
                sim.step(1)
                assert sim.device_errors() == 0
                for k, b in enumerate(both):
                    orc = oracle_for(scene_at(b[which], d))
                    assert orc.step(2) == 0
                    compare(sim.get_state(k), orc.state(), TOL)
            assert sim.pass_info() == (True, launches)


@pytest.mark.gpu
def test_a_sprayed_state_in_a_fresh_handle(gpu):
    """The measure of a full chunk goes with the autotuner's choice: a handle that is created on dense groups and given
    a sprayed state before its first substep, tuned itself or served from the cache, gives its small chunks launches of
    their own if its configuration may."""
    h, rng = 1.0 / 64, np.random.default_rng(7)
    n = 8 * 30 ** 3
    x = h * (17 + 30 * rng.random((n, 3)))
    zero, eye, one = np.zeros((n, 3)), np.tile(np.eye(3), (n, 1, 1)), np.ones(n)
    sc = Scene(dim=3, n=(64,) * 3, h=h, dt=1e-5, bc_type=L.BC_SLIP, bc_lo=3, bc_hi=3,
               groups=[group_from_arrays(S.snow(), h, 8, x, zero, 0 * eye, eye, one)])
    sprayed = np.float32(h * (5 + 54 * rng.random((n, 3))))
    for _ in range(2):
        with Simulation([sc]) as sim:
            sim.set_state(0, x=sprayed)
            sim.step(1)
            sim.step(1)
            rounds = C.c_int()
            L.load().mpm_kernel_config_info(sim.kernel_config(), None, None, C.byref(rounds))
            runs, launches = sim.pass_info()
            assert launches == (2 if runs and rounds.value >= 2 else 1)
