"""Snow's clamp (snow_clamp3) where eigenvalues of the strain are equal, all but equal or at a limit of the elastic
range: stretches along the axes with shears down to subnormal squares, two stretches on both sides of one limit, an
elastic range without width and one without end."""
import dataclasses

import numpy as np
import pytest

from mpm_cuda_b200 import _lib as L
from mpm_cuda_b200 import scenes as S
from mpm_cuda_b200.sim import Scene, Simulation

from helpers import group_from_arrays, oracle_for
from test_polar_stress import rotations

SIDE, H = 52, 1.0 / 52
U = 2.0 ** -24


def one_substep(F, theta_c=None, theta_s=None):
    """One substep of isolated particles at rest without gravity, here and in the oracle: F is the uploaded F clamped."""
    at = np.stack(np.meshgrid(*[np.arange(6, SIDE - 8, 4)] * 3, indexing="ij"), -1).reshape(-1, 3)
    rng = np.random.default_rng(31)
    x = (at + 0.5 + rng.uniform(0.05, 0.95, at.shape)) * H
    n = len(at)
    mat = S.snow()
    if theta_c is not None:
        mat = dataclasses.replace(mat, theta_c=theta_c, theta_s=theta_s)
    g = group_from_arrays(mat, H, 8, x, np.zeros((n, 3)), np.zeros((n, 3, 3)), F[:n], np.ones(n))
    sc = Scene(dim=3, n=(SIDE,) * 3, h=H, dt=1e-6, groups=[g], gravity=(0.0, 0.0, 0.0), bc_type=L.BC_SLIP, bc_lo=3,
               bc_hi=3)
    orc = oracle_for(sc)
    orc.step(1)
    with Simulation([sc]) as sim:
        assert sim.step_status(1) == L.OK
        return sim.get_state(0), orc.state()


def check(got, want):
    """40 u for F, a decomposition's roundings at stretches near 1 (the clamp is a contraction); det Fp 60 u."""
    err = np.abs(got["F"] - want["F"]).max(axis=(1, 2))
    bad = ~(err <= 40 * U)
    assert not bad.any(), (int(bad.sum()), float(np.nanmax(err) / U))
    assert np.all(np.abs(got["aux"] - want["aux"]) <= 60 * U * np.abs(want["aux"]))


def sheared(stretch, rng, n=1000):
    F = np.stack([np.diag(np.roll(stretch, k % 3)) for k in range(n)]).astype(float)
    shear = 10.0 ** rng.uniform(-26, -6, (n, 3, 3)) * rng.choice([-1, 0, 0, 1], (n, 3, 3))
    shear[:, range(3), range(3)] = 0
    return F + shear


@pytest.mark.gpu
@pytest.mark.parametrize("stretch", [(1.02, 1.0, 1.0), (0.96, 1.0, 1.0), (1.02, 1.02, 1.0), (0.96, 0.96, 1.02),
                                     (1.02, 1.02, 1.02)])
def test_all_but_equal_stretches(gpu, stretch):
    check(*one_substep(sheared(stretch, np.random.default_rng(31))))


@pytest.mark.gpu
@pytest.mark.parametrize("theta_c,theta_s", [(0.0, 0.0), (0.0, 1e-2), (1e-2, 0.0)])
@pytest.mark.parametrize("stretch", [(1.0, 1.0, 1.0), (1.02, 1.0, 1.0), (0.98, 1.0, 1.0)])
def test_no_width(gpu, theta_c, theta_s, stretch):
    check(*one_substep(sheared(stretch, np.random.default_rng(32)), theta_c, theta_s))


@pytest.mark.gpu
@pytest.mark.parametrize("theta_c", [2.5e-2, 8e-2, 0.5])
def test_two_stretches_at_one_limit(gpu, theta_c):
    """One inside by 1e-7, one beyond by 1e-5: the sign of the strain's third minor is below its rounding."""
    rng = np.random.default_rng(33)
    n = 1000
    s = np.tile([1.0, 1 - theta_c + 1e-7, 1 - theta_c - 1e-5], (n, 1))
    w = 0.2 * rng.standard_normal((n, 3, 3))
    V = np.linalg.qr(np.eye(3) + w - w.transpose(0, 2, 1))[0]
    V = V * np.sign(np.einsum("nii->ni", V))[:, None, :]
    check(*one_substep(np.einsum("nik,nk,njk->nij", rotations(n, rng), s, V), theta_c, 2e-2))


@pytest.mark.gpu
def test_no_end(gpu):
    """No upper limit and a lower one out of reach: nothing is clamped, so det Fp stays 1 exactly."""
    rng = np.random.default_rng(34)
    n = 1000
    F = np.einsum("nik,nk,njk->nij", rotations(n, rng), rng.uniform(0.7, 1.4, (n, 3)), rotations(n, rng))
    got, want = one_substep(F, 0.99, np.inf)
    check(got, want)
    assert np.all(got["aux"] == 1.0)
