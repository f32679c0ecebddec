"""The polar-iteration stress of the atomic path (kirchhoff_polar3) against the FP64 oracle: one substep of isolated
particles at rest without gravity, whose affine matrix then is the stress times a constant -- near rotations, large
stretches, and both sides of the lines where the iteration hands over to the eigendecomposition (det F outside
(0.02, 50), inverted F)."""
import numpy as np
import pytest

from mpm_cuda_b200 import _lib as L
from mpm_cuda_b200 import scenes as S
from mpm_cuda_b200.sim import Scene, Simulation

from helpers import group_from_arrays, oracle_for


def rotations(n, rng):
    q, r = np.linalg.qr(rng.standard_normal((n, 3, 3)))
    q = q * np.sign(np.diagonal(r, axis1=1, axis2=2))[:, None, :]
    return q * np.linalg.det(q)[:, None, None]


def stretches(kind, n, rng):
    if kind == "two equal":
        s = rng.uniform(0.8, 1.25, (n, 3))
        s[:, 1] = s[:, 0]
        return s
    if kind == "small":
        return np.exp(0.01 * rng.standard_normal((n, 3)))
    if kind == "large":
        return np.exp(rng.uniform(-0.7, 0.7, (n, 3)))
    s = rng.uniform(0.8, 1.25, (n, 3))
    if kind == "inverted":
        s = np.sort(s, axis=1)[:, ::-1].copy()
        s[:, 2] *= -0.8
        return s
    line = {"det 0.02": 0.02, "det 50": 50.0}[kind]  # det F close to the named line
    return s * ((line * rng.uniform(0.9, 1.1, n)) / s.prod(1))[:, None] ** (1 / 3)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["two equal", "small", "large", "det 0.02", "det 50", "inverted"])
def test_stress_of_isolated_particles(gpu, kind):
    """Bound: the rotation and det F are each off by a few roundings times the condition of F, so tau / mu by
    40 u cond (2 (s^2 + s) + l J (J + 1)), u = 2^-24, s the largest stretch; C carries it times C's own constant, and
    its own 27-node sums add 40 u of its size."""
    rng = np.random.default_rng(17)
    side, h, dt = 52, 1.0 / 52, 1e-5
    at = np.stack(np.meshgrid(*[np.arange(6, side - 8, 4)] * 3, indexing="ij"), -1).reshape(-1, 3)
    n = len(at)
    x = (at + 0.5 + rng.uniform(0.05, 0.95, (n, 3))) * h
    s = stretches(kind, n, rng)
    F = np.einsum("nik,nk,njk->nij", rotations(n, rng), s, rotations(n, rng))
    mat = S.jello()
    g = group_from_arrays(mat, h, 8, x, np.zeros((n, 3)), np.zeros((n, 3, 3)), F, np.ones(n))
    sc = Scene(dim=3, n=(side,) * 3, h=h, dt=dt, groups=[g], gravity=(0.0, 0.0, 0.0), bc_type=L.BC_SLIP, bc_lo=3, bc_hi=3)
    orc = oracle_for(sc)
    orc.step(1)
    want = orc.state()["C"]
    with Simulation([sc]) as sim:
        sim.step_status(1)  # inverted F sets the det bit
        got = sim.get_state(0)["C"]
    s, J, lam = np.abs(s), s.prod(1), mat.lam / mat.mu
    top = s.max(1)
    part = 40 * 2.0 ** -24 * (top / s.min(1)) * (2 * (top ** 2 + top) + lam * np.abs(J) * (np.abs(J) + 1))
    # C = -(4 / h) dt vol / mass sum_i (grad w_i . tau) d_i: with |grad w| <= 1 / h, |d| <= 1.5 and 27 nodes of weight
    # ratios grad w / w summed with w, its constant is at most 4 / h * dt * vol / mass * mu * 27 / h
    const = 4 / h * dt * (g.p_vol / g.p_mass) * mat.mu * 27 / h
    bound = const * part + 40 * 2.0 ** -24 * np.abs(want).max(axis=(1, 2))
    assert np.all(np.abs(got - want).max(axis=(1, 2)) <= bound)
