"""Snow's clamp in the 3D fused passes (snow_clamp3) against the FP64 oracle: isolated particles without gravity whose
uploaded F lies inside the elastic range, on both sides of either limit, or outside the range of the polar iteration.
Two substeps: the second one's forces come from the stress the first one kept."""
import numpy as np
import pytest

from mpm_cuda_b200 import _lib as L
from mpm_cuda_b200 import scenes as S
from mpm_cuda_b200.sim import Scene, Simulation

from helpers import group_from_arrays, oracle_for
from test_polar_stress import rotations

LO, HI = 1 - 2.5e-2, 1 + 7.5e-3


def stretches(kind, n, rng):
    inside = rng.uniform(LO + 1e-3, HI - 1e-3, (n, 3))
    if kind == "inside":
        return inside
    if kind == "lower limit":
        inside[:, 0] = LO + rng.uniform(-1e-5, 1e-5, n)
        return inside
    if kind == "upper limit":
        inside[:, 1] = HI + rng.uniform(-1e-5, 1e-5, n)
        return inside
    if kind == "clamped":
        return rng.uniform(0.85, 1.15, (n, 3))
    s = rng.uniform(0.9, 1.1, (n, 3))
    s[:, 2] = 0.015  # "flat": det F under the polar iteration's range
    return s


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["inside", "lower limit", "upper limit", "clamped", "flat"])
def test_clamp_of_isolated_particles(gpu, kind):
    """Bounds, u = 2^-24: F by 40 u cond of the uploaded F (a decomposition's roundings; the clamp itself is a
    contraction), det Fp by 60 u cond of its size; C, whose force is the stress times its constant, by 40 u times the
    condition of the two, the stress being at most mu h (2 * 0.03 * 1.01 + lambda / mu * 0.1), h the hardening."""
    rng = np.random.default_rng(23)
    side, h, dt = 52, 1.0 / 52, 1e-6
    at = np.stack(np.meshgrid(*[np.arange(6, side - 8, 4)] * 3, indexing="ij"), -1).reshape(-1, 3)
    n = len(at)
    x = (at + 0.5 + rng.uniform(0.05, 0.95, (n, 3))) * h
    s = stretches(kind, n, rng)
    F = np.einsum("nik,nk,njk->nij", rotations(n, rng), s, rotations(n, rng))
    mat = S.snow()
    g = group_from_arrays(mat, h, 8, x, np.zeros((n, 3)), np.zeros((n, 3, 3)), F, np.ones(n))
    sc = Scene(dim=3, n=(side,) * 3, h=h, dt=dt, groups=[g], gravity=(0.0, 0.0, 0.0), bc_type=L.BC_SLIP, bc_lo=3, bc_hi=3)
    orc = oracle_for(sc)
    orc.step(2)
    want = orc.state()
    with Simulation([sc]) as sim:
        sim.step(2)
        got = sim.get_state(0)
    u = 2.0 ** -24
    cond = np.abs(s).max(1) / np.abs(s).min(1)
    assert np.all(np.abs(got["F"] - want["F"]).max(axis=(1, 2)) <= 40 * u * cond)
    assert np.all(np.abs(got["aux"] - want["aux"]) <= 60 * u * cond * np.abs(want["aux"]))
    if kind in ("inside", "lower limit", "upper limit", "clamped"):
        hard = np.exp(mat.xi * np.abs(1 - want["aux"]))
        top = hard * (2 * 0.03 * 1.01 + mat.lam / mat.mu * 0.1) + hard * 2  # and F's own 40 u through 2 mu
        const = 4 / h * dt * (g.p_vol / g.p_mass) * mat.mu * 27 / h
        bound = 2 * const * 40 * u * cond * (1 + mat.xi) * top + 40 * u * np.abs(want["C"]).max(axis=(1, 2))
        assert np.all(np.abs(got["C"] - want["C"]).max(axis=(1, 2)) <= bound)
