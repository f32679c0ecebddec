"""The fixed-corotated stress of the plain path (kirchhoff_fcr, through the reference stress of mpm_surrogate_eval)
against 64-bit singular values: near rotations, large stretches, and both sides of the lines where the polar iteration
hands over to the eigendecomposition (det F outside (0.02, 50), inverted F)."""
import numpy as np
import pytest

from mpm_cuda_b200.surrogate import StressSurrogate


def rotations(n, rng):
    q, r = np.linalg.qr(rng.standard_normal((n, 3, 3)))
    q = q * np.sign(np.diagonal(r, axis1=1, axis2=2))[:, None, :]
    return q * np.linalg.det(q)[:, None, None]


def stretches(kind, n, rng):
    if kind == "rigid":
        return np.ones((n, 3))
    if kind == "two equal":
        s = rng.uniform(0.8, 1.25, (n, 3))
        s[:, 1] = s[:, 0]
        return s
    if kind == "small":
        return np.exp(0.01 * rng.standard_normal((n, 3)))
    if kind == "large":
        return np.exp(rng.uniform(-0.7, 0.7, (n, 3)))
    s = rng.uniform(0.8, 1.25, (n, 3))  # det F close to the named line
    line = {"det 0.02": 0.02, "det 50": 50.0, "inverted": 1.0}[kind]
    s *= ((line * rng.uniform(0.9, 1.1, n)) / s.prod(1))[:, None] ** (1 / 3)
    if kind == "inverted":
        s[:, 2] *= -1
    return s


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["rigid", "two equal", "small", "large", "det 0.02", "det 50", "inverted"])
def test_stress_matches_64_bits(gpu, kind):
    """Bound: R and det F are each off by a few roundings times the condition of F, so tau / mu by
    40 u cond (2 (s^2 + s) + l J (J + 1)), u = 2^-24, s the largest stretch."""
    rng = np.random.default_rng(17)
    n, lam = 4099, 1.5
    s = stretches(kind, n, rng)
    if kind == "inverted":  # the smallest stretch carries the sign, as in the singular value decomposition
        s = np.sort(np.abs(s), axis=1)[:, ::-1] * np.array([1, 1, -1])
        s[:, 2] = -0.8 * np.abs(s[:, 2])
    U, V = rotations(n, rng), rotations(n, rng)
    F = np.float32(np.einsum("nik,nk,njk->nij", U, s, V))
    u, sv, vt = np.linalg.svd(np.float64(F))
    d = np.sign(np.linalg.det(np.float64(F)))
    sv[:, 2] *= d
    u[:, :, 2] *= d[:, None]
    J = sv.prod(1)
    want = np.einsum("nik,nk,njk->nij", u, 2 * sv * (sv - 1), u) + (lam * J * (J - 1))[:, None, None] * np.eye(3)
    net = StressSurrogate(seed=1)
    _, got, _ = net.eval(F, lam)
    net.close()
    top = np.abs(sv).max(1)
    bound = 40 * 2.0 ** -24 * (top / np.abs(sv).min(1)) * (2 * (top ** 2 + top) + lam * np.abs(J) * (np.abs(J) + 1))
    assert np.all(np.abs(got - want).max(axis=(1, 2)) <= bound)
