"""State-transition matrices of nearly parabolic hyperbolic orbits at perihelion over short steps,
against complex-step derivatives of the same step in extended precision, its universal functions
by their series.

Tolerance, per 3x3 block relative to its largest entry: the solver leaves the Kepler equation
1e-11 days off, and its rounding adds that of mu (s - g1) / beta (at perihelion the other terms
do not cancel); the anomaly is off by as much of the step, and a block grows with up to its third
power: four times both, over the step."""
import numpy as np
import pytest

from kete_b200.synthetic import EPOCH

pytestmark = pytest.mark.gpu
MU = 0.00029591220828411956


def _series(z):
    """c1, c2, c3 of the universal functions g_k = s^k c_k(beta s^2)."""
    out = []
    for k in (1, 2, 3):
        term = np.clongdouble(1) / (1, 2, 6)[k - 1]
        total = np.clongdouble(0)
        for j in range(20):
            total += term
            term = term * -z / np.clongdouble((2 * j + k + 1) * (2 * j + k + 2))
        out.append(total)
    return out


def _step(x, dt):
    p, v, mu = x[:3], x[3:], np.clongdouble(MU)
    r0, sigma = np.sqrt((p * p).sum()), (p * v).sum()
    beta = 2 * mu / r0 - (v * v).sum()
    s = dt / r0
    for _ in range(40):
        c1, c2, c3 = _series(beta * s * s)
        g1, g2, g3 = s * c1, s * s * c2, s * s * s * c3
        s = s - (r0 * g1 + sigma * g2 + mu * g3 - dt) / (r0 * (1 - beta * g2) + sigma * g1 + mu * g2)
    q = (1 - mu / r0 * g2) * p + (r0 * g1 + sigma * g2) * v
    r = np.sqrt((q * q).sum())
    return np.concatenate([q, -mu / (r * r0) * g1 * p + (1 - mu / r * g2) * v])


def _exact(pos, vel, dt):
    h = np.longdouble("1e-300")
    jac = np.zeros((6, 6), np.longdouble)
    for c in range(6):
        x = np.concatenate([pos, vel]).astype(np.clongdouble)
        x[c] += np.clongdouble(1j) * h
        jac[:, c] = _step(x, np.clongdouble(dt)).imag / h
    return jac


@pytest.mark.parametrize("dt", [0.125, -0.5, 4.0])
def test_near_parabolic(gpu, dt):
    rng = np.random.default_rng(4)
    beta = np.repeat([-1e-6, -1e-7, -3e-8, -1e-8], 6)
    n = beta.size
    r = rng.uniform(0.8, 5.0, n)
    u, w = rng.normal(size=(2, 3, n))
    u /= np.linalg.norm(u, axis=0)
    w = np.cross(u, w, axis=0)  # across the radius
    pos, vel = r * u, np.sqrt(2 * MU / r - beta) * w / np.linalg.norm(w, axis=0)
    jd0 = np.full(n, EPOCH)
    _, _, m, _, st = gpu.state_transition.compute_stm_arrays(pos, vel, jd0, jd0 + dt)
    assert (st == 0).all()
    tol = 4.0 * (1e-11 + 2.0**-52 * MU * (abs(dt) / r) / np.abs(beta)) / abs(dt)
    for i in range(n):
        ref = _exact(pos[:, i], vel[:, i], dt)
        for a in (slice(0, 3), slice(3, 6)):
            for b in (slice(0, 3), slice(3, 6)):
                err = np.abs(m[a, b, i] - ref[a, b]).max() / np.abs(ref[a, b]).max()
                assert err < tol[i], (beta[i], a, b, float(err), tol[i])
