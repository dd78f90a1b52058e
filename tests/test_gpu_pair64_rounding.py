"""Rounding of the FP64 pair kernel: the derivatives of isolated pairs are off
from the exact ones by no more than the reference's arithmetic is (its formulas
with every operation rounded to 64 bits), in the mean square over the pairs.
The mean square of N errors is known to 1 / sqrt(N) or so, which the bar
allows twice.  Errors of the 2 h kernels are weighted by 2 - q, to which the
powers of 2 - q are conditioned."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
CUBIC, GAUSS, WEND = 0, 1, 2
MASS = 0.4


def _pairs(n, h, kernel, seed):
    """n pairs of particles 12 h apart on a square array, q from 0.3 to the
    kernel's support, the second half of each pair after the first halves."""
    from sph.Common import particle_dtype
    rng = np.random.default_rng(seed)
    side = int(np.ceil(np.sqrt(n)))
    k = np.arange(n)
    q = rng.uniform(0.3, 2.9 if kernel == GAUSS else 1.99, n)
    ang = rng.uniform(-1.0, 1.0, n)
    pa = np.zeros(2 * n, dtype=particle_dtype)
    pa["x"][:n], pa["y"][:n] = 12.0 * h * (k % side) + 0.3, 12.0 * h * (k // side) + 0.3
    pa["x"][n:], pa["y"][n:] = pa["x"][:n] + q * h * np.cos(ang), pa["y"][:n] + q * h * np.sin(ang)
    pa["m"] = MASS
    pa["rho"] = rng.uniform(1010.0, 1050.0, 2 * n)
    va = ang + rng.uniform(-1.0, 1.0, n)
    s = rng.uniform(0.1, 1.0, n)
    pa["vx"][n:], pa["vy"][n:] = s * np.cos(va), s * np.sin(va)
    return pa


def _restated(F, s, n, kernel):
    """drho of every particle by the reference's formulas, in the type F, from
    the inputs s and the h that the evaluation had (CubicSpline.py:40-70,
    Gaussian.py:37-59, Wendland.py:36-64, Continuity.py)."""
    j = np.r_[n:2 * n, 0:n]
    x, y, vx, vy, h = (s[k].astype(F) for k in ("x", "y", "vx", "vy", "h"))
    pi = F("3.14159265358979323846264338327950288") if F is not np.float64 else math.pi
    dx, dy = x - x[j], y - y[j]
    r = np.sqrt(dx * dx + dy * dy)
    hij = F(0.5) * (h + h[j])
    q = r / hij
    if kernel == CUBIC:
        al = F(10) / (F(7) * pi) / (hij * hij)
        g = np.where(q > 1, F(-0.75) * ((2 - q) * (2 - q)), F(-3) * q * (1 - F(0.75) * q))
        coef = al * g / (hij * r)
    elif kernel == WEND:
        al = F(9) / (F(4) * pi) / (hij * hij)
        t = 1 - F(0.5) * q
        coef = al * (t * t * t * t * t) * (F(-14) / F(3)) * q * (1 + F(2.5) * q) / (hij * r)
    else:
        al = F(1) / pi / (hij * hij)
        coef = F(-2) * q * al * np.exp(-q * q) / (r * hij)
    vxij, vyij = vx - vx[j], vy - vy[j]
    drho = F(MASS) * (vxij * (coef * dx) + vyij * (coef * dy))
    return q, drho


@pytest.mark.parametrize("kernel", [CUBIC, GAUSS, WEND])
@pytest.mark.parametrize("fixed", [True, False])
@pytest.mark.parametrize("n", [3001, 10007, 35003])
def test_continuity_of_a_pair(kernel, fixed, n):
    """n pairs take 8, 4 and 1 lanes per query."""
    from sph import build, core, state
    build.build()
    h = 0.0325 if fixed else 1.3 * np.sqrt(MASS / 1030.0)
    pa = _pairs(n, h, kernel, n + kernel)
    dp = state.DeviceParticles.from_array(pa)
    dp.h.fill_(h)
    wc = core.wcsph_struct(5.0, 0.01, 1000.0)
    ws = state.DeviceWorkspace(dp.n)
    core.compute(dp, wc, core.config_struct(kernel=kernel, precision="fp64", h_fixed=h if fixed else 0.0), ws)
    ws.check()
    got = dp.soa()
    q, want = _restated(np.longdouble, got, n, kernel)
    _, fp64 = _restated(np.float64, got, n, kernel)
    w = np.minimum(2 - q, 1) if kernel != GAUSS else np.ones_like(q)
    hij = 0.5 * (got["h"] + np.roll(got["h"], n))
    ok = q * hij < 1.99 * got["h"].min()  # the reach of the reference's stencil
    rms = lambda v: np.sqrt(np.mean((((v - want) / want * w)[ok]).astype(np.float64) ** 2))  # noqa: E731
    assert rms(got["drho"]) <= rms(fp64) * (1 + 2 / np.sqrt(ok.sum())), (rms(got["drho"]), rms(fp64))


def test_pressure_term():
    """p / rho^2 has the two roundings of the reference's (WCSPH.py:160-164).
    Pairs at r = h on one line, h a power of two: the gradient factor is 0.75
    and the difference h, both exact, and the constants are the same for every
    pair, so what varies from pair to pair is the rounding of p / rho^2, of the
    sum, and of two products."""
    from sph import build, core, state
    from sph.Common import particle_dtype
    build.build()
    n, h = 10007, 0.03125
    rng = np.random.default_rng(1)
    k = np.arange(n)
    pa = np.zeros(2 * n + 1, dtype=particle_dtype)  # and one alone, which keeps the others off the grid's edge
    pa["x"][:n], pa["y"][:n] = 12 * h * (k % 101), 12 * h * (k // 101)
    pa["x"][n:-1], pa["y"][n:-1] = pa["x"][:n] + h, pa["y"][:n]
    pa["x"][-1], pa["y"][-1] = 3.3 * h, 12 * h * (n // 101) + 6.7 * h
    pa["m"], pa["rho"] = 0.5, rng.uniform(1010.0, 1050.0, 2 * n + 1)
    dp = state.DeviceParticles.from_array(pa)
    dp.h.fill_(h)
    ws = state.DeviceWorkspace(dp.n)
    core.compute(dp, core.wcsph_struct(5.0, 0.01, 1000.0, alpha=0.0), core.config_struct(h_fixed=h), ws)
    ws.check()
    got = {k: v[:-1] for k, v in dp.soa().items()}

    def term(F):
        o = got["p"].astype(F) / (got["rho"].astype(F) * got["rho"].astype(F))
        return F(0.375) * (o + np.roll(o, n)) * F(0.1)
    want = term(np.longdouble)
    rms = lambda v: np.std((np.abs(v) / want / np.mean(np.abs(v) / want) - 1).astype(np.float64))  # noqa: E731
    assert rms(got["ax"]) <= rms(term(np.float64)) * (1 + 2 / np.sqrt(2 * n)), (rms(got["ax"]), rms(term(np.float64)))


@pytest.mark.parametrize("kernel", [CUBIC, GAUSS, WEND])
@pytest.mark.parametrize("fixed", [True, False])
@pytest.mark.parametrize("n", [3001, 10007, 35003])
def test_xsph_of_a_pair(kernel, fixed, n):
    """The XSPH velocity of the pairs' first halves, which are at rest
    (XSPH.py:26-31, the kernels' values)."""
    from sph import build, core, state
    build.build()
    h = 0.0325 if fixed else 1.3 * np.sqrt(MASS / 1030.0)
    pa = _pairs(n, h, kernel, n + kernel)
    dp = state.DeviceParticles.from_array(pa)
    dp.h.fill_(h)
    ws = state.DeviceWorkspace(dp.n)
    core.compute(dp, core.wcsph_struct(5.0, 0.01, 1000.0, use_xsph=True),
                 core.config_struct(kernel=kernel, precision="fp64", h_fixed=h if fixed else 0.0), ws)
    ws.check()
    got = dp.soa()

    def velocity(F):
        x, y, vx, rho, hh = (got[k].astype(F) for k in ("x", "y", "vx", "rho", "h"))
        pi = F("3.14159265358979323846264338327950288") if F is not np.float64 else math.pi
        dx, dy = x[:n] - x[n:], y[:n] - y[n:]
        r = np.sqrt(dx * dx + dy * dy)
        hij = F(0.5) * (hh[:n] + hh[n:])
        q = r / hij
        if kernel == CUBIC:
            w = F(10) / (F(7) * pi) / (hij * hij) * np.where(
                q > 1, F(0.25) * ((2 - q) * (2 - q) * (2 - q)), 1 - F(1.5) * (q * q) * (1 - F(0.5) * q))
        elif kernel == WEND:
            t = 1 - F(0.5) * q
            w = F(9) / (F(4) * pi) / (hij * hij) * (t * t * t * t * t * t) * (F(35) / F(12) * q * q + 3 * q + 1)
        else:
            w = F(1) / pi / (hij * hij) * np.exp(-q * q)
        return q, -F(0.5) * F(MASS) * w / (F(0.5) * (rho[:n] + rho[n:])) * (vx[:n] - vx[n:])
    q, want = velocity(np.longdouble)
    _, fp64 = velocity(np.float64)
    weight = np.minimum(2 - q, 1) if kernel != GAUSS else np.ones_like(q)
    ok = q * got["h"].max() < 1.99 * got["h"].min()
    rms = lambda v: np.sqrt(np.mean((((v - want) / want * weight)[ok]).astype(np.float64) ** 2))  # noqa: E731
    assert rms(got["xsphx"][:n]) <= rms(fp64) * (1 + 2 / np.sqrt(ok.sum())), (rms(got["xsphx"][:n]), rms(fp64))


@pytest.mark.parametrize("n", [3001, 10007, 35003])
def test_boundary_force_of_a_pair(n):
    """The Lennard-Jones force of single boundary particles
    (BoundaryForce.py:6-42)."""
    from sph import build, core, state
    build.build()
    h, r0 = 0.0325, 0.025
    pa = _pairs(n, h, CUBIC, n)
    rng = np.random.default_rng(n)
    r, ang = r0 * rng.uniform(0.3, 0.9, n), rng.uniform(-1.0, 1.0, n)
    pa["x"][n:], pa["y"][n:] = pa["x"][:n] + r * np.cos(ang), pa["y"][:n] + r * np.sin(ang)
    pa["label"][n:], pa["m"][n:], pa["vx"][n:], pa["vy"][n:] = 1, 0.0, 0.0, 0.0
    dp = state.DeviceParticles.from_array(pa)
    wc = core.wcsph_struct(5.0, r0, 1000.0)
    ws = state.DeviceWorkspace(dp.n)
    core.compute(dp, wc, core.config_struct(h_fixed=h), ws)
    ws.check()
    got = dp.soa()

    def force(F):
        x, y = got["x"].astype(F), got["y"].astype(F)
        dx, dy = x[:n] - x[n:], y[:n] - y[n:]
        r = np.sqrt(dx * dx + dy * dy)
        f = F(wc.r0) / r
        f2 = f * f
        return F(wc.D) * (f2 * f2 - f2) * dx / (r * r)
    want = force(np.longdouble)
    rms = lambda v: np.sqrt(np.mean(((v - want) / want).astype(np.float64) ** 2))  # noqa: E731
    assert rms(got["ax"][:n]) <= rms(force(np.float64)) * (1 + 2 / np.sqrt(n)), (rms(got["ax"][:n]), rms(force(np.float64)))
