"""Pairs close to the edge of the kernel support, one by one: isolated pairs at
q = r / h = 2 - t, t from 1e-5 to 1, whose derivatives are that one pair's.

The tolerance is that of the gradient's (2 - q)^2, (2 - q)^3 and
(1 - q / 2)^5, ^6 formed from a q with four roundings on either side: q is off by
at most 9e-16 between the two, and the powers multiply that by at most 6 / t;
1e-13 covers the rest (the EOS at rho / rho0 - 1 >= 1% has 2e-14)."""
import numpy as np
import pytest
import torch
from scipy.spatial import cKDTree

pytestmark = pytest.mark.gpu
CUBIC, WEND = 0, 2


def _tol(t):
    return 1e-13 + 8e-15 / t


def _pairs(n, h, seed):
    """n isolated pairs, 6 h apart, on a square array."""
    from sph.Common import particle_dtype
    rng = np.random.default_rng(seed)
    side = int(np.ceil(np.sqrt(n)))
    k = np.arange(n)
    t = 10.0 ** rng.uniform(-5, 0, n)
    ang = rng.uniform(-1.0, 1.0, n) + np.pi * rng.integers(0, 2, n)
    r = (2.0 - t) * h
    pa = np.zeros(2 * n, dtype=particle_dtype)
    pa["x"][:n], pa["y"][:n] = 6.0 * h * (k % side), 6.0 * h * (k // side)
    pa["x"][n:], pa["y"][n:] = pa["x"][:n] + r * np.cos(ang), pa["y"][:n] + r * np.sin(ang)
    pa["m"] = 0.4
    pa["rho"] = rng.uniform(1010.0, 1050.0, 2 * n)
    # the relative velocity within 1 rad of the pair's line, towards or away
    s = rng.choice([-1.0, 1.0], n) * rng.uniform(0.1, 1.0, n)
    va = ang + rng.uniform(-1.0, 1.0, n)
    pa["vx"][n:], pa["vy"][n:] = s * np.cos(va), s * np.sin(va)
    return pa


@pytest.mark.parametrize("kernel", [CUBIC, WEND])
@pytest.mark.parametrize("fixed", [True, False])
@pytest.mark.parametrize("n", [700, 10007, 35003])
def test_pair_derivatives(kernel, fixed, n):
    """n pairs take 8, 4 and 1 lanes per query."""
    import oracle
    from sph import build, core, state
    build.build()
    # h from the density differs from pair to pair: about 1.3 sqrt(m / rho)
    h = 0.0325 if fixed else 1.3 * np.sqrt(0.4 / 1030.0)
    pa = _pairs(n, h, n + kernel)
    P = oracle.Particles(arrays={k: pa[k] for k in pa.dtype.names if k != "deleted"})
    par = oracle.wcsph_params(5.0, 0.01, 1000.0, kernel=kernel)
    P.h[:] = h
    dp = state.DeviceParticles(P.n)
    dp.upload_soa(P.as_dict())
    wc = core.wcsph_struct(5.0, 0.01, 1000.0)
    cfg = core.config_struct(kernel=kernel, precision="fp64", h_fixed=h if fixed else 0.0)
    ws = state.DeviceWorkspace(dp.n)
    core.compute(dp, wc, cfg, ws)
    ws.check()
    oracle.compute(par, oracle.NN(2.0), P, h if fixed else 0.0, oracle.max_threads())
    got = dp.soa()
    r = np.hypot(P.x[n:] - P.x[:n], P.y[n:] - P.y[:n])
    t = np.tile(2.0 - r / (0.5 * (P.h[:n] + P.h[n:])), 2)
    # of a few pairs, ends lie within each other's support: not these
    near = cKDTree(np.c_[P.x, P.y]).query_ball_point(np.c_[P.x, P.y], 2.1 * P.h.max(), return_length=True)
    inside = (t > 1e-6) & (near == 2)
    assert inside.sum() > n
    for k in ("drho", "ax"):
        want = getattr(P, k)[inside]
        e = np.abs(got[k][inside] - want) / np.abs(want)
        worst = np.argmax(e / _tol(t[inside]))
        assert e[worst] <= _tol(t[inside][worst]), (k, t[inside][worst], e[worst])
    for k in ("drho", "ax"):
        assert np.all(got[k][(t < -1e-6) & (near == 2)] == 0.0)


@pytest.mark.parametrize("t", [1e-2, 1e-3, 1e-4])
@pytest.mark.parametrize("side", [30, 70, 150])
def test_adjoint_of_one_pair(t, side):
    """side^2 groups of a wall particle, a fluid particle in its reach and a
    second fluid particle at 2 - t smoothing lengths from that one: the second
    one's gradients, and alpha's, are that pair's (8, 4 and 1 lanes)."""
    import adjoint_ref
    from sph import adjoint, build
    from sph.Common import particle_dtype
    build.build()
    dx = 0.02
    h = 1.3 * dx
    rng = np.random.default_rng(side)
    n = side * side
    k = np.arange(n)
    pa = np.zeros(3 * n, dtype=particle_dtype)
    wx, wy = 12.0 * h * (1 + k % side), 6.0 * h * (k // side)
    ang = rng.uniform(-0.5, 0.5, n)
    pa["x"][:n], pa["y"][:n] = wx - 0.6 * dx, wy + 0.1 * dx
    pa["x"][n:2 * n] = pa["x"][:n] - (2.0 - t) * h * np.cos(ang)
    pa["y"][n:2 * n] = pa["y"][:n] + (2.0 - t) * h * np.sin(ang)
    pa["x"][2 * n:], pa["y"][2 * n:] = wx, wy
    pa["label"][2 * n:] = 1
    pa["m"][:2 * n] = 1000.0 * dx * dx
    pa["rho"][:2 * n] = 1000.0
    case = adjoint.WallLoadCase(pa, height=6.0 * h * side + 1.0, r0=dx, h=h, dt=1e-6, nsteps=2, wall_x=0.0,
                                checkpoint=2)
    vel = case.velocities()
    # towards each other, by less than a thousandth of t h in the half step
    vel[n:, 0] = torch.as_tensor(rng.uniform(0.5, 1.0, n) * t * h, device="cuda")

    def grads(loss):
        a = torch.tensor(0.01, dtype=torch.float64, device="cuda", requires_grad=True)
        p, v = case.positions().requires_grad_(True), vel.clone().requires_grad_(True)
        return torch.autograd.grad(loss(a, p, v), (a, p, v))
    ga, gp, gv = grads(lambda a, p, v: adjoint.WallLoadLoss.apply(a, p, v, case))
    ra, rp, rv = grads(lambda a, p, v: adjoint_ref.reference_loss(case, a, p, v))
    assert abs(ga - ra).item() <= _tol(t) * abs(ra).item() and ra.item() != 0.0
    for g, w in ((gp, rp), (gv, rv)):
        e = torch.linalg.norm(g[n:] - w[n:], dim=1) / torch.linalg.norm(w[n:], dim=1)
        assert e.max().item() <= _tol(t)
