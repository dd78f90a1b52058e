"""Pairs that straddle a coordinate axis with differences far below the
interaction radius: such positions have more bits than the FP64 kernel's integer
positions hold, and their differences must be the exact ones all the same.
Geometry exact, so the tolerance is that of test_gpu_support_edge at q <= 1.5."""
import numpy as np
import pytest

from test_gpu_support_edge import CUBIC, _pairs, _tol

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fixed", [True, False])
@pytest.mark.parametrize("n", [10007, 35003])
def test_small_differences_near_the_axes(fixed, n):
    """400 pairs along the axes beside n others (4 and 1 lanes): along x = 0
    their ax, along y = 0 (moving in y alone) their drho is proportional to the
    small difference."""
    import oracle
    from sph import build, core, state
    from sph.Common import particle_dtype
    build.build()
    h = 0.0325 if fixed else 1.3 * np.sqrt(0.4 / 1030.0)
    rng = np.random.default_rng(n)
    m = 200
    rest = _pairs(n, h, n)
    rest["x"] += 24 * h
    rest["y"] += 24 * h
    ax = np.zeros(4 * m, dtype=particle_dtype)
    small = rng.choice([-1.0, 1.0], (4, m)) * 10.0 ** rng.uniform(-14, -4, (4, m))
    r = rng.uniform(0.5, 1.5, (2, m)) * h
    along = 24 * h + 12 * h * np.arange(m)
    ax["x"] = np.r_[small[0], small[1], along, along + r[1]]
    ax["y"] = np.r_[along, along + r[0], small[2], small[3]]
    ax["m"], ax["rho"] = 0.4, rng.uniform(1010.0, 1050.0, 4 * m)
    ax["vy"][3 * m:] = rng.uniform(0.1, 1.0, m)
    pa = np.concatenate((ax, rest))
    P = oracle.Particles(arrays={k: pa[k] for k in pa.dtype.names if k != "deleted"})
    P.h[:] = h
    dp = state.DeviceParticles(P.n)
    dp.upload_soa(P.as_dict())
    ws = state.DeviceWorkspace(dp.n)
    core.compute(dp, core.wcsph_struct(5.0, 0.01, 1000.0), core.config_struct(h_fixed=h if fixed else 0.0), ws)
    ws.check()
    oracle.compute(oracle.wcsph_params(5.0, 0.01, 1000.0, kernel=CUBIC), oracle.NN(2.0), P, h if fixed else 0.0,
                   oracle.max_threads())
    got = dp.soa()
    for k, s in (("ax", slice(0, 2 * m)), ("drho", slice(2 * m, 4 * m))):
        want = getattr(P, k)[s]
        assert (np.abs(got[k][s] - want) / np.abs(want)).max() <= _tol(0.4), k
