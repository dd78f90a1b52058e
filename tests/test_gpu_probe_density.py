"""The warp-per-point probe kernel against the oracle: points inside, at the
surface and outside the fluid, search lengths from zero to more than 32 stencil
rows, every kernel, one point and a ragged number of them, and a coarse grid
whose stencil rows span several tiles."""
import numpy as np
import pytest

import sphcases as SC

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", [0, 1, 2])
@pytest.mark.parametrize("max_cells", [0, 64])
@pytest.mark.parametrize("h_search", [0.0, 0.026, 0.9])
def test_probe_density(kernel, max_cells, h_search):
    import oracle
    from sph import build, core, scenarios as S, state
    build.build()
    dx, H = 0.02, 0.5
    pa = S.dam_break(0.3, H, dx, 0.9, 0.7)
    rng = np.random.default_rng(kernel)
    f = pa["label"] == 0
    pa["x"][f] += rng.uniform(-0.002, 0.002, f.sum())
    P = oracle.Particles(arrays={k: pa[k] for k in pa.dtype.names if k != "deleted"})
    par = oracle.wcsph_params(H, dx, 1000.0)
    oracle.setup(P, par, H, 0.026)
    dp = state.DeviceParticles(P.n)
    dp.upload_soa(P.as_dict())
    ws = state.DeviceWorkspace(dp.n, max_cells)
    core.nn_update(dp, core.config_struct(kernel=kernel, h_fixed=0.026), ws)
    nn = oracle.NN(2.0)
    nn.update(P.x, P.y, P.h)
    for n in (1, 37):
        px, py = rng.uniform(0.02, 0.4, n), rng.uniform(0.02, 0.6, n)
        hs, hk = np.full(n, h_search), np.full(n, 0.026)
        rho, p = core.probe_density(dp, core.wcsph_struct(H, dx, 1000.0), kernel, ws, px, py, hs, hk)
        with np.errstate(all="ignore"):
            want, want_p = oracle.probe_density(nn, P, px, py, hs, hk, kernel, 1000.0, par.B, 7.0)
        rho, p = rho.cpu().numpy(), p.cpu().numpy()
        ok = np.isfinite(want)
        assert np.array_equal(np.isfinite(rho), ok)
        assert SC.rel_err(rho[ok], want[ok]) <= 1e-12
        assert SC.rel_err(p[ok], want_p[ok]) <= 1e-9
