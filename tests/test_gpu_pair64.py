"""The FP64 pair kernel (csrc/pair64.cu) against the oracle: one evaluation at
the edges of its rule for lanes per query (particles against the threads of
one wave of blocks), with every smoothing kernel, with a fixed h and an h from
the density, with XSPH and with neighbourhoods that overflow its lists, and on
grids whose stencils span several tiles.  The bar is the FP64 form's 1e-10."""
import numpy as np
import pytest

import sphcases as SC

pytestmark = pytest.mark.gpu
TOL = 1e-10
CUBIC, GAUSS, WEND = 0, 1, 2


def _evaluate(pa, height, dx, h, kernel, xsph, max_cells=0, alpha=0.01, beta=0.0):
    import oracle
    from sph import build, core, state
    build.build()
    P = oracle.Particles(arrays={k: pa[k] for k in pa.dtype.names if k != "deleted"})
    par = oracle.wcsph_params(height, dx, 1000.0, use_xsph=xsph, kernel=kernel, alpha=alpha, beta=beta)
    P.h[P.label == 0] = h if h > 0 else 1.3 * dx
    dp = state.DeviceParticles(P.n)
    dp.upload_soa(P.as_dict())
    wc = core.wcsph_struct(height, dx, 1000.0, use_xsph=xsph, alpha=alpha, beta=beta)
    cfg = core.config_struct(kernel=kernel, precision="fp64", h_fixed=h)
    ws = state.DeviceWorkspace(dp.n, max_cells)
    core.compute(dp, wc, cfg, ws)
    ws.check()
    oracle.compute(par, oracle.NN(2.0), P, h, oracle.max_threads())
    got = dp.soa()
    f = P.label == 0
    bad = {}
    for k in ("drho", "ax", "ay", "h") + (("xsphx", "xsphy") if xsph else ()):
        e = SC.rel_err(got[k][f], getattr(P, k)[f])
        if not e <= TOL:
            bad[k] = e
    assert not bad, bad


@pytest.mark.parametrize("part", [0.125, 0.5, 1.0, 4.0])
@pytest.mark.parametrize("side", [-1, 1])
def test_lanes_per_query_edges(part, side):
    """Lattices just below and just above each edge of the rule."""
    import torch
    from sph import scenarios as S
    wave = torch.cuda.get_device_properties(0).multi_processor_count * 512
    ny = 127
    nx = int(part * wave) // ny + (side > 0)
    pa = S.jittered_lattice(nx, ny, 0.01, seed=int(8 * part) + side)
    _evaluate(pa, 1.27, 0.01, 0.013, CUBIC, False)


@pytest.mark.parametrize("kernel", [CUBIC, GAUSS, WEND])
@pytest.mark.parametrize("h", [0.013, 0.0])
@pytest.mark.parametrize("nx", [7, 90, 260])
def test_kernels_and_h(kernel, h, nx):
    """Every kernel, fixed h and computed h, with XSPH, at each number of
    lanes (7 x 31, 90 x 131 and 260 x 201 particles)."""
    from sph import scenarios as S
    pa = S.jittered_lattice(nx, {7: 31, 90: 131, 260: 201}[nx], 0.01, seed=kernel + nx)
    _evaluate(pa, 1.0, 0.01, h, kernel, True)


@pytest.mark.parametrize("kernel", [CUBIC, GAUSS])
@pytest.mark.parametrize("nx", [24, 120, 230])
def test_lists_overflow(kernel, nx):
    """h = 2.6 dx: about 85 (Gaussian 190) pairs per particle, several lists
    full."""
    from sph import scenarios as S
    pa = S.jittered_lattice(nx, nx + 3, 0.01, seed=nx)
    _evaluate(pa, 1.0, 0.01, 0.026, kernel, False)


@pytest.mark.parametrize("max_cells", [16, 64, 700])
def test_narrow_tiles(max_cells):
    """Coarse grids: tiles of 1 to 4 cells, stencil rows over several tiles;
    a tank, so with boundary neighbours."""
    from sph import scenarios as S
    pa = S.dam_break(0.3, 0.5, 0.02, 0.9, 0.7)
    rng = np.random.default_rng(5)
    f = pa["label"] == 0
    for k in ("x", "y"):
        pa[k][f] += rng.uniform(-0.002, 0.002, f.sum())
        pa["v" + k][f] = rng.normal(0, 0.1, f.sum())
    _evaluate(pa, 0.5, 0.02, 0.026, CUBIC, True, max_cells)
    _evaluate(pa, 0.5, 0.02, 0.0, WEND, False, max_cells, beta=0.02)


@pytest.mark.parametrize("kernel", [CUBIC, GAUSS, WEND])
@pytest.mark.parametrize("offset, scale", [(0.0, 1.0), (-0.6, 1.0), (-37.125, 1.0), (1e3, 1.0), (1e5, 1.0),
                                           (0.0, 1e-4), (0.0, 3e3)])
def test_integer_differences(kernel, offset, scale):
    """The integer positions (at 4 lanes): coordinates around zero, negative,
    far from the origin up to where the FP64 differences take over (1e5 is 4
    million interaction radii), and small and large units."""
    from sph import scenarios as S
    dx = 0.01 * scale
    pa = S.jittered_lattice(121, 131, dx, seed=kernel)
    pa["x"] += offset * scale
    pa["y"] -= 0.5 * offset * scale
    _evaluate(pa, 1.3 * scale, dx, 1.3 * dx, kernel, False)
