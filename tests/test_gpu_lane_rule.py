"""The FP64 kernels and the adjoint's on both sides of every edge of the rule for
lanes per query (lanes_per_query, csrc/pair_common.cuh), with XSPH, with an h
from the density and on coarse grids at 4 and 1 lanes as well.  Bars: 1e-10 for
one evaluation (test_gpu_pair64), 1e-10 and 2e-6 for two steps of the FP64 and
the mixed adjoint (test_gpu_adjoint_lanes)."""
import os
import re

import numpy as np
import pytest

import test_gpu_adjoint_lanes as AL
from test_gpu_pair64 import CUBIC, GAUSS, WEND, _evaluate

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


def _wave():
    """Queries of one wave, from the constants that the rule takes."""
    import torch
    text = open(os.path.join(HERE, "..", "offshore-sph_gb300", "csrc", "pair_common.cuh")).read()
    c = [int(re.search(r"constexpr int %s = (\d+);" % k, text).group(1)) for k in ("kPairBlock", "kPair64Blocks")]
    return torch.cuda.get_device_properties(0).multi_processor_count * c[0] * c[1]


def _lanes(n, wave, kernel=CUBIC, fixed=True, adjoint=False):
    if n < wave // 8:
        return 8
    if n < wave // 2:
        return 4
    if n <= wave or n >= 4 * wave:
        return 1
    if kernel == GAUSS:
        return 4 if adjoint or n % wave <= wave // 2 else 1
    if adjoint or (kernel == CUBIC and fixed):
        return 1
    return 4 if n <= wave + (2 if fixed else 3) * wave // 8 else 1


# (kernel, fixed h, XSPH, edge in eighths of a wave, n at the edge less the edge):
# the last size on one side and the first on the other
EDGES = [(k, f, x, e, -1) for k, f, x in ((CUBIC, True, False), (CUBIC, False, True), (GAUSS, True, True),
                                          (WEND, False, False), (WEND, True, True)) for e in (1, 4)]
EDGES += [(CUBIC, False, True, 8, 0), (CUBIC, False, False, 11, 0), (WEND, False, True, 11, 0), (WEND, True, False, 10, 0),
          (GAUSS, True, False, 8, 0), (GAUSS, False, True, 12, 0), (GAUSS, True, True, 16, -1), (GAUSS, True, False, 28, 0)]


@pytest.mark.parametrize("kernel, fixed, xsph, eighths, last", EDGES)
def test_both_sides_of_an_edge(kernel, fixed, xsph, eighths, last):
    from sph import scenarios as S
    wave = _wave()
    n = eighths * wave // 8 + last
    assert _lanes(n, wave, kernel, fixed) != _lanes(n + 1, wave, kernel, fixed)
    ny = 127
    for size in (n, n + 1):
        pa = S.jittered_lattice(size // ny + 1, ny, 0.01, seed=eighths + kernel)[:size]
        assert len(pa) == size
        _evaluate(pa, 1.27, 0.01, 0.013 if fixed else 0.0, kernel, xsph)


@pytest.mark.parametrize("part", [0.2, 0.7])
@pytest.mark.parametrize("max_cells", [64, 700, 5000])
def test_coarse_grids(part, max_cells):
    """Stencil rows over several tiles of 1 to 4 cells at 4 and 1 lanes, in a
    tank, with XSPH at a fixed h and with an h from the density."""
    from sph import scenarios as S
    wave = _wave()
    ny = int(np.sqrt(part * wave / 0.65))
    dx = 0.02
    pa = S.dam_break(ny * dx / 2, ny * dx, dx, 0.75 * ny * dx, 1.2 * ny * dx)
    assert _lanes(len(pa), wave) == (4 if part < 0.5 else 1)
    rng = np.random.default_rng(max_cells)
    f = pa["label"] == 0
    for k in ("x", "y"):
        pa[k][f] += rng.uniform(-0.002, 0.002, f.sum())
        pa["v" + k][f] = rng.normal(0, 0.1, f.sum())
    _evaluate(pa, ny * dx, dx, 1.3 * dx, CUBIC, True, max_cells)
    _evaluate(pa, ny * dx, dx, 0.0, WEND, False, max_cells, beta=0.02)


@pytest.mark.parametrize("part", [0.2, 0.6, 1.1])
@pytest.mark.parametrize("kernel", [0, 1, 2])
def test_adjoint_at_four_and_one_lanes(part, kernel):
    import adjoint_ref
    from sph import adjoint
    wave = _wave()
    case = AL._case(int(np.sqrt(part * wave / 0.54)), kernel, "fp64")
    lanes = 4 if part < 0.5 or (kernel == GAUSS and part > 1.0) else 1
    assert abs(case.n / wave - part) < 0.1 * part and _lanes(case.n, wave, kernel, adjoint=True) == lanes
    got = AL._grads(case, lambda a, p, v: adjoint.WallLoadLoss.apply(a, p, v, case))
    mixed_case = AL._case(int(np.sqrt(part * wave / 0.54)), kernel, "mixed")
    mixed = AL._grads(mixed_case, lambda a, p, v: adjoint.WallLoadLoss.apply(a, p, v, mixed_case))
    if kernel != 1:
        want = AL._grads(case, lambda a, p, v: adjoint_ref.reference_loss(case, a, p, v))
        for g, w in zip(got, want):
            assert AL._rel(g, w) <= 1e-10
    for m, g in zip(mixed, got):
        assert AL._rel(m, g) <= 2e-6
