"""A batch workspace that other entry points touch between batched runs: a
single-scene neighbour build or evaluation (sph_nn_update, sph_compute) or
sph_workspace_init, which reset or rewrite scratch that both forms use.  The
steps that follow must be those of an ensemble left alone, bit for bit."""
import ctypes as C
import types

import pytest
import torch

pytestmark = pytest.mark.gpu


def _between(E, what):
    from sph import _lib as L, core, state
    ws = types.SimpleNamespace(ws=E.ws)
    dp = state.DeviceParticles(E.dp.n)
    dp._buf.copy_(E.dp._buf)
    dp.label.copy_(E.dp.label)
    cfg = core.config_struct(precision="mixed", h_fixed=E.h[0])
    if what == "init":
        L.check(L.load().sph_workspace_init(C.byref(E.ws), state.current_stream()), "sph_workspace_init")
    elif what == "nn_update":
        core.nn_update(dp, cfg, ws)
    else:
        core.compute(dp, E.wc[0], cfg, ws)
    E.status()  # clears the status of the scene in between


@pytest.mark.parametrize("what", ["init", "nn_update", "compute"])
@pytest.mark.parametrize("count, shift", [(1, 0), (1, 4), (4, 2)])
def test_batched_steps_after_another_entry_point(what, count, shift):
    from sph import batch, build, scenarios
    build.build()
    cases = scenarios.ensemble(count=count, seed=count, width=(0.3, 0.8), height=(0.4, 1.0), dx=(0.02, 0.05))
    alone, touched = batch.Ensemble(cases), batch.Ensemble(cases)
    for E in (alone, touched):
        E.setup(shift)
    for step in range(12):
        _between(touched, what)
        for E in (alone, touched):
            E.run(1)
        assert torch.equal(alone.dp._buf, touched.dp._buf), step
    alone.check()
    touched.check()


def test_more_than_2_to_28_tiles():
    """One-cell tiles over a domain of more than 2^28 cells: particles in its
    corners and its middle step as in a single run."""
    import numpy as np
    from sph import batch, build, core, state
    from sph.Common import particle_dtype
    build.build()
    dx, ext = 0.02, 500.0
    gx, gy = np.meshgrid(np.arange(3) * dx, np.arange(3) * dx)
    at = [(0, 0), (ext, 0), (0, ext), (ext, ext), (ext / 2, ext / 2), (ext / 3, ext)]
    pa = np.zeros(9 * len(at), dtype=particle_dtype)
    pa["x"] = np.concatenate([gx.ravel() + x for x, _ in at])
    pa["y"] = np.concatenate([gy.ravel() + y for _, y in at])
    rng = np.random.default_rng(2)
    pa["vx"], pa["vy"] = rng.normal(0, 0.1, len(pa)), rng.normal(0, 0.1, len(pa))
    pa["m"], pa["rho"] = 1000.0 * dx * dx, 1000.0
    E = batch.Ensemble([(pa, dict(height=ext + 1.0, dx=dx))], max_cells=400_000_000)
    E.setup(0)
    dp = state.DeviceParticles(E.n)
    dp._buf.copy_(E.dp._buf)
    dp.label.copy_(E.dp.label)
    E.run(2)
    cells = E.instance_cells(0)
    E.buf = None
    cfg = core.config_struct(precision="mixed", h_fixed=E.h[0], cfl_c=0.3, cfl_f=0.25)
    ws = state.DeviceWorkspace(E.n, cells)
    core.run(dp, E.wc[0], cfg, ws, 2)
    ws.check()
    assert torch.equal(E.dp._buf, dp._buf)
    assert E.dp.drho.abs().min() > 0
