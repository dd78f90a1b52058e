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
