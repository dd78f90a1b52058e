"""The batched tile kernel's work units: tanks whose tiles come whole, in
halves and in quarters (few tiles: all of them are split) and tanks of tiles
too small to split, with tiles of wall particles alone that are not listed.
The results do not depend on the tile shape, bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 5, 70])
def test_tile_shapes_give_the_same_steps(count):
    from sph import batch, build, scenarios
    build.build()
    cases = scenarios.ensemble(count=count, seed=count, width=(0.3, 1.0), height=(0.4, 1.2), dx=(0.02, 0.05))
    E = batch.Ensemble(cases)
    snap = E.snapshot()
    want = None
    for shift in (4, 3, 2, 1, 0):
        E.setup(shift)
        E.restore(snap)
        E.run(3)
        E.check()
        if want is None:
            want = E.dp._buf.clone()
        assert torch.equal(E.dp._buf, want), shift


@pytest.mark.parametrize("nsteps", [1, 2, 5])
def test_p_c_and_h_end_as_in_a_single_run(nsteps):
    """The steps between the first and the last do not store p, c and h; the
    end is that of a single run, whatever the fields held before."""
    from sph import batch, build, core, scenarios, state
    build.build()
    cases = scenarios.ensemble(count=3, seed=7, width=(0.2, 0.5), height=(0.3, 0.8), dx=(0.02, 0.05))
    E = batch.Ensemble(cases)
    g = torch.Generator().manual_seed(5)
    f = E.dp.fields
    f["p"].copy_(torch.rand(E.dp.n, generator=g, dtype=torch.float64))
    f["c"].mul_(1.0 + 0.1 * torch.rand(E.dp.n, generator=g, dtype=torch.float64).cuda())
    f["h"][E.dp.label == 0] *= 0.9
    start = {k: v.clone() for k, v in f.items()}
    E.run(nsteps)
    E.check()
    for b, (pa, c) in enumerate(cases):
        s, e = int(E.offsets_np[b]), int(E.offsets_np[b + 1])
        dp = state.DeviceParticles.from_array(pa)
        for k, v in start.items():
            dp.fields[k].copy_(v[s:e])
        wc = core.wcsph_struct(c["height"], c["dx"], 1000.0)
        cfg = core.config_struct(precision="mixed", h_fixed=1.3 * c["dx"], cfl_c=0.3, cfl_f=0.25)
        ws = state.DeviceWorkspace(len(pa), E.instance_cells(b))
        core.run(dp, wc, cfg, ws, nsteps)
        for k in start:
            assert torch.equal(f[k][s:e], dp.fields[k]), (b, k)
