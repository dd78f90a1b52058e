"""A run on the sorted copy of the state leaves out of the copy what the run
writes before it reads, and returns by the inverse order; every field of every
particle, walls included, must end as in a run on the caller's arrays, whatever
the fields held before and in whatever order the particles are."""
import pytest

from test_gpu_e2e import _ws_without_copy

pytestmark = pytest.mark.gpu

FIELDS = ("m", "rho", "p", "c", "drho", "h", "x", "y", "vx", "vy", "ax", "ay", "xsphx", "xsphy",
          "x0", "y0", "vx0", "vy0", "rho0")


@pytest.mark.parametrize("steps", [4, 5])
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("form", ["pec", "pec_xsph_damped", "pec_sumdens", "pec_dynamic_h", "euler", "verlet"])
def test_every_field_returns(form, precision, steps):
    import torch
    import bench
    from sph import _lib as L, core, state
    wl = bench.workload("dambreak3200")
    dp, wc, _, _ = bench.prepare(wl, precision)
    g = torch.Generator().manual_seed(11)
    order = torch.randperm(dp.n, generator=g).cuda()
    lab = dp.label[order]
    start = {f: dp.fields[f][order] for f in FIELDS}
    noise = lambda: torch.rand(dp.n, generator=g, dtype=torch.float64).cuda()
    for f in ("x0", "y0", "vx0", "vy0", "rho0", "p", "drho", "xsphx", "xsphy", "ax", "ay"):
        start[f] = noise()
    start["c"] = float(wc.co) * (1.0 + 0.1 * noise())
    integrator = {"euler": L.INTEGRATOR_EULER, "verlet": L.INTEGRATOR_VERLET}.get(form, L.INTEGRATOR_PEC)
    if form == "pec_xsph_damped":
        wc.use_xsph = 1
    if form == "pec_sumdens":
        wc.use_summation_density = 1
    h_fixed = 0.0 if form == "pec_dynamic_h" else float(dp.h[dp.label == 0][0])
    kw = dict(precision=precision, h_fixed=h_fixed, cfl_c=0.25, cfl_f=0.25, integrator=integrator)
    if form == "pec_xsph_damped":
        kw.update(pec_use_xsph=True, damping=0.05)
    cfg = core.config_struct(**kw)
    n, ends = dp.n, []
    for ws in (state.DeviceWorkspace(n), _ws_without_copy(n)):
        dq, *_ = bench.prepare(wl, precision)
        dq.label.copy_(lab)
        for f in FIELDS:
            dq.fields[f].copy_(start[f])
        hist = torch.zeros((steps, 3), dtype=torch.float64, device="cuda")
        core.run(dq, wc, cfg, ws, steps, hist)
        ends.append((hist, {f: dq.fields[f].clone() for f in FIELDS}, dq.label.clone()))
    (h1, a, l1), (h2, b, l2) = ends
    assert torch.equal(h1, h2) and torch.equal(l1, l2)
    for f in FIELDS:
        assert torch.equal(a[f], b[f]), f
    assert not torch.equal(a["x"], start["x"])
