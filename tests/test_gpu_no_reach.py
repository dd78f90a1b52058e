"""A Lennard-Jones length r0 that no distance is below (a negative one,
as r <= r0 decides it) gives no boundary force, in the FP64 form and its adjoint."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ny", [30, 120])
def test_no_boundary_force(ny):
    from sph import adjoint, build, core, scenarios as S, state
    build.build()
    dx = 0.02
    pa = S.dam_break(ny * dx / 2, ny * dx, dx, 0.75 * ny * dx, 1.2 * ny * dx, side="right")
    rng = np.random.default_rng(ny)
    f = pa["label"] == 0
    for k in ("x", "y"):
        pa[k][f] += rng.uniform(-0.1 * dx, 0.1 * dx, f.sum())
        pa["v" + k][f] = rng.normal(0, 0.1, f.sum())

    def evaluate(reach):
        dp = state.DeviceParticles.from_array(pa)
        ws = state.DeviceWorkspace(dp.n)
        core.compute(dp, core.wcsph_struct(ny * dx, reach, 1000.0), core.config_struct(h_fixed=1.3 * dx), ws)
        ws.check()
        return dp.soa(("ax", "ay", "drho"))

    def gradients(reach):
        case = adjoint.WallLoadCase(pa, height=ny * dx, r0=reach, h=1.3 * dx, dt=1e-5, nsteps=2,
                                    wall_x=0.75 * ny * dx, checkpoint=2)
        vel = case.velocities()
        return adjoint.gradients(case, 0.01, None, vel)
    want, got = evaluate(0.0), evaluate(-dx)
    for k in want:
        assert np.array_equal(got[k], want[k]), k
    for w, g in zip(gradients(0.0), gradients(-dx)):
        assert torch.equal(g, w) and not g.any()
