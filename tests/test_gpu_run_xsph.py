"""The XSPH velocity that a run without XSPH leaves: 0 for a particle that had
neighbours (itself included) in any of the run's steps, as steps run one by one
leave it, also when it had none in the first and the last.  A particle at the
right end of the reference's grid, a whole number of cells from the left end,
is in no cell of its own stencil: this one is there in steps 0 and 4 of 5."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("kernel", [0, 1])
def test_neighbours_in_the_middle_steps_alone(precision, kernel):
    from sph import build, core, state
    from sph.Common import particle_dtype
    build.build()
    pa = np.zeros(3, dtype=particle_dtype)
    pa["x"], pa["y"] = [0.0, 0.0, 1.0 - 1.0 / 128], [0.0, 0.51, 0.0]
    pa["vx"] = [0.0, 0.0, 1.0]
    pa["m"], pa["rho"] = 0.5, 1000.0
    pa["xsphx"], pa["xsphy"] = 0.25, -0.5
    wc = core.wcsph_struct(1.0, 0.01, 1000.0)
    cfg = core.config_struct(kernel=kernel, precision=precision, h_fixed=1.0 / 32, dt_fixed=1.0 / 64)

    def run(parts):
        dp = state.DeviceParticles.from_array(pa)
        core.initialize(dp, wc, cfg)
        ws = state.DeviceWorkspace(dp.n)
        left = []
        for n in parts:
            core.run(dp, wc, cfg, ws, n)
            left.append(dp.xsphx.clone())
        ws.check()
        return dp, left
    one, left = run([1] * 5)
    assert left[0].tolist() == [0.0, 0.0, 0.25] and left[1].tolist() == [0.0, 0.0, 0.0]
    for parts in ([5], [3, 2], [1, 4]):
        whole, _ = run(parts)
        assert torch.equal(whole.xsphx, one.xsphx) and torch.equal(whole.xsphy, one.xsphy), parts
