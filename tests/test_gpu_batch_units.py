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
