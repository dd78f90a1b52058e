"""What a wall-load loss holds on the device: beside its checkpoints at most one
set of workspace copies per case, from its forward to its first backward; none
without gradients; and never more than two sets during a backward.  Wherever
the last segment's copies come from, the gradients are the same, bit for bit."""
import gc

import pytest
import torch

pytestmark = pytest.mark.gpu
STEPS, K = 12, 4


def _case():
    from sph import adjoint, build, scenarios as S
    build.build()
    dx = 0.02
    pa = S.dam_break(0.5, 1.0, dx, 0.75, 1.1, side="right")
    return adjoint.WallLoadCase(pa, height=1.0, r0=dx, h=1.3 * dx, dt=1e-5, nsteps=STEPS, wall_x=0.75, checkpoint=K)


def _leaves(case, alpha=0.01):
    a = torch.tensor(alpha, dtype=torch.float64, device="cuda", requires_grad=True)
    return a, case.positions().requires_grad_(True), case.velocities().requires_grad_(True)


def _held():
    gc.collect()
    torch.cuda.synchronize()
    return torch.cuda.memory_allocated()


@pytest.fixture()
def case():
    from sph import adjoint
    c = _case()
    # everything that a first pass allocates once
    torch.autograd.grad(adjoint.WallLoadLoss.apply(*_leaves(c), c), _leaves(c)[:1], allow_unused=True)
    return c


def test_losses_before_their_backward_hold_one_set(case):
    from sph import adjoint
    one = case.ws.buf.numel()
    rows = STEPS // K * 8 * 8 * case.n
    before = _held()
    losses = [adjoint.WallLoadLoss.apply(*_leaves(case, 0.01 + 0.01 * k), case) for k in range(4)]
    assert _held() - before <= K * one + 4 * (2 * rows + (1 << 20))
    torch.autograd.backward(losses)
    assert _held() - before <= 4 * (2 * rows + (1 << 20))  # the losses are still here
    del losses
    assert _held() - before <= 1 << 20


def test_no_copies_without_gradients(case):
    from sph import adjoint
    leaves = _leaves(case)
    before = _held()
    torch.cuda.reset_peak_memory_stats()
    with torch.no_grad():
        loss = adjoint.WallLoadLoss.apply(*leaves, case)
    assert not loss.requires_grad
    assert torch.cuda.max_memory_allocated() - before < case.ws.buf.numel()


def test_backward_needs_two_sets(case):
    from sph import adjoint
    one = case.ws.buf.numel()
    leaves = _leaves(case)
    before = _held()
    torch.cuda.reset_peak_memory_stats()
    torch.autograd.grad(adjoint.WallLoadLoss.apply(*leaves, case), leaves)
    assert torch.cuda.max_memory_allocated() - before < (2 * K + 1) * one


def test_gradients_wherever_the_copies_are(case, monkeypatch):
    from sph import adjoint
    leaves = _leaves(case)
    kept = torch.autograd.grad(adjoint.WallLoadLoss.apply(*leaves, case), leaves)
    # the copies taken over by another loss of the case
    first = adjoint.WallLoadLoss.apply(*leaves, case)
    other = adjoint.WallLoadLoss.apply(*_leaves(case, 0.02), case)
    for g, w in zip(torch.autograd.grad(first, leaves), kept):
        assert torch.equal(g, w) and g.abs().max() > 0
    del other
    # another stream, where the earlier loss's copies are not taken over
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    waiting = adjoint.WallLoadLoss.apply(*_leaves(case, 0.02), case)
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        got = torch.autograd.grad(adjoint.WallLoadLoss.apply(*leaves, case), leaves)
    torch.cuda.current_stream().wait_stream(side)
    del waiting
    for g, w in zip(got, kept):
        assert torch.equal(g, w)
    # a scene whose copies would be too large
    monkeypatch.setattr(adjoint, "KEEP_BYTES", 0, raising=False)
    for g, w in zip(torch.autograd.grad(adjoint.WallLoadLoss.apply(*leaves, case), leaves), kept):
        assert torch.equal(g, w)
