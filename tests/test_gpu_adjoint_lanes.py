"""The adjoint pair kernels at each number of lanes per query (8 below 9.7K
particles on 152 SMs, 4 up to 39K, 1 above) against torch autograd through the
unfused FP64 restatement (tests/adjoint_ref.py), both forms; the Gaussian's
FP64 and mixed forms against each other.  Two steps, so that round-off is not
amplified: 1e-10 for FP64, 2e-6 for the FP32 pair arithmetic."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _case(ny, kernel, precision, beta=0.0):
    from sph import adjoint, build, scenarios as S
    build.build()
    dx, nx = 2.0 / ny, ny // 2
    pa = S.dam_break(nx * dx, 2.0, dx, 1.5 * nx * dx, 2.2, side="right")
    rng = np.random.default_rng(ny)
    f = pa["label"] == 0
    for k in ("x", "y"):
        pa[k][f] += rng.uniform(-0.05 * dx, 0.05 * dx, f.sum())
        pa["v" + k][f] = rng.normal(0, 0.05, f.sum())
    h = 1.3 * dx
    return adjoint.WallLoadCase(pa, height=2.0, r0=dx, h=h, dt=0.2 * h / 62.6, nsteps=2, wall_x=1.5 * nx * dx,
                                checkpoint=2, kernel=kernel, adjoint_precision=precision)


def _rel(a, b):
    return ((a - b).norm() / b.norm()).item()


def _grads(case, loss_fn):
    a = torch.tensor(0.01, dtype=torch.float64, device="cuda", requires_grad=True)
    p, v = case.positions().requires_grad_(True), case.velocities().requires_grad_(True)
    return torch.autograd.grad(loss_fn(a, p, v), (a, p, v))


@pytest.mark.parametrize("ny", [37, 150, 290])
@pytest.mark.parametrize("kernel", [0, 1, 2])
def test_gradients_at_each_lane_count(ny, kernel):
    import adjoint_ref
    from sph import adjoint
    case = _case(ny, kernel, "fp64")
    got = _grads(case, lambda a, p, v: adjoint.WallLoadLoss.apply(a, p, v, case))
    mixed_case = _case(ny, kernel, "mixed")
    mixed = _grads(mixed_case, lambda a, p, v: adjoint.WallLoadLoss.apply(a, p, v, mixed_case))
    if kernel != 1:
        want = _grads(case, lambda a, p, v: adjoint_ref.reference_loss(case, a, p, v))
        for g, w in zip(got, want):
            assert _rel(g, w) <= 1e-10
    for m, g in zip(mixed, got):
        assert _rel(m, g) <= 2e-6


@pytest.mark.parametrize("checkpoint", [1, 2, 5])
def test_last_segment_kept_from_the_forward(checkpoint):
    """The last segment's builds come from the forward: a second backward
    through the same graph, with another forward in between, gives the same
    gradients, and so does every split into segments (a last one of one step
    included), bit for bit."""
    from sph import adjoint

    def loss_and_leaves(case, alpha):
        a = torch.tensor(alpha, dtype=torch.float64, device="cuda", requires_grad=True)
        p, v = case.positions().requires_grad_(True), case.velocities().requires_grad_(True)
        return adjoint.WallLoadLoss.apply(a, p, v, case), (a, p, v)

    def case_of(k):
        case = _case(37, 0, "fp64")
        case.nsteps, case.checkpoint = 5, k
        return case
    case = case_of(checkpoint)
    loss, leaves = loss_and_leaves(case, 0.01)
    first = torch.autograd.grad(loss, leaves, retain_graph=True)
    loss_and_leaves(case, 0.02)
    second = torch.autograd.grad(loss, leaves)
    whole = case_of(5)
    want_loss, want_leaves = loss_and_leaves(whole, 0.01)
    want = torch.autograd.grad(want_loss, want_leaves)
    assert torch.equal(loss, want_loss)
    for f, s, w in zip(first, second, want):
        assert torch.equal(f, s) and torch.equal(f, w)
        assert f.abs().max() > 0
