"""Wide refined solves: every group of columns of the context's width is held to the
tolerance by itself, as when the groups are solved one after the other."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _system(N):
    from magreete_gb300 import engine as E
    from magreete_gb300 import selfterm
    from magreete_gb300 import workloads as W
    prob = W.disk_problem(N, 5, 9.0, n_angles=4)
    pts = prob.points.cuda()
    coef = prob.alpha * prob.k0 ** 2
    shift = selfterm.diagonal_shift(prob.kind, prob.k0, prob.alpha, prob.radius)
    return E.assemble_system(prob.kind, pts, prob.k0, coef, shift, ("cdf", "c64"))


@pytest.mark.parametrize("width,R", [(16, 100), (64, 130), (64, 1100)])
def test_small_group_beside_a_large_one(width, R):
    """A group 1e9 times smaller than the others: its residual, relative to itself, meets
    the tolerance (one norm over all columns is met without a single correction of it)."""
    from magreete_gb300 import engine as E
    Mdf, M32 = _system(400)
    B = torch.randn(800, R, dtype=torch.complex128, generator=torch.Generator().manual_seed(R)).cuda()
    B[:, width:2 * width] *= 1e-9
    f = E.mixed_factor(M32, lambda: None)
    ctx = E.RefineContext(Mdf, width)
    X, it, rr = E.solve_refined(ctx, f, B, tol=1e-12)
    assert it >= 1 and rr <= 1e-12
    Rr = E.residual(Mdf, X, B)
    for c in range(0, R, width):
        rel = torch.linalg.norm(Rr[:, c:c + width]) / torch.linalg.norm(B[:, c:c + width])
        assert rel.item() <= 1.01e-12, c


def test_a_group_that_misses_the_tolerance():
    """A tolerance out of reach is reported, with the residual of the worst group; a zero
    group is met by zero fields."""
    from magreete_gb300 import _lib as L
    from magreete_gb300 import engine as E
    Mdf, M32 = _system(200)
    B = torch.randn(400, 50, dtype=torch.complex128, generator=torch.Generator().manual_seed(1)).cuda()
    B[:, 16:32] = 0
    f = E.mixed_factor(M32, lambda: None)
    ctx = E.RefineContext(Mdf, 16)
    X, _, rr = E.solve_refined(ctx, f, B, tol=1e-30, require=False)
    assert 1e-30 < rr < 1e-13
    with pytest.raises(L.MagreeteError):
        E.solve_refined(ctx, f, B, tol=1e-30)
    X, _, rr = E.solve_refined(ctx, f, B, tol=1e-11)
    assert rr <= 1e-11 and not X[:, 16:32].any()


def test_no_room_for_a_wide_block(monkeypatch):
    """Where the device has no room for a wide block's workspace the columns are
    solved in blocks of the context's width, in its own."""
    from magreete_gb300 import engine as E
    Mdf, M32 = _system(300)
    B = torch.randn(600, 200, dtype=torch.complex128, generator=torch.Generator().manual_seed(2)).cuda()
    f = E.mixed_factor(M32, lambda: None)
    ctx = E.RefineContext(Mdf, 32)
    X0, _, r0 = E.solve_refined(ctx, f, B)
    calls = []

    def full(nbytes, device):
        calls.append(nbytes)
        raise torch.cuda.OutOfMemoryError("no room")

    monkeypatch.setattr(E, "workspace", full)
    X1, _, r1 = E.solve_refined(ctx, f, B)
    assert len(calls) == 1 and r0 <= 1e-10 and r1 <= 1e-10
    assert (torch.linalg.norm(X1 - X0) / torch.linalg.norm(X0)).item() < 1e-8
