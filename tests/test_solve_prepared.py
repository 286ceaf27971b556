"""mgt_solve_prepared (digits in one workspace, a wide solve's scratch in
another) and the refinement's reuse of the factors' inverted diagonal blocks."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,R", [(30, 17), (400, 65), (1400, 130), (300, 1500)])
def test_wide_solve_matches_one_block(N, R):
    """A context prepared for 16 columns, right-hand sides of one column more
    than that up to more than one wide block: residuals meet the tolerance and
    the fields agree with those of a context of full width (both refined to
    1e-10, so within 1e-8)."""
    from magreete_gb300 import engine as E
    from magreete_gb300 import selfterm
    from magreete_gb300 import workloads as W
    prob = W.disk_problem(N, 5, 9.0, n_angles=4)
    pts = prob.points.cuda()
    coef = prob.alpha * prob.k0 ** 2
    shift = selfterm.diagonal_shift(prob.kind, prob.k0, prob.alpha, prob.radius)
    Mdf, M32 = E.assemble_system(prob.kind, pts, prob.k0, coef, shift, ("cdf", "c64"))
    gen = torch.Generator().manual_seed(R)
    B = torch.randn(2 * N, R, dtype=torch.complex128, generator=gen).cuda()
    f = E.mixed_factor(M32, lambda: None)
    full, narrow = E.RefineContext(Mdf, R), E.RefineContext(Mdf, 16)
    X0, _, r0 = E.solve_refined(full, f, B)
    X1, _, r1 = E.solve_refined(narrow, f, B)
    assert r0 <= 1e-10 and r1 <= 1e-10
    assert (torch.linalg.norm(X0 - X1) / torch.linalg.norm(X0)).item() < 1e-8
    # a second right-hand side through the same contexts: nothing of the first solve is reused
    X2, _, r2 = E.solve_refined(narrow, f, 2j * B)
    assert r2 <= 1e-10
    assert (torch.linalg.norm(X2 - 2j * X1) / torch.linalg.norm(X2)).item() < 1e-8
