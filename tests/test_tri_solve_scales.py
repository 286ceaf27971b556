"""complex64 triangular solves with factors whose rows or columns differ in size (U D
and D A for diagonal D up to 2^+-28), with right-hand sides that do, and with one
right-hand side of large entries beside ordinary ones: L U X = B entry by
entry.  FP32 substitution holds each entry to a few rounding errors of its own
terms; 2^-18 is sixteen times the 2^-22 of an operand's last bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu

C = torch.complex128


def _factors(n, seed):
    from magreete_gb300 import engine as E
    gen = torch.Generator().manual_seed(seed)
    A = torch.randn(n, n, dtype=C, generator=gen).cuda() + 4 * n ** 0.5 * torch.eye(n, device="cuda")
    f = E.lu_factor(A)
    assert torch.equal(f.perm.cpu(), torch.arange(n, dtype=torch.int32))
    return torch.tril(f.lu, -1), torch.triu(f.lu)


def _check(L, U, B):
    from magreete_gb300 import _lib as LB
    from magreete_gb300 import engine as E
    n = L.shape[0]
    LU = (L + U).to(torch.complex64)
    f = E.LUFactors(LU, torch.arange(n, dtype=torch.int32, device="cuda"), None, LB.MGT_C64)
    B = B.to(torch.complex64)
    X = E.lu_solve(f, B).to(C)
    assert torch.isfinite(torch.view_as_real(X)).all()
    LU, B = LU.to(C), B.to(C)
    Lm, Um = torch.tril(LU, -1) + torch.eye(n, dtype=C, device="cuda"), torch.triu(LU)
    R = (Lm @ (Um @ X) - B).abs()
    T = Lm.abs() @ (Um.abs() @ X.abs()) + B.abs()
    assert (R / T).max().item() <= 2.0 ** -18


@pytest.mark.parametrize("n,R", [(1200, 40), (300, 3), (2600, 200)])
@pytest.mark.parametrize("bits", [0, 6, 10, 13, 14, 20, 28])
@pytest.mark.parametrize("scaling", ["columns", "rows"])
def test_scaled_factors(n, R, bits, scaling):
    L, U = _factors(n, n)
    gen = torch.Generator().manual_seed(bits)
    s = torch.pow(2.0, ((torch.rand(n, generator=gen, dtype=torch.float64) * 2 - 1) * bits).round()).cuda()
    B = torch.randn(n, R, dtype=C, generator=gen).cuda()
    if scaling == "columns":
        _check(L, U * s[None, :], B)
    else:
        _check(s[:, None] * L / s[None, :], U * s[:, None], s[:, None] * B)


@pytest.mark.parametrize("scale", [1e-32, 1e-26, 1e26, 1e34])
def test_ends_of_the_range(scale):
    """Factors or fields near the ends of FP32's range."""
    L, U = _factors(600, 6)
    B = torch.randn(600, 40, dtype=C, generator=torch.Generator().manual_seed(7)).cuda()
    _check(L, U * scale, B * min(scale, 1.0))
    _check(L, U, B * scale)
    _check(L, U * scale, B * scale)


@pytest.mark.parametrize("coupling", [1.0, 1e-5])
def test_one_large_right_hand_side(coupling):
    L, U = _factors(700, 7)
    d = torch.diagonal(U)
    L, U = coupling * L, coupling * torch.triu(U, 1) + torch.diag(d)
    B = torch.randn(700, 40, dtype=C, generator=torch.Generator().manual_seed(8)).cuda()
    B[::7, 3] *= 1e10
    _check(L, U, B)
    units = torch.zeros(700, 40, dtype=C, device="cuda")
    units[torch.arange(40) * 17, torch.arange(40)] = 1
    _check(L, U, units)
