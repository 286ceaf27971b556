"""complex128 LU and solves where the digit-split products need more than a scale
per row and column: single large entries, pairs of scatterers much nearer to each other
than to the rest, one right-hand side with large entries beside ordinary ones,
columns and rows of U of different size, diagonal blocks with ill-conditioned L.

FP64 elimination keeps the error of every column of P A = L U, and of every
field, within K 2^-53 of |L||U| in that column (K = 64 terms a product, of which
a bound of 64 roundings is taken); so do the products where they are made with
scales, shifted scales or on the FP64 pipe.  Inputs of order 1000, in the blocked
range; each is outside what one scale per column serves by 1e5 or more."""
import pytest
import torch

pytestmark = pytest.mark.gpu

N = 1000
BOUND = 64 * 2.0 ** -53
C = torch.complex128


def _random(n, m, seed):
    return torch.randn(n, m, dtype=C, generator=torch.Generator().manual_seed(seed)).cuda()


def _matrix(name):
    A = _random(N, N, 1)
    gen = torch.Generator().manual_seed(2)
    if name == "large entries":
        p = torch.randperm(N, generator=gen)[:60].cuda()
        A[p[:30], p[30:]] *= 1e9
    elif name == "blocks":
        A[:500, :500] *= 1e8
        A[500:, 500:] *= 1e8
    elif name == "rows and columns":
        k = torch.arange(0, N, 32, device="cuda")
        A[k] *= 1e10
        A[:, k] *= 1e-10
    elif name.startswith("ill-conditioned L"):
        w = 0.5 if name.endswith("0.5") else 0.9
        L = torch.tril(-w * torch.ones(N, N, dtype=torch.float64), -1)
        L = L + 0.1 * w * torch.tril(torch.rand(N, N, generator=gen, dtype=torch.float64), -1)
        L = (L * torch.triu(torch.ones(N, N, dtype=torch.float64), -40)).to(C).cuda()
        eye = torch.eye(N, dtype=C, device="cuda")
        A = (L + eye) @ (0.01 * torch.triu(A, 1) + eye)
    elif name.startswith("pairs"):
        from magreete_gb300 import engine as E
        p = torch.rand(334, 3, dtype=torch.float64, generator=gen)
        near = p[1::10].shape[0]
        p[1::10] = p[0::10][:near] + 1e-4 * torch.randn(near, 3, dtype=torch.float64, generator=gen)
        (A,) = E.assemble_system("3d_vector", p.cuda(), 30.0, 0.9, 0.0, ("c128",))
    return A


@pytest.mark.parametrize("name", ["large entries", "blocks", "rows and columns", "pairs", "ill-conditioned L 0.5",
                                  "ill-conditioned L 0.9"])
def test_columns_of_the_factors(name):
    from magreete_gb300 import engine as E
    A = _matrix(name)
    n = A.shape[0]
    f = E.lu_factor(A.clone())
    L = torch.tril(f.lu, -1) + torch.eye(n, dtype=C, device="cuda")
    U = torch.triu(f.lu)
    D = torch.linalg.norm(A[f.perm.long()] - L @ U, dim=0)
    S = torch.linalg.norm(L.abs() @ U.abs(), dim=0)
    assert (D / S).max().item() <= BOUND


def _rhs(name):
    B = _random(N, 40, 3)
    if name == "one column":
        return B[:, :1].contiguous()
    if name == "large entries in one":
        B[::7, 3] *= 1e10
    elif name == "units":
        B = torch.zeros(N, 40, dtype=C, device="cuda")
        B[torch.arange(40) * 20, torch.arange(40)] = 1
    return B


@pytest.mark.parametrize("system", ["random", "weakly coupled", "columns of U", "rows of U"])
@pytest.mark.parametrize("rhs", ["one column", "plain", "large entries in one", "units"])
def test_columns_of_the_fields(system, rhs):
    """L U X = B, column by column, with factors given as they are."""
    from magreete_gb300 import _lib as LB
    from magreete_gb300 import engine as E
    A = _random(N, N, 4) / N ** 0.5
    eye = torch.eye(N, dtype=C, device="cuda")
    L = torch.tril(A, -1) * (1e-6 if system == "weakly coupled" else 0.5) + eye
    U = torch.triu(A, 1) * (1e-6 if system == "weakly coupled" else 0.5) + eye
    s = torch.pow(2.0, torch.randint(-40, 41, (N,), generator=torch.Generator().manual_seed(5)).double()).cuda()
    B = _rhs(rhs)
    if system == "columns of U":
        U = U * s[None, :]
    elif system == "rows of U":
        U = U * s[:, None]
    f = E.LUFactors((torch.tril(L, -1) + U).contiguous(), torch.arange(N, dtype=torch.int32, device="cuda"), None,
                    LB.MGT_C128)
    X = E.lu_solve(f, B)
    R = (L @ (U @ X) - B).abs()
    T = L.abs() @ (U.abs() @ X.abs()) + B.abs()
    assert (torch.linalg.norm(R, dim=0) / torch.linalg.norm(T, dim=0)).max().item() <= BOUND
    if rhs in ("plain", "one column"):
        # entry by entry as well: no entry of these is small beside its row's terms
        assert (R / T).max().item() <= BOUND
