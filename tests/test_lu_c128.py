"""The complex128 LU and its solves on the tensor cores (csrc/zpanel.cu,
zgemm_tc.cu, zsolve.cu).

The panel kernel (one row per four threads, messages in distributed shared
memory or through L2) picks the pivots of the shared-memory panel and gives
its bits.  From order 768 on, U12 and the trailing update are digit-split
products: backward errors are held to what FP64 arithmetic guarantees,
c n 2^-53 with a small c (random matrices reach about n^0.5).
"""
import pytest
import torch

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


def _random(n, m, seed):
    return torch.randn(n, m, dtype=torch.complex128, generator=torch.Generator().manual_seed(seed)).cuda()


def _split(f):
    n = f.lu.shape[0]
    Lm = torch.tril(f.lu, -1) + torch.eye(n, dtype=torch.complex128, device="cuda")
    return Lm, torch.triu(f.lu)


@pytest.mark.parametrize("n", [1, 4, 31, 32, 33, 65, 200, 513, 767, 768, 1025, 1100, 2500])
def test_panel_matches_shared_memory_panel(n):
    """Orders around the panel width, the cluster's largest panel (1024 rows) and
    the first blocked order; equal largest entries in one column (the lowest
    row wins)."""
    from magreete_gb300 import _lib as L
    from magreete_gb300 import engine as E
    lib = L.load()
    A = _random(n, n, n)
    if n > 64:
        A[5:40, 0] = 10 + 10j
    outs = []
    try:
        for mode, cluster in ((0, 0), (1, 1), (1, 0)):
            lib.mgt_set_tuning(L.MGT_TUNE_PANEL_REGISTERS, mode)
            lib.mgt_set_tuning(L.MGT_TUNE_PANEL_CLUSTER, cluster)
            f = E.lu_factor(A.clone(), check_singular=False)
            assert E.lu_info(f) == (0, 0)
            outs.append(f)
    finally:
        lib.mgt_set_tuning(L.MGT_TUNE_PANEL_REGISTERS, 1)
        lib.mgt_set_tuning(L.MGT_TUNE_PANEL_CLUSTER, 1)
    for f in outs[1:]:
        assert torch.equal(f.perm, outs[0].perm)
        assert torch.equal(f.lu, outs[0].lu)
    if n > 64:
        assert int(outs[1].perm[0]) == 5


@pytest.mark.parametrize("n,pad", [(768, 0), (769, 3), (801, 0), (832, 1), (1000, 0), (2049, 0)])
@pytest.mark.parametrize("scaling", ["none", "rows", "columns"])
def test_blocked_lu_is_a_factorisation(n, pad, scaling):
    """P A = L U row by row (columns scaled) for orders off and on the 64-wide
    block and 128-row tile, leading dimensions beyond n, and rows or columns of
    sizes from 1e-30 to 1e30."""
    from magreete_gb300 import engine as E
    store = torch.zeros(n, n + pad, dtype=torch.complex128, device="cuda")
    A = _random(n, n, 3 * n)
    s = torch.logspace(-30, 30, n, dtype=torch.float64, device="cuda")
    s = s[torch.randperm(n, generator=torch.Generator().manual_seed(n)).cuda()]
    if scaling == "rows":
        A = A * s[:, None]
    elif scaling == "columns":
        A = A * s[None, :]
    store[:, :n] = A
    f = E.lu_factor(store[:, :n], check_singular=False)
    assert E.lu_info(f) == (0, 0)
    Lm, U = _split(f)
    perm = f.perm.long()
    assert torch.equal(torch.sort(perm).values, torch.arange(n, device="cuda"))
    # |l| <= sqrt(2) by the |re| + |im| rule
    assert Lm.abs().max().item() <= 2 ** 0.5 * (1 + 1e-12)
    PA = A[perm]
    if scaling == "columns":
        D = (Lm @ U - PA) / s[None, :]
        ref = PA / s[None, :]
    elif scaling == "rows":
        # L = S_p L0 S_p^-1 and U = S_p U0 for row scales s: compare unscaled
        sp = s[perm]
        D = (Lm / sp[:, None]) @ U - PA / sp[:, None]
        ref = PA / sp[:, None]
    else:
        D, ref = Lm @ U - PA, PA
    err = (torch.linalg.norm(D) / torch.linalg.norm(ref)).item()
    assert err <= 4 * n * EPS, err


@pytest.mark.parametrize("n,R", [(1, 1), (63, 2), (64, 33), (65, 1), (129, 305), (767, 32), (1000, 64), (1153, 700)])
def test_solves(n, R):
    """Backward error of the solves around the 64-row block, with one column,
    columns off the 32-column tile and more columns than twice the SMs."""
    from magreete_gb300 import engine as E
    A, B = _random(n, n, n + R), _random(n, R, 7 * n + R)
    f = E.lu_factor(A.clone())
    X = E.lu_solve(f, B)
    be = torch.linalg.norm(A @ X - B) / (torch.linalg.norm(A) * torch.linalg.norm(X))
    assert be.item() <= 4 * n * EPS, be.item()


def test_solve_with_badly_scaled_rows():
    """Right-hand sides and factors whose rows differ by up to 1e30: the solve of
    a row-scaled system is that of the unscaled one."""
    from magreete_gb300 import engine as E
    n, R = 900, 5
    A, B = _random(n, n, 1), _random(n, R, 2)
    e = torch.randint(-50, 51, (n,), generator=torch.Generator().manual_seed(3)).cuda()
    s = torch.pow(torch.tensor(2.0, dtype=torch.float64), e.to(torch.float64).cpu()).cuda()
    f = E.lu_factor(A * s[:, None])
    X = E.lu_solve(f, B * s[:, None])
    r = torch.linalg.norm(A @ X - B) / (torch.linalg.norm(A) * torch.linalg.norm(X))
    # the pivot order differs (the largest scaled row), the growth with it: n^2 covers both
    assert r.item() <= n * n * EPS, r.item()


@pytest.mark.parametrize("n", [100, 900])
def test_nan_and_singular(n):
    """A NaN entry reaches every field (as an FP64 elimination spreads it); an
    exactly zero column is reported with LAPACK's 1-based index."""
    from magreete_gb300 import engine as E
    A, B = _random(n, n, 5), _random(n, 3, 6)
    Z = A.clone()
    Z[:, 70] = 0
    f = E.lu_factor(Z, check_singular=False)
    assert E.lu_info(f) == (0, 71)
    A[n // 2, n // 3] = float("nan")
    f = E.lu_factor(A, check_singular=False)
    X = E.lu_solve(f, B)
    assert torch.isnan(torch.view_as_real(X)).all()
