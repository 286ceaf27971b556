"""complex64 triangular solves in 256-row blocks (tri_step_kernel): orders and
column counts around the blocks (64, 128, 256 rows, 32 columns), both ways of
sharing the work of a step (a cluster per block row; one CTA per 128 rows once
the launch would not be resident at once), an odd leading dimension, inverted
diagonal blocks with and without their Newton step, and a column of NaN beside
finite ones.

Bound: operands carry 22 bits, sums are FP32, so the residual of L U x = P b is
a few 2^-22 of |L| |U| |x| + |b| for well-conditioned diagonal blocks; 1e-6 is
four of them.  Random factors are ill-conditioned (condition numbers of the
blocks up to 1e4): their bound is the one the substitution in 64-row blocks
meets too, 1e-6 of the same quantity, normwise."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def _solve(lu, perm, B):
    from magreete_gb300 import _lib as L
    lib = L.load()
    n, R = B.shape
    nb = ctypes.c_size_t()
    L.check(lib.mgt_lu_solve_workspace_bytes(L.MGT_C64, n, R, ctypes.byref(nb)))
    work = torch.full((nb.value,), 0x7F, dtype=torch.uint8, device="cuda")
    X = torch.empty_like(B)
    L.check(lib.mgt_lu_solve(L.MGT_C64, ctypes.c_void_p(lu.data_ptr()), n, lu.stride(0),
                             ctypes.c_void_p(perm.data_ptr()), ctypes.c_void_p(B.data_ptr()), R,
                             ctypes.c_void_p(X.data_ptr()), R, R, ctypes.c_void_p(work.data_ptr()), nb.value,
                             ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    torch.cuda.synchronize()
    return X


def _system(n, R, random, lda):
    from magreete_gb300 import engine as E
    gen = torch.Generator(device="cuda").manual_seed(10 * n + R)
    A = torch.randn(n, n, dtype=torch.complex64, device="cuda", generator=gen)
    if not random:
        A += 4 * n ** 0.5 * torch.eye(n, device="cuda")
    f = E.lu_factor(A)
    lu = torch.empty(n, lda, dtype=torch.complex64, device="cuda")[:, :n]
    lu.copy_(f.lu)
    B = torch.randn(n, R, dtype=torch.complex64, device="cuda", generator=gen)
    return lu, f.perm, B


def _residual(lu, perm, X, B):
    LU = lu.to(torch.complex128)
    Lm = torch.tril(LU, -1) + torch.eye(lu.shape[0], dtype=LU.dtype, device="cuda")
    U = torch.triu(LU)
    x, b = X.to(torch.complex128), B.to(torch.complex128)[perm.long()]
    scale = torch.linalg.norm(Lm.abs() @ (U.abs() @ x.abs()) + b.abs())
    return (torch.linalg.norm(Lm @ (U @ x) - b) / scale).item()


@pytest.mark.parametrize("random", [False, True])
@pytest.mark.parametrize("n,R,pad", [(1, 1, 0), (63, 33, 1), (64, 32, 0), (65, 1, 2), (128, 31, 1), (255, 65, 0),
                                     (256, 32, 1), (257, 33, 0), (511, 5, 3), (513, 64, 0), (700, 300, 1),
                                     (1500, 300, 0)])
def test_tri_solve_edges(n, R, pad, random):
    lu, perm, B = _system(n, R, random, n + pad)
    assert _residual(lu, perm, _solve(lu, perm, B), B) < 1e-6


def test_tri_solve_nan_column():
    lu, perm, B = _system(600, 40, False, 600)
    clean = _solve(lu, perm, B)
    B[17, 3] = float("nan")
    B[599, 35] = float("inf")
    X = _solve(lu, perm, B)
    bad = torch.zeros(40, dtype=torch.bool)
    bad[[3, 35]] = True
    assert torch.equal(X[:, ~bad], clean[:, ~bad])
    assert not torch.isfinite(torch.view_as_real(X[:, bad])).all(0).any()
