"""Solves of more columns than one pass takes: 65535 groups of 32 (complex64), 16384
(complex128)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,n,R", [(torch.complex64, 3, 2_200_000), (torch.complex64, 70, 2_097_121),
                                       (torch.complex128, 3, 2_200_000), (torch.complex128, 130, 16_384),
                                       (torch.complex128, 130, 16_385), (torch.complex128, 200, 40_000)])
def test_every_column(dtype, n, R):
    from magreete_gb300 import engine as E
    gen = torch.Generator(device="cuda").manual_seed(R)
    A = torch.randn(n, n, dtype=dtype, device="cuda", generator=gen) + 4 * n ** 0.5 * torch.eye(n, device="cuda")
    B = torch.randn(n, R, dtype=dtype, device="cuda", generator=gen)
    X = E.lu_solve(E.lu_factor(A.clone()), B)
    A, rel = A.to(torch.complex128), 0.0
    for c in range(0, R, 1 << 18):
        x, b = X[:, c:c + (1 << 18)].to(torch.complex128), B[:, c:c + (1 << 18)].to(torch.complex128)
        rel = max(rel, (torch.linalg.norm(A @ x - b, dim=0) / torch.linalg.norm(b, dim=0)).max().item())
    # well conditioned (the diagonal dominates): a few roundings of the type for each of n terms
    assert rel <= 8 * (n + 8) * (2.0 ** -22 if dtype == torch.complex64 else 2.0 ** -53)
