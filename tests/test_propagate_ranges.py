"""The plain method's propagation at the ends of its range: more sources than the
assembled way has slabs for, more detectors than one assembly launch takes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,T,S,R", [("3d_scalar", 3, 4_300_000, 2), ("3d_scalar", 140, 4_200_000, 1),
                                        ("2d_scalar", 300_001, 50, 3), ("2d_scalar", 262_140, 60, 1),
                                        ("2d_scalar", 262_141, 60, 1)])
def test_matches_dense_product(kind, T, S, R):
    from magreete_gb300 import engine as E
    dim = E.KIND_DIMS[kind][0]
    gen = torch.Generator(device="cuda").manual_seed(T)
    tg = torch.rand(T, dim, dtype=torch.float64, device="cuda", generator=gen) + 1.5
    src = torch.rand(S, dim, dtype=torch.float64, device="cuda", generator=gen)
    Ek = torch.randn(S, R, dtype=torch.complex128, device="cuda", generator=gen)
    got = E.propagate(kind, tg, src, 11.0, 1.0, Ek)
    rows = torch.arange(0, T, max(1, T // 7), device="cuda")   # a few detectors, the last block among them
    rows = torch.unique(torch.cat([rows, torch.tensor([T - 1], device="cuda")]))
    G = E.assemble_propagator(kind, tg[rows].contiguous(), src, 11.0)
    err = (got[rows] - G @ Ek).abs()
    # sums of S terms of random phase, in two orders: their roundings grow with the root of S at most
    bound = 4 * (S ** 0.5 + 8) * 2.0 ** -53 * (G.abs() @ Ek.abs())
    assert torch.all(err <= bound)
    assert torch.isfinite(torch.view_as_real(got)).all()
