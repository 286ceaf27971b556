"""The plain method's propagation on the tensor cores (csrc/propagate.cu): the
assembled, digit-split contraction against a dense FP64 product, at sizes on
both sides of the rule that selects it, off the 128-row and 32-column tiles, with
coincident and regularised detectors and non-finite fields."""
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _points(kind, n, seed):
    dim = 2 if kind.startswith("2d") else 3
    return torch.rand(n, dim, dtype=torch.float64, generator=torch.Generator().manual_seed(seed)).cuda()


@pytest.mark.parametrize("kind", O.KINDS)
@pytest.mark.parametrize("T,S,R", [(1, 1, 1), (20, 33, 3), (127, 400, 33), (400, 700, 64), (1025, 350, 5),
                                   (300, 1100, 100)])
def test_matches_dense_product(kind, T, S, R):
    from magreete_gb300 import engine as E
    d = E.KIND_DIMS[kind][1]
    gen = torch.Generator().manual_seed(T + S + R)
    tg, src = _points(kind, T, 1) + 1.5, _points(kind, S, 2)
    Ek = torch.randn(d * S, R, dtype=torch.complex128, generator=gen).cuda()
    E0 = torch.randn(d * T, R, dtype=torch.complex128, generator=gen).cuda()
    coef = 0.3 - 0.2j
    G = E.assemble_propagator(kind, tg, src, 11.0)
    ref = coef * (G @ Ek)
    got = E.propagate(kind, tg, src, 11.0, coef, Ek, E0)
    # a product of K = d S terms, each with its own roundings: (K + 8) 2^-53 of |coef G| |Ek|, and E0's rounding
    bound = 4 * (d * S + 8) * 2.0 ** -53 * abs(coef) * (G.abs() @ Ek.abs()) + 2.0 ** -52 * (E0.abs() + ref.abs())
    assert torch.all((got - (ref + E0)).abs() <= bound)
    assert torch.all((E.propagate(kind, tg, src, 11.0, coef, Ek) - ref).abs() <= bound)


@pytest.mark.parametrize("T,S,R", [(20, 33, 3), (400, 700, 64)])
def test_coincident_points_and_nonfinite_fields(T, S, R):
    """NaN where the reference's G is NaN (a detector on a scatterer, or within
    the radius when regularising), and in every column whose fields hold a NaN."""
    from magreete_gb300 import engine as E
    src = _points("2d_scalar", S, 4)
    tg = _points("2d_scalar", T, 5) + 2.0
    tg[7] = src[3]
    tg[9] = src[5] + 1e-4
    gen = torch.Generator().manual_seed(6)
    Ek = torch.randn(S, R, dtype=torch.complex128, generator=gen).cuda()
    out = E.propagate("2d_scalar", tg, src, 9.0, 1.0, Ek)
    bad = torch.isnan(torch.view_as_real(out)).all(-1)
    assert bad[7].all() and bad.sum().item() == R
    out = E.propagate("2d_scalar", tg, src, 9.0, 1.0, Ek, regularize=True, radius=1e-3)
    bad = torch.isnan(torch.view_as_real(out)).all(-1)
    assert bad[7].all() and bad[9].all() and bad.sum().item() == 2 * R
    Ek[11, 1] = float("nan")
    out = E.propagate("2d_scalar", tg, src, 9.0, 1.0, Ek)
    bad = torch.isnan(torch.view_as_real(out)).all(-1)
    assert bad[:, 1].all() and not bad[0, 0] and not bad[0, 2]


@pytest.mark.parametrize("scale", [1e-200, 1e200])
def test_extreme_scales(scale):
    """Fields near the ends of the FP64 range keep their relative accuracy."""
    from magreete_gb300 import engine as E
    tg, src = _points("3d_scalar", 400, 7) + 1.5, _points("3d_scalar", 600, 8)
    Ek = torch.randn(600, 64, dtype=torch.complex128, generator=torch.Generator().manual_seed(9)).cuda()
    a = E.propagate("3d_scalar", tg, src, 5.0, 1.0, Ek)
    b = E.propagate("3d_scalar", tg, src, 5.0, 1.0, Ek * scale) / scale
    assert (torch.linalg.norm(a - b) / torch.linalg.norm(a)).item() < 1e-13
