"""The plain method's propagation where one scale per 64 sources does not serve:
a field with large entries beside ordinary ones, weak fields at scatterers
that a detector almost touches, rows of the fields that differ in shape.  Every
column of the result is held to what FP64 sums of its own terms guarantee."""
import pytest
import torch

pytestmark = pytest.mark.gpu

T, S, R = 400, 700, 64


@pytest.mark.parametrize("fields", ["large entries in one", "weak beside detectors", "other shapes"])
def test_columns_of_the_result(fields):
    from magreete_gb300 import engine as E
    gen = torch.Generator().manual_seed(3)
    src = torch.rand(S, 3, dtype=torch.float64, generator=gen)
    tg = torch.rand(T, 3, dtype=torch.float64, generator=gen) + 1.5
    Ek = torch.randn(S, 3, R, dtype=torch.complex128, generator=gen)
    if fields == "large entries in one":
        Ek[::7, :, 3] *= 1e10
    elif fields == "weak beside detectors":
        tg[:70] = src[::10] + 1e-3 * torch.randn(70, 3, dtype=torch.float64, generator=gen)
        Ek[::10] *= 1e-8
    else:
        Ek[::5, :, :25] *= 1e10
    Ek = Ek.reshape(3 * S, R).cuda()
    tg, src = tg.cuda(), src.cuda()
    G = E.assemble_propagator("3d_vector", tg, src, 11.0)
    got = E.propagate("3d_vector", tg, src, 11.0, 1.0, Ek)
    err = torch.linalg.norm(got - G @ Ek, dim=0)
    # 3 S terms, each of four real products, here and in the reference: (K + 8) 2^-53 of |G| |Ek| each
    bound = 4 * (3 * S + 8) * 2.0 ** -53 * torch.linalg.norm(G.abs() @ Ek.abs(), dim=0)
    assert torch.all(err <= bound), (err / bound).max()
