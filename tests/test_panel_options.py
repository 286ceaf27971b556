"""Panel options of the complex128 LU: rows per CTA below, at and above what the register
panel holds, and plain launches in flight beside each other (whose CTAs must all
find an SM: the count that panel_rows and panel_max_ctas say)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _matrix(n, seed):
    return torch.randn(n, n, dtype=torch.complex128, generator=torch.Generator().manual_seed(seed)).cuda()


@pytest.mark.parametrize("n", [700, 1500])
@pytest.mark.parametrize("options", [dict(panel_rows=64), dict(panel_rows=128), dict(panel_rows=129),
                                     dict(panel_rows=400), dict(panel_rows=48, panel_max_ctas=9),
                                     dict(cooperative=0), dict(cooperative=0, panel_max_ctas=12),
                                     dict(cooperative=0, panel_rows=100)])
def test_same_factors(n, options):
    from magreete_gb300 import _lib as L
    from magreete_gb300 import engine as E
    A = _matrix(n, n)
    ref = E.lu_factor(A.clone())
    f = E.lu_factor(A.clone(), options=L.LuOptions(**options))
    assert torch.equal(f.perm, ref.perm)
    assert torch.equal(f.lu, ref.lu)


def test_plain_launches_side_by_side():
    """Eight factorisations of eight panel CTAs each, on eight streams."""
    from magreete_gb300 import _lib as L
    from magreete_gb300 import engine as E
    mats = [_matrix(2000, i) for i in range(8)]
    ref = [E.lu_factor(A.clone()) for A in mats]
    streams = [torch.cuda.Stream() for _ in mats]
    for _ in range(3):
        out = []
        torch.cuda.synchronize()
        for A, s in zip(mats, streams):
            with torch.cuda.stream(s):
                out.append(E.lu_factor(A.clone(), check_singular=False, options=L.LuOptions(cooperative=0)))
        torch.cuda.synchronize()
        for f, r in zip(out, ref):
            assert E.lu_info(f) == (0, 0)
            assert torch.equal(f.perm, r.perm) and torch.equal(f.lu, r.lu)
