"""The passes of the tile-pivoting LU at the edges of their tiles: orders around
the 64-row tiles and 128-wide blocks, both schedules (in order, overlapped), and
symmetric factorisations, which update the upper half of the trailing matrix
while its order is at least 4096 and mirror the rest from there.

Bound: P A = L U to 5e-8 n of ||A||, times the growth of U beyond A where there
is any: an FP32 LU's backward error, as for the other tile-pivoting tests."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _check(A, f):
    from magreete_gb300 import engine as E
    n = A.shape[0]
    assert E.lu_info(f) == (0, 0)
    perm, idx = f.perm.long(), torch.arange(n, device="cuda")
    assert torch.equal(perm // 64, idx // 64)
    assert torch.equal(torch.sort(perm).values, idx)
    LU = f.lu.to(torch.complex128)
    U = torch.triu(LU)
    Lm = torch.tril(LU, -1) + torch.eye(n, dtype=LU.dtype, device="cuda")
    Ad = A.to(torch.complex128)
    growth = max(1.0, (U.abs().max() / Ad.abs().max()).item())
    err = (torch.linalg.norm(Lm @ U - Ad[perm]) / torch.linalg.norm(Ad)).item()
    assert err < 5e-8 * n * growth, (err, growth)


def _matrix(n, symmetric):
    gen = torch.Generator(device="cuda").manual_seed(n)
    A = torch.randn(n, n, dtype=torch.complex64, device="cuda", generator=gen)
    if symmetric:
        A = A + A.T
    # a diagonal of the rows' size: pivots move within the tiles, no growth without bound
    return A + 1.5 * n ** 0.5 * torch.eye(n, device="cuda")


def _factor(A, pad, **options):
    from magreete_gb300 import _lib as L
    from magreete_gb300 import engine as E
    W = torch.full((A.shape[0], A.shape[0] + pad), float("nan"), dtype=torch.complex64, device="cuda")[:, :A.shape[0]]
    W.copy_(A)
    return E.lu_factor(W, check_singular=False, options=L.LuOptions(pivoting=L.MGT_PIVOT_TILE, **options))


@pytest.mark.parametrize("lookahead", [0, 1])
@pytest.mark.parametrize("n,pad", [(64, 0), (65, 1), (128, 0), (191, 1), (192, 2), (256, 0), (257, 1), (258, 0),
                                   (300, 4), (320, 0), (384, 0), (385, 1), (450, 2), (641, 1)])
def test_tile_lu_edges(n, pad, lookahead):
    A = _matrix(n, False)
    _check(A, _factor(A, pad, lookahead=lookahead))


@pytest.mark.parametrize("wide_min", [0, 1024])
@pytest.mark.parametrize("lookahead", [0, 1])
@pytest.mark.parametrize("n,pad", [(4096, 0), (4224, 0), (4353, 1), (4608, 2), (4710, 0)])
def test_symmetric_tile_lu(n, pad, lookahead, wide_min):
    """wide_min 1024: paired blocks (K = 256 updates) at these orders too."""
    from magreete_gb300 import _lib as L
    lib = L.load()
    A = _matrix(n, True)
    before = lib.mgt_get_tuning(L.MGT_TUNE_WIDE_UPDATE)
    try:
        L.check(lib.mgt_set_tuning(L.MGT_TUNE_WIDE_UPDATE, wide_min))
        f = _factor(A, pad, lookahead=lookahead, symmetric=1)
    finally:
        lib.mgt_set_tuning(L.MGT_TUNE_WIDE_UPDATE, before)
    _check(A, f)


def test_options_without_symmetric():
    """An options structure of the size before `symmetric` is taken as before."""
    from magreete_gb300 import _lib as L
    from magreete_gb300 import engine as E
    A = _matrix(300, False)
    opt = L.LuOptions(pivoting=L.MGT_PIVOT_TILE, symmetric=1)
    opt.size = L.LuOptions.symmetric.offset
    _check(A, E.lu_factor(A.clone(), check_singular=False, options=opt))
    opt.size = L.LuOptions.symmetric.offset - 4
    with pytest.raises(L.MagreeteError):
        E.lu_factor(A.clone(), options=opt)
