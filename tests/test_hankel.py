"""The table-based Hankel functions of the 2D Green's functions (csrc/hankel.cuh)
against scipy, at and around the table's edges, its interval boundaries and the
argument ranges served by other code."""
import numpy as np
import pytest
import scipy.special as sps
import torch

pytestmark = pytest.mark.gpu

_edges = [3.0, 25.0, 100.0, 512.0]
ARGS = np.unique(np.concatenate(
    [[1e-6, 1e-3, 0.1, 1.0, 2.9, 2.9999999]] +
    [[np.nextafter(e, 0), e, np.nextafter(e, 1e9), e + 0.125, e + 0.0625] for e in _edges] +
    [np.linspace(3.0, 40.0, 1501), np.linspace(40.0, 511.9, 997), np.geomspace(512.0, 5000.0, 101)]))


@pytest.mark.parametrize("kind", ["2d_scalar", "2d_vector"])
def test_greens_blocks_match_scipy(kind):
    """k0 = 1 and separations along x, so that kR is the argument itself: the TM
    value is (i/4) H0, the TE block diag((i/4) H1 / x, (i/4) (H0 - H1 / x)).
    Within 2e-15 of the amplitude for the functions here plus two roundings of
    the phase (x 2^-52) for scipy's, and a few ulp of the singular terms."""
    from magreete_gb300 import engine as E
    x = ARGS
    pts = torch.from_numpy(np.stack([x, np.zeros_like(x)], 1)).cuda()
    origin = torch.zeros(1, 2, dtype=torch.float64, device="cuda")
    G = E.assemble_propagator(kind, pts, origin, 1.0).cpu().numpy()
    h0, h1 = sps.hankel1(0, x), sps.hankel1(1, x)
    amp = np.sqrt(2 / (np.pi * x))
    tol = 0.25 * ((2e-15 + x * 2.0 ** -52) * amp + 8 * 2.0 ** -52 * (np.abs(h0) + np.abs(h1) / x))
    if kind == "2d_scalar":
        assert np.all(np.abs(G[:, 0] - 0.25j * h0) <= tol)
        return
    G = G.reshape(-1, 2, 2)
    assert np.all(np.abs(G[:, 0, 0] - 0.25j * h1 / x) <= tol)
    assert np.all(np.abs(G[:, 1, 1] - 0.25j * (h0 - h1 / x)) <= 2 * tol)
    assert np.all(G[:, 0, 1] == 0) and np.all(G[:, 1, 0] == 0)
