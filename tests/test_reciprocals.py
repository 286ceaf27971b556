"""complex128 pivots at the ends of the range: an infinite part makes zero multipliers (as a
division by it does), the largest and smallest numbers their reciprocals."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _factor(p):
    from magreete_gb300 import engine as E
    A = torch.tensor([[p, 1.0], [0.0, 2.0]], dtype=torch.complex128)
    A[1, 0] = 1.0 if not math.isfinite(abs(p)) else p * 0.25
    f = E.lu_factor(A.cuda(), check_singular=False)
    return f.lu.cpu(), f.perm.cpu()


@pytest.mark.parametrize("p", [complex(math.inf, 0), complex(-math.inf, 3.0), complex(0, math.inf), complex(2.0, -math.inf)])
def test_infinite_pivot(p):
    lu, perm = _factor(p)
    assert perm.tolist() == [0, 1]
    assert lu[1, 0] == 0 and lu[1, 1] == 2


@pytest.mark.parametrize("p", [1e308, 1e308j, complex(3e307, -4e307), complex(1e-300, 1e-300), 5e-309, complex(1e154, 1e-154)])
def test_largest_and_smallest(p):
    lu, perm = _factor(complex(p))
    assert perm.tolist() == [0, 1]
    if abs(p) < 2.0 ** -1024:
        # its reciprocal is beyond the largest number: a multiplier is a product with it
        assert not math.isfinite(abs(lu[1, 0].item()))
        return
    assert abs(lu[1, 0].item() - 0.25) <= 2.0 ** -50
    assert abs(lu[1, 1].item() - 1.75) <= 2.0 ** -48
