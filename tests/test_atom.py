"""Atom positions as the host tables take them."""
import numpy as np
import pytest
import torch

from pyquante_b200.Atom import Atom


@pytest.mark.parametrize("r", [
    np.array([1.0, 2.5, -3.0]), np.array([1.0, 2.5, -3.0], dtype=np.float32), [1, 2.5, -3],
    np.array([1.0, 2.5, -3.0], dtype=object), torch.tensor([1.0, 2.5, -3.0], dtype=torch.float64),
    torch.tensor([1.0, 2.5, -3.0], dtype=torch.float64, requires_grad=True),
])
def test_pos_of_any_three_numbers(r):
    a = Atom(8, 0.0, 0.0, 0.0)
    a.r = r
    p = a.pos()
    assert p == (1.0, 2.5, -3.0) and all(type(c) is float for c in p)
