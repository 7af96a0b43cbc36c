"""autodiff's x + c k takes every plain number a time step can be, and tensors."""
import numpy as np
import pytest
import torch

from openonda_b200.autodiff import _axpy


@pytest.mark.parametrize("c", [0.25, 1, 0, -2, True, False, np.float64(0.5), np.float32(0.5),
                               np.int64(3), torch.tensor(0.5, dtype=torch.float64)])
def test_axpy(c):
    x = torch.tensor([[1.0, -2.0, 4.0]], dtype=torch.float64, requires_grad=True)
    k = torch.tensor([[0.5, 8.0, -1.0]], dtype=torch.float64, requires_grad=True)
    y = _axpy(x, k, c)
    assert y.dtype == torch.float64 and torch.equal(y, x + float(c) * k)
    y.sum().backward()
    assert torch.equal(x.grad, torch.ones_like(x))
    assert torch.equal(k.grad, torch.full_like(k, float(c)))
