"""Calls of the gradient processor that its native path leaves as they were (GPU tests)."""
import numpy as np
import pytest
import torch

from adfwi_gb300.gradient import GradProcessor

pytestmark = pytest.mark.gpu


def planes():
    rng = np.random.default_rng(2)
    return [torch.tensor(rng.random((30, 45)), dtype=torch.float32, device="cuda:0") for _ in range(2)]


def test_no_maximum_velocity_without_scaling():
    """Both sides do the same double-precision operations: a few units in the last place, 1e-13."""
    g, f = planes()
    p, q = (GradProcessor(grad_smooth=2, norm_grad=False) for _ in range(2))
    q._native = lambda *a: None
    out, ref = (r.forward(nx=45, nz=30, vmax=None, grad=g, forw=f) for r in (p, q))
    assert float((out - ref).abs().max()) <= 1e-13 * float(ref.abs().max())


def test_a_mask_with_a_gradient_keeps_it():
    g, f = planes()
    mask = torch.rand((30, 45), device="cuda:0").requires_grad_()
    GradProcessor(grad_mask=mask).forward(nx=45, nz=30, vmax=3000.0, grad=g, forw=f).sum().backward()
    assert float(mask.grad.abs().max()) > 0
