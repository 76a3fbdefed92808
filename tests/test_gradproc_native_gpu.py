"""The gradient processor's native path against the device operations it replaces (GPU tests), over
the forms it accepts. Both sides do the same double-precision operations in the same order except
that PyTorch rounds w x + a once where the compiler fuses it alike, so they agree within a few units
in the last place: 1e-13 of the largest value.
"""
import numpy as np
import pytest
import torch

from adfwi_gb300.gradient import GradProcessor

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nz,nx,mute,smooth,mol,mask,norm,dtype,special", [
    (2, 2, 0, 0, "land", False, True, torch.float32, None),
    (7, 300, 2, 1, "marine", False, True, torch.float64, None),
    (33, 257, 5, 4, "Marine", True, True, torch.float32, None),
    (64, 50, 10, 0, "offshore", False, False, torch.float32, None),
    (90, 121, 12, 7, "Land", True, True, torch.float64, "strided"),
    (41, 43, 3, 3, "marine", False, True, torch.float32, "nan"),
    (41, 43, 0, 3, "land", False, True, torch.float32, "zero"),
])
def test_native_processor_matches_device_operations(nz, nx, mute, smooth, mol, mask, norm, dtype, special):
    rng = np.random.default_rng(nz + nx)
    g = torch.tensor(rng.standard_normal((nz, nx)), dtype=torch.float32, device="cuda:0")
    f = torch.tensor(rng.random((nz, nx)) ** 4, dtype=dtype, device="cuda:0")
    if special == "strided":
        g, f = g.t().contiguous().t(), f.t().contiguous().t()
    if special == "nan":
        g[nz // 2, nx // 2] = float("nan")
    if special == "zero":
        g.zero_()
    m = rng.random((nz, nx)) if mask else None
    make = lambda: GradProcessor(grad_mute=mute, grad_smooth=smooth, grad_mask=m, norm_grad=norm, marine_or_land=mol)  # noqa: E731
    p = make()
    out = p.forward(nx=nx, nz=nz, vmax=3000.0, grad=g, forw=f)
    q = make()
    q._native = lambda *a: None
    ref = q.forward(nx=nx, nz=nz, vmax=3000.0, grad=g, forw=f)
    assert out.dtype == ref.dtype and out.shape == ref.shape
    assert torch.equal(out.isnan(), ref.isnan())
    out, ref = torch.nan_to_num(out), torch.nan_to_num(ref)
    assert float((out - ref).abs().max()) <= 1e-13 * float(ref.abs().max())


def test_wide_spans_read_rows_in_place():
    """A span whose row part exceeds the shared memory of a block: a plane of 4 rows, span 3000."""
    from adfwi_gb300.gradient import smooth2d
    rng = np.random.default_rng(1)
    z = rng.standard_normal((4, 6200))
    span = 3000
    out = smooth2d(torch.tensor(z, device="cuda:0"), span).cpu().numpy()
    x = np.arange(-2.0 * span, 2.0 * span + 1, 2.0) / span
    w = np.exp(-0.5 * x * x)
    w /= w.sum()
    conv = lambda a: np.stack([np.convolve(r, w)[span:span + a.shape[1]] for r in a])  # noqa: E731
    full = lambda a: conv(conv(a).T).T  # noqa: E731
    ref = full(z) / full(np.ones_like(z))
    # two passes of at most 6001 terms: 6001 x 2^-53 each, twice for the normaliser, both sides
    assert np.max(np.abs(out - ref)) <= 8 * 6001 * 2.0 ** -53 * np.max(full(np.abs(z)) / full(np.ones_like(z)))
