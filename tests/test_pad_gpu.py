"""Padding of model planes and its adjoint in the CUDA library against PyTorch's (GPU tests).

Padding copies, so it is exact. A folded cell is a double-precision sum, rounded once to single:
it differs from the double-precision reference by at most 2^-24 of the sum of magnitudes (2^-23
allows for both roundings); in double precision both sides sum at most n values, n 2^-53 each.
"""
import pytest
import torch

from adfwi_gb300.propagator import _fold_planes, _fold_torch, _pad_planes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("shapes,pads", [
    ([(1, 1)], (2, 3, 4, 5)),
    ([(1, 7), (5, 1), (2, 2)], (3, 0, 0, 2)),
    ([(9, 31)], (0, 0, 0, 0)),
    ([(40, 57)] * 12, (2, 25, 25, 25)),
    ([(33, 258), (33, 257), (32, 258), (31, 256)], (50, 50, 50, 50)),
])
def test_pad_and_fold_match_torch(shapes, pads, dtype):
    top, bottom, left, right = pads
    gen = torch.Generator(device="cuda:0").manual_seed(5)
    vs = [torch.randn(s, device="cuda:0", dtype=dtype, generator=gen) for s in shapes]
    if len(vs) == 1:
        vs = [vs[0].t().contiguous().t()]  # strides other than the dense ones
    vs = [v.requires_grad_(k != 1) for k, v in enumerate(vs)]
    outs = _pad_planes(vs, *pads)
    for v, o in zip(vs, outs):
        ref = torch.nn.functional.pad(v[None, None], (left, right, top, bottom), mode="replicate")[0, 0]
        assert torch.equal(o, ref)
    gs = [torch.randn(o.shape, device="cuda:0", dtype=dtype, generator=gen) for o in outs]
    n = max(o.numel() for o in outs)
    eps = 2.0 ** -23 if dtype == torch.float32 else n * 2.0 ** -52
    for g, f in zip(gs, _fold_planes(gs, *pads)):
        bound = eps * _fold_torch(g.double().abs(), *pads)
        assert bool(((f.double() - _fold_torch(g.double(), *pads)).abs() <= bound).all())
    # through autograd, one output unused
    used = [k for k in range(len(outs)) if k != 2]
    torch.autograd.backward([outs[k] for k in used if vs[k].requires_grad], [gs[k] for k in used if vs[k].requires_grad])
    for k, v in enumerate(vs):
        if k == 2 or not v.requires_grad:
            assert v.grad is None
        else:
            assert torch.equal(v.grad, _fold_planes([gs[k]], *pads)[0])
