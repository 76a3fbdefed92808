"""Which planes the padding follows with a graph, and which tensors kernels take by address (CPU tests)."""
import pytest
import torch
from torch.autograd import forward_ad

from adfwi_gb300 import _native as N
from adfwi_gb300.propagator import _fold_torch, _pad_planes, fold_replicate


@pytest.mark.parametrize("need", [(False, False), (True, False), (False, True), (True, True)])
def test_padded_planes_need_gradients_as_their_inputs_do(need):
    vs = [torch.randn(4, 5, dtype=torch.float64).requires_grad_(n) for n in need]
    outs = _pad_planes(vs, 2, 1, 3, 2)
    assert tuple(o.requires_grad for o in outs) == need
    if any(need):
        gs = [torch.randn_like(o) for o in outs]
        torch.autograd.backward([o for o in outs if o.requires_grad], [g for g, n in zip(gs, need) if n])
        for v, g, n in zip(vs, gs, need):
            assert torch.equal(v.grad, _fold_torch(g, 2, 1, 3, 2)) if n else v.grad is None


def test_kernels_take_only_tensors_with_memory_of_their_own():
    x = torch.randn(3, 4)
    assert N.by_address(x) and N.by_address(x.t()) and N.by_address(torch.nn.Parameter(x))
    seen = []
    torch.func.vmap(lambda a: (seen.append(N.by_address(a)), a * 1)[1])(torch.randn(2, 3, 4))
    torch.func.grad(lambda a: (seen.append(N.by_address(a)), a.sum())[1])(x)
    with forward_ad.dual_level():
        seen.append(N.by_address(forward_ad.make_dual(x, x)))
    seen.append(N.by_address(torch._neg_view(x)))
    assert not any(seen) and len(seen) == 4


def test_fold_of_batched_planes():
    g = torch.randn(3, 8, 9, dtype=torch.float64)
    out = torch.func.vmap(lambda a: fold_replicate(a, 2, 1, 3, 2))(g)
    assert torch.equal(out, torch.stack([fold_replicate(a, 2, 1, 3, 2) for a in g]))
