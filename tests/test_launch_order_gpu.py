"""Step kernels that read ahead of the launch before them (GPU tests).

Under a timed profile every launch lies between two recorded events and starts when all work before it
has completed. The same solve without the events has to give the same bits: what a step reads early is
not what the launch before it still writes, at the first step of a loop as well, where that launch
packs coefficients or restores a snapshot.
"""
import pytest
import torch

import adfwi_gb300 as A
from adfwi_gb300 import _native as N
from _cases import ELASTIC_KEYS, acoustic_problem, elastic_problem

pytestmark = pytest.mark.gpu


def ordered_and_not(solve, times=6):
    """The outputs of solve() with every launch ordered, and of `times` solves without."""
    N.profile_start(True)
    try:
        ref = solve()
        torch.cuda.synchronize()
    finally:
        N.profile_stop()
    return ref, [solve() for _ in range(times)]


@pytest.mark.parametrize("precision", ["native", "fp24", "fp16", "bf16"])
@pytest.mark.parametrize("abc_type,free_surface", [("PML", True), ("PML", False), ("gerjan", True)])
def test_elastic_segments_from_snapshots(precision, abc_type, free_surface):
    model, survey, prop = elastic_problem(A, nz=90, nx=150, ns=6, nt=60, abc_type=abc_type, free_surface=free_surface,
                                          seed=5, snapshot_every=3, snapshot_precision=precision)
    gen = torch.Generator().manual_seed(7)
    w = None

    def solve():
        nonlocal w
        for p in ("vp", "vs", "rho", "eps", "delta"):
            getattr(model, p).grad = None
        rec = prop.forward(fd_order=4)
        if w is None:
            w = {k: torch.randn(rec[k].shape, generator=gen).cuda() for k in ELASTIC_KEYS}
        sum((rec[k] * w[k]).sum() for k in ELASTIC_KEYS).backward()
        return [rec[k].detach() for k in rec] + [getattr(model, p).grad for p in ("vp", "vs", "rho", "eps", "delta")]

    ref, got = ordered_and_not(solve)
    for g in got:
        assert all(torch.equal(a, b) for a, b in zip(g, ref))


@pytest.mark.parametrize("every,grad", [(0, False), (0, True), (7, True)])
def test_acoustic_f64_from_its_coefficients(every, grad):
    """Without a gradient nothing lies between the coefficients' kernel and the first step."""
    model, survey, prop = acoustic_problem(A, nz=90, nx=150, ns=5, nt=40, dtype=torch.float64, seed=3, vp_grad=grad,
                                           rho_grad=grad, snapshot_every=every)
    maps = [model.vp.detach().clone(), model.vp.detach() * 1.05]  # other coefficients than the memory held before
    w = torch.randn((5, 40, 20), generator=torch.Generator().manual_seed(7), dtype=torch.float64).cuda()

    def solve():
        out = []
        for vp in maps:
            with torch.no_grad():
                model.vp.copy_(vp)
            model.vp.grad = model.rho.grad = None
            rec = prop.forward()
            out += [rec[k].detach() for k in rec]
            if grad:
                (rec["p"] * w).sum().backward()
                out += [model.vp.grad, model.rho.grad]
        return out

    ref, got = ordered_and_not(solve)
    for g in got:
        assert all(torch.equal(a, b) for a, b in zip(g, ref))
