"""Double-precision acoustic step kernels at the edges of their launches, against the CPU oracle (GPU
tests): partial tiles, several shots per group, more receivers than a block of threads, several in
a cell, receivers on the mirrored row above a free surface, one step, recomputed segments and
boundary saving, and dL/d records of p alone or of p, u and w.

Both sides round every operation of a step a few times in 64 bits, so records stay within steps x 1e-14
< 1e-12 relative L2 and gradients, sums of products of two such fields, within 1e-9.
"""
import numpy as np
import pytest
import torch

import adfwi_gb300 as A
from adfwi_gb300.acoustic import BOUNDARY_SAVING
from _cases import acoustic_problem, oracle_acoustic, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nt,ns,nz,nx,nabc,fs,nr,row,fields,kw", [
    (1, 1, 9, 11, 3, False, 4, 1, "p", {}),
    (2, 2, 12, 21, 4, True, 300, -1, "p", {}),
    (60, 3, 15, 22, 5, False, 300, 2, "puw", {}),
    (60, 3, 17, 33, 6, True, 130, 0, "puw", {"snapshot_every": 13}),
    (60, 5, 21, 40, 8, True, 40, -1, "p", {"shots_per_block": 2}),
    (60, 2, 24, 31, 9, False, 20, 3, "p", {"snapshot_every": BOUNDARY_SAVING}),
])
def test_f64_steps_match_oracle_at_the_edges(nt, ns, nz, nx, nabc, fs, nr, row, fields, kw):
    model, survey, prop = acoustic_problem(A, nz=nz, nx=nx, nabc=nabc, nt=nt, ns=ns, nr=nr, free_surface=fs,
                                           dtype=torch.float64, seed=nt + ns, rcv_z=row, src_z=1, **kw)
    rcv = A.Receiver(nt=nt, dt=survey.receiver.dt)
    rcv.add_receivers(rcv_x=(np.arange(nr) * 5) % (nx - 1), rcv_z=np.full(nr, row), rcv_type="pr")
    prop = A.AcousticPropagator(model, A.Survey(survey.source, rcv), device="cuda:0", dtype=torch.float64, **kw)
    rec = prop.forward()
    ref, vp, rho = oracle_acoustic(prop, model)
    for k in "puw":
        a, b = rec[k].detach().cpu(), ref[k].detach()
        assert float((a - b).norm()) <= 1e-12 * float(b.norm()), k
    gen = torch.Generator().manual_seed(3)
    w = {k: torch.randn(rec[k].shape, generator=gen, dtype=torch.float64) for k in fields}
    sum((rec[k] * w[k].cuda()).sum() for k in fields).backward()
    sum((ref[k] * w[k]).sum() for k in fields).backward()
    if float(vp.grad.norm()) > 0:
        assert rel(model.vp.grad, vp.grad) <= 1e-9
    if float(rho.grad.norm()) > 0:
        assert rel(model.rho.grad, rho.grad) <= 1e-9
