"""Gradients of records on the mirrored row above a free surface, against the CPU oracle (GPU tests).

w[fs-1] = w[fs] closes a step, so what dL/dw asks of row fs-1 belongs to row fs before the step is
reversed, in the last step as in all others: solves of one step and of few show the last one. Float64
gradients stay within 1e-9, float32 within 1e-4 relative L2, as on other rows.
"""
import numpy as np
import pytest
import torch

import adfwi_gb300 as A
from adfwi_gb300.acoustic import BOUNDARY_SAVING
from _cases import acoustic_problem, oracle_acoustic, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,tol", [(torch.float64, 1e-9), (torch.float32, 1e-4)])
@pytest.mark.parametrize("nt,rows,fields,kw", [
    (30, (-1,), "w", {}),
    (60, (-1, 0), "w", {"snapshot_every": 13}),
    (41, (0, -1), "puw", {"snapshot_every": BOUNDARY_SAVING}),
    (30, (-1,), "pu", {}),
])
def test_gradients_of_the_mirrored_row(dtype, tol, nt, rows, fields, kw):
    nx, ns = 37, 2
    model, survey, prop = acoustic_problem(A, nz=17, nx=nx, nabc=6, nt=nt, ns=ns, nr=3, free_surface=True, dtype=dtype,
                                           seed=nt, src_z=1, f0=40.0)
    rcv = A.Receiver(nt=nt, dt=survey.receiver.dt)
    rcv.add_receivers(rcv_x=np.tile(np.arange(nx), len(rows)), rcv_z=np.repeat(rows, nx), rcv_type="pr")
    prop = A.AcousticPropagator(model, A.Survey(survey.source, rcv), device="cuda:0", dtype=dtype, **kw)
    rec = prop.forward()
    ref, vp, rho = oracle_acoustic(prop, model)
    gen = torch.Generator().manual_seed(3)
    w = {k: torch.randn(rec[k].shape, generator=gen, dtype=dtype) for k in fields}
    sum((rec[k] * w[k].cuda()).sum() for k in fields).backward()
    sum((ref[k] * w[k]).sum() for k in fields).backward()
    for got, want in ((model.vp.grad, vp.grad), (model.rho.grad, rho.grad)):
        assert float(want.norm()) > 0 and rel(got, want) <= tol
