"""Double-precision gradients of w-records are the same bits on every run, also where two receiver cells of a
column meet on one row: dL/dw of the mirrored row above a free surface goes to the row below it (GPU test).
"""
import numpy as np
import pytest
import torch

import adfwi_gb300 as A
from _cases import acoustic_problem, oracle_acoustic, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,order", [(40, 1), (333, -1)])
def test_records_that_meet_on_the_surface_row(nx, order):
    nt, ns = 60, 3
    model, survey, prop = acoustic_problem(A, nz=17, nx=nx, nabc=6, nt=nt, ns=ns, nr=3, free_surface=True,
                                           dtype=torch.float64, seed=4, src_z=1)
    rcv = A.Receiver(nt=nt, dt=survey.receiver.dt)
    rcv.add_receivers(rcv_x=np.tile(np.arange(nx), 2)[::order], rcv_z=np.repeat([-1, 0], nx)[::order], rcv_type="pr")
    prop = A.AcousticPropagator(model, A.Survey(survey.source, rcv), device="cuda:0", dtype=torch.float64)
    w = torch.randn((ns, nt, 2 * nx), generator=torch.Generator().manual_seed(3), dtype=torch.float64)
    grads = []
    for _ in range(20):
        model.vp.grad = model.rho.grad = None
        (prop.forward()["w"] * w.cuda()).sum().backward()
        grads.append((model.vp.grad.clone(), model.rho.grad.clone()))
    assert all(torch.equal(a, b) for g in grads[1:] for a, b in zip(g, grads[0]))
    ref, vp, rho = oracle_acoustic(prop, model)
    (ref["w"] * w).sum().backward()
    for got, want in zip(grads[0], (vp.grad, rho.grad)):  # as in test_acoustic_f64_gpu: sums of products of two fields
        assert rel(got, want) <= 1e-9
