"""Elastic step kernels at the edges of their launches, against the CPU oracle (GPU tests).

Receivers on the rows above the free surface (whose velocities the next stress update forms from
the rows below), more receivers than one block of threads, more receiver cells in one tile of the
reverse kernels than a block has threads, an odd number of shots, one and two
steps (the velocity records of the last step are taken after it), grids of a partial tile, and
recomputed segments. In float64 the two sides round differently a few times per step and cell, so
records stay within steps x 1e-14 < 1e-12 relative L2, and gradients, which sum products of two
such fields, within 1e-9.
"""
import numpy as np
import pytest
import torch

import adfwi_gb300 as A
from _cases import ELASTIC_KEYS, elastic_problem, oracle_elastic

pytestmark = pytest.mark.gpu


def close(a, b, tol):
    a, b = a.detach().cpu().double(), b.detach().cpu().double()
    return bool((a - b).norm() <= tol * b.norm())


@pytest.mark.parametrize("nt,ns,nr,nz,nx,fd_order,abc_type,free_surface,every", [
    (1, 1, 5, 12, 20, 4, "PML", True, 0),
    (2, 3, 300, 17, 33, 6, "PML", True, 0),
    (45, 3, 300, 21, 30, 4, "PML", True, 0),
    (45, 2, 40, 24, 41, 6, "PML", True, 11),
    (45, 3, 256, 16, 25, 4, "PML", False, 0),
    (45, 2, 600, 21, 30, 6, "PML", True, 0),
    (1, 2, 5, 12, 20, 4, "gerjan", False, 0),
    (45, 3, 300, 21, 30, 6, "gerjan", False, 0),
    (45, 2, 40, 24, 41, 4, "gerjan", True, 11),
    (45, 3, 257, 19, 30, 6, "sincos", True, 0),
])
def test_steps_match_oracle_at_the_edges(nt, ns, nr, nz, nx, fd_order, abc_type, free_surface, every):
    model, survey, prop = elastic_problem(A, nz=nz, nx=nx, nt=nt, ns=ns, nr=nr, fd_order=fd_order, abc_type=abc_type,
                                          free_surface=free_surface, dtype=torch.float64, seed=nt + nr,
                                          mt=[[1.0, 0.0, 0.4], [0.0, 1.0, 0.0], [0.4, 0.0, 0.6]], snapshot_every=every)
    # receivers on every row from two above the model to its last
    rcv_x = (np.arange(nr) * 7) % nx
    rcv_z = -2 + (np.arange(nr) * 3) % (nz + 2)
    rcv = A.Receiver(nt=nt, dt=survey.receiver.dt)
    rcv.add_receivers(rcv_x=rcv_x, rcv_z=rcv_z, rcv_type="pr")
    prop = A.ElasticPropagator(model, A.Survey(survey.source, rcv), device="cuda:0", dtype=torch.float64,
                               snapshot_every=every)
    rec = prop.forward(fd_order=fd_order)
    ref, pars = oracle_elastic(prop, model, fd_order=fd_order)
    for k in rec:
        assert close(rec[k], ref[k], 1e-12), k
    gen = torch.Generator().manual_seed(7)
    w = {k: torch.randn(rec[k].shape, generator=gen, dtype=torch.float64) for k in ELASTIC_KEYS}
    sum((rec[k] * w[k].cuda()).sum() for k in ELASTIC_KEYS).backward()
    sum((ref[k] * w[k]).sum() for k in ELASTIC_KEYS).backward()
    for p in ("vp", "vs", "rho", "eps", "delta"):
        assert close(getattr(model, p).grad, pars[p].grad, 1e-9), p
