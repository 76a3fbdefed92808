"""Grids with more rows or columns than 16 bits count, against the CPU oracle (GPU tests).

A few rows or columns of 33000 to 131100, with sources and receivers near the far end. Float64 records
stay within steps x 1e-14 < 1e-12 relative L2 and gradients within 1e-9, float32 records
within 1e-5 and gradients within 1e-4, as on small grids.
"""
import numpy as np
import pytest
import torch

import adfwi_gb300 as A
from _cases import ELASTIC_KEYS, acoustic_problem, elastic_problem, oracle_acoustic, oracle_elastic, rel

pytestmark = pytest.mark.gpu
TOL = {torch.float64: (1e-12, 1e-9), torch.float32: (1e-5, 1e-4)}
SHAPES = [(9, 65580), (32780, 9), (9, 131100)]


def survey_at_the_far_end(prop_survey, nz, nx, nt):
    """One source in the last rows and columns, receivers over the last ones and a few over all, two in a cell."""
    src = A.Source(nt=nt, dt=prop_survey.source.dt, f0=prop_survey.source.f0)
    src.add_sources(src_x=np.array([nx - 4]), src_z=np.array([nz - 5]),
                    src_wavelet=np.asarray(prop_survey.source.wavelet).reshape(-1, nt)[0])
    rcv = A.Receiver(nt=nt, dt=prop_survey.receiver.dt)
    z = np.concatenate([np.full(6, nz - 4), nz - 6 + np.arange(5), [nz - 4, nz // 2, 1]])
    x = np.concatenate([nx - 7 + np.arange(6), np.full(5, nx - 4), [nx - 4, nx // 2, 1]])
    rcv.add_receivers(rcv_x=x, rcv_z=z, rcv_type="pr")
    return A.Survey(src, rcv), len(x)


@pytest.mark.parametrize("nz,nx", SHAPES)
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_acoustic_long_grids(nz, nx, dtype):
    nt = 12
    model, survey, prop = acoustic_problem(A, nz=nz, nx=nx, nabc=3, nt=nt, ns=1, nr=3, dtype=dtype, f0=60.0)
    survey, nr = survey_at_the_far_end(survey, nz, nx, nt)
    prop = A.AcousticPropagator(model, survey, device="cuda:0", dtype=dtype)
    rec = prop.forward()
    ref, vp, rho = oracle_acoustic(prop, model)
    w = {k: torch.randn((1, nt, nr), generator=torch.Generator().manual_seed(3), dtype=dtype) for k in "puw"}
    for k in "puw":
        assert float(ref[k].detach()[:, :, :11].abs().max()) > 0
        assert rel(rec[k].detach(), ref[k].detach()) <= TOL[dtype][0], k
    sum((rec[k] * w[k].cuda()).sum() for k in "puw").backward()
    sum((ref[k] * w[k]).sum() for k in "puw").backward()
    for got, want in ((model.vp.grad, vp.grad), (model.rho.grad, rho.grad)):
        assert rel(got, want) <= TOL[dtype][1]


@pytest.mark.parametrize("nz,nx", SHAPES[:2])
@pytest.mark.parametrize("abc_type,free_surface", [("PML", True), ("gerjan", False)])
def test_elastic_long_grids(nz, nx, abc_type, free_surface):
    nt = 8
    kw = dict(nabc=4, nt=nt, ns=1, nr=3, dtype=torch.float64, abc_type=abc_type, free_surface=free_surface)
    model, survey, prop = elastic_problem(A, nz=nz, nx=nx, **kw)
    survey, nr = survey_at_the_far_end(survey, nz, nx, nt)
    prop = A.ElasticPropagator(model, survey, device="cuda:0", dtype=torch.float64)
    rec = prop.forward(fd_order=4)
    ref, pars = oracle_elastic(prop, model, fd_order=4)
    w = {k: torch.randn((1, nt, nr), generator=torch.Generator().manual_seed(3), dtype=torch.float64) for k in ELASTIC_KEYS}
    for k in ELASTIC_KEYS:
        assert float(ref[k].detach()[:, :, :11].abs().max()) > 0
        assert rel(rec[k].detach(), ref[k].detach()) <= 1e-12, k
    sum((rec[k] * w[k].cuda()).sum() for k in ELASTIC_KEYS).backward()
    sum((ref[k] * w[k]).sum() for k in ELASTIC_KEYS).backward()
    for p in ("vp", "vs", "rho", "eps", "delta"):
        assert rel(getattr(model, p).grad, pars[p].grad) <= 1e-9, p
