"""The resident time loop (csrc/acoustic_res.cuh) against the per-step kernels: records bit for bit
and gradients within the rounding of their sums, at the edges of its strips and thread rows.

The per-step kernels are reached through the calls that still take them: a boundary-saving plan's
record solve, and an adjoint that is given dL/d u-records (zeroes).
"""
import numpy as np
import pytest
import torch

import adfwi_gb300 as A
from adfwi_gb300 import _native as N
from adfwi_gb300.acoustic import BOUNDARY_SAVING, AcousticPlan

pytestmark = pytest.mark.gpu

NT = 90
# a gradient is a sum over NT steps: its terms' roundings add up to at most NT eps of the sum's norm
# in either order, and the two orders differ by at most twice that
TOL = 2 * NT * 2.0 ** -24 * 2

# (nz, nx, nabc, shots, free surface, receivers): one block; the smallest strips; strips and thread
# rows of unequal height; every remainder of the columns by four; a cluster; strips that exchange
# rows through global memory; more shots than are resident at a time; one thread row per strip
SHAPES = [
    (4, 5, 2, 1, False, "row"),
    (11, 9, 3, 2, True, "row"),
    (30, 40, 10, 2, False, "row"),
    (37, 58, 9, 3, True, "column"),
    (41, 83, 12, 5, False, "shared"),
    (88, 201, 30, 12, True, "row"),
    (100, 102, 50, 10, False, "column"),
    (120, 420, 40, 9, False, "row"),
    (200, 600, 50, 6, False, "row"),
    (200, 600, 50, 7, True, "shared"),
    (60, 1500, 20, 3, False, "row"),
]


def _case(nz, nx, nabc, ns, fs, rcv, *, seed=0):
    rng = np.random.default_rng(seed)
    if rcv == "row":
        rz, rx = np.full(nx - 1, min(2, nz - 1)), np.arange(nx - 1)
    elif rcv == "column":
        rz, rx = np.arange(1, nz - 1), np.full(nz - 2, nx // 3)
    else:  # several receivers in a cell, in no order
        rz, rx = rng.integers(1, nz - 1, 70), rng.integers(0, nx - 1, 70)
        rz[30:50], rx[30:50] = rz[:20], rx[:20]
    kw = dict(nz=nz, nx=nx, nabc=nabc, free_surface=fs, src_z=rng.integers(1, nz, ns), src_x=rng.integers(0, nx, ns),
              rcv_z=rz, rcv_x=rx, nt=NT, dt=1e-3, dtype=torch.float32)
    nzp, nxp = nz + 2 * nabc, nx + 2 * nabc
    dev = "cuda:0"
    g = torch.Generator(device=dev).manual_seed(seed)
    c = 1500 + 2500 * torch.rand((nzp, nxp), device=dev, generator=g)
    rho = 1800 + 800 * torch.rand((nzp, nxp), device=dev, generator=g)
    a1, a2 = rho * c * c * 1e-4, 1e-4 / rho
    d = torch.zeros((nzp, nxp), device=dev)
    for k in range(nabc):  # a frame as wide as the absorbing strips
        v = 120.0 * ((nabc - k) / nabc) ** 2
        d[k:nzp - k, k] = d[k:nzp - k, nxp - 1 - k] = v
        d[k, k:nxp - k] = d[nzp - 1 - k, k:nxp - k] = v
    wav = torch.randn((ns, NT), device=dev, generator=g)
    wav = torch.nn.functional.avg_pool1d(wav[:, None], 9, 1, 4)[:, 0].contiguous()
    gp = torch.randn((ns, NT, len(rz)), device=dev, generator=g)
    return kw, a1, a2, d, wav, gp


def _rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm())


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "%dx%d_%d_%d%s_%s" % (s[0], s[1], s[2], s[3], "_fs" * s[4], s[5]))
def test_resident_loop_equals_the_per_step_kernels(shape):
    kw, a1, a2, d, wav, gp = _case(*shape)
    n0 = N.launch_count()
    plan = AcousticPlan(**kw)
    got = plan.run_forward(a1, a2, d, wav, True)
    assert N.launch_count() - n0 < NT  # the resident loop ran
    ref = AcousticPlan(**kw, snapshot_every=BOUNDARY_SAVING).run_forward(a1, a2, d, wav, False)
    for k in range(3):
        assert torch.equal(got[k], ref[k]), k
    for k in range(3, 6):
        assert _rel(got[k], ref[k]) <= TOL, k
    g1, g2 = plan.run_backward(a1, a2, d, wav, (gp, None, None), got[6])
    again = AcousticPlan(**kw)  # its adjoint through the per-step kernels
    ws = again.run_forward(a1, a2, d, wav, True)[6]
    r1, r2 = again.run_backward(a1, a2, d, wav, (gp, torch.zeros_like(gp), None), ws)
    assert plan.status(got[6], True) == 0
    assert _rel(g1, r1) <= TOL and _rel(g2, r2) <= TOL


@pytest.mark.parametrize("shape", [SHAPES[3], SHAPES[4]], ids=["fs", "no_fs"])
def test_zero_coefficients_keep_their_gradient(shape):
    """Cells whose alpha is zero pass nothing on, but dL/d alpha there is not zero."""
    kw, a1, a2, d, wav, gp = _case(*shape, seed=3)
    zp, xp = slice(shape[2] + 3, shape[2] + 9), slice(shape[2] + 5, shape[2] + 12)
    a1[zp, xp] = 0.0
    a2[zp.start + 2:zp.stop + 3, xp.start + 3:xp.stop + 4] = 0.0
    for every in (0, 31):
        out = []
        for gu in (None, torch.zeros_like(gp)):
            plan = AcousticPlan(**kw, snapshot_every=every)
            ws = plan.run_forward(a1, a2, d, wav, True)[6]
            out.append(plan.run_backward(a1, a2, d, wav, (gp, gu, None), ws))
        for g, r in zip(*out):
            assert float(r[a1 == 0].abs().max()) > 0
            assert _rel(g, r) <= TOL and _rel(g[a1 == 0], r[a1 == 0]) <= TOL


def test_many_launches_equal_one():
    """The loop is split into launches of bounded length: with enough shots for several hundred
    waves, the steps between two launches continue bit for bit."""
    kw, a1, a2, d, wav, gp = _case(20, 600, 10, 1500, False, "row")
    plan = AcousticPlan(**kw)
    n0 = N.launch_count()
    got = plan.run_forward(a1, a2, d, wav, False)
    launches = N.launch_count() - n0
    ref = AcousticPlan(**kw, snapshot_every=BOUNDARY_SAVING).run_forward(a1, a2, d, wav, False)
    assert launches < NT
    for k in range(3):
        assert torch.equal(got[k], ref[k])


def _solve(plan, a1, a2, d, wav, gp):
    rec = plan.run_forward(a1, a2, d, wav, True)
    return rec[:3] + plan.run_backward(a1, a2, d, wav, (gp, None, None), rec[6])


@pytest.mark.parametrize("shape", [SHAPES[2], SHAPES[7]], ids=["cluster", "global"])
def test_captured_solve_replays_the_same_bits(shape):
    kw, a1, a2, d, wav, gp = _case(*shape)
    plan = AcousticPlan(**kw)
    want = _solve(plan, a1, a2, d, wav, gp)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        graph.capture_begin()
        got = _solve(plan, a1, a2, d, wav, gp)
        graph.capture_end()
    torch.cuda.synchronize()
    for _ in range(2):
        graph.replay()
    torch.cuda.synchronize()
    for x, y in zip(got, want):
        assert torch.equal(x, y)


def test_solves_on_two_streams_at_once():
    """Two threads solve on their own streams; each result is the one it has alone."""
    import threading
    cases = [_case(*SHAPES[7]), _case(*SHAPES[5], seed=4)]
    plans = [AcousticPlan(**c[0]) for c in cases]
    want = [_solve(p, *c[1:]) for p, c in zip(plans, cases)]
    torch.cuda.synchronize()
    got, errors = [None, None], []

    def work(k):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(4):
                    got[k] = _solve(plans[k], *cases[k][1:])
                torch.cuda.current_stream().synchronize()
        except Exception as e:
            errors.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for g, w in zip(got, want):
        for x, y in zip(g, w):
            assert torch.equal(x, y)
