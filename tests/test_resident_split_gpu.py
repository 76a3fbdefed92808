"""The resident time loop at the ends of its launches: solves of more steps than one launch takes, of one
step, and without receivers (GPU tests).

A launch advances at most 16000 steps divided by the waves of shots (at least 64), so each shape here
has some steps more than its first launch takes, forward and in reverse. Records equal the per-step
kernels' bit for bit, and a gradient the one from FP32 snapshots, whose launches end elsewhere.
"""
import pytest
import torch

import test_resident_gpu as R
from adfwi_gb300 import _native as N
from adfwi_gb300.acoustic import BOUNDARY_SAVING, AcousticPlan

pytestmark = pytest.mark.gpu


def counted(solve):
    """solve() and how many forward and reverse step kernels it launched."""
    N.profile_start(False)
    try:
        out = solve()
    finally:
        n = N.profile_stop()
    return out, n.get("acoustic_fwd_step", (0,))[0], n.get("acoustic_adj_step", (0,))[0]


# (shape as in test_resident_gpu, steps, steps between snapshots: 0 for records alone): one block a shot;
# a cluster; strips that exchange rows through global memory; many waves of shots
@pytest.mark.parametrize("shape,nt,every", [
    ((11, 9, 3, 2, True, "row"), 16050, 977),
    ((30, 40, 10, 2, False, "shared"), 16041, 1003),
    ((62, 1500, 5, 1, False, "row"), 16033, 400),
    ((63, 1500, 5, 1, True, "row"), 16033, 400),
    ((20, 600, 10, 1500, False, "shared"), 1700, 0),
], ids=lambda v: "x".join(str(e) for e in v) if isinstance(v, tuple) else str(v))
def test_more_steps_than_a_launch_takes(monkeypatch, shape, nt, every):
    monkeypatch.setattr(R, "NT", nt)
    kw, a1, a2, d, wav, gp = R._case(*shape)
    records, fwd, _ = counted(lambda: AcousticPlan(**kw).run_forward(a1, a2, d, wav, False)[:3])
    assert 1 < fwd < nt // 32
    ref = AcousticPlan(**kw, snapshot_every=BOUNDARY_SAVING).run_forward(a1, a2, d, wav, False)
    for k in range(3):
        assert torch.equal(records[k], ref[k]), k
    del ref, records
    if not every:
        return
    # a launch of the adjoint ends after 16000 steps with the whole history, at the snapshots with these
    grads = []
    for e in (nt, every):
        plan = AcousticPlan(**kw, snapshot_every=e)
        assert plan.snapshot_every == e
        ws = plan.run_forward(a1, a2, d, wav, True)[6]
        g, _, adj = counted(lambda: plan.run_backward(a1, a2, d, wav, (gp, None, None), ws))
        assert plan.status(ws, True) == 0
        assert 1 < adj < nt // 32
        grads.append(g)
        del ws
    for x, y in zip(*grads):
        assert float(x.abs().max()) > 0 and torch.equal(x, y)


@pytest.mark.parametrize("shape", [R.SHAPES[0], R.SHAPES[3], R.SHAPES[7]], ids=["block", "cluster", "global"])
@pytest.mark.parametrize("receivers", [True, False])
def test_one_step_and_no_receivers(monkeypatch, shape, receivers):
    nt = 1 if receivers else 50
    monkeypatch.setattr(R, "NT", nt)
    kw, a1, a2, d, wav, gp = R._case(*shape)
    if not receivers:
        kw["rcv_z"], kw["rcv_x"] = kw["rcv_z"][:0], kw["rcv_x"][:0]
    plan = AcousticPlan(**kw)
    got, fwd, _ = counted(lambda: plan.run_forward(a1, a2, d, wav, True))
    assert fwd < max(2, nt // 4)  # at most one for each snapshot
    ref = AcousticPlan(**kw, snapshot_every=BOUNDARY_SAVING).run_forward(a1, a2, d, wav, False)
    for k in range(3):
        assert got[k] is ref[k] is None or torch.equal(got[k], ref[k]), k
    for k in range(3, 6):
        assert R._rel(got[k], ref[k]) <= 2 * nt * 2.0 ** -24 * 2, k
    g = plan.run_backward(a1, a2, d, wav, (gp if receivers else None, None, None), got[6])
    assert plan.status(got[6], True) == 0
    again = AcousticPlan(**kw)
    ws = again.run_forward(a1, a2, d, wav, True)[6]
    if receivers:  # the adjoint through the per-step kernels
        ref = again.run_backward(a1, a2, d, wav, (gp, torch.zeros_like(gp), None), ws)
        for x, y in zip(g, ref):
            assert float((x - y).double().norm()) <= 2 * nt * 2.0 ** -24 * 2 * float(y.double().norm())
    else:
        assert not any(bool(x.any()) for x in g)
