"""Elastic FP32 forward against the same steps in plain PyTorch on the CPU, bit for bit (GPU tests).

The step kernels evaluate the operations of the reference's step (elastic_kernels.py:339-418 and
709-774) in its order, each rounded by itself, with one rule of their own: where both PML factors are 1
and no surface row is near, the total advances by (t + a) + b instead of the sum of its two parts. The
loop below does the same with elementwise PyTorch operations, so records and the energy maps of one
shot (a sum over shots contracts) are equal, with no tolerance: an operation fused, reordered or
multiplied by a rounded factor shows.
"""
import pytest
import torch

import adfwi_gb300 as A
from _cases import ELASTIC_KEYS, elastic_problem
from oracle.elastic import _apply_fs_stress, _apply_fs_velocity, _dxb, _dxf, _dzb, _dzf, diff_coef

pytestmark = pytest.mark.gpu


def plain_steps(prop, coefs, abc, nn, pml):
    """Records (ns, nt, nr) per component and the last step's fields, from padded CPU planes."""
    c11, c13, c15, c33, c35, c55, bx, bz = coefs
    nzp, nxp = c11.shape
    h, ns, nt = nn + 1, prop.src_n, prop.nt
    fs, dt, dx, dz = bool(prop.free_surface), prop.dt, prop.dx, prop.dz
    fl = list(diff_coef(nn))
    reg = (slice(nn, nzp - nn), slice(nn, nxp - nn))
    R = (slice(None),) + reg
    c11, c13, c15, c33, c35, c55, bx, bz = (a[reg] for a in (c11, c13, c15, c33, c35, c55, bx, bz))
    top = nn if fs else nn + prop.nabc
    sx, sz = (torch.as_tensor(prop.src_loc[:, k]) + o for k, o in ((0, prop.nabc), (1, top)))
    rx, rz = (torch.as_tensor(prop.rcv_loc[:, k]) + o for k, o in ((0, prop.nabc), (1, top)))
    shots, wav, mt = torch.arange(ns), prop.wavelet.cpu(), prop.moment_tensor.cpu()
    m = [mt[:, 0, 0], mt[:, 2, 2], mt[:, 0, 2]]
    t = [torch.zeros((ns, nzp, nxp)) for _ in range(3)]
    v = [torch.zeros((ns, nzp, nxp)) for _ in range(2)]
    if pml:
        bcx, bcz = abc[0][reg], abc[1][reg]
        xd, xn, zd, zn = (1 + 0.5 * dt * bcx, 1 - 0.5 * dt * bcx, 1 + 0.5 * dt * bcz, 1 - 0.5 * dt * bcz)
        split = (bcx != 0) | (bcz != 0)
        if fs:
            split[:h + 2 - nn] = True
        ts = [torch.zeros((ns, nzp, nxp)) for _ in range(6)]
        vs = [torch.zeros((ns, nzp, nxp)) for _ in range(4)]
    rec = {k: [] for k in ELASTIC_KEYS}
    for it in range(nt):
        vx, vz = v
        d = [_dxb(vx, fl, nn), _dxb(vz, fl, nn), _dzb(vx, fl, nn), _dzb(vz, fl, nn), _dxf(vx, fl, nn), _dxf(vz, fl, nn),
             _dzf(vx, fl, nn), _dzf(vz, fl, nn)]
        a = [c11 * d[0] + c15 * d[1], c15 * d[2] + c13 * d[3], c13 * d[0] + c35 * d[1], c35 * d[2] + c33 * d[3],
             c15 * d[4] + c55 * d[5], c55 * d[6] + c35 * d[7]]
        for k in range(3):
            if pml:
                x, z = (dt / dx) * a[2 * k], (dt / dz) * a[2 * k + 1]
                total, src = (t[k][R] + x) + z, -(m[k] / 2) * wav[:, it]
                ts[2 * k][R] = (xn * ts[2 * k][R] + x) * (1.0 / xd)
                ts[2 * k + 1][R] = (zn * ts[2 * k + 1][R] + z) * (1.0 / zd)
                t[k] = torch.zeros((ns, nzp, nxp))
                t[k][R] = total
                t[k][shots, sz, sx] += 2 * src
                for q in (2 * k, 2 * k + 1):
                    ts[q][shots, sz, sx] += src
                t[k][R] = torch.where(split, ts[2 * k][R] + ts[2 * k + 1][R], t[k][R])
            else:
                t[k][R] += dt * (a[2 * k] / dx + a[2 * k + 1] / dz)
                t[k][shots, sz, sx] += (-1 / 3) * m[k] * wav[:, it]
        if fs:
            t[1], t[2] = _apply_fs_stress(t[1], t[2], h)
        b = [_dxf(t[0], fl, nn), _dzb(t[2], fl, nn), _dxb(t[2], fl, nn), _dzf(t[1], fl, nn)]
        for k in range(2):
            c = dt * (bx, bz)[k]
            if pml:
                x, z = c * b[2 * k] / dx, c * b[2 * k + 1] / dz
                vs[2 * k][R] = (xn * vs[2 * k][R] + x) / xd
                vs[2 * k + 1][R] = (zn * vs[2 * k + 1][R] + z) / zd
                total = torch.where(split, vs[2 * k][R] + vs[2 * k + 1][R], (v[k][R] + x) + z)
                v[k] = torch.zeros((ns, nzp, nxp))
                v[k][R] = total
            else:
                v[k][R] += c * (b[2 * k] / dx + b[2 * k + 1] / dz)
        if fs:
            v = list(_apply_fs_velocity(v[0], v[1], h, nn, nxp - nn - 1))
        if not pml:
            v = [f * abc[0] for f in v]
        for k, f in zip(ELASTIC_KEYS, t + v):
            rec[k].append(f[:, rz, rx].clone())
    inner = (slice(None), slice(top, top + prop.nz), slice(prop.nabc, prop.nabc + prop.nx))
    return {k: torch.stack(r, dim=1) for k, r in rec.items()}, {k: f[inner] for k, f in zip(ELASTIC_KEYS, t + v)}


@pytest.mark.parametrize("ns,nz,nx,nt,dx,fd_order,abc_type,free_surface", [
    (1, 30, 40, 160, 5.0, 4, "PML", True),
    (1, 21, 33, 90, 7.3, 6, "PML", False),
    (2, 17, 70, 120, 12.5, 6, "PML", True),
    (1, 30, 40, 160, 5.0, 4, "gerjan", True),
    (2, 33, 21, 120, 7.3, 6, "gerjan", False),
    (1, 19, 45, 90, 1.0 / 3.0, 4, "sincos", False),
    (1, 12, 20, 40, 3.0e18, 4, "PML", False),  # a spacing beyond the range of the quick division
])
def test_fp32_forward_rounds_every_operation_by_itself(ns, nz, nx, nt, dx, fd_order, abc_type, free_surface):
    model, survey, prop = elastic_problem(A, nz=nz, nx=nx, nt=nt, ns=ns, nr=nx - 4, dx=dx, dt=1e-4 * dx, f0=0.07 / (1e-4 * dx),
                                          fd_order=fd_order, abc_type=abc_type, free_surface=free_surface,
                                          mt=[[1.0, 0.0, 0.4], [0.0, 1.0, 0.0], [0.4, 0.0, 0.6]])
    with torch.no_grad():
        rec = prop.forward(fd_order=fd_order)
        coefs, abc = prop.padded_coefficients(model, fd_order)
    ref, last = plain_steps(prop, [c.cpu() for c in coefs], [a if a is None else a.cpu() for a in abc], fd_order // 2,
                            abc_type == "PML")
    for k in ELASTIC_KEYS:
        got = rec[k].cpu()
        assert bool(got.abs().max() > 0) and torch.equal(got, ref[k]), k
        if ns == 1:
            assert torch.equal(rec["forward_wavefield_" + k].cpu(), last[k][0] * last[k][0]), k
