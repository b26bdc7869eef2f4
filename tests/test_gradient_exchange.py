"""The viscous gradient as callers see it: cb_solver_pack, cb_solver_unpack and
the face traces carry (Np, fields, directions) per element whatever form the
passes keep, and a kernel choice made between two passes changes no result.

The gradient is compared with the per-kernel calls on the same state (volume_grad,
flux_grad, update_gradQ).  Tolerances, relative L2 per component: a derivative is
a sum of N + 1 products of entries of D (up to N^2 per element) and values of
order one, against gradients of order 0.1, so rounding eps of the values becomes
eps (N + 1) N^2 / 0.1: 1e-12 in FP64 (N <= 10) and 3e-4 in FP32 (N <= 7).  After a run both
sides have advanced the state, each to 1e-13; the same factor gives 1e-10.  States
against states: 1e-12, the bar of the viscous passes."""
import ctypes as C
import math

import numpy as np
import pytest

from conftest import cuda_available
from dg_cases import relerr_fields
from canary_b200 import _lib, dg, ic
from canary_b200 import partition as P
from canary_b200._lib import check
from canary_b200.metric import warp_sinusoidal

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not cuda_available(), reason="needs a CUDA GPU")]

PHYS = dict(dg.WORKLOAD_PHYS, visc=0.02)
RKA = (0.0, -567301805773.0 / 1357537059087.0, -2404267990393.0 / 2016746695238.0,
       -3550918686646.0 / 2091501179385.0, -1275806237668.0 / 842570457699.0)
RKB = (1432997174477.0 / 9575080441755.0, 5161836677717.0 / 13612068292357.0,
       1720146321549.0 / 2090206949498.0, 3134564353537.0 / 4481467310338.0,
       2277821191437.0 / 14882151754819.0)


def box(N, n, walls=True, gravity=0.0):
    m = dg.build_mesh(3, N, tuple(np.linspace(0, 2 * math.pi, k + 1) for k in n), (True, True, not walls),
                      meshwarp=lambda X: warp_sinusoidal(X, 0.05))
    Q = np.asfortranarray(np.stack(ic.fourier_state(*m.coords(), seed=N), axis=1))
    return m, Q, 0.1 * ic.fourier_dt(Q, N, h=2 * math.pi / max(n)), dict(PHYS, gravity=gravity)


def stage_pass(s, st, dt, pass_):
    nxt = C.c_void_p()
    check(_lib.lib().cb_solver_stage_pass(s._h, st, dt, pass_, C.byref(nxt)))


def packed(s, m, idx, real):
    """Gradient of elements idx, (Np, 5, 3, len(idx))."""
    import torch
    buf = torch.full((len(idx) * 15 * m.Np,), 7.0, dtype=real, device="cuda")
    ids = torch.as_tensor(idx, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    check(_lib.lib().cb_solver_pack(s._h, 1, C.c_void_p(ids.data_ptr()), len(idx), C.c_void_p(buf.data_ptr())))
    torch.cuda.synchronize()
    return dg.from_device(buf.double(), (m.Np, 5, 3, len(idx)))


def plain_run(m, Q, dt, steps, phys, stages=None):
    """State and last gradient of the per-kernel calls (FP64)."""
    import torch
    dm, ph = dg.DeviceMesh.upload(m), dg.make_phys(**phys)
    q, E, N = dg.to_device(Q), m.nelem, m.N
    rhs, rg = torch.zeros_like(q), torch.zeros(3 * q.numel(), dtype=torch.float64, device="cuda")
    g = torch.zeros_like(rg)
    maps = (dm.vmapM, dm.vmapP, dm.elemtobndy)
    for k in range(5 * steps if stages is None else stages):
        st = k % 5
        dg.volumerhs(3, N, rhs, q, dm.vgeo, dm.D, E, ph)
        dg.fluxrhs(3, N, rhs, q, dm.sgeo, dm.vgeo, E, *maps, ph)
        dg.volume_grad(3, N, rg, q, dm.vgeo, dm.D, E, ph)
        dg.flux_grad(3, N, rg, q, dm.sgeo, dm.vgeo, E, *maps, ph)
        dg.update_gradQ(3, N, g, rg, dm.vgeo, E)
        dg.volume_div(3, N, rg, g, q, dm.vgeo, dm.D, E, ph)
        dg.flux_div(3, N, rg, g, q, dm.sgeo, E, *maps, ph)
        dg.updatesolution(3, N, rhs, rg, q, dm.vgeo, E, RKA[(st + 1) % 5], RKB[st], dt, ph.visc)
    return dg.from_device(q, Q.shape), dg.from_device(g, (m.Np, 5, 3, E))


def gradient_error(a, b):
    return max(np.linalg.norm(a[:, s, d] - b[:, s, d]) / np.linalg.norm(b[:, s, d])
               for s in range(5) for d in range(3))


def solver(m, Q, precision, phys, kernel=0, offset=None):
    s = dg.LSRK.for_state(dg.DeviceMesh.upload(m), Q, precision, phys=dg.make_phys(**phys), offset=offset)
    s.set_kernel(kernel)
    return s


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("kernel", [5, 1, 3])
@pytest.mark.parametrize("N,n,gravity", [(1, (3, 4, 3), 0.0), (2, (3, 3, 3), 0.0), (4, (3, 2, 3), 0.3),
                                         (7, (2, 2, 3), 0.0)])
def test_packed_gradient_of_a_pass(N, n, gravity, kernel, precision):
    import torch
    m, Q, dt, phys = box(N, n, gravity=gravity)
    real = torch.float64 if precision == 64 else torch.float32
    tol = 1e-12 if precision == 64 else 3e-4
    _, ref = plain_run(m, Q, dt, 0, phys, stages=1)
    s = solver(m, Q, precision, phys, kernel)
    stage_pass(s, 0, dt, 0)
    idx = np.random.default_rng(N).permutation(m.nelem)
    got = packed(s, m, idx, real)
    assert gradient_error(got, ref[..., idx]) < tol
    # face traces: the same values at the face's nodes, component after component
    Nq, Nfp = N + 1, (N + 1) ** 2
    e = np.repeat(np.arange(m.nelem), 6)
    f = np.tile(np.arange(6), m.nelem)
    codes = torch.as_tensor(e * 8 + f, dtype=torch.int64, device="cuda")
    buf = torch.full((len(e) * 15 * Nfp,), 7.0, dtype=real, device="cuda")
    torch.cuda.synchronize()
    check(_lib.lib().cb_solver_pack_faces(s._h, 1, C.c_void_p(codes.data_ptr()), len(e), C.c_void_p(buf.data_ptr())))
    torch.cuda.synchronize()
    faces = buf.double().cpu().numpy().reshape(len(e), 3, 5, Nfp)
    byel = np.empty_like(got)
    byel[..., idx] = got
    nodes = np.arange(m.Np).reshape(Nq, Nq, Nq)  # [k, j, i]
    of = [nodes[:, :, 0], nodes[:, :, -1], nodes[:, 0, :], nodes[:, -1, :], nodes[0], nodes[-1]]
    for i in range(len(e)):
        want = byel[of[f[i]].ravel(), :, :, e[i]]  # (Nfp, 5, 3)
        assert np.array_equal(faces[i], want.transpose(2, 1, 0)), (e[i], f[i])
    s.close()


@pytest.mark.parametrize("N,kernel", [(3, 5), (3, 1), (6, 5), (8, 0), (10, 0)])
@pytest.mark.parametrize("steps", [1, 2, 3])
def test_packed_gradient_after_a_run(N, kernel, steps):
    """The buffer holds the gradient of the last stage, as a pass leaves it;
    odd and even step counts end in different buffers.  Then again after calls that
    may come first: another offset, another kernel choice."""
    import torch
    m, Q, dt, phys = box(N, (2, 3, 2))
    state, ref = plain_run(m, Q, dt, steps, phys)
    idx = np.arange(m.nelem)[::-1].copy()
    for between in ("none", "offset", "kernel", "pass"):
        if N > 7 and between == "pass":
            continue  # (no stage calls)
        s = solver(m, Q, 64, phys, kernel)
        s.run(steps, dt)
        assert max(relerr_fields(s.state(), state)) < 1e-12
        if between == "offset" and N <= 7:
            s.set_offset([0.0, 0.0, 0.0, 0.5, 0.0])
        if between == "kernel":
            s.set_kernel({0: 3, 5: 3, 1: 5}[kernel])
        if between == "pass":
            stage_pass(s, 0, dt, 1)  # (on the gradient at hand: its values stay)
        assert gradient_error(packed(s, m, idx, torch.float64), ref[..., idx]) < 1e-10, between
        s.close()


@pytest.mark.parametrize("between", ["none", "settle", "offset", "pass"])
@pytest.mark.parametrize("stages", [1, 2, 3])
@pytest.mark.parametrize("N,kernel", [(3, 5), (3, 1), (6, 5)])
def test_packed_gradient_after_stage_calls(N, kernel, stages, between):
    """The gradient of the last stage call, also once its input has been overwritten."""
    import torch
    m, Q, dt, phys = box(N, (2, 3, 2))
    _, ref = plain_run(m, Q, dt, 0, phys, stages=stages)
    s = solver(m, Q, 64, phys, kernel)
    nxt = C.c_void_p()
    for st in range(stages):
        check(_lib.lib().cb_solver_stage(s._h, st, dt, C.byref(nxt)))
    if between == "settle":
        check(_lib.lib().cb_solver_settle(s._h))
    if between == "offset":
        s.set_offset([0.0, 0.0, 0.0, 0.5, 0.0])
    if between == "pass":
        stage_pass(s, stages, dt, 1)
    idx = np.arange(m.nelem)
    assert gradient_error(packed(s, m, idx, torch.float64), ref) < 1e-10
    s.close()


@pytest.mark.parametrize("precision,tol", [(64, 1e-12), (32, 1e-5)])
@pytest.mark.parametrize("first,second", [(5, 1), (1, 5), (5, 3), (3, 5)])
@pytest.mark.parametrize("N", [2, 5])
def test_kernel_choice_between_two_passes(N, first, second, precision, tol):
    m, Q, dt, phys = box(N, (3, 3, 2))
    want, _ = plain_run(m, Q, dt, 0, phys, stages=2)
    s = solver(m, Q, precision, phys, first)
    for st in range(2):
        stage_pass(s, st, dt, 0)
        s.set_kernel(second)
        stage_pass(s, st, dt, 1)
        s.set_kernel(first)
    check(_lib.lib().cb_solver_settle(s._h))
    import torch
    torch.cuda.synchronize()
    assert max(relerr_fields(s.state(), want)) < tol
    s.close()


@pytest.mark.parametrize("faces", [True, False])
@pytest.mark.parametrize("precision,tol", [(64, 1e-12), (32, 1e-5)])
def test_parts_with_different_kernel_choices(precision, tol, faces):
    """Ranks exchange gradients in one layout whatever each one runs."""
    import torch
    m, Q, dt, phys = box(3, (4, 3, 3))
    want, _ = plain_run(m, Q, dt, 2, phys)
    stream = torch.cuda.Stream()
    parts = [P.GhostedLSRK(m, P.plan(m, r, 3), Q, precision, dg.make_phys(**phys), stream=stream) for r in range(3)]
    for part, kernel in zip(parts, (5, 1, 3)):
        check(_lib.lib().cb_solver_set_kernel(part._h, kernel))
    P.run_parts(parts, 2, dt, faces=faces)
    got = np.concatenate([p.state() for p in parts], axis=2)
    for p in parts:
        p.close()
    assert max(relerr_fields(got, want)) < tol


@pytest.mark.parametrize("before,after", [(5, 1), (1, 5)])
def test_ghost_gradients_outlive_a_kernel_choice(before, after):
    """Ghost gradients stored under one choice are read by a stage of another."""
    import torch
    m, Q, dt, phys = box(3, (4, 3, 3))
    stream = torch.cuda.Stream()
    out = []
    for choices in ((before, after), (after, after)):
        parts = [P.GhostedLSRK(m, P.plan(m, r, 2), Q, 64, dg.make_phys(**phys), stream=stream) for r in range(2)]
        p = parts[0]
        with torch.cuda.stream(stream):
            for part in parts:
                check(_lib.lib().cb_solver_set_kernel(part._h, choices[0]))
            for what in (0, 1):  # the state, then the gradient of the first pass
                for q, first, n in p.plan.recv:
                    idx = torch.as_tensor(dict(parts[q].plan.send)[0], dtype=torch.int64, device="cuda")
                    buf = torch.empty(n * max(p.widths), dtype=torch.float64, device="cuda")
                    if what:
                        for r, f1, n1 in parts[q].plan.recv:
                            back = torch.as_tensor(dict(p.plan.send)[q], dtype=torch.int64, device="cuda")
                            b1 = torch.empty(n1 * p.widths[0], dtype=torch.float64, device="cuda")
                            p.pack(back, b1, 0)
                            parts[q].unpack(b1, f1, n1, 0)
                        parts[q].stage(0, dt, 0)
                    b = buf[:n * p.widths[what]]
                    parts[q].pack(idx, b, what)
                    p.unpack(b, first, n, what)
            check(_lib.lib().cb_solver_set_kernel(p._h, choices[1]))
            p.stage(0, dt, 0)
            p.stage(0, dt, 1)
        out.append(p.state())
        for part in parts:
            part.close()
    assert max(relerr_fields(out[0], out[1])) < 1e-12


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("kernel", [5, 1])
@pytest.mark.parametrize("stages", [0, 1])
def test_gradient_is_of_the_state_its_pass_read(stages, kernel, precision):
    """What a caller writes over the current state after the gradient pass (in Q, or
    in the twin after an odd number of stages) does not reach a packed gradient."""
    import torch
    m, Q, dt, phys = box(3, (3, 2, 3))
    _, ref = plain_run(m, Q, dt, 0, phys, stages=stages + 1)
    real = torch.float64 if precision == 64 else torch.float32
    s = solver(m, Q, precision, phys, kernel)
    for st in range(stages):
        stage_pass(s, st, dt, 0)
        stage_pass(s, st, dt, 1)
    stage_pass(s, stages, dt, 0)
    torch.cuda.synchronize()
    if stages == 0:
        s.Q.mul_(2.0).add_(1.0)
    else:  # (unpack, what = 0, needs ghosts: an even stage call overwrites the buffer instead)
        stage_pass(s, stages, dt, 1)
        stage_pass(s, stages + 1, dt, 1)
    torch.cuda.synchronize()
    got = packed(s, m, np.arange(m.nelem), real)
    assert gradient_error(got, ref) < (1e-10 if precision == 64 else 3e-4)
    s.close()
