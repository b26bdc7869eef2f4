"""Stages of small meshes (geometry and codes loaded before the wait for the
preceding stage), chained launches, and the per-kernel calls on meshes with partial
blocks.

Tolerances, relative L2 per field: FP64 runs 1e-12, FP32 runs 1e-5, single calls
1e-13 in FP64 (the bars of the other parity tests); single FP32 calls 1e-5: their
values are sums of up to 3·(N + 1) products, each rounded to 6e-8 of fluxes about
ten times the sum."""
import math

import numpy as np
import pytest

from conftest import cuda_available
from dg_cases import oracle_phys, oracle_run, relerr_fields, vortex_case
from oracle import pyoracle as O
from canary_b200 import dg, ic
from canary_b200.metric import warp_sinusoidal

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not cuda_available(), reason="needs a CUDA GPU")]

TOL = {64: 1e-12, 32: 1e-5}


def cube(N, n, walls, seed):
    m = dg.build_mesh(3, N, tuple(np.linspace(0, 2 * math.pi, k + 1) for k in n), (True, True, not walls),
                      meshwarp=lambda X: warp_sinusoidal(X, 0.05))
    Q = np.asfortranarray(np.stack(ic.fourier_state(*m.coords(), seed=seed), axis=1))
    return m, Q, 0.1 * ic.fourier_dt(Q, N, h=2 * math.pi / max(n))


def solver(m, Q, precision, phys):
    return dg.LSRK.for_state(dg.DeviceMesh.upload(m), Q, precision, phys=dg.make_phys(**phys))


# below and above the block counts at which the small-mesh form ends (148 and 592
# blocks: N=1 blocks hold 32 elements, N=3 four, N>=5 one; 2-D N=4 ten)
@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("N,n", [(1, (3, 3, 3)), (2, (5, 4, 3)), (3, (1, 1, 1)), (3, (8, 8, 9)), (3, (13, 13, 14)),
                                 (4, (7, 5, 3)), (5, (5, 5, 5)), (6, (3, 4, 3)), (7, (3, 2, 2)), (8, (2, 3, 3))])
def test_small_stage_3d(N, n, precision):
    m, Q, dt = cube(N, n, True, seed=N)
    phys = dict(dg.WORKLOAD_PHYS, gravity=0.3)
    ref = oracle_run(m, Q, dt, 3, phys=phys)  # two steps as a graph, one launched directly
    s = solver(m, Q, precision, phys)
    s.run(3, dt)
    assert max(relerr_fields(s.state(), ref)) < TOL[precision]
    s.sums()
    s.close()


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("N,side", [(1, 5), (4, 3), (4, 10), (4, 39), (7, 12), (7, 13), (10, 6)])
def test_small_stage_2d(N, side, precision):
    m, Q = vortex_case(N, side)
    dt = 0.1 * (10 / side) / (N * N * 3.0)
    ref = oracle_run(m, Q, dt, 3)
    s = solver(m, Q, precision, dg.WORKLOAD_PHYS)
    s.run(3, dt)
    assert max(relerr_fields(s.state(), ref)) < TOL[precision]
    s.close()


@pytest.mark.parametrize("dim,N,side,precision", [(2, 4, 10, 64), (2, 7, 30, 32), (3, 3, 8, 32), (3, 4, 9, 64),
                                                  (3, 6, 5, 64), (3, 7, 6, 64), (3, 8, 5, 64)])
def test_chained_launches(dim, N, side, precision):
    """In a graph a stage is launched while the one before it finishes; a single
    step is launched directly, its first stage after all earlier work.  The same
    kernels on the same data: the same bits."""
    m, Q, dt = cube(N, (side,) * 3, True, seed=N) if dim == 3 else (*vortex_case(N, side), 1e-4)
    a, b = (solver(m, Q, precision, dg.WORKLOAD_PHYS) for _ in range(2))
    a.run(20, dt)
    for _ in range(20):
        b.run(1, dt)
    assert np.array_equal(a.state(), b.state())
    a.close()
    b.close()


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("dim,N,n", [(2, 1, 3), (2, 10, 2), (3, 1, 3), (3, 2, 3), (3, 3, 3), (3, 5, 3), (3, 6, 2),
                                     (3, 8, 2), (3, 9, 2), (3, 10, 1)])
def test_stage_by_calls(dim, N, n, precision):
    import torch
    L = 2 * math.pi
    m = dg.build_mesh(dim, N, (np.linspace(0, L, n + 1),) * dim, (True,) * (dim - 1) + (False,),
                      meshwarp=lambda X: warp_sinusoidal(X, 0.05))
    X = m.coords()
    f = ic.fourier_state(*X, seed=N) if dim == 3 else ic.isentropic_vortex(X[0] * (10 / L), X[1] * (10 / L))
    real = np.float64 if precision == 64 else np.float32
    g = np.random.default_rng(N)
    h = {k: np.asfortranarray(v.astype(real)) for k, v in
         (("Q", np.stack(f, axis=1)), ("vgeo", np.asarray(m.vgeo)), ("sgeo", np.asarray(m.sgeo)),
          ("D", np.asarray(m.D)))}
    h["r"] = np.asfortranarray(g.standard_normal(h["Q"].shape).astype(real))
    h["rg"] = np.asfortranarray(g.standard_normal(h["Q"].shape[:2] + (dim,) + h["Q"].shape[2:]).astype(real))
    d = {k: dg.to_device(v) for k, v in h.items()}
    assert d["Q"].dtype == (torch.float64 if precision == 64 else torch.float32)
    phys = dict(dg.WORKLOAD_PHYS, gravity=0.3)
    ph, op = dg.make_phys(**phys), oracle_phys(phys)
    dm = dg.DeviceMesh.upload(m)
    w = {k: np.asfortranarray(v.astype(np.float64)) for k, v in h.items()}
    tol = 1e-13 if precision == 64 else 1e-5
    r, Q = w["r"], w["Q"]
    # (each call is compared on its own: the oracle continues from the device's values)
    O.volumerhs(dim, N, r, Q, w["vgeo"], w["D"], op, 4)
    dg.volumerhs(dim, N, d["r"], d["Q"], d["vgeo"], d["D"], m.nelem, ph)
    out = dg.from_device(d["r"], Q.shape)
    assert max(relerr_fields(out, r)) < tol
    r = np.asfortranarray(out.astype(np.float64))
    O.fluxrhs(dim, N, r, Q, w["sgeo"], w["vgeo"], m.vmapM, m.vmapP, m.elemtobndy, op, 4)
    dg.fluxrhs(dim, N, d["r"], d["Q"], d["sgeo"], d["vgeo"], m.nelem, dm.vmapM, dm.vmapP, dm.elemtobndy, ph)
    dg.device_status()
    out = dg.from_device(d["r"], Q.shape)
    assert max(relerr_fields(out, r)) < tol
    r = out.astype(np.float64)
    rka, rkb, dt, visc = -0.7, 0.4, 1e-2, 0.3
    dg.updatesolution(dim, N, d["r"], d["rg"], d["Q"], d["vgeo"], m.nelem, rka, rkb, dt, visc)
    r = r + visc * w["rg"][:, :, 0, :]
    Qn = Q + rkb * dt * r * w["vgeo"][:, dim * dim + 1, :][:, None, :]
    assert max(relerr_fields(dg.from_device(d["Q"], Q.shape), Qn)) < tol
    assert max(relerr_fields(dg.from_device(d["r"], Q.shape), rka * r)) < tol
    if precision == 64:
        grad = torch.full_like(d["rg"], 7.0)
        dg.update_gradQ(dim, N, grad, d["rg"], d["vgeo"], m.nelem)
        want = w["rg"] * w["vgeo"][:, dim * dim + 1, :][:, None, None, :]
        assert np.array_equal(dg.from_device(grad, want.shape), want)


def test_calls_report_entries_off_the_element():
    """fluxrhs checks both maps of a face entry: a node of another element in vmapM
    and ids outside the mesh in vmapP are skipped and reported."""
    import torch
    from canary_b200 import CanaryError
    from canary_b200._lib import CB_ERR_MESH
    m, Q = vortex_case(3, 4)
    dm = dg.DeviceMesh.upload(m)
    dQ = dg.to_device(Q)
    last = m.Np * m.nelem
    for key, value in (("vmapM", 0), ("vmapM", m.Np + 1), ("vmapP", 0), ("vmapP", last + 1), ("vmapP", (1 << 32) + 1)):
        maps = {"vmapM": dm.vmapM.clone(), "vmapP": dm.vmapP.clone()}
        maps[key].view(-1)[0] = value
        r = torch.zeros_like(dQ)
        dg.fluxrhs(2, 3, r, dQ, dm.sgeo, dm.vgeo, m.nelem, maps["vmapM"], maps["vmapP"], dm.elemtobndy)
        with pytest.raises(CanaryError) as ei:
            dg.device_status()
        assert ei.value.code == CB_ERR_MESH, (key, value)
    dg.device_status()
