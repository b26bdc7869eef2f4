"""The default stage kernel by mesh size: on both sides of each rule's line the solver
reports the kernel of that side and agrees with the oracle (FP64 1e-12, FP32 1e-5
relative L2 per field, the bars of the stages).  Lines are in element groups per SM, so
the sides follow from the device."""
import math

import numpy as np
import pytest

from conftest import cuda_available
from dg_cases import oracle_run, relerr_fields
from canary_b200 import dg, ic
from canary_b200.metric import warp_sinusoidal

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not cuda_available(), reason="needs a CUDA GPU")]


def sms():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


def groups(N, nelem):
    Np = (N + 1) ** 3
    return -(-nelem // (1 if Np >= 200 else 256 // Np))


# (order, precision, groups per SM up to which the pipelined passes run, sides on
# both sides of it with 148 SMs)
@pytest.mark.parametrize("N,precision,limit,sides", [
    (1, 64, 0, (2, 4)), (2, 64, 1, (11, 12)), (2, 32, 1, (11, 12)), (3, 32, 2, (10, 11)), (4, 64, 2, (8, 9)),
    (4, 32, 1, (6, 7)), (5, 32, 3, (7, 8)), (6, 64, 1, (5, 6)), (7, 64, 1, (5, 6)), (7, 32, 2, (6, 7)),
    (8, 64, 0, (2,))])
def test_viscous_passes(N, precision, limit, sides):
    for n in sides:
        m = dg.build_mesh(3, N, (np.linspace(0, 2 * math.pi, n + 1),) * 3, (True, True, False),
                          meshwarp=lambda X: warp_sinusoidal(X, 0.05))
        Q = np.asfortranarray(np.stack(ic.fourier_state(*m.coords(), seed=N), axis=1))
        dt = 0.1 * ic.fourier_dt(Q, N, h=2 * math.pi / n)
        phys = dict(dg.WORKLOAD_PHYS, visc=0.02, gravity=0.02)
        s = dg.LSRK.for_state(dg.DeviceMesh.upload(m), Q, precision, phys=dg.make_phys(**phys),
                              offset=np.zeros(5) if N > 7 else None)
        assert s.kernel == (1 if groups(N, m.nelem) <= limit * sms() else 5), n
        s.run(2, dt)
        assert max(relerr_fields(s.state(), oracle_run(m, Q, dt, 2, phys=phys))) < (1e-12 if precision == 64 else 1e-5), n
        s.close()


@pytest.mark.parametrize("N,precision,sides", [(8, 64, (5, 6)), (9, 64, (5, 6)), (10, 64, (5,)), (10, 32, (5, 6))])
def test_inviscid_high_orders(N, precision, sides):
    for n in sides:
        m = dg.build_mesh(3, N, (np.linspace(0, 2 * math.pi, n + 1),) * 3, (True, True, False),
                          meshwarp=lambda X: warp_sinusoidal(X, 0.05))
        Q = np.asfortranarray(np.stack(ic.fourier_state(*m.coords(), seed=N), axis=1))
        dt = 0.1 * ic.fourier_dt(Q, N, h=2 * math.pi / n)
        phys = dict(dg.WORKLOAD_PHYS, gravity=0.02)
        s = dg.LSRK.for_state(dg.DeviceMesh.upload(m), Q, precision, phys=dg.make_phys(**phys))
        assert s.kernel == (3 if m.nelem <= sms() else 5), n
        s.run(2, dt)
        assert max(relerr_fields(s.state(), oracle_run(m, Q, dt, 2, phys=phys))) < (1e-12 if precision == 64 else 1e-5), n
        s.close()


@pytest.mark.parametrize("n,gravity", [(5, 0.3), (15, 0.3), (16, 0.3), (5, 0.0), (16, 0.0)])
def test_gravity_at_order_six(n, gravity):
    m = dg.build_mesh(3, 6, (np.linspace(0, 1, n + 1),) * 3, (True, True, False))
    Q = np.zeros((m.Np, 5, m.nelem), order="F")
    Q[:, 3], Q[:, 4] = 1.0, 2.5
    phys = dict(dg.WORKLOAD_PHYS, gravity=gravity)
    s = dg.LSRK.for_state(dg.DeviceMesh.upload(m), Q, 64, phys=dg.make_phys(**phys))
    assert s.kernel == (4 if gravity and m.nelem > 24 * sms() else 1)
    if n == 5:
        s.run(2, 1e-4)
        assert max(relerr_fields(s.state() + 1.0, oracle_run(m, Q, 1e-4, 2, phys=phys) + 1.0)) < 1e-12
    s.close()
