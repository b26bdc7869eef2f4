"""The 3-D stages in which a thread owns grid lines (cb_march.cuh): the viscous
passes of every order and the inviscid stage of N = 9 (FP64) and N = 10.

Element counts (27, 12, 1) leave partial blocks at every order (1 to 32
elements per block).  Tolerances: FP64 against the FP64 oracle 1e-12 relative L2
per field, the bar of the other fused stages; FP32 1e-5, its form's bar (states
of order one rounded once per stage: 15 stages of 6e-8 relative)."""
import math

import numpy as np
import pytest

from conftest import cuda_available
from dg_cases import oracle_run, relerr_fields
from canary_b200 import CanaryError, dg, ic
from canary_b200._lib import CB_ERR_BC
from canary_b200.metric import warp_sinusoidal

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not cuda_available(), reason="needs a CUDA GPU")]


def box(N, n, walls, seed):
    per = (True, not walls, not walls)
    m = dg.build_mesh(3, N, tuple(np.linspace(0, 2 * math.pi, k + 1) for k in n), per,
                      meshwarp=lambda X: warp_sinusoidal(X, 0.05))
    x, y, z = m.coords()
    Q = np.asfortranarray(np.stack(ic.fourier_state(x, y, z, seed=seed), axis=1))
    return m, Q, 0.1 * ic.fourier_dt(Q, N, h=2 * math.pi / max(n))


def run(m, Q, dt, steps, precision, phys, kernel=0):
    s = dg.LSRK.for_state(dg.DeviceMesh.upload(m), Q, precision, phys=dg.make_phys(**phys),
                          offset=np.zeros(5) if precision == 64 or m.N > 7 else None)
    s.set_kernel(kernel)
    s.run(steps, dt)
    out = s.state()
    s.sums()
    s.close()
    return out


@pytest.mark.parametrize("precision,tol", [(64, 1e-12), (32, 1e-5)])
@pytest.mark.parametrize("N,n,walls", [(1, (3, 3, 3), True), (2, (3, 3, 3), True), (3, (3, 3, 3), False), (4, (3, 3, 3), True),
                                       (5, (2, 2, 3), True), (6, (3, 2, 2), True), (7, (3, 3, 3), True),
                                       (8, (3, 2, 2), True), (9, (2, 2, 3), True), (10, (2, 3, 2), True),
                                       (10, (1, 1, 1), True)])
def test_viscous_passes(N, n, walls, precision, tol):
    m, Q, dt = box(N, n, walls, seed=N)
    phys = dict(dg.WORKLOAD_PHYS, visc=0.02, gravity=0.3)
    ref = oracle_run(m, Q, dt, 3, phys=phys)
    assert max(relerr_fields(run(m, Q, dt, 3, precision, phys), ref)) < tol


@pytest.mark.parametrize("precision,tol", [(64, 1e-12), (32, 1e-5)])
@pytest.mark.parametrize("N,n", [(9, (3, 2, 2)), (10, (2, 3, 2)), (10, (1, 1, 1))])
def test_inviscid_stage(N, n, precision, tol):
    m, Q, dt = box(N, n, True, seed=N)
    phys = dict(dg.WORKLOAD_PHYS, gravity=0.3)
    ref = oracle_run(m, Q, dt, 3, phys=phys)
    for kernel in (0, 3):
        assert max(relerr_fields(run(m, Q, dt, 3, precision, phys, kernel), ref)) < tol, kernel


def test_high_viscous_orders_accept_any_boundary_code_at_creation():
    """3-D N >= 8 runs the reference's sequence of passes where the maps give no
    neighbour table: an unknown boundary code is reported by the run, as
    there."""
    m, Q, dt = box(8, (2, 2, 2), True, seed=1)
    m.elemtobndy = np.array(m.elemtobndy, order="F")
    m.elemtobndy[tuple(np.argwhere(m.elemtobndy == 1)[0])] = 2
    s = dg.LSRK.for_state(dg.DeviceMesh.upload(m), Q, 64, phys=dg.make_phys(visc=0.02))
    s.run(2, dt)
    with pytest.raises(CanaryError) as ei:
        s.sums()
    assert ei.value.code == CB_ERR_BC
    s.close()


def test_high_viscous_orders_off_the_neighbour_table():
    """The same orders take face maps of another orientation (one face's vmapP
    reversed), which the neighbour table cannot express; the oracle follows the
    same maps."""
    m, Q, dt = box(8, (2, 2, 2), False, seed=2)
    m.vmapP = np.array(m.vmapP, order="F")
    m.vmapP[:, 0, 0] = m.vmapP[::-1, 0, 0].copy()
    phys = dict(dg.WORKLOAD_PHYS, visc=0.02)
    ref = oracle_run(m, Q, dt, 2, phys=phys)
    assert max(relerr_fields(run(m, Q, dt, 2, 64, phys), ref)) < 1e-12
