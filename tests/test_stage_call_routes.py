"""Stage calls and runs take the same kernels, and report them.

Bit for bit: a stage run in two halves against the stage in one call; a run of a graph
of programmatic launches against plainly launched stage calls; a run under the
kernel that the solver reports against a run under its default."""
import ctypes as C
import math

import numpy as np
import pytest

from conftest import cuda_available
from dg_cases import vortex_case
from canary_b200 import _lib, dg, ic
from canary_b200._lib import check
from canary_b200.metric import warp_sinusoidal

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not cuda_available(), reason="needs a CUDA GPU")]


def case(dim, N, n):
    if dim == 2:
        return (*vortex_case(N, n), 1e-4)
    m = dg.build_mesh(3, N, (np.linspace(0, 2 * math.pi, n + 1),) * 3, (True, True, False),
                      meshwarp=lambda X: warp_sinusoidal(X, 0.05))
    Q = np.asfortranarray(np.stack(ic.fourier_state(*m.coords(), seed=N), axis=1))
    return m, Q, 0.1 * ic.fourier_dt(Q, N, h=2 * math.pi / n)


def solver(m, Q, precision, phys):
    off = np.zeros(Q.shape[1]) if phys["visc"] > 0 and m.dim == 3 and m.N > 7 else None
    return dg.LSRK.for_state(dg.DeviceMesh.upload(m), Q, precision, phys=dg.make_phys(**phys), offset=off)


def state(s):
    import torch
    check(_lib.lib().cb_solver_settle(s._h))
    torch.cuda.synchronize()
    return s.state()


# (2-D: the heights reach 10, so that gravity 0.02 keeps the pressure positive)
# the second size of a shape lies above the block count at which the small-mesh form
# ends (148 blocks FP64, 592 FP32)
@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("gravity", [0.0, 0.02])
@pytest.mark.parametrize("dim,N,n", [(2, 1, 5), (2, 4, 10), (2, 4, 42), (2, 5, 6), (2, 7, 12), (2, 10, 7), (3, 1, 3),
                                     (3, 3, 4), (3, 4, 4), (3, 5, 4), (3, 6, 3), (3, 7, 3), (3, 8, 3), (3, 9, 2)])
def test_split_stage_equals_the_stage(dim, N, n, gravity, precision):
    m, Q, dt = case(dim, N, n)
    phys = dict(dg.WORKLOAD_PHYS, gravity=gravity)
    a, b = (solver(m, Q, precision, phys) for _ in range(2))
    nxt = C.c_void_p()
    check(_lib.lib().cb_solver_set_split(b._h, m.nelem // 3))
    for k in range(6):
        check(_lib.lib().cb_solver_stage(a._h, k % 5, dt, C.byref(nxt)))
        for half in (0, 1):
            check(_lib.lib().cb_solver_stage_split(b._h, k % 5, dt, half, C.byref(nxt)))
    assert np.array_equal(state(a), state(b))
    a.close()
    b.close()


# chained launches by kernel: the small-mesh form, the grouped stage above eight
# blocks an SM (3-D N=4 FP32, two elements a block: 14^3), the pipelined, lean,
# tensor-core and grid-line stages, both viscous passes of each
@pytest.mark.parametrize("dim,N,n,precision,visc", [
    (2, 4, 10, 64, 0.0), (2, 7, 40, 64, 0.0), (2, 4, 60, 32, 0.0), (2, 7, 30, 64, 0.02), (2, 4, 20, 32, 0.02),
    (3, 3, 9, 64, 0.0), (3, 4, 14, 32, 0.0), (3, 4, 8, 64, 0.0), (3, 5, 8, 64, 0.0), (3, 7, 8, 64, 0.0),
    (3, 7, 8, 32, 0.0), (3, 10, 4, 64, 0.0), (3, 3, 4, 64, 0.02), (3, 3, 17, 32, 0.02), (3, 5, 4, 32, 0.02),
    (3, 7, 10, 64, 0.02), (3, 5, 10, 32, 0.02), (3, 6, 4, 64, 0.02)])
def test_run_equals_stage_calls(dim, N, n, precision, visc):
    m, Q, dt = case(dim, N, n)
    a, b = (solver(m, Q, precision, dict(dg.WORKLOAD_PHYS, visc=visc)) for _ in range(2))
    a.run(4, dt)
    nxt = C.c_void_p()
    for k in range(20):
        check(_lib.lib().cb_solver_stage(b._h, k % 5, dt, C.byref(nxt)))
    assert np.array_equal(state(a), state(b))
    a.close()
    b.close()


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("gravity", [0.0, 0.02])
@pytest.mark.parametrize("dim,N,n,visc", [(2, 4, 10, 0.0), (2, 4, 42, 0.0), (2, 4, 10, 0.02), (3, 2, 4, 0.0),
                                          (3, 4, 4, 0.0), (3, 6, 4, 0.0), (3, 7, 3, 0.0), (3, 8, 2, 0.0), (3, 8, 7, 0.0),
                                          (3, 10, 2, 0.0), (3, 10, 6, 0.0), (3, 1, 5, 0.02), (3, 5, 3, 0.02),
                                          (3, 4, 12, 0.02), (3, 8, 3, 0.02)])
def test_the_reported_kernel_is_the_one_that_runs(dim, N, n, visc, gravity, precision):
    m, Q, dt = case(dim, N, n)
    phys = dict(dg.WORKLOAD_PHYS, visc=visc, gravity=gravity)
    a, b = (solver(m, Q, precision, phys) for _ in range(2))
    b.set_kernel(b.kernel)
    assert b.kernel == a.kernel
    for s in (a, b):
        s.run(3, dt)
    assert np.array_equal(a.state(), b.state())
    a.close()
    b.close()
