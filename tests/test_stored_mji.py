"""The viscous passes scale the gradient by the caller's MJI, as the update does,
not by a reciprocal of MJ: a caller may pass geometry whose MJI is not 1/MJ (a
filtered or masked inverse mass).  Against the oracle on the same geometry; the bars
are those of the viscous passes (FP64 1e-12, FP32 1e-5 relative L2 per field)."""
import math

import numpy as np
import pytest

from conftest import cuda_available
from dg_cases import oracle_run, relerr_fields
from canary_b200 import dg, ic
from canary_b200.metric import warp_sinusoidal

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not cuda_available(), reason="needs a CUDA GPU")]


@pytest.mark.parametrize("precision,tol", [(64, 1e-12), (32, 1e-5)])
@pytest.mark.parametrize("N,n", [(1, 4), (4, 3), (5, 6), (7, 2), (8, 2), (10, 2)])
def test_gradient_is_scaled_by_the_stored_mji(N, n, precision, tol):
    m = dg.build_mesh(3, N, (np.linspace(0, 2 * math.pi, n + 1),) * 3, (True, True, False),
                      meshwarp=lambda X: warp_sinusoidal(X, 0.05))
    m.vgeo = np.array(m.vgeo, order="F")
    scale = np.random.default_rng(N).uniform(0.5, 1.0, (m.Np, m.nelem))
    m.vgeo[:, 10, :] *= scale  # MJI: fields are nine metric terms, MJ, MJI, coordinates
    Q = np.asfortranarray(np.stack(ic.fourier_state(*m.coords(), seed=N), axis=1))
    dt = 0.1 * ic.fourier_dt(Q, N, h=2 * math.pi / n)
    phys = dict(dg.WORKLOAD_PHYS, visc=0.1)
    ref = oracle_run(m, Q, dt, 3, phys=phys)
    off = np.zeros(5) if precision == 64 or N > 7 else None
    for kernel in (0, 1, 5):  # the shape's default, the pipelined passes, the grid-line passes
        s = dg.LSRK.for_state(dg.DeviceMesh.upload(m), Q, precision, phys=dg.make_phys(**phys), offset=off)
        s.set_kernel(kernel)
        s.run(3, dt)
        assert max(relerr_fields(s.state(), ref)) < tol, kernel
        s.close()
