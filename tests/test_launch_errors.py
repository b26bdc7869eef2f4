"""An error of one call is returned by that call and not by a later one.

A stage call on a stream whose capture was invalidated is refused by the runtime (no
kernel runs); once the capture has been ended, other calls work."""
import ctypes as C

import pytest

from conftest import cuda_available
from dg_cases import fourier_case
from canary_b200 import _lib, dg
from canary_b200._lib import CB_OK

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not cuda_available(), reason="needs a CUDA GPU")]


# the grouped small-mesh, pipelined, lean, tensor-core and column-march stages
@pytest.mark.parametrize("N,precision", [(3, 32), (5, 64), (3, 64), (7, 64), (7, 32), (10, 64)])
def test_a_refused_stage_leaves_no_error_behind(N, precision):
    import torch
    m, Q, dt = fourier_case(N, 2)
    stream = torch.cuda.Stream()
    dm = dg.DeviceMesh.upload(m)
    s = dg.LSRK.for_state(dm, Q, precision, stream=stream)
    r = torch.zeros_like(dg.to_device(Q))
    q = dg.to_device(Q)
    torch.cuda.synchronize()
    rt, h, nxt, graph = C.CDLL("libcudart.so.12"), C.c_void_p(stream.cuda_stream), C.c_void_p(), C.c_void_p()
    assert rt.cudaStreamBeginCapture(h, 1) == 0  # thread-local mode
    assert rt.cudaStreamSynchronize(h) != 0      # not allowed: invalidates the capture
    refused = _lib.lib().cb_solver_stage(s._h, 0, dt, C.byref(nxt))
    rt.cudaStreamEndCapture(h, C.byref(graph))
    rt.cudaGetLastError()
    assert refused != CB_OK
    dg.updatesolution(3, N, r, None, q, dm.vgeo, m.nelem, 0.0, 0.0, 0.0)
    torch.cuda.synchronize()
    s.close()
