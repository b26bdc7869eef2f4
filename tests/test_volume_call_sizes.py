"""volumerhs in 3-D on both sides of the mesh size from which it runs by grid lines
(1, 3 or 8 blocks of the grouped kernel per SM, by order), with odd element counts that
leave partial blocks.  Against the oracle; 1e-13 (FP64) and 1e-5 (FP32) relative L2 per
field, the bars of single calls."""
import math

import numpy as np
import pytest

from conftest import cuda_available
from dg_cases import oracle_phys, relerr_fields
from oracle import pyoracle as O
from canary_b200 import dg, ic
from canary_b200.metric import warp_sinusoidal

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not cuda_available(), reason="needs a CUDA GPU")]


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("N,n", [(2, (7, 5, 3)), (3, (7, 7, 9)), (3, (13, 12, 13)), (4, (7, 7, 7)), (4, (13, 13, 15)),
                                 (5, (7, 5, 7)), (5, (9, 7, 9)), (6, (5, 5, 5)), (6, (9, 7, 9)), (7, (5, 5, 5)),
                                 (7, (9, 7, 9)), (8, (5, 5, 3)), (8, (7, 5, 5)), (9, (5, 5, 3)), (9, (7, 5, 5)),
                                 (10, (5, 3, 3)), (10, (7, 5, 5))])
def test_volume_integral(N, n, precision):
    m = dg.build_mesh(3, N, tuple(np.linspace(0, 2 * math.pi, k + 1) for k in n), (True, True, False),
                      meshwarp=lambda X: warp_sinusoidal(X, 0.05))
    real = np.float64 if precision == 64 else np.float32
    f = ic.fourier_state(*m.coords(), seed=N)
    h = {k: np.asfortranarray(np.asarray(v).astype(real)) for k, v in
         (("Q", np.stack(f, axis=1)), ("vgeo", m.vgeo), ("D", m.D))}
    h["r"] = np.asfortranarray(np.random.default_rng(N).standard_normal(h["Q"].shape).astype(real))
    d = {k: dg.to_device(v) for k, v in h.items()}
    phys = dict(dg.WORKLOAD_PHYS, gravity=0.02)
    w = {k: np.asfortranarray(v.astype(np.float64)) for k, v in h.items()}
    O.volumerhs(3, N, w["r"], w["Q"], w["vgeo"], w["D"], oracle_phys(phys), 4)
    dg.volumerhs(3, N, d["r"], d["Q"], d["vgeo"], d["D"], m.nelem, dg.make_phys(**phys))
    out = dg.from_device(d["r"], h["Q"].shape).astype(np.float64)
    assert max(relerr_fields(out, w["r"])) < (1e-13 if precision == 64 else 1e-5)


# elements on both sides of the block count from which the march runs
@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("gravity", [0.0, 0.02])
@pytest.mark.parametrize("N,few,many", [(2, 33, 7000), (3, 33, 4500), (4, 301, 2900), (5, 101, 1500), (6, 51, 700),
                                        (7, 37, 700), (8, 31, 400), (9, 21, 300), (10, 17, 300)])
def test_an_element_does_not_depend_on_the_count(N, few, many, gravity, precision):
    """Bit for bit: the first elements of a large call against a call for them alone."""
    import torch
    real = torch.float64 if precision == 64 else torch.float32
    g = torch.Generator(device="cuda").manual_seed(N)
    Np = (N + 1) ** 3
    def rand(*shape):
        return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)
    Q = rand(many, 5, Np) - 0.5
    Q[:, 3] += 1.5  # density and total energy: positive pressure
    Q[:, 4] += 4.0
    Q, vgeo, D, r = (t.to(real).reshape(-1).contiguous() for t in
                     (Q, rand(many, 14, Np) + 0.1, rand(N + 1, N + 1) - 0.5, rand(many, 5, Np) - 0.5))
    a, b = r.clone(), r.clone()
    ph = dg.make_phys(**dict(dg.WORKLOAD_PHYS, gravity=gravity))
    dg.volumerhs(3, N, a, Q, vgeo, D, many, ph)
    dg.volumerhs(3, N, b, Q, vgeo, D, few, ph)
    k = few * 5 * Np
    assert torch.isfinite(a).all()
    assert torch.equal(a[:k], b[:k])
    assert torch.equal(b[k:], r[k:])
