"""Timed workloads of the nodal-DG path, each through a public entry point.

Three kinds of case:

  solver    one mesh advanced by LSRK.run: isentropic vortex (2-D), Euler and
            LDG Navier-Stokes cubes (3-D, warped, periodic), and the bubble
            set-up of the reference's drivers (walls below and above, gravity,
            its physical constants)
  calls     one RK stage through the per-kernel calls, as a host program that
            keeps its own time loop makes it
  ensemble  many independent instances of uneven order and size in one Batch

A pass advances the state in place and returns it with the residual carry, so
repeated passes follow the solution in time; the time steps are small enough
that it stays smooth.

`exact` evaluates the same scheme with plain torch operations in FP64 on the
same inputs (mesh arrays and initial state).
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "canary.jl_b200"))

from canary_b200 import dg, ic  # noqa: E402
from canary_b200.batch import Batch, BatchMesh  # noqa: E402

TWO_PI = 2.0 * math.pi
VISC = 1e-3  # viscosity of the Navier-Stokes cases
RKA = (0.0, -567301805773.0 / 1357537059087.0, -2404267990393.0 / 2016746695238.0,
       -3550918686646.0 / 2091501179385.0, -1275806237668.0 / 842570457699.0)
RKB = (1432997174477.0 / 9575080441755.0, 5161836677717.0 / 13612068292357.0,
       1720146321549.0 / 2090206949498.0, 3134564353537.0 / 4481467310338.0,
       2277821191437.0 / 14882151754819.0)


def _solver(name, dim, N, n, bits, steps, flow):
    return {"name": name, "kind": "solver", "flow": flow, "dim": dim, "N": N, "nx": n[0], "ny": n[1],
            "nz": n[2] if dim == 3 else 0, "bits": bits, "steps": steps}


def listed():
    return [
        # the 2-D verification run: tiny, all launch latency
        _solver("vortex2d_n4_10x10_f64", 2, 4, (10, 10), 64, 20, "euler"),
        # a small 3-D request of the served mix, as one solver
        _solver("euler3d_n3_8_f32", 3, 3, (8, 8, 8), 32, 10, "euler"),
        # the precision study: low order, FP32
        _solver("euler3d_n4_32_f32", 3, 4, (32, 32, 32), 32, 4, "euler"),
        # the headline workload and its FP32 form
        _solver("euler3d_n7_32_f64", 3, 7, (32, 32, 32), 64, 4, "euler"),
        _solver("euler3d_n7_32_f32", 3, 7, (32, 32, 32), 32, 4, "euler"),
        # the reference drivers' set-up: walls, gravity, a ragged brick, one
        # step a call (a program that looks at the state after every step)
        _solver("bubble3d_n6_ragged_f64", 3, 6, (23, 17, 19), 64, 1, "bubble"),
        # the precision study: highest order
        _solver("euler3d_n10_20_f64", 3, 10, (20, 20, 20), 64, 2, "euler"),
        # Navier-Stokes: middle order FP64, the order of the headline in FP32,
        # the highest order in FP32
        _solver("ns3d_n4_24_f64", 3, 4, (24, 24, 24), 64, 4, "ns"),
        _solver("ns3d_n7_16_f32", 3, 7, (16, 16, 16), 32, 4, "ns"),
        _solver("ns3d_n10_16_f32", 3, 10, (16, 16, 16), 32, 2, "ns"),
        # volumerhs + fluxrhs + updatesolution from a host's own time loop
        {"name": "calls3d_n5_ragged_f64", "kind": "calls", "flow": "euler", "dim": 3, "N": 5, "nx": 24, "ny": 20,
         "nz": 22, "bits": 64},
        # a quarter of the 512-instance vortex ensemble, FP32
        {"name": "ensemble_vortex_128_f32", "kind": "ensemble", "flow": "euler", "dim": 2, "count": 128, "sizes": 0,
         "bits": 32, "steps": 4},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """A case of the same kinds: orders 2 to 10, sizes over the logarithm up to
    the listed ones, both precisions."""
    limit = max(work(c)["bytes"] for c in listed())
    while True:
        u = rng.random()
        bits = rng.choice((64, 32))
        if u < 0.15:
            dim = rng.choice((2, 2, 3))
            c = {"kind": "ensemble", "flow": rng.choice(("euler", "ns")) if dim == 3 else "euler", "dim": dim,
                 "count": _log_int(rng, 4, 128) if dim == 2 else _log_int(rng, 2, 24),
                 "sizes": rng.randrange(1, 1 << 20), "bits": bits, "steps": 2 * rng.randint(1, 3)}
        elif u < 0.30:
            flow = rng.choice(("euler", "euler", "bubble", "ns"))
            dim = rng.choice((2, 3, 3)) if flow == "euler" else 3
            n = _log_int(rng, 4, 32) if dim == 3 else _log_int(rng, 8, 200)
            c = {"kind": "calls", "flow": flow, "dim": dim, "N": rng.randint(2, 10), "nx": n,
                 "ny": max(3, n - rng.randint(0, 3)), "nz": max(3, n - rng.randint(0, 3)) if dim == 3 else 0,
                 "bits": 64 if flow == "ns" else bits}
        elif u < 0.45:
            n = _log_int(rng, 8, 200)
            c = _solver("", 2, rng.randint(2, 10), (n, max(4, n - rng.randint(0, 5))), bits, rng.randint(1, 20),
                        "euler")
        else:
            flow = rng.choice(("euler", "euler", "euler", "bubble", "ns", "ns"))
            n = _log_int(rng, 4, 32)
            c = _solver("", 3, rng.randint(2, 10), (n, max(3, n - rng.randint(0, 3)), max(3, n - rng.randint(0, 3))),
                        bits, rng.randint(1, 6), flow)
        c.pop("name", None)
        if work(c)["bytes"] <= limit and (c["kind"] == "ensemble" or _held(c) < 12e9):
            return c


# ------------------------------------------------------------------- sizes
def _counts(dim, N):
    """(state fields, nodes, face nodes of all faces) per element."""
    Nq = N + 1
    return (5 if dim == 3 else 4), Nq ** dim, 2 * dim * Nq ** (dim - 1)


def _elems(c):
    return [c["nx"], c["ny"]] + ([c["nz"]] if c["dim"] == 3 else [])


def _held(c):
    """Device bytes of one state (geometry in FP64, maps, states, gradient)."""
    ns, Np, nf = _counts(c["dim"], c["N"])
    E, d = math.prod(_elems(c)), c["dim"]
    return E * (Np * 8 * ((14 if d == 3 else 8) * 1.5 + 4 * ns + 2 * d * ns) + nf * 8 * 10)


def _members(c):
    """(order, elements a side) of an ensemble's instances: the vortex
    ensemble in 2-D, the served stream's 3-D ranges in 3-D."""
    if c["dim"] == 2:
        return [(p["N"], p["n_side"]) for p in ic.vortex_ensemble(c["count"], c["sizes"])]
    g = np.random.Generator(np.random.PCG64(c["sizes"]))
    return [(int(g.integers(3, 8)), int(g.integers(4, 17))) for _ in range(c["count"])]


def _stage_work(dim, N, E, bits, visc):
    """Bytes and operations of one RK stage of one mesh: state and carry read
    and written, metric, MJ, MJI and the face normals and sMJ read, once.  The
    viscous form has the same inputs and outputs (its gradient is an
    intermediate) and about three times the contractions."""
    ns, Np, nf = _counts(dim, N)
    words = Np * (4 * ns + dim * dim + 2) + nf * (dim + 1)
    flops = Np * ns * dim * 2 * (N + 1) * ((2 + dim) if visc else 1) + Np * 60 + nf * 80
    return bits // 8 * words * E, flops * E


def work(case):
    c = case
    visc = c["flow"] == "ns"
    if c["kind"] == "ensemble":
        parts = [_stage_work(c["dim"], N, n ** c["dim"], c["bits"], visc) for N, n in _members(c)]
    else:
        parts = [_stage_work(c["dim"], c["N"], math.prod(_elems(c)), c["bits"], visc)]
    stages = 1 if c["kind"] == "calls" else 5 * c["steps"]
    return {"bytes": stages * sum(p[0] for p in parts), "flops": stages * sum(p[1] for p in parts)}


# ------------------------------------------------------------------ inputs
def _phys(c):
    if c["flow"] == "bubble":
        return dict(dg.REFERENCE_PHYS)
    return dict(dg.WORKLOAD_PHYS, visc=VISC if c["flow"] == "ns" else 0.0)


def _mesh(flow, dim, N, n):
    """Device mesh: [0,10]^2 in 2-D, the warped periodic cube [0,2pi]^3 in 3-D,
    a 1 km box with walls at the bottom and the top for the bubble."""
    if flow == "bubble":
        return dg.DeviceMesh.build(dim, N, [np.linspace(0.0, 1000.0, k + 1) for k in n],
                                   (True,) * (dim - 1) + (False,))
    L = 10.0 if dim == 2 else TWO_PI
    return dg.DeviceMesh.build(dim, N, [np.linspace(0.0, L, k + 1) for k in n], (True,) * dim,
                               warp_amp=0.05 if dim == 3 else 0.0)


def _fields(flow, dim, X, seed, vortex=None):
    """Conserved fields on the nodes X: an isentropic vortex (2-D), a random
    Fourier state of velocity peak 0.1 (3-D), a warm bubble in air at rest."""
    g = np.random.Generator(np.random.PCG64(seed))
    if flow == "bubble":
        cx, cy, cz, r0 = g.uniform(300, 700), g.uniform(300, 700), g.uniform(300, 500), g.uniform(150, 300)
        x, y, z = X
        r = torch.sqrt((x - cx) ** 2 + (y - cy) ** 2 + (z - cz) ** 2)
        warm = torch.where(r < r0, 0.5 * (1.0 + torch.cos(math.pi * r / r0)), torch.zeros_like(r))
        p = 1e5 * torch.exp(-1.2 * 10.0 * z / 1e5)
        rho = 1.2 * torch.exp(-1.2 * 10.0 * z / 1e5) / (1.0 + 0.01 * warm)
        u, v = 5.0 * torch.sin(TWO_PI * y / 1000.0), 5.0 * torch.sin(TWO_PI * x / 1000.0 + float(g.uniform(0, 6)))
        E = p * (717.5 / 287.17) + 0.5 * rho * (u * u + v * v) + rho * 10.0 * z
        return [rho * u, rho * v, torch.zeros_like(rho), rho, E]
    if dim == 2:
        beta, xc, yc = vortex or (float(g.uniform(1, 5)), float(g.uniform(2, 8)), float(g.uniform(2, 8)))
        return list(ic.isentropic_vortex_t(X[0], X[1], beta, xc, yc))
    return list(ic.fourier_state_t(X[0], X[1], X[2], seed=seed % (1 << 32), vel_peak=0.1))


def _offset(flow, dim, N, bits):
    """Constants the stored FP32 state is relative to (the free stream); the
    highest viscous orders and FP64 have none."""
    if bits == 64 or (flow == "ns" and dim == 3 and N > 7):
        return [0.0] * (5 if dim == 3 else 4)
    if flow == "bubble":
        return [0.0, 0.0, 0.0, 1.2, 2.5e5]
    return [1.0, 0.0, 1.0, 3.0] if dim == 2 else [0.0, 0.0, 0.0, 1.0, 2.5]


def _dt(flow, dim, N, n):
    if flow == "bubble":
        return 0.1 * (1000.0 / max(n)) / (N * N * 400.0)
    if dim == 2:
        return min(0.002, 0.2 * (10.0 / max(n)) / (N * N * 3.0))
    return min(1e-4, 0.2 * (TWO_PI / max(n)) / (N * N * 1.6))


def _inputs(flow, dim, N, n, bits, seed):
    """(device mesh, stored state, offset, dt) of one instance."""
    dm = _mesh(flow, dim, N, n)
    off = _offset(flow, dim, N, bits)
    real = torch.float64 if bits == 64 else torch.float32
    Q = ic.device_state(_fields(flow, dim, dm.coords(), seed), real, off)
    return dm, Q, off, _dt(flow, dim, N, n)


def _arena(c):
    """First value of every instance of an ensemble and one zeroed array for
    all their states, each on a 16-byte boundary."""
    begin, total = [], 0
    for N, n in _members(c):
        ns, Np, _ = _counts(c["dim"], N)
        begin.append(total)
        total += -(-ns * Np * n ** c["dim"] // 4) * 4
    real = torch.float64 if c["bits"] == 64 else torch.float32
    return begin, torch.zeros(total, dtype=real, device="cuda")


def prepare(case, seed):
    c = case
    phys = dg.make_phys(**_phys(c))
    if c["kind"] == "ensemble":
        b = Batch(c["bits"], max_instances=c["count"], phys=phys)
        meshes = {}
        begin, states = _arena(c)
        carries = torch.zeros_like(states)
        for i, (N, n) in enumerate(_members(c)):
            dm, Q, off, dt = _inputs(c["flow"], c["dim"], N, (n,) * c["dim"], c["bits"], seed * 1009 + i)
            if (N, n) not in meshes:  # instances of one order and size share their mesh
                meshes[N, n] = BatchMesh(dm, c["bits"])
            own = slice(begin[i], begin[i] + Q.numel())
            states[own] = Q
            b.add(meshes[N, n], states[own], carries[own], dt, 10 ** 9, off)
        return {"case": c, "batch": b, "meshes": meshes, "Q": states, "rhs": carries}
    dm, Q, off, dt = _inputs(c["flow"], c["dim"], c["N"], _elems(c), c["bits"], seed)
    rhs = torch.zeros_like(Q)
    if c["kind"] == "solver":
        s = dg.LSRK(dm, Q, rhs, c["bits"], phys)
        if any(off):
            s.set_offset(off)
        return {"case": c, "solver": s, "Q": Q, "rhs": rhs, "dt": dt}
    geo = {k: getattr(dm, k) for k in ("vgeo", "sgeo", "D")}
    if c["bits"] == 32:  # the FP32 calls take FP32 geometry and the full state
        geo = {k: v.float() for k, v in geo.items()}
        Q = (Q.view(-1, len(off), (c["N"] + 1) ** c["dim"]).double()
             + torch.tensor(off, dtype=torch.float64, device=Q.device)[None, :, None]).float().reshape(-1)
    st = {"case": c, "dm": dm, "Q": Q, "rhs": rhs, "dt": dt, "phys": phys, **geo}
    if c["flow"] == "ns":
        st["grad"] = torch.zeros(Q.numel() * c["dim"], dtype=torch.float64, device=Q.device)
        st["rhs_grad"] = torch.zeros_like(st["grad"])
    return st


def run(state):
    c = state["case"]
    if c["kind"] == "solver":
        state["solver"].run(c["steps"], state["dt"])
        return {"Q": state["Q"], "rhs": state["rhs"]}
    if c["kind"] == "ensemble":
        state["batch"].run(c["steps"])  # an even number: every state is back in its caller's buffer
        return {"Q": state["Q"], "rhs": state["rhs"]}
    d, N, dm, Q, rhs, ph = c["dim"], c["N"], state["dm"], state["Q"], state["rhs"], state["phys"]
    E = dm.mesh.nelem
    maps = (dm.vmapM, dm.vmapP, dm.elemtobndy)
    dg.volumerhs(d, N, rhs, Q, state["vgeo"], state["D"], E, ph)
    dg.fluxrhs(d, N, rhs, Q, state["sgeo"], state["vgeo"], E, *maps, ph)
    rg = None
    if c["flow"] == "ns":
        g, rg = state["grad"], state["rhs_grad"]
        dg.volume_grad(d, N, rg, Q, state["vgeo"], state["D"], E, ph)
        dg.flux_grad(d, N, rg, Q, state["sgeo"], state["vgeo"], E, *maps, ph)
        dg.update_gradQ(d, N, g, rg, state["vgeo"], E)
        dg.volume_div(d, N, rg, g, Q, state["vgeo"], state["D"], E, ph)
        dg.flux_div(d, N, rg, g, Q, state["sgeo"], E, *maps, ph)
    dg.updatesolution(d, N, rhs, rg, Q, state["vgeo"], E, RKA[1], RKB[0], state["dt"], ph.visc)
    out = {"Q": Q, "rhs": rhs}
    if rg is not None:
        out["gradQ"] = state["grad"]
    return out


# ------------------------------------------------- the scheme in plain torch
class _Plain:
    """One mesh's LSRK stage in FP64 with plain torch operations."""

    def __init__(self, dm, dim, N, phys):
        self.dim, self.N, self.p = dim, N, phys
        Nq = N + 1
        self.ns, self.Np, _ = _counts(dim, N)
        self.Nfp, self.nf = Nq ** (dim - 1), 2 * dim
        E = self.E = dm.mesh.nelem
        self.vgeo = dm.vgeo.view(E, 14 if dim == 3 else 8, self.Np)
        self.sgeo = dm.sgeo.view(E, self.nf, self.Nfp, 5 if dim == 3 else 4)
        self.vM = dm.vmapM.view(E, self.nf, self.Nfp) - 1
        self.vP = dm.vmapP.view(E, self.nf, self.Nfp) - 1
        self.wall = dm.elemtobndy.view(E, self.nf) == 1
        self.D = dm.D.view(Nq, Nq)  # [i, m] = D[m, i]
        self.MJ, self.MJI = self.vgeo[:, dim * dim], self.vgeo[:, dim * dim + 1]
        self.height = self.vgeo[:, dim * dim + 2 + dim - 1]

    def metric(self, r, c):
        return self.vgeo[:, r + self.dim * c]

    def pressure(self, q, h):
        d = self.dim
        ke = sum(q[c] * q[c] for c in range(d)) / (2.0 * q[d])
        return (self.p["R_gas"] / self.p["c_v"]) * (q[d + 1] - ke - q[d] * self.p["gravity"] * h)

    def flux(self, q, P):
        d = self.dim
        f = [[q[a] * q[c] / q[d] + (P if a == c else 0.0) for c in range(d)] for a in range(d)]
        f.append([q[c] for c in range(d)])
        f.append([q[c] / q[d] * (q[d + 1] + P) for c in range(d)])
        return f

    def contract(self, F, r):
        """Sum over m of D[m, index r] F[.., m, ..] along reference direction r."""
        Nq = self.N + 1
        V = F.reshape((self.E,) + (Nq,) * self.dim)  # (e, [k,] j, i)
        ax = self.dim - r
        return torch.movedim(torch.tensordot(V, self.D, dims=([ax], [1])), -1, ax).reshape(self.E, self.Np)

    def at(self, field, idx):
        return field.reshape(-1)[idx.reshape(-1)].view(idx.shape)

    def scatter(self, out, f, v):
        out.view(-1).index_add_(0, self.vM[:, f].reshape(-1), v.reshape(-1))

    def inviscid(self, q):
        d, ns = self.dim, self.ns
        P = self.pressure(q, self.height)
        f = self.flux(q, P)
        R = []
        for s in range(ns):
            acc = torch.zeros_like(q[0])
            for r in range(d):
                acc += self.contract(self.MJ * sum(self.metric(r, c) * f[s][c] for c in range(d)), r)
            R.append(acc)
        R[d - 1] -= self.MJ * q[d] * self.p["gravity"]
        g = self.p["gamma"]
        for f_ in range(self.nf):
            n = [self.sgeo[:, f_, :, c] for c in range(d)]
            sMJ, w = self.sgeo[:, f_, :, d], self.wall[:, f_, None]
            qM = [self.at(x, self.vM[:, f_]) for x in q]
            qP = [self.at(x, self.vP[:, f_]) for x in q]
            un = sum(n[c] * qM[c] for c in range(d))
            qP = [torch.where(w, qM[s] - 2.0 * un * n[s] if s < d else qM[s], qP[s]) for s in range(ns)]
            PM, PP = self.at(P, self.vM[:, f_]), self.at(P, self.vP[:, f_])
            PP = torch.where(w, PM, PP)
            fM, fP = self.flux(qM, PM), self.flux(qP, PP)
            sp = [abs(sum(n[c] * x[c] for c in range(d))) / x[d] + torch.sqrt(g * p / x[d])
                  for x, p in ((qM, PM), (qP, PP))]
            lam = torch.maximum(*sp)
            for s in range(ns):
                a = sum(n[c] * (fM[s][c] + fP[s][c]) for c in range(d))
                self.scatter(R[s], f_, -sMJ * 0.5 * (a - lam * (qP[s] - qM[s])))
        return R

    def primitives(self, q, P):
        d = self.dim
        return [q[c] / q[d] for c in range(d)] + [q[d], P / (self.p["R_gas"] * q[d])]

    def stress(self, g, vel):
        d = self.dim
        div = sum(g[c][c] for c in range(d))
        out = [[2.0 * g[a][a] + self.p["lam"] * div if a == c else g[a][c] + g[c][a] for c in range(d)]
               for a in range(d)]
        out.append([torch.zeros_like(div)] * d)
        out.append([sum(vel[a] * out[a][c] for a in range(d)) + self.p["c_p"] / self.p["Pr"] * g[d + 1][c]
                    for c in range(d)])
        return out

    def gradient(self, q):
        d, ns = self.dim, self.ns
        pr = self.primitives(q, self.pressure(q, self.height))
        G = [[-sum(self.contract(self.MJ * self.metric(r, c) * pr[s], r) for r in range(d)) for c in range(d)]
             for s in range(ns)]
        for f_ in range(self.nf):
            n = [self.sgeo[:, f_, :, c] for c in range(d)]
            sMJ, w = self.sgeo[:, f_, :, d], self.wall[:, f_, None]
            pM = [self.at(x, self.vM[:, f_]) for x in pr]
            pP = [self.at(x, self.vP[:, f_]) for x in pr]
            un = sum(n[c] * pM[c] for c in range(d))
            for s in range(ns):
                wallv = pM[s] - 2.0 * un * n[s] if s < d else pM[s]
                avg = 0.5 * (pM[s] + torch.where(w, wallv, pP[s]))
                for c in range(d):
                    self.scatter(G[s][c], f_, sMJ * n[c] * avg)
        return [[x * self.MJI for x in row] for row in G]

    def viscous(self, q, G):
        """Divergence of the viscous flux (to be multiplied by visc)."""
        d, ns = self.dim, self.ns
        vel = [q[c] / q[d] for c in range(d)]
        fv = self.stress(G, vel)
        R = [-sum(self.contract(self.MJ * sum(self.metric(r, c) * fv[s][c] for c in range(d)), r) for r in range(d))
             for s in range(ns)]
        for f_ in range(self.nf):
            n = [self.sgeo[:, f_, :, c] for c in range(d)]
            sMJ, w = self.sgeo[:, f_, :, d], self.wall[:, f_, None]
            gM = [[self.at(x, self.vM[:, f_]) for x in row] for row in G]
            vM = [self.at(x, self.vM[:, f_]) for x in vel]
            un = sum(n[c] * vM[c] for c in range(d))
            gP, vP = [], []
            for s in range(ns):
                sn = sum(n[c] * gM[s][c] for c in range(d))
                gP.append([torch.where(w, gM[s][c] if s == d + 1 else gM[s][c] - 2.0 * sn * n[c],
                                       self.at(G[s][c], self.vP[:, f_])) for c in range(d)])
            for c in range(d):
                vP.append(torch.where(w, vM[c] - 2.0 * un * n[c], self.at(vel[c], self.vP[:, f_])))
            fM, fP = self.stress(gM, vM), self.stress(gP, vP)
            for s in range(ns):
                self.scatter(R[s], f_, sMJ * 0.5 * sum(n[c] * (fM[s][c] + fP[s][c]) for c in range(d)))
        return R

    def stage(self, q, rhs, rka, rkb, dt):
        """New state and carry; the gradient as well in the viscous form."""
        R, G = self.inviscid(q), None
        if self.p["visc"] > 0:
            G = self.gradient(q)
            R = [a + self.p["visc"] * b for a, b in zip(R, self.viscous(q, G))]
        R = [a + b for a, b in zip(R, rhs)]
        return [a + rkb * dt * r * self.MJI for a, r in zip(q, R)], [rka * r for r in R], G

    def step(self, q, dt, steps):
        rhs = [torch.zeros_like(x) for x in q]
        for _ in range(steps):
            for k in range(5):
                q, rhs, _ = self.stage(q, rhs, RKA[(k + 1) % 5], RKB[k], dt)
        return q


def _full(Q, off, E, Np):
    V = Q.view(E, len(off), Np).double()
    return [V[:, s] + off[s] for s in range(len(off))]


def _stored(q, off):
    return torch.stack([x - o for x, o in zip(q, off)], dim=1).reshape(-1)


def exact(case, seed):
    c = case
    ph = _phys(c)
    if c["kind"] == "ensemble":
        begin, states = _arena(dict(c, bits=64))
        for i, (N, n) in enumerate(_members(c)):
            dm, Q, off, dt = _inputs(c["flow"], c["dim"], N, (n,) * c["dim"], c["bits"], seed * 1009 + i)
            p = _Plain(dm, c["dim"], N, ph)
            states[begin[i]:begin[i] + Q.numel()] = _stored(p.step(_full(Q, off, p.E, p.Np), dt, c["steps"]), off)
        return {"Q": states, "rhs": None}
    dm, Q, off, dt = _inputs(c["flow"], c["dim"], c["N"], _elems(c), c["bits"], seed)
    p = _Plain(dm, c["dim"], c["N"], ph)
    q = _full(Q, off, p.E, p.Np)
    if c["kind"] == "solver":
        q = p.step(q, dt, c["steps"])
        return {"Q": _stored(q, off), "rhs": None}
    if c["bits"] == 32:
        q = [x.float().double() for x in q]
        off = [0.0] * len(off)
    z = [0.0] * len(off)
    q, rhs, G = p.stage(q, [torch.zeros_like(x) for x in q], RKA[1], RKB[0], dt)
    out = {"Q": _stored(q, z), "rhs": _stored(rhs, z)}
    if G is not None:  # (Np, fields, dim, elements), as the calls keep it
        out["gradQ"] = torch.stack([torch.stack([G[s][k] for s in range(p.ns)], 1) for k in range(p.dim)], 1).reshape(-1)
    return out
