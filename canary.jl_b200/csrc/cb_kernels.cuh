// Kernel templates of the nodal-DG hot path and their host launchers.
// Included once per (dim, precision) translation unit; see cb_inst.cuh.
#pragma once
#include "cb_dg.cuh"
#include "cb_march.h"

namespace cb {

// Face-neighbour code of the fused path: for an interior face
// (e2 << 3) | f2 with 0-based neighbour element e2 and face f2;
// NBR_WALL for a reflective wall (elemtobndy == 1).
constexpr int32_t NBR_WALL = -1;

template <typename T>
__device__ __forceinline__ void load_D(T *Ds, const T *__restrict__ D, int nq2) {
  for (int t = threadIdx.x; t < nq2; t += blockDim.x) Ds[t] = D[t];
}

// Reflective wall state (euler3d_set3c.jl:382-389).
template <int DIM, typename T>
__device__ __forceinline__ void wall_state(const T *qM, const T *nrm, T *qP) {
  constexpr int NS = Lay<DIM>::NS;
  T un = nrm[0] * qM[0] + nrm[1] * qM[1];
  if (DIM == 3) un = un + nrm[2] * qM[2];
#pragma unroll
  for (int s = 0; s < NS; ++s) qP[s] = qM[s];
#pragma unroll
  for (int c = 0; c < DIM; ++c) qP[c] = qM[c] - T(2) * un * nrm[c];
}

// ======================================================================
// Stateless volume RHS: rhs += volume integral (volumerhs!).
// ======================================================================
template <int DIM, int Nq, typename T>
__global__ void __launch_bounds__(Cfg<DIM, Nq>::THREADS)
k_volumerhs(T *__restrict__ rhs, const T *__restrict__ Q,
            const T *__restrict__ vgeo, const T *__restrict__ D, int64_t nelem,
            PhysT<T> p) {
  using C = Cfg<DIM, Nq>;
  constexpr int NS = Lay<DIM>::NS, NVG = Lay<DIM>::NVG, Np = C::Np, IR = Lay<DIM>::IR;
  // where large meshes run the march, its order of summation: a result does not
  // depend on how many elements a call has
  constexpr bool PLANES = DIM == 3 && march_volume_built(Nq, sizeof(T));
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T *Ds = reinterpret_cast<T *>(smem_raw);
  T *sF = Ds + Nq * Nq;
  load_D(Ds, D, Nq * Nq);
  const int64_t e0 = (int64_t)blockIdx.x * C::EPB;
  T R[C::NPT][NS], rhoMJ[PLANES ? C::NPT : 1];
#pragma unroll
  for (int u = 0; u < C::NPT; ++u) {
    const int slot = threadIdx.x + u * C::THREADS;
    const int el = slot / Np, n = slot % Np;
    const int64_t e = e0 + el;
    if (slot < C::SLOTS && e < nelem) {
      T q[NS];
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        q[s] = Q[n + Np * (s + NS * e)];
        R[u][s] = rhs[n + Np * (s + NS * e)];
      }
      T met[DIM][DIM], MJ;
      const T *vg = vgeo + (int64_t)Np * NVG * e;
      load_metric<DIM, T>(vg, n, Np, met, MJ);
      if constexpr (PLANES) {
        T unused[NS] = {};
        pointwise_euler<DIM, Nq, C::EPB, T>(q, met, MJ, vg, n, el, sF, p, unused);
        rhoMJ[u] = MJ * q[IR];
      } else {
        pointwise_euler<DIM, Nq, C::EPB, T>(q, met, MJ, vg, n, el, sF, p, R[u]);
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int u = 0; u < C::NPT; ++u) {
    const int slot = threadIdx.x + u * C::THREADS;
    const int el = slot / Np, n = slot % Np;
    const int64_t e = e0 + el;
    if (slot < C::SLOTS && e < nelem) {
      if constexpr (PLANES) contract_planes<Nq, C::EPB, T>(sF, Ds, el, n, rhoMJ[u], p.grav, R[u]);
      else contract<DIM, Nq, C::EPB, T>(sF, Ds, el, n, R[u]);
#pragma unroll
      for (int s = 0; s < NS; ++s) rhs[n + Np * (s + NS * e)] = R[u][s];
    }
  }
}

// Nodes of a face entry's 1-based ids: vM in element e, and element eP and node
// vP of idP, eP = -1 if idP is not a node of the mesh (32-bit division where the
// node count allows it).  Whether idM is a node of element e.
__device__ __forceinline__ bool face_ids(int64_t idM, int64_t idP, int64_t e, int64_t nelem, int Np, int &vM,
                                         int64_t &eP, int &vP) {
  const int64_t oM = idM - 1 - e * Np, oP = idP - 1, all = nelem * Np;
  vM = (int)oM;
  if (all <= 0xffffffffll) {
    eP = (uint32_t)oP / (uint32_t)Np;
    vP = (int)((uint32_t)oP % (uint32_t)Np);
  } else {
    eP = oP / Np;
    vP = (int)(oP % Np);
  }
  if (oP < 0 || oP >= all) eP = -1;
  return oM >= 0 && oM < Np;
}

// ======================================================================
// Stateless face RHS with the reference's int64 vmaps (fluxrhs!).
// Face fluxes of the block's elements go to shared memory first and are then
// subtracted per node in face order, which reproduces the reference's
// sequential f = 1..nface update without atomics.
// ======================================================================
template <int DIM, int Nq, typename T>
__global__ void __launch_bounds__(Cfg<DIM, Nq>::THREADS)
k_fluxrhs(T *__restrict__ rhs, const T *__restrict__ Q,
          const T *__restrict__ sgeo, const T *__restrict__ vgeo,
          int64_t nelem, const int64_t *__restrict__ vmapM,
          const int64_t *__restrict__ vmapP,
          const int64_t *__restrict__ elemtobndy, PhysT<T> p,
          unsigned *status) {
  using C = Cfg<DIM, Nq>;
  constexpr int NS = Lay<DIM>::NS, NVG = Lay<DIM>::NVG, NSG = Lay<DIM>::NSG, IR = Lay<DIM>::IR;
  constexpr int Np = C::Np, Nfp = C::Nfp, NF = C::NFACE, FS = C::EPB * Nfp;
  constexpr int GC = DIM * DIM + 2 + DIM - 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T *FF = reinterpret_cast<T *>(smem_raw);  // [NF][NS][EPB*Nfp]
  const int64_t e0 = (int64_t)blockIdx.x * C::EPB;
#pragma unroll
  for (int u = 0; u < C::FPT; ++u) {
    const int fs = threadIdx.x + u * C::THREADS;
    if (fs >= C::FSLOTS) break;
    const int el = fs / (NF * Nfp), f = (fs / Nfp) % NF, fn = fs % Nfp;
    const int64_t e = e0 + el;
    if (e >= nelem) continue;
    const int64_t fidx = fn + (int64_t)Nfp * (f + NF * e);
    const T *sg = sgeo + (int64_t)NSG * fidx;
    T nrm[DIM];
#pragma unroll
    for (int c = 0; c < DIM; ++c) nrm[c] = sg[c];
    const T sMJ = sg[DIM];
    const int64_t idM = vmapM[fidx], idP = vmapP[fidx];
    const int64_t bc = elemtobndy[f + NF * e];
    int vM, vP;
    int64_t eP;
    const bool mapped = face_ids(idM, idP, e, nelem, Np, vM, eP, vP);
    if (!mapped || (bc == 0 && eP < 0)) {
      atomicOr(status, ST_MESH);  // vmapP points outside the mesh: skip the face
#pragma unroll
      for (int s = 0; s < NS; ++s) FF[(f * NS + s) * FS + el * Nfp + fn] = T(0);
      continue;
    }
    T qM[NS], qP[NS], out[NS];
#pragma unroll
    for (int s = 0; s < NS; ++s) qM[s] = Q[vM + Np * (s + NS * e)];
    const T gM = p.grav != T(0) ? vgeo[vM + Np * (GC + NVG * e)] : T(0);
    const T riM = T(1) / qM[IR];
    const T PM = pressure_ri<DIM, T>(qM, riM, gM, p);
    T PP, riP;
    if (bc == 0) {
#pragma unroll
      for (int s = 0; s < NS; ++s) qP[s] = Q[vP + Np * (s + NS * eP)];
      const T gP = p.grav != T(0) ? vgeo[vP + Np * (GC + NVG * eP)] : T(0);
      riP = T(1) / qP[IR];
      PP = pressure_ri<DIM, T>(qP, riP, gP, p);
    } else if (bc == 1) {
      wall_state<DIM, T>(qM, nrm, qP);
      riP = riM;
      PP = PM;
    } else {
      atomicOr(status, ST_BC);
#pragma unroll
      for (int s = 0; s < NS; ++s) FF[(f * NS + s) * FS + el * Nfp + fn] = T(0);
      continue;
    }
    rusanov_n<DIM, T>(qM, riM, PM, qP, riP, PP, nrm, p, out);
#pragma unroll
    for (int s = 0; s < NS; ++s) FF[(f * NS + s) * FS + el * Nfp + fn] = sMJ * out[s];
  }
  __syncthreads();
#pragma unroll
  for (int u = 0; u < C::NPT; ++u) {
    const int slot = threadIdx.x + u * C::THREADS;
    const int el = slot / Np, n = slot % Np;
    const int64_t e = e0 + el;
    if (slot < C::SLOTS && e < nelem) {
      const int i = n % Nq, j = (n / Nq) % Nq, k = DIM == 3 ? n / (Nq * Nq) : 0;
      const bool onface = i == 0 || i == Nq - 1 || j == 0 || j == Nq - 1 ||
                          (DIM == 3 && (k == 0 || k == Nq - 1));
      if (!onface) continue;
      T R[NS];
#pragma unroll
      for (int s = 0; s < NS; ++s) R[s] = rhs[n + Np * (s + NS * e)];
      gather_face_terms<DIM, Nq, C::EPB, T>(FF, el, n, R);
#pragma unroll
      for (int s = 0; s < NS; ++s) rhs[n + Np * (s + NS * e)] = R[s];
    }
  }
}

// ======================================================================
// Stateless update (updatesolution!).  BY_NODE: one thread per node takes all
// its fields, the index is divided once and eleven loads are in flight per
// thread instead of three (B200, 2.3 M nodes, N=5: FP64 75.6 -> 66.5 us, FP32
// 49.4 -> 33.1).  FP64 elements of fewer than 64 nodes take one thread per value:
// a field of theirs is too short a run for a warp (N=2 FP64: 78 us by value, 99
// by node).
// ======================================================================
template <int DIM, int Nq, typename T>
constexpr bool update_by_node = sizeof(T) == 4 || ipow(Nq, DIM) >= 64;
template <int DIM, int Nq, typename T>
__global__ void __launch_bounds__(256) k_update(T *__restrict__ rhs, const T *__restrict__ rhs_gradQ,
                                                T *__restrict__ Q, const T *__restrict__ vgeo, int64_t nelem, T rka,
                                                T rkb, T dt, T visc) {
  constexpr int NS = Lay<DIM>::NS, NVG = Lay<DIM>::NVG, MJI = DIM * DIM + 1, Np = ipow(Nq, DIM);
  const int64_t g = blockIdx.x * (int64_t)256 + threadIdx.x;
  if constexpr (!update_by_node<DIM, Nq, T>) {
    if (g >= nelem * (Np * NS)) return;
    const int64_t e = g / (Np * NS);
    const int m = (int)(g - e * (Np * NS)), n = m % Np;
    T r = rhs[g];
    if (rhs_gradQ) r += visc * rhs_gradQ[m + e * (Np * NS * DIM)];
    Q[g] += rkb * dt * r * vgeo[n + Np * (MJI + (int64_t)NVG * e)];
    rhs[g] = r * rka;
    return;
  }
  if (g >= nelem * Np) return;
  const int64_t e = g / Np;
  const int n = (int)(g - e * Np);
  T *r0 = rhs + n + e * (Np * NS), *q0 = Q + n + e * (Np * NS);
  T r[NS], q[NS];
#pragma unroll
  for (int s = 0; s < NS; ++s) {
    r[s] = r0[Np * s];
    q[s] = q0[Np * s];
  }
  const T mji = vgeo[n + Np * (MJI + (int64_t)NVG * e)];
  if (rhs_gradQ) {
    const T *v = rhs_gradQ + n + e * ((int64_t)Np * NS * DIM);
#pragma unroll
    for (int s = 0; s < NS; ++s) r[s] += visc * v[Np * s];
  }
#pragma unroll
  for (int s = 0; s < NS; ++s) {
    q0[Np * s] = q[s] + rkb * dt * r[s] * mji;
    r0[Np * s] = r[s] * rka;
  }
}

// ======================================================================
// Fused LSRK stage: volume + face + update in one pass over the element.
//   Qin   state at the start of the stage (read, also for neighbour traces)
//   Qout  state after the stage (distinct buffer)
//   rhs   residual carry: read, then overwritten with rka_next * residual
// EARLY: for launches of a block or two per SM, whose time is one block's
// latency: metric, normals and neighbour codes are loaded before the wait for
// the preceding stage and the neighbours' traces with the state, at the price of
// registers that a full SM could not spare (see Launch::EARLY_BLOCKS).
// ======================================================================
template <int DIM, int Nq, typename T, bool EARLY = false>
__global__ void __launch_bounds__(Cfg<DIM, Nq>::THREADS)
k_stage(const T *Qin_, T *Qout_, T *rhs_,
        const T *__restrict__ vgeo, const T *__restrict__ sgeo,
        const int32_t *__restrict__ nbr, const T *__restrict__ D,
        int64_t nelem, PhysT<T> p, Offs<T, Lay<DIM>::NS> qref, T rka, T rkbdt,
        unsigned *status, int64_t ebeg) {
  using C = Cfg<DIM, Nq>;
  constexpr int NS = Lay<DIM>::NS, NVG = Lay<DIM>::NVG, NSG = Lay<DIM>::NSG, IR = Lay<DIM>::IR;
  constexpr int Np = C::Np, Nfp = C::Nfp, NF = C::NFACE, SP = C::SLOTS;
  constexpr int FS = C::EPB * Nfp, MJI = DIM * DIM + 1;
  constexpr int GC = DIM * DIM + 2 + DIM - 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T *Ds = reinterpret_cast<T *>(smem_raw);
  T *sQ = Ds + ((Nq * Nq + 1) & ~1);  // [NS][SP]
  T *sF = sQ + NS * SP;               // [DIM][NS][SP], reused as FF
  load_D(Ds, D, Nq * Nq);
  const int64_t e0 = ebeg + (int64_t)blockIdx.x * C::EPB;
  // EARLY: what no stage writes, while the preceding one finishes
  T met[EARLY ? C::NPT : 1][DIM][DIM], MJ[EARLY ? C::NPT : 1], mjis[EARLY ? C::NPT : 1];
  int32_t nbs[EARLY ? C::FPT : 1];
  T nrms[EARLY ? C::FPT : 1][DIM + 1], qNb[EARLY ? C::FPT : 1][NS];
  if constexpr (EARLY) {
#pragma unroll
    for (int u = 0; u < C::NPT; ++u) {
      const int slot = threadIdx.x + u * C::THREADS;
      const int el = slot / Np, n = slot % Np;
      if (slot < C::SLOTS && e0 + el < nelem) {
        const T *vg = vgeo + (int64_t)Np * NVG * (e0 + el);
        load_metric<DIM, T>(vg, n, Np, met[u], MJ[u]);
        mjis[u] = vg[n + Np * MJI];
      }
    }
#pragma unroll
    for (int u = 0; u < C::FPT; ++u) {
      const int fs = threadIdx.x + u * C::THREADS;
      const int el = fs / (NF * Nfp), f = (fs / Nfp) % NF, fn = fs % Nfp;
      nbs[u] = NBR_WALL;
      if (fs < C::FSLOTS && e0 + el < nelem) {
        nbs[u] = nbr[f + NF * (e0 + el)];
        const T *sg = sgeo + (int64_t)NSG * (fn + (int64_t)Nfp * (f + NF * (e0 + el)));
#pragma unroll
        for (int c = 0; c <= DIM; ++c) nrms[u][c] = sg[c];
      }
    }
  }
  grid_wait(Qin_, Qout_, rhs_);
  const T *__restrict__ Qin = Qin_;
  T *__restrict__ Qout = Qout_;
  T *__restrict__ rhs = rhs_;
  if constexpr (EARLY) {  // the neighbours' traces, in flight with the state
#pragma unroll
    for (int u = 0; u < C::FPT; ++u) {
      const int fn = (threadIdx.x + u * C::THREADS) % Nfp;
      if (nbs[u] >= 0) {
        const T *q2 = Qin + face_node<DIM, Nq>(nbs[u] & 7, fn) + (int64_t)(nbs[u] >> 3) * (Np * NS);
#pragma unroll
        for (int s = 0; s < NS; ++s) qNb[u][s] = q2[Np * s];
      }
    }
  }
  T R[C::NPT][NS];
  // ---- pointwise fluxes
#pragma unroll
  for (int u = 0; u < C::NPT; ++u) {
    const int slot = threadIdx.x + u * C::THREADS;
    const int el = slot / Np, n = slot % Np;
    const int64_t e = e0 + el;
    if (slot < C::SLOTS && e < nelem) {
      T q[NS];
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        const T d = Qin[n + Np * (s + NS * e)];
        sQ[s * SP + slot] = d;
        q[s] = d + qref.v[s];
        R[u][s] = rhs[n + Np * (s + NS * e)];
      }
      const T *vg = vgeo + (int64_t)Np * NVG * e;
      if constexpr (EARLY) {
        pointwise_euler<DIM, Nq, C::EPB, T>(q, met[u], MJ[u], vg, n, el, sF, p, R[u]);
      } else {
        T m[DIM][DIM], mj;
        load_metric<DIM, T>(vg, n, Np, m, mj);
        pointwise_euler<DIM, Nq, C::EPB, T>(q, m, mj, vg, n, el, sF, p, R[u]);
      }
    }
  }
  __syncthreads();
  // ---- volume contraction
#pragma unroll
  for (int u = 0; u < C::NPT; ++u) {
    const int slot = threadIdx.x + u * C::THREADS;
    const int el = slot / Np, n = slot % Np;
    if (slot < C::SLOTS && e0 + el < nelem) contract<DIM, Nq, C::EPB, T>(sF, Ds, el, n, R[u]);
  }
  __syncthreads();
  // ---- face fluxes (sF reused as FF[NF][NS][EPB*Nfp])
  T *FF = sF;
#pragma unroll
  for (int u = 0; u < C::FPT; ++u) {
    const int fs = threadIdx.x + u * C::THREADS;
    if (fs >= C::FSLOTS) break;
    const int el = fs / (NF * Nfp), f = (fs / Nfp) % NF, fn = fs % Nfp;
    const int64_t e = e0 + el;
    if (e >= nelem) continue;
    const int vM = face_node<DIM, Nq>(f, fn);
    const T *sg = sgeo + (int64_t)NSG * (fn + (int64_t)Nfp * (f + NF * e));
    T nrm[DIM];
#pragma unroll
    for (int c = 0; c < DIM; ++c) nrm[c] = EARLY ? nrms[EARLY ? u : 0][c] : sg[c];
    const T sMJ = EARLY ? nrms[EARLY ? u : 0][DIM] : sg[DIM];
    T qM[NS], qP[NS];
#pragma unroll
    for (int s = 0; s < NS; ++s) qM[s] = sQ[s * SP + el * Np + vM] + qref.v[s];
    const T gM = p.grav != T(0) ? vgeo[vM + Np * (GC + NVG * e)] : T(0);
    const T riM = T(1) / qM[IR];
    const T PM = pressure_ri<DIM, T>(qM, riM, gM, p);
    const int32_t nb = EARLY ? nbs[EARLY ? u : 0] : nbr[f + NF * e];
    T PP, riP;
    if (nb >= 0) {
      const int64_t e2 = nb >> 3;
      const int vP = face_node<DIM, Nq>(nb & 7, fn);
#pragma unroll
      for (int s = 0; s < NS; ++s) qP[s] = (EARLY ? qNb[EARLY ? u : 0][s] : Qin[vP + Np * (s + NS * e2)]) + qref.v[s];
      const T gP = p.grav != T(0) ? vgeo[vP + Np * (GC + NVG * e2)] : T(0);
      riP = T(1) / qP[IR];
      PP = pressure_ri<DIM, T>(qP, riP, gP, p);
    } else {
      wall_state<DIM, T>(qM, nrm, qP);
      riP = riM;
      PP = PM;
    }
    T out[NS];
    rusanov_n<DIM, T>(qM, riM, PM, qP, riP, PP, nrm, p, out);
#pragma unroll
    for (int s = 0; s < NS; ++s) FF[(f * NS + s) * FS + el * Nfp + fn] = sMJ * out[s];
  }
  __syncthreads();
  // ---- face accumulation and LSRK update
  bool bad = false;
#pragma unroll
  for (int u = 0; u < C::NPT; ++u) {
    const int slot = threadIdx.x + u * C::THREADS;
    const int el = slot / Np, n = slot % Np;
    const int64_t e = e0 + el;
    if (slot < C::SLOTS && e < nelem) {
      gather_face_terms<DIM, Nq, C::EPB, T>(FF, el, n, R[u]);
      const T mji = EARLY ? mjis[EARLY ? u : 0] : vgeo[n + Np * (MJI + (int64_t)NVG * e)];
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        const T qn = sQ[s * SP + slot] + rkbdt * R[u][s] * mji;
        bad |= !isfinite(qn);
        Qout[n + Np * (s + NS * e)] = qn;
        rhs[n + Np * (s + NS * e)] = R[u][s] * rka;
      }
    }
  }
  if (bad) atomicOr(status, ST_NONFINITE);
}

// Build the compact face-neighbour table from the reference vmaps and
// validate that they describe a conforming mesh with orientation 1.
template <int DIM, int Nq>
__global__ void k_build_nbr(int32_t *__restrict__ nbr,
                            const int64_t *__restrict__ vmapM,
                            const int64_t *__restrict__ vmapP,
                            const int64_t *__restrict__ elemtobndy,
                            int64_t nelem, int64_t nall, unsigned *status) {
  // nall: elements a neighbour may be (nelem, plus the ghost elements that a
  // partitioned solve appends after its own)
  using C = Cfg<DIM, Nq>;
  constexpr int Np = C::Np, Nfp = C::Nfp, NF = C::NFACE;
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= nelem * NF) return;
  const int64_t e = t / NF;
  const int f = (int)(t % NF);
  const int64_t bc = elemtobndy[t];
  const int64_t *vm = vmapM + (int64_t)Nfp * t, *vp = vmapP + (int64_t)Nfp * t;
  bool ok = true;
  for (int fn = 0; fn < Nfp; ++fn)
    ok &= vm[fn] == Np * e + face_node<DIM, Nq>(f, fn) + 1;
  if (bc == 1) {
    nbr[t] = NBR_WALL;
  } else if (bc == 0) {
    const int64_t id0 = vp[0] - 1;
    const int64_t e2 = id0 / Np;
    int f2 = -1;
    for (int g = 0; g < NF; ++g)
      if (face_node<DIM, Nq>(g, 0) == (int)(id0 % Np)) {
        bool m = true;
        for (int fn = 0; fn < Nfp; ++fn) m &= vp[fn] == Np * e2 + face_node<DIM, Nq>(g, fn) + 1;
        if (m) { f2 = g; break; }
      }
    ok &= f2 >= 0 && e2 >= 0 && e2 < nall && e2 < (1ll << 28);
    nbr[t] = ok ? (int32_t)((e2 << 3) | f2) : NBR_WALL;
  } else {
    atomicOr(status, ST_BC);
    nbr[t] = NBR_WALL;
  }
  if (!ok) atomicOr(status, ST_MESH);
}

// ======================================================================
// LDG Navier–Stokes passes (nse2d.jl / nse3d.jl).  Stateless.
// ======================================================================

// primitives (u, v, [w], ρ, T) in state slots (nse3d.jl:509-522)
template <int DIM, typename T>
__device__ __forceinline__ void primitives(const T *q, T gc, const PhysT<T> &p, T *prim) {
  constexpr int IR = Lay<DIM>::IR, IE = Lay<DIM>::IE;
  const T P = pressure<DIM, T>(q, gc, p);
#pragma unroll
  for (int c = 0; c < DIM; ++c) prim[c] = q[c] / q[IR];
  prim[IR] = q[IR];
  prim[IE] = P / (p.R * q[IR]);
}

// volume_grad!: rhs[:, s, c, e] = -Σ Dᵀ (MJ ξ_c prim_s) per reference direction.
template <int DIM, int Nq, typename T>
__global__ void __launch_bounds__(Cfg<DIM, Nq>::THREADS)
k_volume_grad(T *__restrict__ rhs, const T *__restrict__ Q,
              const T *__restrict__ vgeo, const T *__restrict__ D,
              int64_t nelem, PhysT<T> p) {
  using C = Cfg<DIM, Nq>;
  constexpr int NS = Lay<DIM>::NS, NVG = Lay<DIM>::NVG, Np = C::Np, SP = C::SLOTS;
  constexpr int GC = DIM * DIM + 2 + DIM - 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T *Ds = reinterpret_cast<T *>(smem_raw);
  T *sF = Ds + ((Nq * Nq + 1) & ~1);
  load_D(Ds, D, Nq * Nq);
  const int64_t e0 = (int64_t)blockIdx.x * C::EPB;
  T prim[C::NPT][NS], met[C::NPT][DIM][DIM], MJ[C::NPT];
#pragma unroll
  for (int u = 0; u < C::NPT; ++u) {
    const int slot = threadIdx.x + u * C::THREADS;
    const int el = slot / Np, n = slot % Np;
    const int64_t e = e0 + el;
    if (slot < C::SLOTS && e < nelem) {
      T q[NS];
#pragma unroll
      for (int s = 0; s < NS; ++s) q[s] = Q[n + Np * (s + NS * e)];
      const T *vg = vgeo + (int64_t)Np * NVG * e;
      load_metric<DIM, T>(vg, n, Np, met[u], MJ[u]);
      const T gc = p.grav != T(0) ? vg[n + Np * GC] : T(0);
      primitives<DIM, T>(q, gc, p, prim[u]);
    }
  }
  for (int c = 0; c < DIM; ++c) {
#pragma unroll
    for (int u = 0; u < C::NPT; ++u) {
      const int slot = threadIdx.x + u * C::THREADS;
      const int el = slot / Np, n = slot % Np;
      if (slot < C::SLOTS && e0 + el < nelem)
#pragma unroll
        for (int r = 0; r < DIM; ++r)
#pragma unroll
          for (int s = 0; s < NS; ++s)
            sF[(r * NS + s) * SP + el * Np + n] = MJ[u] * (met[u][r][c] * prim[u][s]);
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < C::NPT; ++u) {
      const int slot = threadIdx.x + u * C::THREADS;
      const int el = slot / Np, n = slot % Np;
      const int64_t e = e0 + el;
      if (slot < C::SLOTS && e < nelem) {
        T R[NS];
#pragma unroll
        for (int s = 0; s < NS; ++s) R[s] = T(0);
        contract_sub<DIM, Nq, C::EPB, T>(sF, Ds, el, n, R);
#pragma unroll
        for (int s = 0; s < NS; ++s) rhs[n + Np * (s + NS * (c + (int64_t)DIM * e))] = R[s];
      }
    }
    __syncthreads();
  }
}

// flux_grad!: rhs[vM, s, c] += sMJ n_c (prim⁻ + prim⁺)/2 in face order.
template <int DIM, int Nq, typename T>
__global__ void __launch_bounds__(Cfg<DIM, Nq>::THREADS)
k_flux_grad(T *__restrict__ rhs, const T *__restrict__ Q,
            const T *__restrict__ sgeo, const T *__restrict__ vgeo,
            int64_t nelem, const int64_t *__restrict__ vmapM,
            const int64_t *__restrict__ vmapP,
            const int64_t *__restrict__ elemtobndy, PhysT<T> p,
            unsigned *status) {
  using C = Cfg<DIM, Nq>;
  constexpr int NS = Lay<DIM>::NS, NVG = Lay<DIM>::NVG, NSG = Lay<DIM>::NSG;
  constexpr int Np = C::Np, Nfp = C::Nfp, NF = C::NFACE, FS = C::EPB * Nfp;
  constexpr int GC = DIM * DIM + 2 + DIM - 1, IR = Lay<DIM>::IR, IE = Lay<DIM>::IE;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T *FF = reinterpret_cast<T *>(smem_raw);  // [NF][NS*DIM][FS]
  const int64_t e0 = (int64_t)blockIdx.x * C::EPB;
  for (int fs = threadIdx.x; fs < C::FSLOTS; fs += C::THREADS) {
    const int el = fs / (NF * Nfp), f = (fs / Nfp) % NF, fn = fs % Nfp;
    const int64_t e = e0 + el;
    if (e >= nelem) continue;
    const int64_t fidx = fn + (int64_t)Nfp * (f + NF * e);
    const T *sg = sgeo + (int64_t)NSG * fidx;
    T nrm[DIM];
#pragma unroll
    for (int c = 0; c < DIM; ++c) nrm[c] = sg[c];
    const T sMJ = sg[DIM];
    const int64_t idM = vmapM[fidx], idP = vmapP[fidx];
    int vM, vP;
    int64_t eP;
    const bool mapped = face_ids(idM, idP, e, nelem, Np, vM, eP, vP);
    if (!mapped) vM = 0;
    T qM[NS], pM[NS], pP[NS];
#pragma unroll
    for (int s = 0; s < NS; ++s) qM[s] = Q[vM + Np * (s + NS * e)];
    const T gM = p.grav != T(0) ? vgeo[vM + Np * (GC + NVG * e)] : T(0);
    primitives<DIM, T>(qM, gM, p, pM);
    const int64_t bc = elemtobndy[f + NF * e];
    if (!mapped || (bc == 0 && eP < 0)) {
      atomicOr(status, ST_MESH);
      for (int s = 0; s < NS * DIM; ++s) FF[(f * NS * DIM + s) * FS + el * Nfp + fn] = T(0);
      continue;
    }
    if (bc == 0) {
      T qP[NS];
#pragma unroll
      for (int s = 0; s < NS; ++s) qP[s] = Q[vP + Np * (s + NS * eP)];
      const T gP = p.grav != T(0) ? vgeo[vP + Np * (GC + NVG * eP)] : T(0);
      primitives<DIM, T>(qP, gP, p, pP);
    } else if (bc == 1) {
      T qP[NS];
      wall_state<DIM, T>(qM, nrm, qP);
#pragma unroll
      for (int c = 0; c < DIM; ++c) pP[c] = qP[c] / qM[IR];
      pP[IR] = qM[IR];
      pP[IE] = pM[IE];
    } else {
      atomicOr(status, ST_BC);
      for (int s = 0; s < NS * DIM; ++s) FF[(f * NS * DIM + s) * FS + el * Nfp + fn] = T(0);
      continue;
    }
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      const T fsv = T(0.5) * (pM[s] + pP[s]);
#pragma unroll
      for (int c = 0; c < DIM; ++c)
        FF[(f * NS * DIM + s * DIM + c) * FS + el * Nfp + fn] = sMJ * nrm[c] * fsv;
    }
  }
  __syncthreads();
  for (int slot = threadIdx.x; slot < C::SLOTS; slot += C::THREADS) {
    const int el = slot / Np, n = slot % Np;
    const int64_t e = e0 + el;
    if (e >= nelem) continue;
    const int i = n % Nq, j = (n / Nq) % Nq, k = DIM == 3 ? n / (Nq * Nq) : 0;
    int fl[3], fnl[3], nf = 0;
    if (i == 0) { fl[nf] = 0; fnl[nf++] = DIM == 3 ? j + Nq * k : j; }
    if (i == Nq - 1) { fl[nf] = 1; fnl[nf++] = DIM == 3 ? j + Nq * k : j; }
    if (j == 0) { fl[nf] = 2; fnl[nf++] = DIM == 3 ? i + Nq * k : i; }
    if (j == Nq - 1) { fl[nf] = 3; fnl[nf++] = DIM == 3 ? i + Nq * k : i; }
    if (DIM == 3 && k == 0) { fl[nf] = 4; fnl[nf++] = i + Nq * j; }
    if (DIM == 3 && k == Nq - 1) { fl[nf] = 5; fnl[nf++] = i + Nq * j; }
    if (nf == 0) continue;
    for (int s = 0; s < NS; ++s)
      for (int c = 0; c < DIM; ++c) {
        T *dst = rhs + n + Np * (s + NS * (c + (int64_t)DIM * e));
        T v = *dst;
        for (int a = 0; a < nf; ++a) v += FF[(fl[a] * NS * DIM + s * DIM + c) * FS + el * Nfp + fnl[a]];
        *dst = v;
      }
  }
}

// update_gradQ!: gradQ = rhs * MJI, one thread per node.
template <int DIM, int Nq, typename T>
__global__ void __launch_bounds__(256) k_update_gradQ(T *__restrict__ gradQ, const T *__restrict__ rhs,
                                                      const T *__restrict__ vgeo, int64_t nelem) {
  constexpr int NS = Lay<DIM>::NS, NVG = Lay<DIM>::NVG, MJI = DIM * DIM + 1, Np = ipow(Nq, DIM);
  const int64_t g = blockIdx.x * (int64_t)256 + threadIdx.x;
  if (g >= nelem * Np) return;
  const int64_t e = g / Np;
  const int n = (int)(g - e * Np);
  const int64_t o = n + e * ((int64_t)Np * NS * DIM);
  const T mji = vgeo[n + Np * (MJI + (int64_t)NVG * e)];
#pragma unroll
  for (int s = 0; s < NS * DIM; ++s) gradQ[o + Np * s] = rhs[o + Np * s] * mji;
}

// Viscous flux of one node (nse3d.jl:717-742 / nse2d.jl:598-614).
// g[s][c] = gradient component c of primitive slot s; vel = (u,v,[w]).
template <int DIM, typename T>
__device__ __forceinline__ void visc_flux(const T (*g)[DIM], const T *vel,
                                          const PhysT<T> &p, T (*out)[DIM]) {
  constexpr int IR = Lay<DIM>::IR, IE = Lay<DIM>::IE;
  T div = g[0][0] + g[1][1];
  if (DIM == 3) div = div + g[2][DIM - 1];
#pragma unroll
  for (int c = 0; c < DIM; ++c) out[IR][c] = T(0) * g[IR][c];
  // momentum rows: τ_ac = ∂_c u_a + ∂_a u_c (+ λ div δ_ac); reference order
#pragma unroll
  for (int a = 0; a < DIM; ++a)
#pragma unroll
    for (int c = 0; c < DIM; ++c)
      out[a][c] = a == c ? T(2) * g[a][a] + p.lambda * div : g[a][c] + g[c][a];
#pragma unroll
  for (int c = 0; c < DIM; ++c) {
    T e = vel[0] * out[0][c] + vel[1] * out[1][c];
    if (DIM == 3) e = e + vel[2] * out[2][c];
    out[IE][c] = e + p.cpPr * g[IE][c];
  }
}

// volume_div!: rhs[:, s, 1, e] = -Σ Dᵀ (MJ ξ·F_visc); other components zeroed.
template <int DIM, int Nq, typename T>
__global__ void __launch_bounds__(Cfg<DIM, Nq>::THREADS)
k_volume_div(T *__restrict__ rhs, const T *__restrict__ gradQ,
             const T *__restrict__ Q, const T *__restrict__ vgeo,
             const T *__restrict__ D, int64_t nelem, PhysT<T> p) {
  using C = Cfg<DIM, Nq>;
  constexpr int NS = Lay<DIM>::NS, NVG = Lay<DIM>::NVG, Np = C::Np, SP = C::SLOTS;
  constexpr int IR = Lay<DIM>::IR;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T *Ds = reinterpret_cast<T *>(smem_raw);
  T *sF = Ds + ((Nq * Nq + 1) & ~1);
  load_D(Ds, D, Nq * Nq);
  const int64_t e0 = (int64_t)blockIdx.x * C::EPB;
#pragma unroll
  for (int u = 0; u < C::NPT; ++u) {
    const int slot = threadIdx.x + u * C::THREADS;
    const int el = slot / Np, n = slot % Np;
    const int64_t e = e0 + el;
    if (slot < C::SLOTS && e < nelem) {
      T g[NS][DIM], out[NS][DIM], vel[DIM], met[DIM][DIM], MJ;
#pragma unroll
      for (int s = 0; s < NS; ++s)
#pragma unroll
        for (int c = 0; c < DIM; ++c) g[s][c] = gradQ[n + Np * (s + NS * (c + (int64_t)DIM * e))];
      const T rho = Q[n + Np * (IR + NS * e)];
#pragma unroll
      for (int c = 0; c < DIM; ++c) vel[c] = Q[n + Np * (c + NS * e)] / rho;
      load_metric<DIM, T>(vgeo + (int64_t)Np * NVG * e, n, Np, met, MJ);
      visc_flux<DIM, T>(g, vel, p, out);
#pragma unroll
      for (int r = 0; r < DIM; ++r)
#pragma unroll
        for (int s = 0; s < NS; ++s) {
          T a = met[r][0] * out[s][0] + met[r][1] * out[s][1];
          if (DIM == 3) a = a + met[r][2] * out[s][2];
          sF[(r * NS + s) * SP + el * Np + n] = MJ * a;
        }
    }
  }
  __syncthreads();
#pragma unroll
  for (int u = 0; u < C::NPT; ++u) {
    const int slot = threadIdx.x + u * C::THREADS;
    const int el = slot / Np, n = slot % Np;
    const int64_t e = e0 + el;
    if (slot < C::SLOTS && e < nelem) {
      T R[NS];
#pragma unroll
      for (int s = 0; s < NS; ++s) R[s] = T(0);
      contract_sub<DIM, Nq, C::EPB, T>(sF, Ds, el, n, R);
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        rhs[n + Np * (s + NS * (0 + (int64_t)DIM * e))] = R[s];
#pragma unroll
        for (int c = 1; c < DIM; ++c) rhs[n + Np * (s + NS * (c + (int64_t)DIM * e))] = T(0);
      }
    }
  }
}

// flux_div!: rhs[vM, s, 1] += sMJ · n·(F⁻+F⁺)/2 in face order.
template <int DIM, int Nq, typename T>
__global__ void __launch_bounds__(Cfg<DIM, Nq>::THREADS)
k_flux_div(T *__restrict__ rhs, const T *__restrict__ gradQ,
           const T *__restrict__ Q, const T *__restrict__ sgeo,
           int64_t nelem, const int64_t *__restrict__ vmapM,
           const int64_t *__restrict__ vmapP,
           const int64_t *__restrict__ elemtobndy, PhysT<T> p,
           unsigned *status) {
  using C = Cfg<DIM, Nq>;
  constexpr int NS = Lay<DIM>::NS, NSG = Lay<DIM>::NSG, IR = Lay<DIM>::IR, IE = Lay<DIM>::IE;
  constexpr int Np = C::Np, Nfp = C::Nfp, NF = C::NFACE, FS = C::EPB * Nfp;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T *FF = reinterpret_cast<T *>(smem_raw);  // [NF][NS][FS]
  const int64_t e0 = (int64_t)blockIdx.x * C::EPB;
  for (int fs = threadIdx.x; fs < C::FSLOTS; fs += C::THREADS) {
    const int el = fs / (NF * Nfp), f = (fs / Nfp) % NF, fn = fs % Nfp;
    const int64_t e = e0 + el;
    if (e >= nelem) continue;
    const int64_t fidx = fn + (int64_t)Nfp * (f + NF * e);
    const T *sg = sgeo + (int64_t)NSG * fidx;
    T nrm[DIM];
#pragma unroll
    for (int c = 0; c < DIM; ++c) nrm[c] = sg[c];
    const T sMJ = sg[DIM];
    const int64_t idM = vmapM[fidx], idP = vmapP[fidx];
    int vM, vP;
    int64_t eP;
    const bool mapped = face_ids(idM, idP, e, nelem, Np, vM, eP, vP);
    if (!mapped) vM = 0;
    T gm[NS][DIM], gp[NS][DIM], vM_[DIM], vP_[DIM];
#pragma unroll
    for (int s = 0; s < NS; ++s)
#pragma unroll
      for (int c = 0; c < DIM; ++c) gm[s][c] = gradQ[vM + Np * (s + NS * (c + (int64_t)DIM * e))];
    const T rhoM = Q[vM + Np * (IR + NS * e)];
#pragma unroll
    for (int c = 0; c < DIM; ++c) vM_[c] = Q[vM + Np * (c + NS * e)] / rhoM;
    const int64_t bc = elemtobndy[f + NF * e];
    if (!mapped || (bc == 0 && eP < 0)) {
      atomicOr(status, ST_MESH);
      for (int s = 0; s < NS; ++s) FF[(f * NS + s) * FS + el * Nfp + fn] = T(0);
      continue;
    }
    if (bc == 0) {
#pragma unroll
      for (int s = 0; s < NS; ++s)
#pragma unroll
        for (int c = 0; c < DIM; ++c) gp[s][c] = gradQ[vP + Np * (s + NS * (c + (int64_t)DIM * eP))];
      const T rhoP = Q[vP + Np * (IR + NS * eP)];
#pragma unroll
      for (int c = 0; c < DIM; ++c) vP_[c] = Q[vP + Np * (c + NS * eP)] / rhoP;
    } else if (bc == 1) {
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        T sn = nrm[0] * gm[s][0] + nrm[1] * gm[s][1];
        if (DIM == 3) sn = sn + nrm[2] * gm[s][2];
#pragma unroll
        for (int c = 0; c < DIM; ++c) gp[s][c] = gm[s][c] - T(2) * sn * nrm[c];
      }
      T un = nrm[0] * vM_[0] + nrm[1] * vM_[1];
      if (DIM == 3) un = un + nrm[2] * vM_[2];
#pragma unroll
      for (int c = 0; c < DIM; ++c) vP_[c] = vM_[c] - T(2) * un * nrm[c];
#pragma unroll
      for (int c = 0; c < DIM; ++c) gp[IE][c] = gm[IE][c];
    } else {
      atomicOr(status, ST_BC);
      for (int s = 0; s < NS; ++s) FF[(f * NS + s) * FS + el * Nfp + fn] = T(0);
      continue;
    }
    T fM[NS][DIM], fP[NS][DIM];
    visc_flux<DIM, T>(gm, vM_, p, fM);
    visc_flux<DIM, T>(gp, vP_, p, fP);
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      T a = nrm[0] * (fM[s][0] + fP[s][0]) + nrm[1] * (fM[s][1] + fP[s][1]);
      if (DIM == 3) a = a + nrm[2] * (fM[s][2] + fP[s][2]);
      FF[(f * NS + s) * FS + el * Nfp + fn] = sMJ * (T(0.5) * a);
    }
  }
  __syncthreads();
  for (int slot = threadIdx.x; slot < C::SLOTS; slot += C::THREADS) {
    const int el = slot / Np, n = slot % Np;
    const int64_t e = e0 + el;
    if (e >= nelem) continue;
    const int i = n % Nq, j = (n / Nq) % Nq, k = DIM == 3 ? n / (Nq * Nq) : 0;
    const bool onface = i == 0 || i == Nq - 1 || j == 0 || j == Nq - 1 ||
                        (DIM == 3 && (k == 0 || k == Nq - 1));
    if (!onface) continue;
    // rhs += Σ_f FF, faces in reference order
    for (int s = 0; s < NS; ++s) {
      T *dst = rhs + n + Np * (s + NS * (0 + (int64_t)DIM * e));
      T v = *dst;
      if (i == 0) v += FF[(0 * NS + s) * FS + el * Nfp + (DIM == 3 ? j + Nq * k : j)];
      if (i == Nq - 1) v += FF[(1 * NS + s) * FS + el * Nfp + (DIM == 3 ? j + Nq * k : j)];
      if (j == 0) v += FF[(2 * NS + s) * FS + el * Nfp + (DIM == 3 ? i + Nq * k : i)];
      if (j == Nq - 1) v += FF[(3 * NS + s) * FS + el * Nfp + (DIM == 3 ? i + Nq * k : i)];
      if (DIM == 3 && k == 0) v += FF[(4 * NS + s) * FS + el * Nfp + i + Nq * j];
      if (DIM == 3 && k == Nq - 1) v += FF[(5 * NS + s) * FS + el * Nfp + i + Nq * j];
      *dst = v;
    }
  }
}

// Compensated FP64 sums of MJ·Q and MJ·Q² per state field.  Every thread
// keeps Neumaier (sum, compensation) pairs; pairs are merged with an exact
// two-sum across the warp and the block, and each block writes 4*NS doubles
// (sum, comp for MJ·Q and for MJ·Q²) that the host merges the same way.
__device__ __forceinline__ void neu_add(double &sum, double &comp, double v) {
  const double t = sum + v;
  if (fabs(sum) >= fabs(v)) comp += (sum - t) + v;
  else comp += (v - t) + sum;
  sum = t;
}
__device__ __forceinline__ void neu_merge(double &sum, double &comp, double s2, double c2) {
  neu_add(sum, comp, s2);
  comp += c2;
}
template <int DIM, typename T>
__global__ void __launch_bounds__(256) k_cons_sums(const T *__restrict__ Q, const T *__restrict__ vgeo,
                                                   int64_t nelem, int Np, Offs<double, Lay<DIM>::NS> qref,
                                                   double *__restrict__ part) {
  constexpr int NS = Lay<DIM>::NS, NVG = Lay<DIM>::NVG, MJ = DIM * DIM;
  double acc[4 * NS];
  for (int s = 0; s < 4 * NS; ++s) acc[s] = 0.0;
  const int64_t total = (int64_t)Np * nelem;
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < total;
       q += (int64_t)gridDim.x * blockDim.x) {
    const int64_t n = q % Np, e = q / Np;
    const double mj = (double)vgeo[n + Np * (MJ + (int64_t)NVG * e)];
    for (int s = 0; s < NS; ++s) {
      const double v = (double)Q[n + Np * (s + (int64_t)NS * e)] + qref.v[s];
      neu_add(acc[4 * s + 0], acc[4 * s + 1], mj * v);
      neu_add(acc[4 * s + 2], acc[4 * s + 3], mj * (v * v));
    }
  }
  for (int off = 16; off > 0; off >>= 1)
    for (int s = 0; s < 2 * NS; ++s) {
      const double so = __shfl_down_sync(0xffffffffu, acc[2 * s], off);
      const double co = __shfl_down_sync(0xffffffffu, acc[2 * s + 1], off);
      neu_merge(acc[2 * s], acc[2 * s + 1], so, co);
    }
  __shared__ double red[8][4 * NS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0)
    for (int s = 0; s < 4 * NS; ++s) red[warp][s] = acc[s];
  __syncthreads();
  if (threadIdx.x == 0) {
    const int nw = (blockDim.x + 31) >> 5;
    for (int w = 1; w < nw; ++w)
      for (int s = 0; s < 2 * NS; ++s) neu_merge(red[0][2 * s], red[0][2 * s + 1], red[w][2 * s], red[w][2 * s + 1]);
    for (int s = 0; s < 4 * NS; ++s) part[blockIdx.x * (int64_t)(4 * NS) + s] = red[0][s];
  }
}

// Rounds an FP64 array to FP32.
__global__ void k_round_f32(float *__restrict__ dst, const double *__restrict__ src, int64_t n);

}  // namespace cb
#include "cb_pipe.cuh"
#include "cb_pipe2.cuh"
#include "cb_mma.cuh"
#include "cb_ns_pipe.cuh"
#include "cb_lean.cuh"
namespace cb {

// ---------------------------------------------------------------- launchers
template <int DIM, int Nq, typename T>
struct Launch {
  using C = Cfg<DIM, Nq>;
  static constexpr int NS = Lay<DIM>::NS;
  static size_t smem_volume() { return sizeof(T) * (((Nq * Nq + 1) & ~1) + (size_t)DIM * NS * C::SLOTS); }
  static size_t smem_stage() { return sizeof(T) * (((Nq * Nq + 1) & ~1) + (size_t)NS * C::SLOTS + (size_t)DIM * NS * C::SLOTS); }
  static size_t smem_face() { return sizeof(T) * (size_t)C::NFACE * NS * C::EPB * C::Nfp; }
  static size_t smem_face_grad() { return sizeof(T) * (size_t)C::NFACE * NS * DIM * C::EPB * C::Nfp; }
  static int grid(int64_t nelem) { return (int)((nelem + C::EPB - 1) / C::EPB); }

  template <typename K>
  static cudaError_t prep(K kernel, size_t smem) {
    if (smem > 48 * 1024) return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    return cudaSuccess;
  }

  static cudaError_t volumerhs(T *rhs, const T *Q, const T *vgeo, const T *D, int64_t nelem,
                               const PhysT<T> &p, cudaStream_t st) {
    // 3-D N >= 3 (FP64: 4): the march (B200, 2.3 M nodes, us: FP64 N=4 98.9 ->
    // 90.0, N=8 190.8 -> 166.2, N=10 188.6 -> 149.9, FP32 N=7 72.4 -> 57.9; below,
    // the grouped kernel is the faster one: FP64 N=3 72.5, march 74.1).  The grouped
    // kernel spreads a node's work over more threads and is the faster one up to so
    // many of its blocks per SM (us a call, grouped / march: FP64 N=4 5^3 3.2 / 6.4, 12^3
    // 10.2 / 11.3, 20^3 46.6 / 44.3; N=5 7^3 5.2 / 6.1, 10^3 9.8 / 9.1; N=7 5^3 5.3 / 6.2, 8^3
    // 15.4 / 11.2; N=10 5^3 13.7 / 14.4; FP32 N=3 10^3 2.8 / 3.0, 15^3 4.8 / 4.5; N=6 6^3 4.5 /
    // 6.6, 9^3 8.3 / 8.3; N=9 4^3 6.0 / 6.7, 6^3 9.8 / 8.5).
    if constexpr (DIM == 3 && march_volume_built(Nq, sizeof(T))) {
      constexpr int GROUPED_BLOCKS = Nq >= 9 ? 1 : Nq == 5 ? 8 : 3;
      if (grid(nelem) > GROUPED_BLOCKS * num_sms()) return march_volume<T>(Nq, rhs, Q, vgeo, D, nelem, p, st);
    }
    size_t sm = smem_volume();
    cudaError_t err = prep(k_volumerhs<DIM, Nq, T>, sm);
    if (err != cudaSuccess) return err;
    k_volumerhs<DIM, Nq, T><<<grid(nelem), C::THREADS, sm, st>>>(rhs, Q, vgeo, D, nelem, p);
    return cudaGetLastError();
  }
  static cudaError_t fluxrhs(T *rhs, const T *Q, const T *sgeo, const T *vgeo, int64_t nelem,
                             const int64_t *vmapM, const int64_t *vmapP, const int64_t *bnd,
                             const PhysT<T> &p, unsigned *status, cudaStream_t st) {
    size_t sm = smem_face();
    cudaError_t err = prep(k_fluxrhs<DIM, Nq, T>, sm);
    if (err != cudaSuccess) return err;
    k_fluxrhs<DIM, Nq, T><<<grid(nelem), C::THREADS, sm, st>>>(rhs, Q, sgeo, vgeo, nelem, vmapM,
                                                                vmapP, bnd, p, status);
    return cudaGetLastError();
  }
  // Whether the tensor-core (DMMA) stage is built for this shape.
  static constexpr bool MMA_OK = DIM == 3 && Nq == 8;
  // Whether kernel 0 (the shape's default) is the tensor-core stage: the
  // faster of the two on B200 at the benchmark size.
  static constexpr bool MMA_DEFAULT = MMA_OK && PipeMT<T>::DEFAULT;
  // Whether the lean pipelined stage is built for this shape, and whether it
  // is the shape's default (where the tensor-core stage is not).
  static constexpr bool LEAN_OK = Lean<DIM, Nq, T>::OK;
  // Whether the default is the column march (cb_march.cuh): where the all-at-once plan
  // leaves one block per SM (B200, one mesh of 5.8-6.5 M nodes, ms per step:
  // N=10 FP64 4.28 -> 3.35, FP32 1.92 -> 1.61; N=9 FP64 2.96 -> 2.72; N=8 FP64
  // 16^3 1.58 -> 1.43, under gravity 1.64 -> 1.45).  Below,
  // the other stages are the faster ones (N=9 FP32 grouped 1.36, march 1.51;
  // N=4 FP32 1.21, 1.24; N=7 FP64 tensor-core 1.75, march 2.34).  Meshes of up to an
  // element per SM keep the grouped stage, whose block spreads an element over 512
  // threads (5^3, us a step, grouped / march: FP64 N=8 52 / 83, N=9 65 / 84, N=10 100 /
  // 116, FP32 N=10 64 / 75; 6^3: 99 / 106, 125 / 118, 196 / 174, 106 / 97).
  static constexpr bool MARCH = DIM == 3 && march_inviscid(Nq, sizeof(T));
  // Default stage kernel per shape, from B200 timings of one mesh (ms per
  // step, warped 3-D cubes of 7-17 M nodes; pipelined CUDA-core / grouped /
  // lean): FP64 N=3 3.66 / 3.34 / 2.76, N=4 4.95 / 4.20 / 3.78, N=5 2.37 /
  // 3.45 / 2.67, N=6 3.37 / 5.13 / 3.83, N=8 5.78 / 5.71 / 5.33; FP32 N=3
  // 1.34 / 1.31 / 1.66, N=4 2.61 / 1.75 / 2.26, N=5 1.65 / 1.44 / 1.72, N=6
  // 2.02 / 1.68 / 2.61, N=8 3.08 / 2.61 / 3.44, N=9 2.22 / 1.93 / 2.45 (the
  // FP32 pipelined plans fit fewer blocks per SM than the grouped stage;
  // FP64 N=8, 9 have no pipelined plan that fits shared memory, so their
  // first figure is the grouped stage as well).  N=2, 6.1 M nodes: FP64 4.30 /
  // 3.18 / 3.42, FP32 1.83 / 1.33 / 1.64; N=1: FP64 4.52 / 3.30 / 3.90, FP32
  // 2.87 / 1.36 / 2.43.  3-D N=7 runs the tensor-core stage in both precisions.
  // (N=3 to 9: timed before the stages formed contravariant fluxes directly, which
  // took 1 to 10 % off each and kept their order.)
  static constexpr int DEFAULT_KERNEL =
      MARCH         ? 5
      : MMA_DEFAULT ? 2
      : DIM == 3 && sizeof(T) == 8 && LEAN_OK && (Nq == 4 || Nq == 5) ? 4
      : DIM == 3 && (Nq <= 3 || (sizeof(T) == 4 && Nq <= 10)) ? 3
      : 1;
  // The same under gravity, whose heights are a dependent load in every phase:
  // where more warps are in flight than in the default (B200, ms per step: FP64
  // N=6 19^3 pipelined 1.12, lean 1.08, without gravity 1.00 and 1.04; N=4 28^3
  // lean 1.39, grouped 1.33, without gravity 1.30 and 1.32; N=4 is so at every size, 5^3
  // 31 us and 29).  N=6 in large meshes only: up to two dozen elements per SM the blocks of
  // the pipelined stage, one per SM and each the whole SM's, are the faster ones (us a
  // step, pipelined / lean: 5^3 32 / 39, 9^3 117 / 145, 12^3 301 / 302, 15^3 565 / 566,
  // 16^3 682 / 664, 24^3 2241 / 2145).
  static constexpr int GRAVITY_LEAN_GROUPS = 24;
  static constexpr int GRAVITY_KERNEL = DIM == 3 && sizeof(T) == 8 && Nq == 7   ? 4
                                        : DIM == 3 && sizeof(T) == 8 && Nq == 5 ? 3
                                                                                : DEFAULT_KERNEL;
  // The grouped stage of small meshes is its EARLY form, and small 2-D meshes
  // default to it: up to EARLY_BLOCKS blocks per SM.
  static constexpr bool EARLY_OK = C::NPT == 1 && !MARCH && (DIM == 2 || DEFAULT_KERNEL == 3);
  // (us a stage, stages in a row on one solver: FP32 3-D N=3 8^3 4.9 -> 3.0, 12^3
  // 6.4 -> 5.6, N=4 8^3 5.9 -> 4.4, N=6 6^3 6.8 -> 5.3, 2-D N=4 48^2 5.7 -> 3.2;
  // FP64 2-D N=4 10^2 4.9 -> 2.9, but N=7 32^2 4.5 at one block, 5.6 at two; 2-D
  // against the pipelined stage, time ratios over N=1 to 10: 10^2 FP64 0.57 to 0.84,
  // FP32 0.56 to 0.93, 32^2 FP32 0.55 to 0.89, 48^2 FP32 at N <= 7 0.56 to 0.96)
  static constexpr int EARLY_BLOCKS = sizeof(T) == 4 ? 4 : 1;
  static bool small_mesh(int64_t nelem) {
    return EARLY_OK && (nelem + C::EPB - 1) / C::EPB <= (int64_t)EARLY_BLOCKS * num_sms();
  }
  // Whether a chained launch of a persistent kernel of `grid` blocks is
  // programmatic.  What overlaps is its prologue; what it costs is the even spread
  // of the blocks: they start wherever an SM has room, so that blocks with a group
  // more than the others meet on one SM.  Worth it where few or nearly all blocks of a wave
  // have a group more, or the prologue zeroes padded flux rows (us a step plain /
  // programmatic, groups a block in brackets.  Unpadded: 2-D FP64 N=3 72^2 36.3 / 33.8
  // (1.1), 3-D FP64 N=5 7^3 42.9 / 41.0 (1.2); 2-D N=7 FP64 40^2 35.9 / 37.9 (1.35), FP32 60^2
  // 35.9 / 38.9 (1.5); 3-D FP64 N=5 8^3 49.2 / 47.2 (1.7), 2-D FP64 N=3 100^2 50.4 / 48.2
  // (2.1), FP32 N=7 72^2 48.1 / 45.2 (2.2); 3-D FP64 N=7 9^3 128.1 / 130.3 (2.5), N=3 17^3
  // 141 / 152 (4.2), 2-D FP64 N=5 130^2 139 / 144 (8.2).  Padded: 2-D FP32 N=5 85^2 55.4 / 46.5
  // (1.7), 200^2 203 / 189 (9.7)).
  static constexpr bool PADDED = Pipe2<DIM, Nq, T>::MV > Nq;
  static int chain_pays(int chained, int64_t groups, int64_t grid) {
    return chained && (PADDED || 4 * groups <= 5 * grid || (10 * groups >= 16 * grid && 10 * groups <= 22 * grid));
  }
  // The stage kernel that choice 0 resolves to on a mesh of nelem elements.
  static int choice(int64_t nelem, bool gravity) {
    if (MARCH) return nelem <= num_sms() ? 3 : 5;
    if (DIM == 2 && small_mesh(nelem)) return 3;
    if (GRAVITY_KERNEL == 4 && DEFAULT_KERNEL == 1 && nelem <= GRAVITY_LEAN_GROUPS * num_sms()) return 1;
    return gravity ? GRAVITY_KERNEL : DEFAULT_KERNEL;
  }
  // Resident blocks per SM of a kernel at `smem` bytes, from the occupancy
  // calculator, cached per device in `cache`.
  template <typename K>
  static cudaError_t blocks_per_sm(K kernel, int threads, size_t smem, int *cache, int *out) {
    int dev = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err != cudaSuccess) return err;
    if (dev < 0 || dev >= MAX_DEVICES) return cudaErrorInvalidDevice;
    if (!cache[dev]) {
      err = prep(kernel, smem);
      if (err != cudaSuccess) return err;
      int v = 0;
      err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, kernel, threads, smem);
      if (err != cudaSuccess) return err;
      cache[dev] = v < 1 ? 1 : v;
    }
    *out = cache[dev];
    return cudaSuccess;
  }
  // kernel: 0 = the default for the mesh (choice), 1 = the CUDA-core stages
  // only, 2 = the tensor-core stage (cudaErrorNotSupported where it is not
  // built), 3 = the unpipelined grouped stage k_stage, 4 = the lean pipelined
  // stage k_stage_lean (state-only staging; the pipelined stage where the
  // arrays are not 16-byte aligned), 5 = the column march (where it is the
  // default).  probe != 0: the timeout test hook of the pipelined, lean and
  // tensor-core stages (see MeshSrc); shapes without one return
  // cudaErrorNotSupported for it.
  // ebeg: the launch covers elements ebeg .. nelem - 1 (neighbour indices
  // stay absolute); only the pipelined, lean and tensor-core stages, the march
  // and the default grouped stage take ebeg > 0, the others return
  // cudaErrorNotSupported for it.  nall: elements of the whole mesh, by which
  // the default is chosen: a stage in parts runs the kernel of the stage in one
  // call.  chained: the stream's preceding launch is a stage of the same solve
  // (see grid_wait).
  static cudaError_t stage(const T *Qin, T *Qout, T *rhs, const T *vgeo, const T *sgeo,
                           const int32_t *nbr, const T *D, int64_t nelem, const PhysT<T> &p,
                           const Offs<T, NS> &qref, T rka, T rkbdt, unsigned *status,
                           cudaStream_t st, int probe, int kernel, int64_t ebeg, int chained, int64_t nall) {
    constexpr bool pipe_ok = Pipe<DIM, Nq, T>::OK;
    static_assert(Pipe2<DIM, Nq, T>::OK || (DEFAULT_KERNEL != 1 && GRAVITY_KERNEL != 1),
                  "choice 1 as the default takes element ranges");
    const bool aligned = ((reinterpret_cast<uintptr_t>(Qin) | reinterpret_cast<uintptr_t>(vgeo)) & 15) == 0;
    const bool aligned2 = aligned && ((reinterpret_cast<uintptr_t>(rhs) | reinterpret_cast<uintptr_t>(sgeo)) & 15) == 0;
    if (ebeg < 0 || ebeg > nelem) return cudaErrorInvalidValue;
    const bool by_default = kernel == 0 || (kernel == 5 && probe);
    if (by_default) {
      // the grouped stage and the march take no test hook: that call takes the
      // pipelined stage, or the lean one where the pipelined plan does not fit
      // shared memory (3-D N=9 FP64, N=10 FP32)
      kernel = !probe                                             ? choice(nall, p.grav != T(0))
               : DEFAULT_KERNEL == 2 || DEFAULT_KERNEL == 4        ? DEFAULT_KERNEL
               : Pipe2<DIM, Nq, T>::OK || !LEAN_OK                 ? 1
                                                                   : 4;
      if (kernel == 2 && !aligned2) kernel = 1;
    }
    if constexpr (MARCH) {
      if (kernel == 5) {
        MarchArgs<T> a{Qin, Qout, rhs, vgeo, sgeo, nbr, D, nullptr, ebeg, nelem, {}, rka, rkbdt, status};
        for (int s = 0; s < NS; ++s) a.qref.v[s] = qref.v[s];
        return march_stage<T>(Nq, false, a, p, st);
      }
    }
    if (kernel == 5 || (kernel == 2 && !(MMA_OK && aligned2))) return cudaErrorNotSupported;
    if (kernel == 3 && (probe || (ebeg && !by_default))) return cudaErrorNotSupported;
    if (kernel == 4 && !LEAN_OK) return cudaErrorNotSupported;
    if (kernel == 4 && !aligned2) kernel = 1;  // bulk copies need 16-byte aligned slabs
    const int64_t groups = (nelem - ebeg + C::EPB - 1) / C::EPB;
    if (groups == 0) return cudaSuccess;
    if constexpr (EARLY_OK) {
      if (kernel == 3 && small_mesh(nall)) {
        const size_t sm = smem_stage();
        const cudaError_t err = prep(k_stage<DIM, Nq, T, true>, sm);
        if (err != cudaSuccess) return err;
        // (2-D: plain above 2.5 blocks per SM, where they no longer spread evenly, FP32
        // N=7 40^2 20.2 us a step against 23.6, N=4 60^2, 2.4 blocks per SM, 23.2 against 20.5)
        const int chain = chained && (DIM == 3 || 2 * groups <= 5 * num_sms());
        return launch_stage_kernel(k_stage<DIM, Nq, T, true>, (unsigned)groups, C::THREADS, sm, st, chain, Qin, Qout,
                                   rhs, vgeo, sgeo, nbr, D, nelem, p, qref, rka, rkbdt, status, ebeg);
      }
    }
    if constexpr (MMA_OK) {
      if (kernel == 2) {
        using S = MeshSrc<T, NS, C::EPB>;  // MeshSrc<T, 5, 1> here
        using PM = PipeMT<T>;
        static int per_sm[MAX_DEVICES] = {0};
        int bps = 0;
        cudaError_t err = blocks_per_sm(k_stage_mma<S, PM::MINB>, PM::THREADS, PM::smem(), per_sm, &bps);
        if (err != cudaSuccess) return err;
        int64_t g = (int64_t)num_sms() * bps;
        if (g > groups) g = groups;
        const S src{Qin, Qout, rhs, vgeo, sgeo, nbr, D, nelem, qref, rkbdt, status, probe, ebeg};
        return launch_stage_kernel(k_stage_mma<S, PM::MINB>, (unsigned)g, PM::THREADS, PM::smem(), st,
                                   chain_pays(chained, groups, g), src, p, rka);
      }
    }
    if constexpr (LEAN_OK) {
      if (kernel == 4) {
        using S = MeshSrc<T, NS, C::EPB>;
        using PL = Lean<DIM, Nq, T>;
        static int per_sm[MAX_DEVICES] = {0};
        int bps = 0;
        cudaError_t err = blocks_per_sm(k_stage_lean<DIM, Nq, T, S>, C::THREADS, PL::smem(), per_sm, &bps);
        if (err != cudaSuccess) return err;
        int64_t g = (int64_t)num_sms() * bps;
        if (g > groups) g = groups;
        const S src{Qin, Qout, rhs, vgeo, sgeo, nbr, D, nelem, qref, rkbdt, status, probe, ebeg};
        return launch_stage_kernel(k_stage_lean<DIM, Nq, T, S>, (unsigned)g, C::THREADS, PL::smem(), st,
                                   chain_pays(chained, groups, g), src, p, rka);
      }
    }
    if (Pipe2<DIM, Nq, T>::OK && aligned2 && kernel != 3) {
      using PP = Pipe2<DIM, Nq, T>;
      using S = MeshSrc<T, NS, C::EPB>;
      const size_t sm = PP::smem();
      static int per_sm[MAX_DEVICES] = {0};
      int bps = 0;
      cudaError_t err = blocks_per_sm(k_stage_pipe2<DIM, Nq, T, S>, C::THREADS, sm, per_sm, &bps);
      if (err != cudaSuccess) return err;
      int64_t g = (int64_t)num_sms() * bps;
      if (g > groups) g = groups;
      const S src{Qin, Qout, rhs, vgeo, sgeo, nbr, D, nelem, qref, rkbdt, status, probe, ebeg};
      return launch_stage_kernel(k_stage_pipe2<DIM, Nq, T, S>, (unsigned)g, C::THREADS, sm, st,
                                 chain_pays(chained, groups, g), src, p, rka);
    } else if (probe || (ebeg && kernel != 3)) {
      return cudaErrorNotSupported;
    } else if (pipe_ok && aligned && kernel != 3) {
      using PP = Pipe<DIM, Nq, T>;
      size_t sm = PP::smem();
      cudaError_t err = prep(k_stage_pipe<DIM, Nq, T>, sm);
      if (err != cudaSuccess) return err;
      int g = num_sms();
      if ((int64_t)g > groups) g = (int)groups;
      k_stage_pipe<DIM, Nq, T><<<g, C::THREADS, sm, st>>>(Qin, Qout, rhs, vgeo, sgeo, nbr, D, nelem,
                                                          p, qref, rka, rkbdt, status);
      return cudaGetLastError();
    } else {
      size_t sm = smem_stage();
      cudaError_t err = prep(k_stage<DIM, Nq, T>, sm);
      if (err != cudaSuccess) return err;
      // (plain up to a wave: the next stage's blocks would crowd onto the SMs that
      // have room, FP32 N=4 10^3: 9.5 us a stage against 7.6; from 2000 blocks on,
      // FP32 N=2 to 6, both within 1 %)
      return launch_stage_kernel(k_stage<DIM, Nq, T>, (unsigned)groups, C::THREADS, sm, st, chained && groups > 8 * num_sms(),
                                 Qin, Qout, rhs, vgeo, sgeo, nbr, D, nelem, p, qref, rka, rkbdt, status, ebeg);
    }
  }
  // Whether stage() takes an element range (ebeg > 0) for arrays aligned
  // like these.
  static bool ranged(const void *Qin, const void *rhs, const void *vgeo, const void *sgeo) {
    const bool a = ((reinterpret_cast<uintptr_t>(Qin) | reinterpret_cast<uintptr_t>(rhs) |
                     reinterpret_cast<uintptr_t>(vgeo) | reinterpret_cast<uintptr_t>(sgeo)) & 15) == 0;
    return a && (Pipe2<DIM, Nq, T>::OK || MMA_OK || LEAN_OK);
  }
  static cudaError_t build_nbr(int32_t *nbr, const int64_t *vmapM, const int64_t *vmapP,
                               const int64_t *bnd, int64_t nelem, unsigned *status,
                               cudaStream_t st) {
    const int64_t n = nelem * C::NFACE;
    k_build_nbr<DIM, Nq><<<(int)((n + 255) / 256), 256, 0, st>>>(nbr, vmapM, vmapP, bnd, nelem, nelem, status);
    return cudaGetLastError();
  }
  static cudaError_t build_nbr_ghost(int32_t *nbr, const int64_t *vmapM, const int64_t *vmapP,
                                     const int64_t *bnd, int64_t nelem, int64_t nall, unsigned *status,
                                     cudaStream_t st) {
    const int64_t n = nelem * C::NFACE;
    k_build_nbr<DIM, Nq><<<(int)((n + 255) / 256), 256, 0, st>>>(nbr, vmapM, vmapP, bnd, nelem, nall, status);
    return cudaGetLastError();
  }
  static cudaError_t volume_grad(T *rhs, const T *Q, const T *vgeo, const T *D, int64_t nelem,
                                 const PhysT<T> &p, cudaStream_t st) {
    size_t sm = smem_volume();
    cudaError_t err = prep(k_volume_grad<DIM, Nq, T>, sm);
    if (err != cudaSuccess) return err;
    k_volume_grad<DIM, Nq, T><<<grid(nelem), C::THREADS, sm, st>>>(rhs, Q, vgeo, D, nelem, p);
    return cudaGetLastError();
  }
  static cudaError_t flux_grad(T *rhs, const T *Q, const T *sgeo, const T *vgeo, int64_t nelem,
                               const int64_t *vmapM, const int64_t *vmapP, const int64_t *bnd,
                               const PhysT<T> &p, unsigned *status, cudaStream_t st) {
    size_t sm = smem_face_grad();
    cudaError_t err = prep(k_flux_grad<DIM, Nq, T>, sm);
    if (err != cudaSuccess) return err;
    k_flux_grad<DIM, Nq, T><<<grid(nelem), C::THREADS, sm, st>>>(rhs, Q, sgeo, vgeo, nelem, vmapM,
                                                                  vmapP, bnd, p, status);
    return cudaGetLastError();
  }
  static cudaError_t volume_div(T *rhs, const T *gradQ, const T *Q, const T *vgeo, const T *D,
                                int64_t nelem, const PhysT<T> &p, cudaStream_t st) {
    size_t sm = smem_volume();
    cudaError_t err = prep(k_volume_div<DIM, Nq, T>, sm);
    if (err != cudaSuccess) return err;
    k_volume_div<DIM, Nq, T><<<grid(nelem), C::THREADS, sm, st>>>(rhs, gradQ, Q, vgeo, D, nelem, p);
    return cudaGetLastError();
  }
  static cudaError_t flux_div(T *rhs, const T *gradQ, const T *Q, const T *sgeo, int64_t nelem,
                              const int64_t *vmapM, const int64_t *vmapP, const int64_t *bnd,
                              const PhysT<T> &p, unsigned *status, cudaStream_t st) {
    size_t sm = smem_face();
    cudaError_t err = prep(k_flux_div<DIM, Nq, T>, sm);
    if (err != cudaSuccess) return err;
    k_flux_div<DIM, Nq, T><<<grid(nelem), C::THREADS, sm, st>>>(rhs, gradQ, Q, sgeo, nelem, vmapM,
                                                                 vmapP, bnd, p, status);
    return cudaGetLastError();
  }
};

}  // namespace cb
