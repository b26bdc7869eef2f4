// Stages of the 3-D hexahedra in which a thread owns grid lines (sm_100a).
//
// The derivative contractions of an element run along its grid lines.  A thread
// that owns a whole line multiplies each flux value by a row of D where it is
// made, straight into the line's accumulators: no exchange, and D is read
// uniformly by the block.  (The node-owner stages read Nq flux values per node,
// field and direction from shared memory; they are bound by that pipe.)  Both
// kernels below read the state, the carry and the geometry by plain and cp.async
// accesses of single values, so there is no rule on the alignment of the caller's
// arrays or of element slabs; the neighbour codes (read in pairs) and the gradient
// records (in 16-byte vectors) are the solver's own allocations.
//
// k_march_stage: the fused stage, inviscid or (VISC) with the viscous flux.  The
// thread (i, j) owns the ζ line (i, j, 0..N) and the block marches through the
// planes k of its elements: at plane k every thread forms the contravariant
// fluxes of its node (the flux normal to the rows of MJ ξ_r, about half the
// operations of the full tensor dotted with the metric).  The ζ flux goes into
// the line's accumulators; the ξ and η fluxes to a double-buffered plane in
// shared memory, rows along their contraction index, one barrier per plane.
// Face terms of the ξ and η faces pass through a face buffer, those of the ζ
// faces belong to the thread's own nodes.  Two planes are staged instead of the
// element (3-D N=10 FP64: 97 KB with the state against 213 KB for the
// all-at-once grouped stage it replaced, one block per SM), and the loads of
// plane k + 1 are in flight while plane k is contracted.
//
// k_line_grad: the gradient pass of the viscous form, nine steps (direction r of
// gradient component c), in each of which a thread owns a line of direction r;
// the primitives and one metric field per step lie in shared memory, the fields
// copied three steps ahead by cp.async, which takes no registers.  36
// contractions a node make this pass bound by the shared-memory pipe and by
// latency; per node it moves 100 words through shared memory at N=7 where the
// node-owner pass moved about 330.  B200, one gradient pass, 6.2 M nodes (N=7),
// FP32: 282 us, marching like the stage 440 us, the pipelined node-owner pass
// about 600 us.
#pragma once
#include "cb_kernels.cuh"

namespace cb {

// Elements per block: the lines of EPB elements fill the block's warps (threads
// in use: 32·4, 14·9, 8·16, 5·25, 5·36, 3·49, 2·64, 81, 100, 121).  FP64 takes
// fewer elements at N=5, 6 and 7 (2·36, 49, 64): of its 230 to 255 registers a
// thread, few large blocks fit an SM (B200, ms per viscous step: N=5 20^3 three
// elements 2.58, two 2.18, four 2.30; N=6 17^3 two 2.15, one 2.06; N=7 16^3 two
// 2.54, one 2.40).
__host__ __device__ constexpr int march_epb(int nq, int w) {
  return nq == 2   ? 32
         : nq == 3 ? 14
         : nq == 4 ? 8
         : nq == 5 ? 5
         : nq == 6 ? (w == 4 ? 5 : 2)
         : nq == 7 ? (w == 4 ? 3 : 1)
         : nq == 8 ? (w == 4 ? 2 : 1)
                   : 1;
}

template <int Nq, typename T>
struct March {
  static constexpr int Np = Nq * Nq * Nq, N2 = Nq * Nq, NS = 5, NVG = 14, NSG = 5;
  static constexpr int EPB = march_epb(Nq, sizeof(T));
  static constexpr int THREADS = cdiv(EPB * N2, 32) * 32;
  static constexpr int VW = 16 / (int)sizeof(T);  // values per 16-byte vector
  static constexpr int RS = row_stride<T>(Nq);    // plane rows: distinct banks for the rows of a warp
  static constexpr int ROW = N2 * EPB / Nq * RS;  // one field's rows of a plane
  static constexpr int FS = EPB * N2;
  static constexpr size_t pad16(size_t b) { return (b + 15) & ~size_t(15); }
  // D[m + Nq i] by rows i (DT) and by rows m (DZ)
  static constexpr size_t OFF_DT = 0, DB = pad16(sizeof(T) * Nq * RS);
  static constexpr size_t OFF_DZ = DB;
  static constexpr size_t OFF_P = 2 * DB;                                    // [2][2][NS][ROW]
  static constexpr size_t OFF_FF = OFF_P + pad16(sizeof(T) * 4 * NS * ROW);  // [4][NS][FS]
  // the elements' state, [EPB][NS][Nq][Nq][QR]: rows of an odd length, so that
  // the ξ faces (one value a row) fall into distinct banks
  static constexpr int QR = Nq | 1, QE = N2 * QR;
  static constexpr size_t OFF_Q = OFF_FF + pad16(sizeof(T) * 4 * NS * FS);
  static constexpr size_t smem_stage() { return OFF_Q + pad16(sizeof(T) * EPB * NS * QE); }
  // gradient pass: four primitives, four sums, three metric fields per node
  static constexpr int RD = cdiv(Nq, VW) * VW, GSLABS = 11;
  static constexpr size_t OFF_S = pad16(sizeof(T) * Nq * RD);
  static constexpr size_t smem_grad() { return OFF_S + pad16(sizeof(T) * EPB * GSLABS * (size_t)QE); }
  // the two D rows of a thread stay in registers where they take few
  static constexpr bool DREG = sizeof(T) * Nq <= 48;
  // resident blocks the registers are sized for
  static constexpr int blocks_for(int regs) { return 65536 / (THREADS * regs) < 1 ? 1 : 65536 / (THREADS * regs); }
  // (fewer registers and more blocks spill; more registers lose a block: FP64
  // N=8 16^3 inviscid step 1.68 ms at 255, 1.43 ms at 168, the lean stage 1.58;
  // viscous passes at 168 instead of 255: N=4 2.06 -> 2.69, N=9 2.31 -> 2.96; FP32
  // N=7 viscous stage step 3.06 ms at 168, 3.57 ms at 128)
  static constexpr int REGS_STAGE = sizeof(T) == 4 ? (Nq <= 5 ? 96 : Nq <= 8 ? 128 : 168) : (Nq <= 5 || Nq == 9 ? 168 : 255);
  static constexpr int REGS_NS = sizeof(T) == 4 ? (Nq <= 5 ? 128 : 168) : Nq == 6 ? 224 : 255;
  static constexpr int REGS_VOLUME = sizeof(T) == 4 ? (Nq <= 8 ? 96 : 128) : (Nq <= 5 ? 128 : Nq <= 8 ? 168 : 255);
  static constexpr size_t smem_volume() { return OFF_FF; }
  static constexpr int REGS_GRAD = sizeof(T) == 4 ? (Nq <= 5 ? 96 : 128) : (Nq <= 9 ? 168 : 255);
};

// Loads that stay where the march issues them (volatile), ahead of the barrier
// that their latency overlaps.
__device__ __forceinline__ float ld_here(const float *p) {
  float v;
  asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ double ld_here(const double *p) {
  double v;
  asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}

// Pointers that the compiler cannot take for read-only parameters, whose loads it
// otherwise schedules over the whole kernel at the price of registers (us a step
// without / with: viscous FP64 N=2 33^3 1520 / 1478, N=5 25^3 4180 / 4113, Euler FP64 N=8
// 17^3 1699 / 1682).
template <typename... P>
__device__ __forceinline__ void here_pointers(P *&...ptr) {
  int64_t zero;
  asm volatile("mov.s64 %0, 0;" : "=l"(zero)::"memory");
  ((void)(ptr += zero), ...);
}

// D by rows i (DT[i][m] = D[m + Nq i]) and by rows m (DZ[m][i]).
template <int Nq, int RS, int THREADS, typename T>
__device__ __forceinline__ void march_load_D(T *DT, T *DZ, const T *__restrict__ D) {
  for (int t = threadIdx.x; t < Nq * Nq; t += THREADS) {
    const int m = t % Nq, i = t / Nq;
    const T d = D[t];
    DT[i * RS + m] = d;
    DZ[m * RS + i] = d;
  }
}

// Σ_m row[m] d[m] over the Nq values of a shared-memory row, 16 bytes a load.
template <int Nq, typename T>
__device__ __forceinline__ T march_dot(const T *row, const T *d, T acc) {
  constexpr int VW = 16 / (int)sizeof(T);
  using V = typename Vec16<T>::type;
#pragma unroll
  for (int c = 0; c < cdiv(Nq, VW); ++c) {
    T v[VW];
    *reinterpret_cast<V *>(v) = *reinterpret_cast<const V *>(row + c * VW);
#pragma unroll
    for (int x = 0; x < VW; ++x)
      if (c * VW + x < Nq) acc += v[x] * d[c * VW + x];
  }
  return acc;
}
template <int Nq, typename T>
__device__ __forceinline__ void march_row(const T *row, T *d) {
  constexpr int VW = 16 / (int)sizeof(T);
  using V = typename Vec16<T>::type;
#pragma unroll
  for (int c = 0; c < cdiv(Nq, VW); ++c) {
    T v[VW];
    *reinterpret_cast<V *>(v) = *reinterpret_cast<const V *>(row + c * VW);
#pragma unroll
    for (int x = 0; x < VW; ++x)
      if (c * VW + x < Nq) d[c * VW + x] = v[x];
  }
}

// The six face-neighbour codes of an element (24 bytes, 8-byte aligned).
__device__ __forceinline__ void march_codes(const int32_t *__restrict__ nbr, int32_t *code) {
#pragma unroll
  for (int h = 0; h < 3; ++h) {
    const int2 v = *reinterpret_cast<const int2 *>(nbr + 2 * h);
    code[2 * h] = v.x;
    code[2 * h + 1] = v.y;
  }
}

// Position of face node (a, b) of face f in a state slab with rows of QR.
template <int Nq, int QR>
__device__ __forceinline__ int march_node(int f, int a, int b) {
  const int side = (f & 1) * (Nq - 1);
  return f < 2 ? side + QR * (a + Nq * b) : f < 4 ? a + QR * (side + Nq * b) : a + QR * (b + Nq * side);
}

// Viscous traction of one side: t = τ·n (momentum) and n·(τ·u + c_p/Pr ∇T),
// τ = ∇u + ∇uᵀ + λ div u (nse3d.jl:717-742).  g[s][c]: gradient component c of
// u, v, w, T.
template <typename T>
__device__ __forceinline__ void visc_normal(const T (*g)[3], const T *vel, const T *n, const PhysT<T> &p, T *t) {
  const T ld = p.lambda * (g[0][0] + g[1][1] + g[2][2]);
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    T v = ld * n[a];
#pragma unroll
    for (int c = 0; c < 3; ++c) v += (g[a][c] + g[c][a]) * n[c];
    t[a] = v;
  }
  t[3] = vel[0] * t[0] + vel[1] * t[1] + vel[2] * t[2] + p.cpPr * (g[3][0] * n[0] + g[3][1] * n[1] + g[3][2] * n[2]);
}

template <typename T>
__device__ __forceinline__ void load_grad(const T *rec, T (*g)[3]) {
  constexpr int VW = 16 / (int)sizeof(T);
  using V = typename Vec16<T>::type;
  T v[GREC];
#pragma unroll
  for (int c = 0; c < GREC / VW; ++c) *reinterpret_cast<V *>(v + c * VW) = *reinterpret_cast<const V *>(rec + c * VW);
#pragma unroll
  for (int c = 0; c < GREC; ++c) g[c % 4][c / 4] = v[c];
}
// State slot of primitive s (u, v, w, T).
__device__ __forceinline__ constexpr int grad_slot(int s) { return s < 3 ? s : 4; }

// One fused stage: volume + face + LSRK update of elements ebeg .. eend - 1.
// VISC: with the viscous flux of the gradient gq (the second viscous pass).
template <int Nq, typename T, bool VISC>
__global__ void __launch_bounds__(March<Nq, T>::THREADS,
                                  March<Nq, T>::blocks_for(VISC ? March<Nq, T>::REGS_NS : March<Nq, T>::REGS_STAGE))
    k_march_stage(MarchArgs<T> a, PhysT<T> p) {
  using C = March<Nq, T>;
  constexpr int Np = C::Np, N2 = C::N2, NS = 5, NVG = 14, NSG = 5, IR = 3, RS = C::RS, ROW = C::ROW, FS = C::FS;
  constexpr int MJF = 9, MJIF = 10, GC = 13, EPB = C::EPB, QR = C::QR, QE = C::QE;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T *DT = reinterpret_cast<T *>(smem_raw + C::OFF_DT), *DZ = reinterpret_cast<T *>(smem_raw + C::OFF_DZ);
  T *PL = reinterpret_cast<T *>(smem_raw + C::OFF_P);
  T *FF = reinterpret_cast<T *>(smem_raw + C::OFF_FF);
  here_pointers(a.Qin, a.Qout, a.rhs, a.gq);
  const int tid = threadIdx.x, el = tid / N2, ij = tid % N2, i = ij % Nq, j = ij / Nq;
  const int64_t e0 = a.ebeg + (int64_t)blockIdx.x * EPB, e = e0 + el;
  const bool act = el < EPB && e < a.eend;
  const int64_t ec = act ? e : e0;  // idle threads keep valid addresses
  const T *__restrict__ Q = a.Qin + ec * (Np * NS);
  const T *__restrict__ vg = a.vgeo + ec * (Np * NVG);
  const T *__restrict__ gq = VISC ? a.gq + ec * (Np * GREC) : nullptr;
  T *__restrict__ rhs = a.rhs + ec * (Np * NS);
  // the column's state into shared memory
  T *Qs = reinterpret_cast<T *>(smem_raw + C::OFF_Q) + (act ? el : 0) * (NS * QE);
  const int qij = i + QR * j;
  if (act) {
#pragma unroll
    for (int k = 0; k < Nq; ++k)
#pragma unroll
      for (int s = 0; s < NS; ++s)
        cp_async<sizeof(T)>(Qs + s * QE + qij + QR * Nq * k, Q + ij + N2 * k + Np * s);
  }
  cp_async_commit();
  march_load_D<Nq, RS, C::THREADS, T>(DT, DZ, a.D);
  T qr[NS];
#pragma unroll
  for (int s = 0; s < NS; ++s) qr[s] = a.qref.v[s];

  int32_t code[6];
  march_codes(a.nbr + 6 * ec, code);
  T acc[Nq][NS];  // the column's residual, from the carry on
#pragma unroll
  for (int k = 0; k < Nq; ++k)
#pragma unroll
    for (int s = 0; s < NS; ++s) acc[k][s] = ld_here(rhs + ij + N2 * k + Np * s);
  cp_async_wait<0>();
  __syncthreads();  // D and the state

  // ---- face terms: thread (a, b) = (i, j) takes face node a + Nq b of all
  // six.  No branch on the kind of face: at a wall the neighbour is the node
  // itself and the mirrored state is selected afterwards, so that the loads of
  // several faces can be in flight.
#pragma unroll
  for (int f = 0; f < 6; ++f) {
    const bool wall = code[f] < 0;
    const int64_t e2 = wall ? ec : (int64_t)(code[f] >> 3);
    const int vM = face_node<3, Nq>(f, ij), vP = face_node<3, Nq>(wall ? f : code[f] & 7, ij);
    const T *sg = a.sgeo + NSG * (ij + (int64_t)N2 * (f + 6 * ec));
    const T *Q2 = a.Qin + e2 * (Np * NS) + vP;
    T n[3], qM[NS], qP[NS];
#pragma unroll
    for (int s = 0; s < NS; ++s) qP[s] = Q2[Np * s] + qr[s];
#pragma unroll
    for (int s = 0; s < NS; ++s) qM[s] = Qs[s * QE + march_node<Nq, QR>(f, i, j)] + qr[s];
#pragma unroll
    for (int c = 0; c < 3; ++c) n[c] = sg[c];
    const T sMJ = sg[3];
    T gM = T(0), gP = T(0);
    if (p.grav != T(0)) {
      gM = vg[vM + Np * GC];
      gP = a.vgeo[vP + Np * (GC + NVG * e2)];
    }
    const T riM = T(1) / qM[IR], riP = T(1) / qP[IR];
    const T PM = pressure_ri<3, T>(qM, riM, gM, p);
    T PP = pressure_ri<3, T>(qP, riP, gP, p);
    const T un2 = wall ? T(2) * (n[0] * qM[0] + n[1] * qM[1] + n[2] * qM[2]) : T(0);
    PP = wall ? PM : PP;
#pragma unroll
    for (int c = 0; c < 3; ++c) qP[c] -= un2 * n[c];
    T out[NS];
    rusanov_n<3, T>(qM, riM, PM, qP, riP, PP, n, p, out);
    if constexpr (VISC) {
      T g[4][3], vel[3], t0[4], t1[4];
      load_grad<T>(gq + GREC * vM, g);
#pragma unroll
      for (int c = 0; c < 3; ++c) vel[c] = qM[c] * riM;
      visc_normal<T>(g, vel, n, p, t0);
      load_grad<T>(a.gq + (e2 * Np + vP) * GREC, g);
#pragma unroll
      for (int s = 0; s < 3; ++s) {  // reflective wall: mirrored velocity gradients (nse3d.jl:880-900)
        const T sn = wall ? T(2) * (n[0] * g[s][0] + n[1] * g[s][1] + n[2] * g[s][2]) : T(0);
#pragma unroll
        for (int c = 0; c < 3; ++c) g[s][c] -= sn * n[c];
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) vel[c] = qP[c] * riP;  // a wall mirrors the momentum
      visc_normal<T>(g, vel, n, p, t1);
#pragma unroll
      for (int s = 0; s < 4; ++s) out[grad_slot(s)] -= p.visc * (T(0.5) * (t0[s] + t1[s]));
    }
    if (f < 4) {
      if (act)
#pragma unroll
        for (int s = 0; s < NS; ++s) FF[(f * NS + s) * FS + tid] = sMJ * out[s];
    } else {
#pragma unroll
      for (int s = 0; s < NS; ++s) acc[f == 4 ? 0 : Nq - 1][s] -= sMJ * out[s];
    }
  }

  // ---- the march
  T m[9], MJ, hz = T(0);
  T g[4][3];  // VISC only
  auto load_plane = [&](int k) {
    const int nn = ij + N2 * k;
#pragma unroll
    for (int c = 0; c < 9; ++c) m[c] = ld_here(vg + nn + Np * c);
    MJ = ld_here(vg + nn + Np * MJF);
    if (p.grav != T(0)) hz = vg[nn + Np * GC];
    if constexpr (VISC) load_grad<T>(gq + GREC * nn, g);
  };
  load_plane(0);
  T dx[C::DREG ? Nq : 1], dy[C::DREG ? Nq : 1];
  __syncthreads();  // FF
  if constexpr (C::DREG) {
    march_row<Nq, T>(DT + i * RS, dx);
    march_row<Nq, T>(DT + j * RS, dy);
  }
  const int elr = (act ? el : 0) * Nq;
#pragma unroll
  for (int k = 0; k < Nq; ++k) {
    T *F = PL + (k & 1) * (2 * NS * ROW), *G = F + NS * ROW;
    if (act) {
      T q[NS];
#pragma unroll
      for (int s = 0; s < NS; ++s) q[s] = Qs[s * QE + qij + QR * Nq * k] + qr[s];
      const T ri = T(1) / q[IR];
      const T P = pressure_ri<3, T>(q, ri, hz, p);
      T vel[3];
      if constexpr (VISC)
#pragma unroll
        for (int c = 0; c < 3; ++c) vel[c] = q[c] * ri;
      T f[3][NS];
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        const T nr[3] = {MJ * m[r], MJ * m[r + 3], MJ * m[r + 6]};
        T un;
        normal_flux<3, T>(q, ri, P, nr, un, f[r]);
        if constexpr (VISC) {
          T t[4];
          visc_normal<T>(g, vel, nr, p, t);
#pragma unroll
          for (int s = 0; s < 4; ++s) f[r][grad_slot(s)] -= p.visc * t[s];
        }
      }
      acc[k][2] -= MJ * q[IR] * p.grav;
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        F[s * ROW + (elr + j) * RS + i] = f[0][s];
        G[s * ROW + (elr + i) * RS + j] = f[1][s];
      }
      if (k + 1 < Nq) load_plane(k + 1);
      T dz[Nq];
      march_row<Nq, T>(DZ + k * RS, dz);
#pragma unroll
      for (int x = 0; x < Nq; ++x)
#pragma unroll
        for (int s = 0; s < NS; ++s) acc[x][s] += dz[x] * f[2][s];
    }
    __syncthreads();
    if (act) {
      if constexpr (C::DREG) {
#pragma unroll
        for (int s = 0; s < NS; ++s) {
          acc[k][s] = march_dot<Nq, T>(F + s * ROW + (elr + j) * RS, dx, acc[k][s]);
          acc[k][s] = march_dot<Nq, T>(G + s * ROW + (elr + i) * RS, dy, acc[k][s]);
        }
      } else {
        T d[Nq];
        march_row<Nq, T>(DT + i * RS, d);
#pragma unroll
        for (int s = 0; s < NS; ++s) acc[k][s] = march_dot<Nq, T>(F + s * ROW + (elr + j) * RS, d, acc[k][s]);
        march_row<Nq, T>(DT + j * RS, d);
#pragma unroll
        for (int s = 0; s < NS; ++s) acc[k][s] = march_dot<Nq, T>(G + s * ROW + (elr + i) * RS, d, acc[k][s]);
      }
      const int fb = el * N2 + Nq * k;
      if (i == 0 || i == Nq - 1) {
        const T *ff = FF + (i == 0 ? 0 : NS * FS) + fb + j;
#pragma unroll
        for (int s = 0; s < NS; ++s) acc[k][s] -= ff[s * FS];
      }
      if (j == 0 || j == Nq - 1) {
        const T *ff = FF + (j == 0 ? 2 : 3) * NS * FS + fb + i;
#pragma unroll
        for (int s = 0; s < NS; ++s) acc[k][s] -= ff[s * FS];
      }
    }
  }
  // ---- LSRK update
  if (!act) return;
  T *__restrict__ Qo = a.Qout + e * (Np * NS);
  bool bad = false;
#pragma unroll
  for (int k = 0; k < Nq; ++k) {
    const int nn = ij + N2 * k;
    const T mji = a.rkbdt * vg[nn + Np * MJIF];
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      const T qn = Qs[s * QE + qij + QR * Nq * k] + acc[k][s] * mji;
      bad |= !isfinite(qn);
      Qo[nn + Np * s] = qn;
      rhs[nn + Np * s] = acc[k][s] * a.rka;
    }
  }
  if (bad) atomicOr(a.status, ST_NONFINITE);
}

// The volume integral alone (volumerhs!): the march without faces and update,
// rhs += volume terms.  The grouped kernel reads every flux value Nq times per
// direction from shared memory and is bound by that pipe (3-D N=5 FP64, 2.3 M
// nodes: 96 us, 84 % of its wavefronts).
template <int Nq, typename T>
__global__ void __launch_bounds__(March<Nq, T>::THREADS, March<Nq, T>::blocks_for(March<Nq, T>::REGS_VOLUME))
    k_march_volume(T *__restrict__ rhs_, const T *__restrict__ Q_, const T *__restrict__ vgeo, const T *__restrict__ D,
                   int64_t nelem, PhysT<T> p) {
  using C = March<Nq, T>;
  constexpr int Np = C::Np, N2 = C::N2, NS = 5, NVG = 14, IR = 3, RS = C::RS, ROW = C::ROW, MJF = 9, GC = 13, EPB = C::EPB;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T *DT = reinterpret_cast<T *>(smem_raw + C::OFF_DT), *DZ = reinterpret_cast<T *>(smem_raw + C::OFF_DZ);
  T *PL = reinterpret_cast<T *>(smem_raw + C::OFF_P);
  const int tid = threadIdx.x, el = tid / N2, ij = tid % N2, i = ij % Nq, j = ij / Nq;
  const int64_t e0 = (int64_t)blockIdx.x * EPB, e = e0 + el;
  const bool act = el < EPB && e < nelem;
  const int64_t ec = act ? e : e0;
  const T *__restrict__ Q = Q_ + ec * (Np * NS) + ij;
  const T *__restrict__ vg = vgeo + ec * (Np * NVG) + ij;
  T *__restrict__ rhs = rhs_ + ec * (Np * NS) + ij;
  T q[NS], m[9], MJ, hz = T(0);
  auto load_plane = [&](int k) {
#pragma unroll
    for (int s = 0; s < NS; ++s) q[s] = ld_here(Q + N2 * k + Np * s);
#pragma unroll
    for (int c = 0; c < 9; ++c) m[c] = ld_here(vg + N2 * k + Np * c);
    MJ = ld_here(vg + N2 * k + Np * MJF);
    if (p.grav != T(0)) hz = vg[N2 * k + Np * GC];
  };
  load_plane(0);
  march_load_D<Nq, RS, C::THREADS, T>(DT, DZ, D);
  T acc[Nq][NS];
#pragma unroll
  for (int k = 0; k < Nq; ++k)
#pragma unroll
    for (int s = 0; s < NS; ++s) acc[k][s] = ld_here(rhs + N2 * k + Np * s);
  __syncthreads();  // D
  T dx[C::DREG ? Nq : 1], dy[C::DREG ? Nq : 1];
  if constexpr (C::DREG) {
    march_row<Nq, T>(DT + i * RS, dx);
    march_row<Nq, T>(DT + j * RS, dy);
  }
  const int elr = (act ? el : 0) * Nq;
#pragma unroll
  for (int k = 0; k < Nq; ++k) {
    T *F = PL + (k & 1) * (2 * NS * ROW), *G = F + NS * ROW;
    if (act) {
      const T ri = T(1) / q[IR];
      const T P = pressure_ri<3, T>(q, ri, hz, p);
      T f[3][NS];
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        const T row[3] = {m[r], m[r + 3], m[r + 6]};
        contravariant_flux<3, T>(q, ri, P, MJ, row, f[r]);
      }
      acc[k][2] -= MJ * q[IR] * p.grav;
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        F[s * ROW + (elr + j) * RS + i] = f[0][s];
        G[s * ROW + (elr + i) * RS + j] = f[1][s];
      }
      if (k + 1 < Nq) load_plane(k + 1);
      T dz[Nq];
      march_row<Nq, T>(DZ + k * RS, dz);
#pragma unroll
      for (int x = 0; x < Nq; ++x)
#pragma unroll
        for (int s = 0; s < NS; ++s) acc[x][s] += dz[x] * f[2][s];
    }
    __syncthreads();
    if (act) {
      // the ξ and η terms are summed by themselves: each cancels to a small value
      // (the rows of D have the sum 0), the ζ sum is half done
      T d[Nq], t[NS];
      if constexpr (!C::DREG) march_row<Nq, T>(DT + i * RS, d);
#pragma unroll
      for (int s = 0; s < NS; ++s) t[s] = march_dot<Nq, T>(F + s * ROW + (elr + j) * RS, C::DREG ? dx : d, T(0));
      if constexpr (!C::DREG) march_row<Nq, T>(DT + j * RS, d);
#pragma unroll
      for (int s = 0; s < NS; ++s)
        acc[k][s] += march_dot<Nq, T>(G + s * ROW + (elr + i) * RS, C::DREG ? dy : d, t[s]);
    }
  }
  if (!act) return;
#pragma unroll
  for (int k = 0; k < Nq; ++k)
#pragma unroll
    for (int s = 0; s < NS; ++s) rhs[N2 * k + Np * s] = acc[k][s];
}

// Node x of the thread's line in direction R in a slab with rows of QR.
template <int Nq, int QR, int R>
__device__ __forceinline__ int line_slab(int a, int b, int x) {
  return R == 0 ? x + QR * (a + Nq * b) : R == 1 ? a + QR * (x + Nq * b) : a + QR * (b + Nq * x);
}

// What a thread of the gradient pass works with.
template <int Nq, typename T>
struct LineCtx {
  const T *Q, *vg, *DS;  // its element's state and geometry; D by rows m
  T *Qs, *Rs;            // its element's slabs
  int64_t e;
  int a, b;
  bool act;
};

// Step t = R + 3 cc of the gradient pass, direction R of component cc: the
// thread's line of -Σ_m D[m, i] ξ_R,cc (MJ prim) + face terms into acc.
template <int Nq, typename T, int R>
__device__ __forceinline__ void line_grad_dir(const LineCtx<Nq, T> &c, const T *__restrict__ sgeo, const T *M, int cc,
                                              const T (*av)[4], T (*acc)[4]) {
  using C = March<Nq, T>;
  constexpr int N2 = C::N2, NSG = 5, QR = C::QR, QE = C::QE;
  const T *sg = sgeo + NSG * (c.a + Nq * c.b + (int64_t)N2 * (2 * R + 6 * c.e)) + cc;
  const T n0 = sg[0], n1 = sg[NSG * N2];
#pragma unroll
  for (int i = 0; i < Nq; ++i)
#pragma unroll
    for (int s = 0; s < 4; ++s) acc[i][s] = T(0);
#pragma unroll
  for (int x = 0; x < Nq; ++x) {
    const int l = line_slab<Nq, QR, R>(c.a, c.b, x);
    const T h = -M[l];
    T f[4], d[Nq];
#pragma unroll
    for (int s = 0; s < 4; ++s) f[s] = h * c.Qs[s * QE + l];
    march_row<Nq, T>(c.DS + x * C::RD, d);
#pragma unroll
    for (int i = 0; i < Nq; ++i)
#pragma unroll
      for (int s = 0; s < 4; ++s) acc[i][s] += d[i] * f[s];
  }
#pragma unroll
  for (int s = 0; s < 4; ++s) {
    acc[0][s] += n0 * av[2 * R][s];
    acc[Nq - 1][s] += n1 * av[2 * R + 1][s];
  }
}

// Gradient pass of the viscous form: the records ∂_c prim = MJI (-Σ_r Dᵀ(MJ
// ξ_r,c prim) + Σ_f sMJ n_c (prim⁻ + prim⁺)/2), prim = u, v, w, T: nine steps,
// direction r of component c after the other, one metric field each, copied
// three steps ahead (cp.async) in the order in which the fields lie.
template <int Nq, typename T>
__global__ void __launch_bounds__(March<Nq, T>::THREADS, March<Nq, T>::blocks_for(March<Nq, T>::REGS_GRAD))
    k_line_grad(MarchArgs<T> A, PhysT<T> p) {
  using C = March<Nq, T>;
  constexpr int Np = C::Np, N2 = C::N2, NS = 5, NVG = 14, NSG = 5, IR = 3, MJF = 9, MJIF = 10, GC = 13, EPB = C::EPB, QR = C::QR,
                QE = C::QE, VW = C::VW;
  using V = typename Vec16<T>::type;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T *DS = reinterpret_cast<T *>(smem_raw), *S = reinterpret_cast<T *>(smem_raw + C::OFF_S);
  here_pointers(A.Qin, A.gq);
  const int tid = threadIdx.x, el = tid / N2, ab = tid % N2;
  const int64_t e0 = A.ebeg + (int64_t)blockIdx.x * EPB;
  LineCtx<Nq, T> c;
  c.act = el < EPB && e0 + el < A.eend;
  c.e = c.act ? e0 + el : e0;
  c.a = ab % Nq;
  c.b = ab / Nq;
  c.Q = A.Qin + c.e * (Np * NS);
  c.vg = A.vgeo + c.e * (Np * NVG);
  c.DS = DS;
  c.Qs = S + (c.act ? el : 0) * (C::GSLABS * QE);  // u, v, w, T, later times MJ
  c.Rs = c.Qs + 4 * QE;                            // four sums
  T *M = c.Rs + 4 * QE;                            // three metric fields
  auto copy_field = [&](int t) {
    if (c.act && t < 9) {
#pragma unroll
      for (int x = 0; x < Nq; ++x)
        cp_async<sizeof(T)>(M + (t % 3) * QE + line_slab<Nq, QR, 2>(c.a, c.b, x), c.vg + ab + N2 * x + Np * t);
    }
    cp_async_commit();
  };
  int32_t code[6];
  march_codes(A.nbr + 6 * c.e, code);
#pragma unroll
  for (int t = 0; t < 3; ++t) copy_field(t);
  for (int t = tid; t < Nq * Nq; t += C::THREADS) DS[(t % Nq) * C::RD + t / Nq] = A.D[t];
  T qr[NS];
#pragma unroll
  for (int s = 0; s < NS; ++s) qr[s] = A.qref.v[s];
  const T rR = T(1) / p.R;
  // primitives of a state, u, v, w and T
  auto prims = [&](const T *q, T hz, T *w) {
    const T ri = T(1) / q[IR];
#pragma unroll
    for (int d = 0; d < 3; ++d) w[d] = q[d] * ri;
    w[3] = pressure_ri<3, T>(q, ri, hz, p) * ri * rR;
  };
  T MJ[Nq];
#pragma unroll
  for (int x = 0; x < Nq; ++x) {
    const int n = ab + N2 * x, l = line_slab<Nq, QR, 2>(c.a, c.b, x);
    T q[NS], w[4];
#pragma unroll
    for (int s = 0; s < NS; ++s) q[s] = c.Q[n + Np * s] + qr[s];
    MJ[x] = c.vg[n + Np * MJF];
    prims(q, p.grav != T(0) ? c.vg[n + Np * GC] : T(0), w);
    if (c.act)
#pragma unroll
      for (int s = 0; s < 4; ++s) c.Qs[s * QE + l] = w[s];
  }
  // neighbours' half of the face averages
  T av[6][4];
#pragma unroll
  for (int f = 0; f < 6; ++f) {
    const bool wall = code[f] < 0;
    const int64_t e2 = wall ? c.e : (int64_t)(code[f] >> 3);
    const int vP = face_node<3, Nq>(wall ? f : code[f] & 7, ab);
    const T *Q2 = A.Qin + e2 * (Np * NS) + vP;
    T q[NS];
#pragma unroll
    for (int s = 0; s < NS; ++s) q[s] = Q2[Np * s] + qr[s];
    prims(q, p.grav != T(0) ? A.vgeo[vP + Np * (GC + NVG * e2)] : T(0), av[f]);
  }
  __syncthreads();  // D and the primitives
#pragma unroll
  for (int f = 0; f < 6; ++f) {  // sMJ (prim⁻ + prim⁺)/2; a wall mirrors the velocity
    const T *sg = A.sgeo + NSG * (ab + (int64_t)N2 * (f + 6 * c.e));
    const int x = (f & 1) * (Nq - 1);
    const T *w = c.Qs + (f < 2 ? line_slab<Nq, QR, 0>(c.a, c.b, x) : f < 4 ? line_slab<Nq, QR, 1>(c.a, c.b, x)
                                                                            : line_slab<Nq, QR, 2>(c.a, c.b, x));
    const T un2 = code[f] < 0 ? T(2) * (sg[0] * w[0] + sg[1] * w[QE] + sg[2] * w[2 * QE]) : T(0);
    const T h = T(0.5) * sg[3];
#pragma unroll
    for (int s = 0; s < 4; ++s) av[f][s] = h * (av[f][s] + w[s * QE] - (s < 3 ? un2 * sg[s] : T(0)));
  }
  __syncthreads();
  if (c.act)
#pragma unroll
    for (int x = 0; x < Nq; ++x)
#pragma unroll
      for (int s = 0; s < 4; ++s) c.Qs[s * QE + line_slab<Nq, QR, 2>(c.a, c.b, x)] *= MJ[x];
#pragma unroll
  for (int x = 0; x < Nq; ++x) MJ[x] = c.vg[ab + N2 * x + Np * MJIF];  // from here on MJI
  cp_async_wait<2>();
  __syncthreads();  // MJ prim and the first field
  T *__restrict__ gq = A.gq + c.e * (Np * GREC);
#pragma unroll 1
  for (int cc = 0; cc < 3; ++cc) {
    T acc[Nq][4];
    line_grad_dir<Nq, T, 0>(c, A.sgeo, M, cc, av, acc);
    if (c.act)
#pragma unroll
      for (int x = 0; x < Nq; ++x)
#pragma unroll
        for (int s = 0; s < 4; ++s) c.Rs[s * QE + line_slab<Nq, QR, 0>(c.a, c.b, x)] = acc[x][s];
    cp_async_wait<1>();
    __syncthreads();  // the ξ terms; the next field
    copy_field(3 * cc + 3);
    line_grad_dir<Nq, T, 1>(c, A.sgeo, M + QE, cc, av, acc);
    if (c.act)
#pragma unroll
      for (int x = 0; x < Nq; ++x)
#pragma unroll
        for (int s = 0; s < 4; ++s) c.Rs[s * QE + line_slab<Nq, QR, 1>(c.a, c.b, x)] += acc[x][s];
    cp_async_wait<1>();
    __syncthreads();  // the η terms; the next field
    copy_field(3 * cc + 4);
    line_grad_dir<Nq, T, 2>(c, A.sgeo, M + 2 * QE, cc, av, acc);
    if (c.act)
#pragma unroll
      for (int x = 0; x < Nq; ++x) {
        const int l = line_slab<Nq, QR, 2>(c.a, c.b, x);
        T v[4];
#pragma unroll
        for (int s = 0; s < 4; ++s) v[s] = (c.Rs[s * QE + l] + acc[x][s]) * MJ[x];
#pragma unroll
        for (int y = 0; y < 4 / VW; ++y)
          *reinterpret_cast<V *>(gq + GREC * (ab + N2 * x) + 4 * cc + y * VW) = *reinterpret_cast<const V *>(v + y * VW);
      }
    cp_async_wait<1>();
    __syncthreads();  // the sums are rewritten for the next direction; the next field
    copy_field(3 * cc + 5);
  }
  // (read again at the end: a store in the loop above, also one never taken, cost FP32
  // N=5 20^3 3 % of a step, 1111 -> 1148 us)
  if (A.rho && c.act)
#pragma unroll
    for (int x = 0; x < Nq; ++x) A.rho[c.e * Np + ab + N2 * x] = c.Q[ab + N2 * x + Np * IR] + qr[IR];
}

template <int Nq, typename T>
struct MarchLaunch {
  using M = March<Nq, T>;
  template <typename K>
  static cudaError_t launch(K kernel, size_t smem, const MarchArgs<T> &a, const PhysT<T> &p, cudaStream_t st) {
    const int64_t g = (a.eend - a.ebeg + M::EPB - 1) / M::EPB;
    if (g <= 0) return cudaSuccess;
    if (smem > 48 * 1024) {
      const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e != cudaSuccess) return e;
    }
    // (plain: a programmatic launch of either kernel starts its blocks unevenly and gains
    // nothing, us a viscous step plain / programmatic: N=7 FP32 8^3 157 / 231, 20^3 2020 / 2330,
    // N=4 FP32 10^3 121 / 173, N=7 FP64 20^3 4080 / 4540)
    kernel<<<(unsigned)g, M::THREADS, smem, st>>>(a, p);
    return cudaGetLastError();
  }
  static cudaError_t stage(bool visc, const MarchArgs<T> &a, const PhysT<T> &p, cudaStream_t st) {
    if (visc) return launch(k_march_stage<Nq, T, true>, M::smem_stage(), a, p, st);
    if constexpr (march_inviscid(Nq, sizeof(T))) return launch(k_march_stage<Nq, T, false>, M::smem_stage(), a, p, st);
    return cudaErrorNotSupported;
  }
  static cudaError_t volume(T *rhs, const T *Q, const T *vgeo, const T *D, int64_t nelem, const PhysT<T> &p,
                            cudaStream_t st) {
    if constexpr (march_volume_built(Nq, sizeof(T))) {
      const int64_t g = (nelem + M::EPB - 1) / M::EPB;
      if (g <= 0) return cudaSuccess;
      if (M::smem_volume() > 48 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(k_march_volume<Nq, T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   (int)M::smem_volume());
        if (e != cudaSuccess) return e;
      }
      k_march_volume<Nq, T><<<(unsigned)g, M::THREADS, M::smem_volume(), st>>>(rhs, Q, vgeo, D, nelem, p);
      return cudaGetLastError();
    }
    return cudaErrorNotSupported;
  }
  static cudaError_t grad(const MarchArgs<T> &a, const PhysT<T> &p, cudaStream_t st) {
    return launch(k_line_grad<Nq, T>, M::smem_grad(), a, p, st);
  }
};

}  // namespace cb

// Defines the launchers of precision T_ (included by cb_march_<prec>.cu).
#define CB_MARCH_DEFINE(T_)                                                                                         \
  namespace cb {                                                                                                    \
  template <>                                                                                                       \
  cudaError_t march_stage<T_>(int Nq, bool visc, const MarchArgs<T_> &a, const PhysT<T_> &p, cudaStream_t st) {     \
    static cudaError_t (*const f[])(bool, const MarchArgs<T_> &, const PhysT<T_> &, cudaStream_t) = {               \
        &MarchLaunch<2, T_>::stage, &MarchLaunch<3, T_>::stage, &MarchLaunch<4, T_>::stage,                         \
        &MarchLaunch<5, T_>::stage, &MarchLaunch<6, T_>::stage, &MarchLaunch<7, T_>::stage,                         \
        &MarchLaunch<8, T_>::stage, &MarchLaunch<9, T_>::stage, &MarchLaunch<10, T_>::stage,                        \
        &MarchLaunch<11, T_>::stage};                                                                               \
    return Nq < 2 || Nq > 11 ? cudaErrorInvalidValue : f[Nq - 2](visc, a, p, st);                                   \
  }                                                                                                                 \
  template <>                                                                                                       \
  cudaError_t march_volume<T_>(int Nq, T_ *rhs, const T_ *Q, const T_ *vgeo, const T_ *D, int64_t nelem,            \
                               const PhysT<T_> &p, cudaStream_t st) {                                               \
    static cudaError_t (*const f[])(T_ *, const T_ *, const T_ *, const T_ *, int64_t, const PhysT<T_> &,           \
                                    cudaStream_t) = {                                                               \
        &MarchLaunch<2, T_>::volume, &MarchLaunch<3, T_>::volume, &MarchLaunch<4, T_>::volume,                      \
        &MarchLaunch<5, T_>::volume, &MarchLaunch<6, T_>::volume, &MarchLaunch<7, T_>::volume,                      \
        &MarchLaunch<8, T_>::volume, &MarchLaunch<9, T_>::volume, &MarchLaunch<10, T_>::volume,                     \
        &MarchLaunch<11, T_>::volume};                                                                              \
    return Nq < 2 || Nq > 11 ? cudaErrorInvalidValue : f[Nq - 2](rhs, Q, vgeo, D, nelem, p, st);                    \
  }                                                                                                                 \
  template <>                                                                                                       \
  cudaError_t march_grad<T_>(int Nq, const MarchArgs<T_> &a, const PhysT<T_> &p, cudaStream_t st) {                 \
    static cudaError_t (*const f[])(const MarchArgs<T_> &, const PhysT<T_> &, cudaStream_t) = {                     \
        &MarchLaunch<2, T_>::grad, &MarchLaunch<3, T_>::grad, &MarchLaunch<4, T_>::grad, &MarchLaunch<5, T_>::grad, \
        &MarchLaunch<6, T_>::grad, &MarchLaunch<7, T_>::grad, &MarchLaunch<8, T_>::grad, &MarchLaunch<9, T_>::grad, \
        &MarchLaunch<10, T_>::grad, &MarchLaunch<11, T_>::grad};                                                    \
    return Nq < 2 || Nq > 11 ? cudaErrorInvalidValue : f[Nq - 2](a, p, st);                                         \
  }                                                                                                                 \
  }
