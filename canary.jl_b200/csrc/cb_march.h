// Launchers of the 3-D column-march stages (cb_march.cuh), compiled in their
// own translation units (cb_march_f32.cu, cb_march_f64.cu).
#pragma once
#include "cb_dg.cuh"

namespace cb {

// The gradient of a node is one record of 12 values, ∂_c of u, v, w, T for each
// direction c: a neighbour's face node is then 48 (FP32) or 96 contiguous bytes
// instead of twelve lines of which the ξ faces use one value each.
constexpr int GREC = 12;

// One launch: elements ebeg .. eend - 1 (neighbour indices are absolute).
template <typename T>
struct MarchArgs {
  const T *Qin;
  T *Qout, *rhs;
  const T *vgeo, *sgeo;
  const int32_t *nbr;
  const T *D;
  T *gq;  // gradient records [element][Np][GREC]: written by the gradient pass, read by the viscous stage
  int64_t ebeg, eend;
  Offs<T, 5> qref;
  T rka, rkbdt;
  unsigned *status;
  T *rho = nullptr;  // where given, the gradient pass leaves the density of its input there, [element][Np]
};

// The shapes whose inviscid stage and whose volume integral are built (where
// Launch chooses them); the viscous passes are built for every order.
constexpr bool march_inviscid(int Nq, size_t w) { return Nq >= 11 || (Nq >= 9 && w == 8); }
constexpr bool march_volume_built(int Nq, size_t w) { return Nq >= (w == 4 ? 4 : 5); }

// Fused stage of order Nq - 1 (visc: the second viscous pass) and the
// gradient pass.
template <typename T>
cudaError_t march_stage(int Nq, bool visc, const MarchArgs<T> &a, const PhysT<T> &p, cudaStream_t st);
// rhs += volume integral (volumerhs!).
template <typename T>
cudaError_t march_volume(int Nq, T *rhs, const T *Q, const T *vgeo, const T *D, int64_t nelem, const PhysT<T> &p,
                         cudaStream_t st);
template <typename T>
cudaError_t march_grad(int Nq, const MarchArgs<T> &a, const PhysT<T> &p, cudaStream_t st);

}  // namespace cb
