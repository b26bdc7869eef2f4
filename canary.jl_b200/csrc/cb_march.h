// Launchers of the 3-D column-march stages (cb_march.cuh), compiled in their
// own translation units (cb_march_f32.cu, cb_march_f64.cu).
#pragma once
#include "cb_dg.cuh"

namespace cb {

// One launch: elements ebeg .. eend - 1 (neighbour indices are absolute).
template <typename T>
struct MarchArgs {
  const T *Qin;
  T *Qout, *rhs;
  const T *vgeo, *sgeo;
  const int32_t *nbr;
  const T *D;
  T *gq;  // gradient (Np, 5, 3, nelem): written by the gradient pass, read by the viscous stage
  int64_t ebeg, eend;
  Offs<T, 5> qref;
  T rka, rkbdt;
  unsigned *status;
};

// Fused stage of order Nq - 1 (visc: the second viscous pass) and the
// gradient pass (chained: see launch_stage_kernel).
template <typename T>
cudaError_t march_stage(int Nq, bool visc, const MarchArgs<T> &a, const PhysT<T> &p, cudaStream_t st, int chained);
// rhs += volume integral (volumerhs!).
template <typename T>
cudaError_t march_volume(int Nq, T *rhs, const T *Q, const T *vgeo, const T *D, int64_t nelem, const PhysT<T> &p,
                         cudaStream_t st);
template <typename T>
cudaError_t march_grad(int Nq, const MarchArgs<T> &a, const PhysT<T> &p, cudaStream_t st, int chained);

}  // namespace cb
