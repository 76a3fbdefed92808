// Grid description shared by the acoustic kernels: explicitly rounded arithmetic, geometry and
// update regions, the misfit's adjoint source at a receiver, and the coefficient planes.
#pragma once
#include "common.cuh"
#include "l2.cuh"

namespace adfwi {
namespace ac {

// Explicitly rounded arithmetic (keeps the reference's operation order; no FMA contraction).
__device__ __forceinline__ float radd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float rsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float rmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double radd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double rsub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double rmul(double a, double b) { return __dmul_rn(a, b); }

template <typename T>
struct Geo {
  Layout L;
  int ns, nt, nr;
  int fs;     // first stencil row of u/w (nabc with a free surface, else 1)
  int fsurf;  // free surface on / off
  int zbeg;   // first tiled row (fs-1 with a free surface: rows above never change)
  int tiles_x;
  int nabc, nz, nx;
  T dt;
  T c1, c2;
  const int* src_z;          // padded source rows (ns)
  const int* src_x;          // padded source columns (ns)
  const int* tile_rcv_beg;   // ntiles+1 offsets into trcv_*
  const int* trcv_cell;      // (local row << 16) | local column
  const int* trcv_id;        // receiver index
  const int* tile_cell_beg;  // ntiles+1 offsets into tcell_*
  const int* tcell_cell;     // unique receiver cells of a tile, packed like trcv_cell
  const int* tcell_rbeg;     // ncells+1 offsets into cell_rcv
  const int* cell_rcv;       // receiver indices grouped by unique cell
  const int* grp_beg;        // ngroups+1 offsets: shots of each shot group (a group has one model)
  const int* grp_model;      // model of each shot group
  // Fused misfit: when fz_tr is set, the dL/d p-records handed to the adjoint are the
  // normalised L2 misfit's adjoint source, formed from the synthetic records (the p-record
  // gradient pointer then holds them) and fz_obs with the per-trace factors fz_tr.
  const T* fz_obs;
  const l2::TraceFactors<T>* fz_tr;
  const double* fz_gmul;     // device scale of the source (the objective's gradient w.r.t. the loss)
  int fz_norm_obs;
};

// dL/d p-record of shot sh, step t, receiver rid: from the gradient array gp, or formed from the
// records (gp) and the observed data with the misfit's factors when the misfit is fused. In two
// parts, the loads (RecPIn) and the value from them, so that a caller handling several
// receivers issues every load before the arithmetic (the IEEE divisions of the source have an
// out-of-line slow path, across which later loads are not hoisted).
// (gmul: the source's scale, read once by the caller with fused_scale)
template <typename T>
struct RecPIn {
  T v, o;
  l2::TraceFactors<T> f;
};
template <typename T>
__device__ __forceinline__ RecPIn<T> grad_rec_p_load(const Geo<T>& g, const T* gp, int sh, int t, int rid) {
  RecPIn<T> r;
  const int64_t o = ((int64_t)sh * g.nt + t) * g.nr + rid;
  r.v = gp[o];
  if (g.fz_tr != nullptr) {
    r.o = g.fz_obs[o];
    r.f = g.fz_tr[(int64_t)sh * g.nr + rid];
  }
  return r;
}
template <typename T>
__device__ __forceinline__ T grad_rec_p_value(const Geo<T>& g, const RecPIn<T>& r, int t, T gmul) {
  return g.fz_tr == nullptr ? r.v : l2::source(r.f, r.v, r.o, t, g.fz_norm_obs, gmul);
}
template <typename T>
__device__ __forceinline__ T grad_rec_p(const Geo<T>& g, const T* gp, int sh, int t, int rid, T gmul) {
  return grad_rec_p_value(g, grad_rec_p_load(g, gp, sh, t, rid), t, gmul);
}
template <typename T>
__device__ __forceinline__ T fused_scale(const Geo<T>& g) {
  return g.fz_gmul != nullptr ? (T)*g.fz_gmul : T(1);
}

// Update regions of acoustic_kernels.py:115, 139, 151.
template <typename T>
__device__ __forceinline__ bool in_p(const Geo<T>& g, int i, int j) {
  return i >= g.fs + 1 && i <= g.L.nzp - 3 && j >= 2 && j <= g.L.nxp - 3;
}
template <typename T>
__device__ __forceinline__ bool in_u(const Geo<T>& g, int i, int j) {
  return i >= g.fs && i <= g.L.nzp - 2 && j >= 1 && j <= g.L.nxp - 3;
}
template <typename T>
__device__ __forceinline__ bool in_w(const Geo<T>& g, int i, int j) {
  return i >= g.fs && i <= g.L.nzp - 3 && j >= 1 && j <= g.L.nxp - 2;
}
template <typename T>
__device__ __forceinline__ bool in_window(const Geo<T>& g, int i, int j) {
  return i >= g.nabc && i < g.nabc + g.nz && j >= g.nabc && j < g.nabc + g.nx;
}

// Masked coefficient planes for the branch-free pipelined kernels, computed with the
// reference's own operations (acoustic_kernels.py:257-265, and 1 - kappa of 115-160):
//   A1M = alpha1 on the p region, 0 elsewhere;  B1 = 1 - damp*dt on the p region, 1 elsewhere;
//   A2U / A2W = alpha2 on the u / w regions, 0 elsewhere;
//   B2 / B3 = 1 - 0.5*(d + d_right)*dt / 1 - 0.5*(d + d_below)*dt on the u / w regions, 1 elsewhere.
// Ghost cells stay 0. Planes follow the raw a1, a2, damp planes in the coefficient block.
enum { kA1 = 0, kA2 = 1, kDamp = 2, kA1M = 3, kB1 = 4, kA2U = 5, kA2W = 6, kB2 = 7, kB3 = 8, kNumCoef = 9 };

}  // namespace ac
}  // namespace adfwi
