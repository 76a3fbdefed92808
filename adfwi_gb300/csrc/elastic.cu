// 2-D velocity-stress elastic propagator (vx, vz, txx, tzz, txz), 4th / 6th order staggered
// grid, split-field PML or multiplicative absorbing layer, free surface, moment-tensor
// sources, 5-component receivers; exact discrete adjoint for the coefficient gradients;
// checkpoint / recompute driver and the C ABI.
//
// Reference algorithm (paths inside liufeng2317/ADFWI):
//   ADFWI/propagator/elastic_kernels.py:20-108    DiffCoef and the half-cell operators Dxfm/Dxbm/Dzfm/Dzbm
//   ADFWI/propagator/elastic_kernels.py:339-418   PML step (split stresses, source -MT/2 on both parts,
//                                                 totals, free-surface rows h-3..h-1, split velocities,
//                                                 totals, free-surface velocity rows, receivers, energy)
//   ADFWI/propagator/elastic_kernels.py:709-774   absorbing-layer step (unsplit, -MT/3 source, v *= damp)
//   ADFWI/propagator/elastic_kernels.py:917-1037  padding, index shifts, chunked loop, record dict
//
// One time step is two launches over (cell, shot), stresses and velocities (four with an absorbing layer
// under a free surface). Split fields are kept where the scheme needs them and updated in place, every
// other cell advances its totals; free-surface rows are written with the rows they mirror. A reverse
// step is two launches over tiles and groups of shots (three there): a block takes the shots of its group one
// after another and sums their coefficient gradients in a fixed order (deterministic, no atomics). The
// forward arithmetic uses explicitly rounded operations in the reference's order.
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <cmath>
#include <new>
#include <vector>

#include "../../include/adfwi_gb300.h"
#include "common.cuh"
#include "snapshot.cuh"

namespace adfwi {
namespace el {

__device__ __forceinline__ float radd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float rsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float rmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double radd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double rsub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double rmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float rdiv(float a, float b) { return __fdiv_rn(a, b); }
__device__ __forceinline__ double rdiv(double a, double b) { return __ddiv_rn(a, b); }
// Division by a number d that many are divided by, correctly rounded (P. Markstein, Computation of elementary
// functions on the IBM RISC System/6000 processor, 1990): with r = 1 / d rounded and e = 1 / d - r, y = x r + x e
// is one of the two numbers next to x / d, x - y d is exact, and y + (x - y d) r rounds to x / d. A numerator
// below `low`, where these would underflow, is scaled up first (tiny); zero needs nothing. It replaces the
// division because that takes a path of tens of instructions for numerators near zero, which some
// warp of every launch has at the front of a wave (300 steps of a shot on a 122 x 140 grid: 2.2 ms, with
// divisions 3.0).
template <typename T>
struct Divisor {
  static constexpr bool kF = sizeof(T) == 4;
  static constexpr T low = kF ? T(0x1p-95) : T(0x1p-900), most = kF ? T(0x1p90) : T(0x1p900), range = T(0x1p20);
  static constexpr T up = kF ? T(0x1p100) : T(0x1p900), down = T(1) / up;
  static constexpr T tie = kF ? T(0x1p-50) : T(0x1p-175);  // half of the least number, scaled up
  T d, r, e;
  T hi;  // numerators up to this; -1: the divisor is out of range and none is
  Divisor() = default;
  __host__ __device__ __forceinline__ explicit Divisor(T d_) : d(d_) {
    r = T(1) / d;
    e = fma(-r, d, T(1)) * r;
    hi = d >= T(1) / range && d <= range ? most : T(-1);
  }
  __device__ __forceinline__ bool takes(T x) const { return fabs(x) <= hi; }
  static __device__ __forceinline__ bool small(T x) { return fabs(x) < low && x != T(0); }
  __device__ __forceinline__ T of(T x) const {
    const T y = fma(x, r, x * e);
    return fma(fma(-y, d, x), r, y);
  }
  // Numerators of any size that is taken. Scaling a subnormal quotient back rounds a second time: half
  // way between two numbers, the remainder of the first rounding decides.
  __device__ __forceinline__ T tiny(T x) const {
    const bool s = fabs(x) < low;
    x = s ? x * up : x;
    const T y = of(x), z = s ? y * down : y, rem = fma(-y, d, x);
    if (s && fabs(y - z * up) == tie && rem != T(0)) return (y + copysign(tie, rem)) * down;
    return z;
  }
};

// Field indices inside the state blocks (each field = ns consecutive planes).
enum { TXX_X = 0, TXX_Z, TZZ_X, TZZ_Z, TXZ_X, TXZ_Z };  // split stresses (PML)
enum { VX_X = 0, VX_Z, VZ_X, VZ_Z };                    // split velocities (PML)
enum { TXX = 0, TZZ, TXZ };                             // stress totals / ABL stresses
enum { VX = 0, VZ };                                    // velocity totals / ABL velocities
enum { C11 = 0, C13, C15, C33, C35, C55, BX, BZ, BCX, BCZ, DAMP = 8 };  // coefficient planes

template <typename T>
struct Geo {
  Layout L;
  int ns, nt, nr;
  int fsurf, h;                // free surface; h = NN + 1
  int ilo, ihi, jlo, jhi;      // update region I = [NN, nzp-NN-1] x [NN, nxp-NN-1]
  int top, nabc, nz, nx;       // energy window
  T dt, dt_dx, dt_dz, hdt;
  Divisor<T> dx, dz;
  T f0, f1, f2;                // staggered coefficients
  const int* src_z;
  const int* src_x;
  const T* src_m;              // ns x 3 source weights (xx, zz, xz) already scaled for the mode
  const int* rcv_z;
  const int* rcv_x;
  const int* ucell_z;          // rows and columns of the unique receiver cells
  const int* ucell_x;
  const int* ucell_beg;        // ncells+1 offsets into ucell_rcv
  const int* ucell_rcv;
  const int* tile_beg;         // first unique receiver cell of each tile of the reverse kernels, and the end
  int ncells;
};

template <typename T>
__device__ __forceinline__ bool in_I(const Geo<T>& g, int i, int j) {
  return i >= g.ilo && i <= g.ihi && j >= g.jlo && j <= g.jhi;
}

// The cell of this thread in the per-cell kernels: a block of 256 threads covers a tile of
// 32 x 8 cells (full 128-byte rows of a plane; most rows that the vertical stencils read belong
// to the same block, so they come from L1), tiles row-major over the padded grid.
constexpr int kTileX = 32, kTileZ = 8, kTileThreads = kTileX * kTileZ;
#define EL_TILE_IJ                                                                   \
  const int tiles_x_ = (g.L.nxp + kTileX - 1) / kTileX;                              \
  const int ti_ = (int)blockIdx.x / tiles_x_, tj_ = (int)blockIdx.x - ti_ * tiles_x_; \
  const int i = ti_ * kTileZ + (int)threadIdx.x / kTileX;                            \
  const int j = tj_ * kTileX + (int)threadIdx.x % kTileX;                            \
  if (i >= g.L.nzp || j >= g.L.nxp) return;

#define EL_CELL_SHOT                                                                 \
  EL_TILE_IJ                                                                         \
  const int s = blockIdx.y;                                                          \
  const int64_t PL = g.L.plane, NSP = (int64_t)g.ns * PL;                            \
  const int64_t o = (int64_t)s * PL + g.L.off(i, j);                                 \
  (void)NSP;

// 1 / d of a PML denominator d = 1 + dt/2 d(x): exactly 1 where d is (outside the absorbing frame),
// so the division runs only inside the frame.
template <typename T>
__device__ __forceinline__ T pml_inv(T d) {
  return d == T(1) ? T(1) : T(1) / d;
}

// Gradient kernels: blockIdx.y picks a group of `eg` consecutive shots; the group's gradient
// partials (8 planes) start at gpart + blockIdx.y * 8 * PL and are summed over the groups in a
// fixed order at the end of the backward pass (deterministic).
#define EL_SHOT_GROUP                                                                \
  const int s_beg = blockIdx.y * eg, s_end = min(g.ns, s_beg + eg);                  \
  T* gbase = gpart + (int64_t)blockIdx.y * 8 * PL;

// ---- a thread takes kVW consecutive columns of a row, read and written as one vector of 8 bytes (16
// in double precision; columns start at a multiple of kVW, planes at multiples of 128 bytes with a
// ghost frame of 4 columns, so every vector is aligned). In the forward kernels a warp covers 32
// columns of 2 rows and a block of 128 threads 32 columns of 8 rows. One column per thread moves the
// same bytes with twice the instructions, four leave too few warps: 12.1, 10.5 and 12.7 ms for 200
// forward steps of 20 shots on a 242 x 480 grid with 1, 2 and 4.
constexpr int kVecThreads = 128, kVecX = 32;
constexpr int kVW = 2;
template <int B>
struct Bytes;
template <>
struct Bytes<8> {
  using t = int2;
};
template <>
struct Bytes<16> {
  using t = int4;
};
template <typename T>
using VecBits = typename Bytes<kVW * (int)sizeof(T)>::t;
template <typename T>
constexpr int kVecRows = kVecThreads * kVW / kVecX;
template <typename T>
struct Vec {
  T v[kVW];
};
template <typename T>
__device__ __forceinline__ Vec<T> ldv(const T* p) {
  Vec<T> r;
  *reinterpret_cast<VecBits<T>*>(r.v) = *reinterpret_cast<const VecBits<T>*>(p);
  return r;
}
template <typename T>
__device__ __forceinline__ void stv(T* p, const Vec<T>& x) {
  *reinterpret_cast<VecBits<T>*>(p) = *reinterpret_cast<const VecBits<T>*>(x.v);
}
// The vector at p of a row with the whole vectors that hold its NN neighbours on each side.
template <typename T, int NN>
struct Row {
  static constexpr int H = (NN + kVW - 1) / kVW * kVW;
  T v[kVW + 2 * H];
  __device__ __forceinline__ explicit Row(const T* p) {
#pragma unroll
    for (int k = 0; k < kVW + 2 * H; k += kVW)
      *reinterpret_cast<VecBits<T>*>(v + k) = *reinterpret_cast<const VecBits<T>*>(p - H + k);
  }
  __device__ __forceinline__ T operator()(int k) const { return v[H + k]; }
};
// Half-cell difference (elastic_kernels.py:66-108): `at(m)` is the value m cells from the lower of the two
// middle ones. `rounded` keeps the reference's operations, each rounded by itself, for the forward
// kernels; `diff` is contracted to multiply-adds, for the gradients' sums.
template <typename T>
struct Fd {
  T f0, f1, f2;
  template <int NN, typename A>
  __device__ __forceinline__ T rounded(const A& at) const {
    T r = radd(rmul(f0, rsub(at(1), at(0))), rmul(f1, rsub(at(2), at(-1))));
    if (NN == 3) r = radd(r, rmul(f2, rsub(at(3), at(-2))));
    return r;
  }
  template <int NN, typename A>
  __device__ __forceinline__ T diff(const A& at) const {
    T r = f0 * (at(1) - at(0)) + f1 * (at(2) - at(-1));
    if (NN == 3) r += f2 * (at(3) - at(-2));
    return r;
  }
};
// Vectors over their divisors by(k, e).
template <int N, typename T, typename By>
__device__ __forceinline__ void divide(Vec<T> (&a)[N], const By& by) {
  bool taken = true, small = false;
#pragma unroll
  for (int k = 0; k < N; ++k)
#pragma unroll
    for (int e = 0; e < kVW; ++e) {
      taken = taken && by(k, e).takes(a[k].v[e]);
      small = small || Divisor<T>::small(a[k].v[e]);
    }
  if (!taken) {
#pragma unroll
    for (int k = 0; k < N; ++k)
#pragma unroll
      for (int e = 0; e < kVW; ++e) a[k].v[e] = rdiv(a[k].v[e], by(k, e).d);
  } else if (small) {
#pragma unroll
    for (int k = 0; k < N; ++k)
#pragma unroll
      for (int e = 0; e < kVW; ++e) a[k].v[e] = by(k, e).tiny(a[k].v[e]);
  } else {
#pragma unroll
    for (int k = 0; k < N; ++k)
#pragma unroll
      for (int e = 0; e < kVW; ++e) a[k].v[e] = by(k, e).of(a[k].v[e]);
  }
}
// the x parts (even planes) over dx, the z parts over dz
template <int N, typename T>
__device__ __forceinline__ void over_dx_dz(const Geo<T>& g, Vec<T> (&a)[N]) {
  divide(a, [&](int k, int) -> const Divisor<T>& { return k & 1 ? g.dz : g.dx; });
}
template <typename T>
__host__ __device__ __forceinline__ int vec_tiles(const Layout& L) {
  return ((L.nxp + kVecX - 1) / kVecX) * ((L.nzp + kVecRows<T> - 1) / kVecRows<T>);
}
// this thread's row i and first column j
#define EL_VEC_IJ                                                               \
  constexpr int W = kVW;                                                     \
  const int tiles_x_ = (g.L.nxp + kVecX - 1) / kVecX;                           \
  const int ti_ = (int)blockIdx.x / tiles_x_, tj_ = (int)blockIdx.x - ti_ * tiles_x_; \
  const int i = ti_ * kVecRows<T> + (int)threadIdx.x / (kVecX / W);             \
  const int j = tj_ * kVecX + (int)threadIdx.x % (kVecX / W) * W;               \
  if (i >= g.L.nzp || j >= g.L.nxp) return;                                     \
  const int64_t PL = g.L.plane, NSP = (int64_t)g.ns * PL, P = g.L.pitch;        \
  const int64_t occ = g.L.off(i, j);

// The velocity rows above a free surface (elastic_kernels.py:395-402) from the totals of rows h-1
// and h: vz[h-3] = vz[h-2] = vz[h-1] and vx[h-2] from vz[h-1] and vx[h], on columns J; zero
// elsewhere. The stress update reads them through this function (vx, vz: a shot's planes), so they
// need no pass of their own before it.
template <typename T>
__device__ __forceinline__ T vel_above(const Geo<T>& g, const T* vx, const T* vz, bool x, int r, int j) {
  const int h = g.h;
  if (r >= h - 1) return (x ? vx : vz)[g.L.off(r, j)];
  if (j < g.jlo || j > g.jhi || r < h - 3) return T(0);
  const T up = vz[g.L.off(h - 1, j)];
  if (!x) return up;
  if (r == h - 3) return T(0);
  const T right = vz[g.L.off(h - 1, j + 1)];
  return radd(rsub(radd(rsub(j + 1 <= g.jhi ? right : T(0), up), right), up), vx[g.L.off(h, j)]);
}
// Receiver records taken by extra blocks of the step kernels (elastic_kernels.py:407-411): the
// blocks of a launch after its tiles gather `ncomp` components of step `it` from fields that the
// launch only reads, so recording costs no launch of its own. src: the first component's planes;
// c0: its index in the record array; rows_above: the velocity rows above the free surface are not
// in `src` (a receiver there reads vel_above).
template <typename T>
__device__ __forceinline__ void record_block(const Geo<T>& g, int tiles, int it, const T* src, int ncomp, int c0,
                                             T* rec, bool rows_above = false) {
  const int r = ((int)blockIdx.x - tiles) * (int)blockDim.x + (int)threadIdx.x;
  if (r >= g.nr) return;
  const int64_t NSP = (int64_t)g.ns * g.L.plane, RS = (int64_t)g.ns * g.nt * g.nr;
  const int i = g.rcv_z[r], j = g.rcv_x[r];
  const int64_t oc = g.L.off(i, j);
  rows_above = rows_above && g.fsurf && i < g.h - 1;
  const int s = blockIdx.y;
  const int64_t o = (int64_t)s * g.L.plane + oc, e = ((int64_t)s * g.nt + it) * g.nr + r;
  if (rows_above) {
    const T *vx = src + o - oc, *vz = vx + NSP;
    rec[c0 * RS + e] = vel_above(g, vx, vz, true, i, j);
    rec[(c0 + 1) * RS + e] = vel_above(g, vx, vz, false, i, j);
    return;
  }
  for (int c = 0; c < ncomp; ++c) rec[(c0 + c) * RS + e] = src[c * NSP + o];
}

// Stress totals of a vector (offset o, row i) with the free-surface rows h-3 .. h-1
// (elastic_kernels.py:375-384, 738-742): tzz[h-1] = 0, tzz[h-2] = -tzz[h], txz[h-2] = -txz[h-1],
// txz[h-3] = -txz[h]. Rows h-1 and h write the mirrored values; the rows they mirror to leave
// theirs out.
template <typename T>
__device__ __forceinline__ void store_stress(const Geo<T>& g, int i, int64_t o, int64_t NSP, const Vec<T>& xx, Vec<T> zz,
                                             const Vec<T>& xz, T* tt) {
  const int64_t P = g.L.pitch;
  const int h = g.h;
  stv(tt + TXX * NSP + o, xx);
  if (!g.fsurf || i > h || i < h - 3) {
    stv(tt + TZZ * NSP + o, zz);
    stv(tt + TXZ * NSP + o, xz);
    return;
  }
  Vec<T> nz, nx;
#pragma unroll
  for (int e = 0; e < kVW; ++e) {
    if (i == h - 1) zz.v[e] = T(0);
    nz.v[e] = -zz.v[e];
    nx.v[e] = -xz.v[e];
  }
  if (i != h - 2) stv(tt + TZZ * NSP + o, zz);
  if (i >= h - 1) stv(tt + TXZ * NSP + o, xz);
  if (i == h - 1) stv(tt + TXZ * NSP + o - P, nx);
  if (i == h) {
    stv(tt + TZZ * NSP + o - 2 * P, nz);
    stv(tt + TXZ * NSP + o - 3 * P, nx);
  }
}

// ======================================================================= forward
// Split-field update with PML (elastic_kernels.py:351-402) or unsplit update with an absorbing
// layer (:733-774), fields and totals in one pass, two launches per step: the stress rows that
// mirror others at the free surface are written by the rows they mirror; with PML the velocity rows
// above it are formed and written by the next stress update (with an absorbing layer they are inputs
// of the damping and take two small launches).
//
// What bounds them is latency: a thread's chain of loads from L2 and the launch boundary, not L2 or
// DRAM bandwidth (30 % of either) nor issue slots (32 %). So a thread has all its loads in flight at
// once and reads what the launch before does not write ahead of that launch's end; with two columns a
// thread that takes 96 registers, five blocks per SM (six and eight spill and measured 7 and 30 %
// slower). 300 steps of one shot on a 122 x 140 grid: 4.56 -> 3.0 ms; 200 steps of 20 shots on a
// 242 x 480 grid: 16.3 -> 10.5 ms, against one cell and two shots per thread with scalar loads and
// divisions by dx.
//
// Every operation is the reference's, rounded by itself and in its order. Products and sums fused, with
// dt / dx rounded into the difference coefficients, took as long (2.2 to 2.3 ms for the 300 steps either way)
// and left the energy maps of some short solves two to four times further from 64 bits.
//
// Cells that keep split fields: outside the update region, where a PML factor differs from 1,
// and in the surface rows that mirror others or are mirrored (h-3 .. h) plus one. Every other cell
// advances its totals directly: there the split update is x' = x + a, z' = z + b, total = x' + z'
// (the factors are exactly 1), so the unsplit t' = (t + a) + b differs only by one rounding of the
// sum and moves half the bytes.
template <typename T>
__device__ __forceinline__ bool keeps_split(const Geo<T>& g, int i, T bcx, T bcz) {
  return bcx != T(0) || bcz != T(0) || (g.fsurf && i <= g.h + 1);
}

// tprev: stress totals at the start of the step (tt itself when the totals advance in place);
// tt: where the new totals go; rec: the velocity records of step it - 1 are taken (null: none).
template <typename T, int NN, bool PML>
__global__ void __launch_bounds__(kVecThreads, 5)
    stress_step(Geo<T> g, int it, const T* __restrict__ cf, T* __restrict__ v, T* __restrict__ ts, T* tt, const T* tprev,
                const T* __restrict__ wav, T* __restrict__ rec) {
  if (const int tiles = vec_tiles<T>(g.L); (int)blockIdx.x >= tiles) {
    griddep_wait();
    griddep_launch_dependents();
    record_block(g, tiles, it - 1, (const T*)v, 2, 3, rec, PML);
    return;
  }
  EL_VEC_IJ
  const int s = blockIdx.y;
  const int64_t so = (int64_t)s * PL, o = so + occ;
  const int src_row = g.src_z[s], src_col = g.src_x[s];
  // What the launch before this one (the velocity update, or work that the stream has completed) does not
  // write is read ahead of its end.
  Vec<T> c[6], bcx, bcz, t[3], px[3], pz[3];
#pragma unroll
  for (int k = 0; k < 6; ++k) c[k] = ldv(cf + (C11 + k) * PL + occ);
#pragma unroll
  for (int k = 0; k < 3; ++k) t[k] = ldv(tprev + k * NSP + o);
  bool in[W], sp[W], any = false;
  if (PML) {
    bcx = ldv(cf + BCX * PL + occ);
    bcz = ldv(cf + BCZ * PL + occ);
  }
#pragma unroll
  for (int e = 0; e < W; ++e) {
    in[e] = in_I(g, i, j + e);
    sp[e] = PML && (!in[e] || keeps_split(g, i, bcx.v[e], bcz.v[e]));
    any = any || sp[e];
  }
  griddep_wait();  // launched with programmatic serialisation in the time loops
  griddep_launch_dependents();
  {
    const Row<T, NN> x(v + VX * NSP + o), z(v + VZ * NSP + o);
    Vec<T> rx[2 * NN + 1], rz[2 * NN + 1];  // rows i - NN .. i + NN
#pragma unroll
    for (int k = 0; k <= 2 * NN; ++k)
      if (k != NN) {
        rx[k] = ldv(v + VX * NSP + o + (k - NN) * P);
        rz[k] = ldv(v + VZ * NSP + o + (k - NN) * P);
      }
    if (any) {
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        px[k] = ldv(ts + (2 * k) * NSP + o);
        pz[k] = ldv(ts + (2 * k + 1) * NSP + o);
      }
    }
    // source of the step on the cell of this vector that holds it
    T w[3] = {T(0), T(0), T(0)};
    const int se = i == src_row ? src_col - j : -1;
    const bool has_src = se >= 0 && se < W;
    if (has_src) {
      const T wv = wav[(int64_t)s * g.nt + it];
#pragma unroll
      for (int k = 0; k < 3; ++k) w[k] = rmul(g.src_m[3 * s + k], wv);
    }
    if (PML && g.fsurf && i <= g.h + NN - 2) {  // rows above the surface are read: form them
      Vec<T> ax, az;
#pragma unroll
      for (int e = 0; e < W; ++e) {
        ax.v[e] = vel_above(g, v + VX * NSP + so, v + VZ * NSP + so, true, g.h - 2, j + e);
        az.v[e] = vel_above(g, v + VX * NSP + so, v + VZ * NSP + so, false, g.h - 2, j + e);
      }
#pragma unroll
      for (int k = 0; k < NN; ++k) {
        const int r = i + k - NN;
#pragma unroll
        for (int e = 0; e < W; ++e) {
          if (r < g.h - 1) rx[k].v[e] = r == g.h - 2 ? ax.v[e] : T(0);
          if (r < g.h - 1) rz[k].v[e] = r >= g.h - 3 ? az.v[e] : T(0);
        }
      }
      if (i == g.h - 1) {  // and kept for whoever reads the velocities later
        stv(v + VX * NSP + o - P, ax);
        stv(v + VZ * NSP + o - P, az);
#pragma unroll
        for (int e = 0; e < W; ++e) ax.v[e] = T(0);
        stv(v + VX * NSP + o - 2 * P, ax);
        stv(v + VZ * NSP + o - 2 * P, az);
      }
    }
    const Fd<T> fd{g.f0, g.f1, g.f2};
    // the increments of the split parts xx_x, xx_z, zz_x, zz_z, xz_x, xz_z: times dt / dx or dt / dz with
    // PML, as sums of coefficient and difference products otherwise
    Vec<T> a[6];
#pragma unroll
    for (int e = 0; e < W; ++e) {
      auto zx = [&](int m) { return m == 0 ? x(e) : rx[NN + m].v[e]; };
      auto zz = [&](int m) { return m == 0 ? z(e) : rz[NN + m].v[e]; };
      const T dxbm_vx = fd.template rounded<NN>([&](int m) { return x(e - 1 + m); });
      const T dxbm_vz = fd.template rounded<NN>([&](int m) { return z(e - 1 + m); });
      const T dzbm_vx = fd.template rounded<NN>([&](int m) { return zx(m - 1); });
      const T dzbm_vz = fd.template rounded<NN>([&](int m) { return zz(m - 1); });
      const T dxfm_vx = fd.template rounded<NN>([&](int m) { return x(e + m); });
      const T dxfm_vz = fd.template rounded<NN>([&](int m) { return z(e + m); });
      const T dzfm_vx = fd.template rounded<NN>(zx);
      const T dzfm_vz = fd.template rounded<NN>(zz);
      const T c11 = c[0].v[e], c13 = c[1].v[e], c15 = c[2].v[e], c33 = c[3].v[e], c35 = c[4].v[e], c55 = c[5].v[e];
      a[0].v[e] = radd(rmul(c11, dxbm_vx), rmul(c15, dxbm_vz));
      a[1].v[e] = radd(rmul(c15, dzbm_vx), rmul(c13, dzbm_vz));
      a[2].v[e] = radd(rmul(c13, dxbm_vx), rmul(c35, dxbm_vz));
      a[3].v[e] = radd(rmul(c35, dzbm_vx), rmul(c33, dzbm_vz));
      a[4].v[e] = radd(rmul(c15, dxfm_vx), rmul(c55, dxfm_vz));
      a[5].v[e] = radd(rmul(c55, dzfm_vx), rmul(c35, dzfm_vz));
      if (PML) {
#pragma unroll
        for (int k = 0; k < 6; ++k) a[k].v[e] = rmul(k & 1 ? g.dt_dz : g.dt_dx, a[k].v[e]);
      }
    }
    if (!PML) {
      over_dx_dz(g, a);
#pragma unroll
      for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int e = 0; e < W; ++e) {
          if (in[e]) t[k].v[e] = radd(t[k].v[e], rmul(g.dt, radd(a[2 * k].v[e], a[2 * k + 1].v[e])));
          if (has_src && e == se) t[k].v[e] = radd(t[k].v[e], w[k]);
        }
    } else {
#pragma unroll
      for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int e = 0; e < W; ++e)
          if (!sp[e]) {
            t[k].v[e] = radd(radd(t[k].v[e], a[2 * k].v[e]), a[2 * k + 1].v[e]);
            if (has_src && e == se) t[k].v[e] = radd(t[k].v[e], rmul(T(2), w[k]));  // -MT/2 w on both split parts
          }
      if (any) {
        T pxn[W], pxi[W], pzn[W], pzi[W];
#pragma unroll
        for (int e = 0; e < W; ++e) {
          pxn[e] = rsub(T(1), rmul(g.hdt, bcx.v[e]));
          pzn[e] = rsub(T(1), rmul(g.hdt, bcz.v[e]));
          pxi[e] = pml_inv(radd(T(1), rmul(g.hdt, bcx.v[e])));
          pzi[e] = pml_inv(radd(T(1), rmul(g.hdt, bcz.v[e])));
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) {
#pragma unroll
          for (int e = 0; e < W; ++e)
            if (sp[e]) {
              if (in[e]) {
                px[k].v[e] = rmul(radd(rmul(pxn[e], px[k].v[e]), a[2 * k].v[e]), pxi[e]);
                pz[k].v[e] = rmul(radd(rmul(pzn[e], pz[k].v[e]), a[2 * k + 1].v[e]), pzi[e]);
              }
              if (has_src && e == se) {
                px[k].v[e] = radd(px[k].v[e], w[k]);
                pz[k].v[e] = radd(pz[k].v[e], w[k]);
              }
              t[k].v[e] = radd(px[k].v[e], pz[k].v[e]);
            }
          stv(ts + (2 * k) * NSP + o, px[k]);
          stv(ts + (2 * k + 1) * NSP + o, pz[k]);
        }
      }
    }
    store_stress(g, i, o, NSP, t[TXX], t[TZZ], t[TXZ], tt);
  }
}

// vprev: velocity totals at the start of the step (v itself when they advance in place); rec: the
// stress records of step it are taken (null: none). Without a free surface the absorbing layer's
// damping is applied here; with one it follows the surface rows.
template <typename T, int NN, bool PML>
__global__ void __launch_bounds__(kVecThreads, 5)
    vel_step(Geo<T> g, int it, const T* __restrict__ cf, const T* __restrict__ tt, T* __restrict__ vs, T* v,
             const T* vprev, T* __restrict__ rec) {
  if (const int tiles = vec_tiles<T>(g.L); (int)blockIdx.x >= tiles) {
    griddep_wait();
    griddep_launch_dependents();
    record_block(g, tiles, it, tt, 3, 0, rec);
    return;
  }
  EL_VEC_IJ
  const int64_t o = (int64_t)blockIdx.y * PL + occ;
  // What the launch before this one (the stress update) does not write is read ahead of its end.
  const Vec<T> bx = ldv(cf + BX * PL + occ), bz = ldv(cf + BZ * PL + occ);
  Vec<T> nx = ldv(vprev + VX * NSP + o), nz = ldv(vprev + VZ * NSP + o);
  Vec<T> bcx, bcz, damp, f[4];
  if (PML) {
    bcx = ldv(cf + BCX * PL + occ);
    bcz = ldv(cf + BCZ * PL + occ);
  } else {
    damp = ldv(cf + DAMP * PL + occ);
  }
  bool in[W], sp[W], any = false;
#pragma unroll
  for (int e = 0; e < W; ++e) {
    in[e] = in_I(g, i, j + e);
    sp[e] = PML && (!in[e] || keeps_split(g, i, bcx.v[e], bcz.v[e]));
    any = any || sp[e];
  }
  griddep_wait();  // launched with programmatic serialisation in the time loops
  griddep_launch_dependents();
  {
    const Row<T, NN> xx(tt + TXX * NSP + o), xz(tt + TXZ * NSP + o);
    Vec<T> rxz[2 * NN], rzz[2 * NN];  // rows i - NN .. i + NN - 1 of txz, i - NN + 1 .. i + NN of tzz
#pragma unroll
    for (int k = 0; k < 2 * NN; ++k) {
      if (k != NN) rxz[k] = ldv(tt + TXZ * NSP + o + (k - NN) * P);
      rzz[k] = ldv(tt + TZZ * NSP + o + (k - NN + 1) * P);
    }
    if (any) {
#pragma unroll
      for (int k = 0; k < 4; ++k) f[k] = ldv(vs + k * NSP + o);
    }
    const Fd<T> fd{g.f0, g.f1, g.f2};
    // the increments of the split parts vx_x, vx_z, vz_x, vz_z with PML, the differences over dx or dz otherwise
    Vec<T> a[4];
#pragma unroll
    for (int e = 0; e < W; ++e) {
      a[0].v[e] = fd.template rounded<NN>([&](int m) { return xx(e + m); });
      a[1].v[e] = fd.template rounded<NN>([&](int m) { return m == 1 ? xz(e) : rxz[NN + m - 1].v[e]; });
      a[2].v[e] = fd.template rounded<NN>([&](int m) { return xz(e - 1 + m); });
      a[3].v[e] = fd.template rounded<NN>([&](int m) { return rzz[NN + m - 1].v[e]; });
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (PML) a[k].v[e] = rmul(rmul(g.dt, (k < 2 ? bx : bz).v[e]), a[k].v[e]);
    }
    over_dx_dz(g, a);
#pragma unroll
    for (int e = 0; e < W; ++e) {
      if (!PML) {
        if (in[e]) {
          nx.v[e] = radd(nx.v[e], rmul(rmul(g.dt, bx.v[e]), radd(a[0].v[e], a[1].v[e])));
          nz.v[e] = radd(nz.v[e], rmul(rmul(g.dt, bz.v[e]), radd(a[2].v[e], a[3].v[e])));
        }
        if (!g.fsurf) {
          nx.v[e] = rmul(nx.v[e], damp.v[e]);
          nz.v[e] = rmul(nz.v[e], damp.v[e]);
        }
      } else if (!sp[e]) {
        nx.v[e] = radd(radd(nx.v[e], a[0].v[e]), a[1].v[e]);
        nz.v[e] = radd(radd(nz.v[e], a[2].v[e]), a[3].v[e]);
      }
    }
    if (PML) {
      if (any) {
        Divisor<T> d[2][W];
#pragma unroll
        for (int e = 0; e < W; ++e) {
          d[0][e] = Divisor<T>(radd(T(1), rmul(g.hdt, bcx.v[e])));
          d[1][e] = Divisor<T>(radd(T(1), rmul(g.hdt, bcz.v[e])));
        }
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
          for (int e = 0; e < W; ++e)
            a[k].v[e] = radd(rmul(rsub(T(1), rmul(g.hdt, (k & 1 ? bcz : bcx).v[e])), f[k].v[e]), a[k].v[e]);
        divide(a, [&](int k, int e) -> const Divisor<T>& { return d[k & 1][e]; });
#pragma unroll
        for (int k = 0; k < 4; ++k) {
#pragma unroll
          for (int e = 0; e < W; ++e)
            if (sp[e] && in[e]) f[k].v[e] = a[k].v[e];
          stv(vs + k * NSP + o, f[k]);
        }
#pragma unroll
        for (int e = 0; e < W; ++e)
          if (sp[e]) {
            nx.v[e] = radd(f[VX_X].v[e], f[VX_Z].v[e]);
            nz.v[e] = radd(f[VZ_X].v[e], f[VZ_Z].v[e]);
          }
      }
      if (g.fsurf && (i == g.h - 2 || i == g.h - 3)) return;  // the next stress update's
    }
    stv(v + VX * NSP + o, nx);
    stv(v + VZ * NSP + o, nz);
  }
}

// Free-surface velocity rows in place (elastic_kernels.py:753-756); one thread per column in J.
// Reads only rows h-1, h and the cell (h-2, jhi+1), none of which any thread writes.
template <typename T>
__global__ void vel_fs_abl(Geo<T> g, T* __restrict__ v) {
  griddep_wait();
  griddep_launch_dependents();
  const int j = g.jlo + blockIdx.x * blockDim.x + threadIdx.x;
  if (j > g.jhi) return;
  const int s = blockIdx.y, h = g.h;
  const int64_t NSP = (int64_t)g.ns * g.L.plane, so = (int64_t)s * g.L.plane;
  T* vx = v + VX * NSP + so;
  T* vz = v + VZ * NSP + so;
  const T vz_up = vz[g.L.off(h - 1, j)];
  const T vzn_r = (j + 1 <= g.jhi) ? vz[g.L.off(h - 1, j + 1)] : vz[g.L.off(h - 2, j + 1)];
  const T vxh = vx[g.L.off(h, j)];
  const T vz_up_r = vz[g.L.off(h - 1, j + 1)];
  vz[g.L.off(h - 2, j)] = vz_up;
  vx[g.L.off(h - 2, j)] = radd(rsub(radd(rsub(vzn_r, vz_up), vz_up_r), vz_up), vxh);
  vz[g.L.off(h - 3, j)] = vz_up;
}

template <typename T>
__global__ void damp_v(Geo<T> g, const T* __restrict__ cf, T* __restrict__ v) {
  griddep_wait();
  griddep_launch_dependents();
  EL_CELL_SHOT
  const T d = cf[DAMP * PL + g.L.off(i, j)];
  v[VX * NSP + o] = rmul(v[VX * NSP + o], d);
  v[VZ * NSP + o] = rmul(v[VZ * NSP + o], d);
}

// The velocity records of step it, after the last step (the stress update of the next one would
// have taken them).
template <typename T>
__global__ void record_v(Geo<T> g, int it, const T* __restrict__ v, T* __restrict__ rec, bool rows_above) {
  griddep_wait();
  griddep_launch_dependents();
  record_block(g, 0, it, v, 2, 3, rec, rows_above);
}

// forward_wavefield_* += sum_s X^2 of the last step of a chunk (elastic_kernels.py:414-418, 1016-1021).
template <typename T>
__global__ void energy(Geo<T> g, const T* __restrict__ tt, const T* __restrict__ v, T* fw) {
  const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (e >= (int64_t)g.nz * g.nx) return;
  const int i = (int)(e / g.nx) + g.top, j = (int)(e % g.nx) + g.nabc;
  const int64_t NSP = (int64_t)g.ns * g.L.plane, oc = g.L.off(i, j);
  const int64_t n = (int64_t)g.nz * g.nx;
  const T* src[5] = {tt + TXX * NSP, tt + TZZ * NSP, tt + TXZ * NSP, v + VX * NSP, v + VZ * NSP};
  for (int c = 0; c < 5; ++c) {
    T acc = T(0);
    for (int s = 0; s < g.ns; ++s) {
      T x = src[c][(int64_t)s * g.L.plane + oc];
      acc += x * x;
    }
    fw[c * n + e] += acc;
  }
}

// ======================================================================= adjoint
// dL/d velocity records of step it added to lv, before the first reverse step (each adj_v_step adds
// those of the step before its own). One thread per (unique receiver cell, shot).
template <typename T>
__global__ void adj_inject(Geo<T> g, int it, const T* __restrict__ grec, T* lv) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= g.ncells) return;
  const int s = blockIdx.y;
  const int64_t NSP = (int64_t)g.ns * g.L.plane;
  const int64_t o = (int64_t)s * g.L.plane + g.L.off(g.ucell_z[q], g.ucell_x[q]);
  const int64_t RS = (int64_t)g.ns * g.nt * g.nr, base = ((int64_t)s * g.nt + it) * g.nr;
  for (int c = 0; c < 2; ++c) {
    T a = T(0);
    for (int m = g.ucell_beg[q]; m < g.ucell_beg[q + 1]; ++m) a += grec[(3 + c) * RS + base + g.ucell_rcv[m]];
    lv[c * NSP + o] += a;
  }
}

// Adjoint of the free-surface velocity rows (reverse of elastic_kernels.py:400-402, 753-756): lambda
// of the velocities BEFORE the rows h-3 / h-2 were overwritten, at cell (i, j). l(comp, ii, jj) is
// the lambda after; ax, az hold l at (i, j) on entry.
template <typename T, typename F>
__device__ __forceinline__ void vfs_adjoint(const Geo<T>& g, int i, int j, const F& l, T& ax, T& az) {
  const int h = g.h;
  auto inJ = [&](int m) { return m >= g.jlo && m <= g.jhi; };
  if (i == h - 3) {
    if (inJ(j)) az = T(0);
  } else if (i == h - 2) {
    if (inJ(j)) {
      ax = T(0);
      az = T(0);
    } else if (inJ(j - 1)) {
      az += l(VX, i, j - 1);
    }
  } else if (i == h - 1) {
    const T a_l = inJ(j - 1) ? l(VX, h - 2, j - 1) : T(0);
    const T a_c = inJ(j) ? l(VX, h - 2, j) : T(0);
    T r = az + a_l - a_c;
    if (inJ(j)) r += l(VZ, h - 2, j) + l(VZ, h - 3, j) + a_l - a_c;
    az = r;
  } else if (i == h) {
    if (inJ(j)) ax += l(VX, h - 2, j);
  }
}

// Adjoint of the free-surface stress rows (reverse of elastic_kernels.py:381-384) at a cell of row i:
// azz, axz hold the lambda there on entry, lzz and lxz point to it in planes of pitch P.
template <typename T>
__device__ __forceinline__ void tfs_adjoint(const Geo<T>& g, const T* lzz, const T* lxz, int i, int P, T& azz, T& axz) {
  const int h = g.h;
  if (i == h - 3) axz = T(0);
  if (i == h - 2) {
    axz = T(0);
    azz = T(0);
  }
  if (i == h - 1) {
    azz = T(0);
    axz -= lxz[-P];
  }
  if (i == h) {
    azz -= lzz[-2 * P];
    axz -= lxz[-3 * P];
  }
}

// The reverse step is two launches. Each takes a group of shots per block, a tile of kAR rows x 32
// columns with a vector of kVW columns per thread, and per shot: forms in shared memory the adjoint
// sources of the update that it reverses (lambda after the step times coefficient times dt/dx or
// dt/dz, zero outside I) on the tile and on the NN rows or 4 columns around it that the transposed
// differences read, then applies the transposes and adds to the gradients in registers.
//
// Cells that keep split fields in the forward step have a lambda per split part, advanced here as
// S * lambda + lambda of the total (read from one copy and written to the other, so that no block
// reads a halo cell another block has already advanced), and the transposes overwrite the lambda
// of the totals. In every other cell both parts of a field have the same lambda for all time (S = 1 and
// equal increments): only its running sum is kept, in the plane of the total, to which the transposes
// add. That is the case of all cells with an absorbing layer, whose update is unsplit.
//
// dL/d records: stresses are added by adj_t_step after its transposes, the velocities of the step
// before by adj_v_step after its own.
//
// What bounds them is the latency of a shot's chain: copies, sources, barrier, transposes. All that a
// shot reads is copied to shared memory while the shot before is evaluated (loads into registers
// instead were moved to their uses by the compiler: 66 and 75 us a launch for 20 shots on a 282 x 480
// grid, with copies 50 and 57); histories and records are copied ahead of the end of the launch
// before. Shared memory (75 and 91 KB) and registers (80 and 128) allow three and two blocks of 256
// threads per SM; with 3 shots per block and more the copies of all but the first shot are hidden.
// 400 gradient steps of 20 shots on a 242 x 480 grid take 62 ms (75 with a lambda per split part in
// every cell, tiles of 8 rows, and two launches for the dL/d records).
constexpr int kAR = 16;
template <typename T>
constexpr int kAdjThreads = kAR * kVecX / kVW;
constexpr int kAXW = kVecX + 8;                             // an x plane's row: columns j0-4 .. j0+35
constexpr int kAX = kAR * kAXW, kAZ = (kAR + 6) * kVecX;  // x plane: tile rows; z plane: rows i0-3 ..
constexpr int kAH = (kAR + 6) * kAXW;                       // a history plane: z plane's rows, x plane's columns
constexpr int kAI = kAR * kVecX;                            // a plane of the tile alone
// one of two buffers (split lambda, then sources; lambda of the totals; history; lambda to add to), and
// all shared memory (two buffers, dL/d records)
constexpr int kAdjTBuf = 2 * kAX + 2 * kAZ + 2 * kAH + 3 * kAH + 3 * kAI, kAdjT = 2 * kAdjTBuf + 3 * kAI;
constexpr int kAdjVBuf = 4 * kAX + 4 * kAZ + 3 * kAH + 2 * kAH + 2 * kAI, kAdjV = 2 * kAdjVBuf + 2 * kAI;

// f_k (q[-k] - q[1+k]): a transposed half-cell difference (gather form); `at(m)` as in Fd
template <int NN, typename T, typename A>
__device__ __forceinline__ T diff_t(const Geo<T>& g, const A& at) {
  T r = g.f0 * (at(0) - at(1)) + g.f1 * (at(-1) - at(2));
  if (NN == 3) r += g.f2 * (at(-2) - at(3));
  return r;
}

// A thread's vector of the tile and the vector of the tile's halo that it also forms sources for.
template <typename T, int NN>
struct AdjTile {
  static constexpr int W = kVW, NX = kAR * 8 / W, NZ = 2 * NN * kVecX / W;  // halo vectors beside, above and below
  static_assert(NX + NZ <= kAdjThreads<T>, "one halo vector per thread");
  int i0, j0;            // the tile's first cell
  int i, j, px, pz, ph, pi;  // own vector; its place in an x, a z and a history plane and in the tile
  int hi, hj, hp, hph;   // halo vector, its place (x plane if hx, else z plane) and in a history plane
  bool valid, halo, hx;  // on the grid; has a halo vector on the grid or beside it
  __device__ __forceinline__ explicit AdjTile(const Layout& L) {
    const int tiles_x = (L.nxp + kVecX - 1) / kVecX, t = threadIdx.x;
    i0 = ((int)blockIdx.x / tiles_x) * kAR;
    j0 = ((int)blockIdx.x % tiles_x) * kVecX;
    const int r = t / (kVecX / W), c = t % (kVecX / W) * W;
    i = i0 + r;
    j = j0 + c;
    px = r * kAXW + c + 4;
    pz = (r + 3) * kVecX + c;
    ph = (r + 3) * kAXW + c + 4;
    pi = r * kVecX + c;
    valid = i < L.nzp && j < L.nxp;
    hx = t < NX;
    halo = t < NX + NZ;
    if (hx) {
      const int hr = t / (8 / W), k = t % (8 / W) * W;
      hi = i0 + hr;
      hj = j0 + (k < 4 ? k - 4 : kVecX + k - 4);
      hp = hr * kAXW + hj - j0 + 4;
    } else {
      const int u = t - NX, k = u / (kVecX / W);
      const int hr = k < NN ? k - NN : kAR + k - NN;
      hi = i0 + hr;
      hj = j0 + u % (kVecX / W) * W;
      hp = (hr + 3) * kVecX + hj - j0;
    }
    hph = (hi - i0 + 3) * kAXW + hj - j0 + 4;
  }
};

// Copies of N planes (`stride` apart) around the tile into shared memory planes of ROWS rows and COLS
// columns, from row i0 - ZH and column j0 - XH, left in flight. Every copy is 16 bytes on a 16-byte
// boundary (j0 is a multiple of 32, rows start at multiples of 128 bytes, the ghost frame is 4 columns
// wide) and lies in the plane's allocation, which keeps 4 rows and columns before the grid and 20 rows
// and 64 columns after it.
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
template <int N, int ROWS, int COLS, int ZH, int XH, typename T>
__device__ __forceinline__ void stage(const Geo<T>& g, T* dst, const T* src, int64_t stride, int i0, int j0) {
  constexpr int E = 16 / (int)sizeof(T), C = COLS / E;
#pragma unroll
  for (int t0 = 0; t0 < ROWS * C; t0 += kAdjThreads<T>) {
    const int t = t0 + (int)threadIdx.x;
    if (t >= ROWS * C) break;
    const int r = t / C, c = t % C * E;
    const T* from = src + g.L.off(i0 - ZH + r, j0 - XH + c);
#pragma unroll
    for (int k = 0; k < N; ++k) cp_async16(dst + k * (ROWS * COLS) + r * COLS + c, from + k * stride);
  }
}
template <int N, typename T>
__device__ __forceinline__ void stage_full(const Geo<T>& g, T* dst, const T* src, int64_t stride, int i0, int j0) {
  stage<N, kAR + 6, kAXW, 3, 4>(g, dst, src, stride, i0, j0);
}

// The factors of a vector: 1 + dt/2 d inverted times dt/dx (k) and the decay S of a split lambda.
// unit: bit e set where cell e keeps no split fields (only cells of I can); in: cells of I.
template <typename T, bool PML>
struct AdjFactors {
  T kx[kVW], kz[kVW], sx[kVW], sz[kVW];
  unsigned in = 0, unit = 0;
  __device__ __forceinline__ AdjFactors(const Geo<T>& g, const T* cf, int i, int j) {
    Vec<T> bx, bz;
    const bool near = i >= g.ilo && i <= g.ihi && j + kVW > g.jlo && j <= g.jhi;
    if (PML && near) {
      bx = ldv(cf + BCX * g.L.plane + g.L.off(i, j));
      bz = ldv(cf + BCZ * g.L.plane + g.L.off(i, j));
    }
#pragma unroll
    for (int e = 0; e < kVW; ++e) {
      const bool ok = in_I(g, i, j + e);
      kx[e] = ok ? g.dt_dx : T(0);
      kz[e] = ok ? g.dt_dz : T(0);
      sx[e] = sz[e] = T(1);
      if (ok) in |= 1u << e;
      if (PML && ok) {
        const T ix = pml_inv(T(1) + g.hdt * bx.v[e]), iz = pml_inv(T(1) + g.hdt * bz.v[e]);
        kx[e] *= ix;
        kz[e] *= iz;
        sx[e] = (T(1) - g.hdt * bx.v[e]) * ix;
        sz[e] = (T(1) - g.hdt * bz.v[e]) * iz;
        if (!keeps_split(g, i, bx.v[e], bz.v[e])) unit |= 1u << e;
      }
    }
    if (!PML) unit = (1u << kVW) - 1u;
  }
  __device__ __forceinline__ bool split() const { return PML && (in & ~unit) != 0u; }
};

// Lambda of the velocities of the vector at (i, j) (place ph in the staged planes l, j0 the tile's first
// column) with the reverse of the damping (d) and of the free-surface rows, which lie in the first
// row of tiles.
template <typename T, bool PML>
__device__ __forceinline__ void adj_vel_totals(const Geo<T>& g, const T* cf, const T* l, int ph, int j0, const Vec<T>& d,
                                               int i, int j, Vec<T>& ax, Vec<T>& az) {
  ax = ldv(l + VX * kAH + ph);
  az = ldv(l + VZ * kAH + ph);
  if (!PML) {
#pragma unroll
    for (int e = 0; e < kVW; ++e) {
      ax.v[e] *= d.v[e];
      az.v[e] *= d.v[e];
    }
  }
  if (g.fsurf && i >= g.h - 3 && i <= g.h) {
    auto at = [&](int comp, int ii, int jj) {
      const T v = l[comp * kAH + (ii + 3) * kAXW + max(jj - j0 + 4, 0)];
      return PML ? v : cf[DAMP * g.L.plane + g.L.off(ii, jj)] * v;
    };
#pragma unroll
    for (int e = 0; e < kVW; ++e) vfs_adjoint(g, i, j + e, at, ax.v[e], az.v[e]);
  }
}

// dL/d records of one step at the receivers of this block's tile, NC components of them: each thread
// takes a receiver cell (unique cells, so no two threads share one), reads its traces ahead of their
// use and leaves their sum in shared memory planes of the tile's cells, from which the owner of the
// cell adds it to its lambda. Read where they were needed, they were a chain of five dependent loads
// that every shot of a tile with receivers waited for (12 us of a launch of one shot).
template <typename T, int NC>
struct Inject {
  int beg, end, cell = 0, m0 = 0, m1 = 0;
  const T* grec;  // the first component's records of the step, shot 0
  T a[NC] = {};
  __device__ __forceinline__ Inject(const Geo<T>& g, const T* gr, int c0, int it) : beg((int)threadIdx.x), end(0) {
    if (gr == nullptr || it < 0) return;
    grec = gr + ((int64_t)c0 * g.ns * g.nt + it) * g.nr;
    beg = g.tile_beg[blockIdx.x] + (int)threadIdx.x;
    end = g.tile_beg[blockIdx.x + 1];
    if (beg < end) take(g, beg);
  }
  __device__ __forceinline__ void take(const Geo<T>& g, int q) {
    cell = g.ucell_z[q] % kAR * kVecX + g.ucell_x[q] % kVecX;
    m0 = g.ucell_beg[q];
    m1 = g.ucell_beg[q + 1];
  }
  // whether the tile has receivers (uniform over the block)
  __device__ __forceinline__ bool any() const { return end - beg + (int)threadIdx.x > 0; }
  __device__ __forceinline__ void fetch(const Geo<T>& g, int s) {
    if (beg >= end) return;
    const int64_t RS = (int64_t)g.ns * g.nt * g.nr;
    const T* e = grec + (int64_t)s * g.nt * g.nr;
#pragma unroll
    for (int c = 0; c < NC; ++c) a[c] = T(0);
    for (int m = m0; m < m1; ++m) {
      const int r = g.ucell_rcv[m];
#pragma unroll
      for (int c = 0; c < NC; ++c) a[c] += e[c * RS + r];
    }
  }
  // the fetched sums into the planes; a tile with more receiver cells than threads reads the rest here
  __device__ __forceinline__ void put(const Geo<T>& g, int s, T* planes) {
    for (int q = beg; q < end;) {
#pragma unroll
      for (int c = 0; c < NC; ++c) planes[c * kAI + cell] = a[c];
      q += kAdjThreads<T>;
      if (q < end) take(g, q), fetch(g, s);
    }
    if (end - beg > kAdjThreads<T>) take(g, beg);
  }
};

// Reverse of the velocity update: lambda of the (split) velocities after the step (lvs_in -> lvs_out
// with PML; lv -> lv_out with an absorbing layer), lt from the transposes of its stress differences,
// dL/d stress records of step it, and the bx, bz gradients.
template <typename T, int NN, bool PML>
__global__ void __launch_bounds__(kAdjThreads<T>, sizeof(T) == 4 ? (PML ? 3 : 2) : 1)
    adj_t_step(Geo<T> g, int it, const T* __restrict__ cf, const T* __restrict__ lv, T* __restrict__ lv_out,
               const T* __restrict__ lvs_in, T* __restrict__ lvs_out, T* lt, const T* __restrict__ tt_hist,
               const T* __restrict__ grec, T* gpart, int eg) {
  extern __shared__ __align__(16) unsigned char el_smem[];
  constexpr int W = kVW;
  const AdjTile<T, NN> p(g.L);
  const int64_t PL = g.L.plane, NSP = (int64_t)g.ns * PL;
  const int64_t oc = g.L.off(p.i, p.j), oh = g.L.off(p.hi, p.hj);
  EL_SHOT_GROUP
  // coefficients are not written by the launches before
  const AdjFactors<T, PML> f(g, cf, p.i, p.j), fh(g, cf, p.halo ? p.hi : -1, p.hj);
  Vec<T> bx{}, bz{}, hbx{}, hbz{};
  if (f.in) {
    bx = ldv(cf + BX * PL + oc);
    bz = ldv(cf + BZ * PL + oc);
  }
  if (fh.in) {
    hbx = ldv(cf + BX * PL + oh);
    hbz = ldv(cf + BZ * PL + oh);
  }
  Vec<T> gx{}, gz{};
  Vec<T> damp{}, hdamp{};
  if (!PML) {
    if (p.valid) damp = ldv(cf + DAMP * PL + oc);
    if (fh.in) hdamp = ldv(cf + DAMP * PL + oh);
  }
  auto buffer = [&](int s) { return reinterpret_cast<T*>(el_smem) + ((s - s_beg) & 1) * kAdjTBuf; };
  const bool any_split = PML && __syncthreads_or(f.split() || fh.split());
  const bool any_unit = !PML || __syncthreads_or(f.unit);
  auto stage_shot = [&](int s) {
    T* b = buffer(s);
    const int64_t so = (int64_t)s * PL;
    if (any_split) {
      stage<2, kAR, kAXW, 0, 4>(g, b, lvs_in + VX_X * NSP + so, (VZ_X - VX_X) * NSP, p.i0, p.j0);
      stage<2, kAR + 6, kVecX, 3, 0>(g, b + 2 * kAX, lvs_in + VX_Z * NSP + so, (VZ_Z - VX_Z) * NSP, p.i0, p.j0);
    }
    b += 2 * kAX + 2 * kAZ;
    stage_full<2>(g, b, lv + so, NSP, p.i0, p.j0);
    if (any_unit) stage<3, kAR, kVecX, 0, 0>(g, b + 5 * kAH, (const T*)lt + so, NSP, p.i0, p.j0);
  };
  auto stage_history = [&](int s) {
    stage_full<3>(g, buffer(s) + 2 * kAX + 2 * kAZ + 2 * kAH, tt_hist + (int64_t)s * PL, NSP, p.i0, p.j0);
  };
  T* sI = reinterpret_cast<T*>(el_smem) + 2 * kAdjTBuf;
  Inject<T, 3> inj(g, grec, 0, it);
  if (inj.any()) {
    for (int t = threadIdx.x; t < 3 * kAI; t += kAdjThreads<T>) sI[t] = T(0);
    inj.fetch(g, s_beg);
  }
  stage_history(s_beg);  // nor are the histories
  griddep_wait();  // launched with programmatic serialisation
  griddep_launch_dependents();
  stage_shot(s_beg);
  for (int s = s_beg; s < s_end; ++s) {
    T* sX = buffer(s);
    T* sZ = sX + 2 * kAX;
    const T* sV = sZ + 2 * kAZ;
    const T* sH = sV + 2 * kAH + p.ph;
    const T* sO = sV + 5 * kAH + p.pi;
    cp_async_wait_all();
    __syncthreads();  // the copies of all threads; the other buffer's readers
    if (s + 1 < s_end) {
      stage_shot(s + 1);
      stage_history(s + 1);
    }
    const int64_t so = (int64_t)s * PL, o = so + oc;
    Vec<T> vx_x{}, vz_x{}, vx_z{}, vz_z{};  // lambda after the step times k
    if (p.valid) {
      Vec<T> ax, az;
      adj_vel_totals<T, PML>(g, cf, sV, p.ph, p.j0, damp, p.i, p.j, ax, az);
      if (!PML) {
        stv(lv_out + VX * NSP + o, ax);
        stv(lv_out + VZ * NSP + o, az);
      }
      vx_x = vx_z = ax;
      vz_x = vz_z = az;
      if (f.split()) {
        Vec<T> sp[4];
        sp[VX_X] = ldv(sX + p.px);
        sp[VZ_X] = ldv(sX + kAX + p.px);
        sp[VX_Z] = ldv(sZ + p.pz);
        sp[VZ_Z] = ldv(sZ + kAZ + p.pz);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
#pragma unroll
          for (int e = 0; e < W; ++e) {
            const T n = ((k & 1) ? f.sz[e] : f.sx[e]) * sp[k].v[e] + (k < 2 ? ax.v[e] : az.v[e]);
            (k == VX_X ? vx_x : k == VX_Z ? vx_z : k == VZ_X ? vz_x : vz_z).v[e] = n;
            sp[k].v[e] = (f.unit >> e & 1u) ? T(0) : n;
          }
          stv(lvs_out + k * NSP + o, sp[k]);
        }
      }
#pragma unroll
      for (int e = 0; e < W; ++e) {
        vx_x.v[e] = f.in >> e & 1u ? vx_x.v[e] * f.kx[e] : T(0);
        vz_x.v[e] = f.in >> e & 1u ? vz_x.v[e] * f.kx[e] : T(0);
        vx_z.v[e] = f.in >> e & 1u ? vx_z.v[e] * f.kz[e] : T(0);
        vz_z.v[e] = f.in >> e & 1u ? vz_z.v[e] * f.kz[e] : T(0);
      }
    }
    {
      Vec<T> q[4];
#pragma unroll
      for (int e = 0; e < W; ++e) {
        q[0].v[e] = vx_x.v[e] * bx.v[e];
        q[1].v[e] = vz_x.v[e] * bz.v[e];
        q[2].v[e] = vx_z.v[e] * bx.v[e];
        q[3].v[e] = vz_z.v[e] * bz.v[e];
      }
      stv(sX + p.px, q[0]);
      stv(sX + kAX + p.px, q[1]);
      stv(sZ + p.pz, q[2]);
      stv(sZ + kAZ + p.pz, q[3]);
    }
    if (p.halo) {
      Vec<T> q0{}, q1{};
      if (fh.in) {
        Vec<T> ax, az, l0{}, l1{};
        adj_vel_totals<T, PML>(g, cf, sV, p.hph, p.j0, hdamp, p.hi, p.hj, ax, az);
        if (fh.split()) {
          l0 = ldv((p.hx ? sX : sZ) + p.hp);
          l1 = ldv((p.hx ? sX + kAX : sZ + kAZ) + p.hp);
        }
#pragma unroll
        for (int e = 0; e < W; ++e) {
          const T sh = p.hx ? fh.sx[e] : fh.sz[e], k = p.hx ? fh.kx[e] : fh.kz[e];
          q0.v[e] = fh.in >> e & 1u ? (sh * l0.v[e] + ax.v[e]) * k * hbx.v[e] : T(0);
          q1.v[e] = fh.in >> e & 1u ? (sh * l1.v[e] + az.v[e]) * k * hbz.v[e] : T(0);
        }
      }
      stv((p.hx ? sX : sZ) + p.hp, q0);
      stv((p.hx ? sX + kAX : sZ + kAZ) + p.hp, q1);
    }
    if (inj.any()) inj.put(g, s, sI);
    __syncthreads();
    if (s + 1 < s_end) inj.fetch(g, s + 1);
    if (p.valid) {
      Vec<T> n[3];
      {
        const Row<T, NN> qx(sX + p.px), qz(sX + kAX + p.px);
        Vec<T> rx[2 * NN + 1], rz[2 * NN + 1];
#pragma unroll
        for (int k = 0; k <= 2 * NN; ++k) {
          rx[k] = ldv(sZ + p.pz + (k - NN) * kVecX);
          rz[k] = ldv(sZ + kAZ + p.pz + (k - NN) * kVecX);
        }
#pragma unroll
        for (int e = 0; e < W; ++e) {
          n[TXX].v[e] = diff_t<NN>(g, [&](int m) { return qx(e - 1 + m); });
          n[TXZ].v[e] = diff_t<NN>(g, [&](int m) { return rx[NN + m].v[e]; }) +
                        diff_t<NN>(g, [&](int m) { return qz(e + m); });
          n[TZZ].v[e] = diff_t<NN>(g, [&](int m) { return rz[NN + m - 1].v[e]; });
        }
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        if (f.unit) {
          const Vec<T> old = ldv(sO + c * kAI);
#pragma unroll
          for (int e = 0; e < W; ++e)
            if (f.unit >> e & 1u) n[c].v[e] += old.v[e];
        }
        if (inj.any()) {
          const Vec<T> a = ldv(sI + c * kAI + p.pi);
#pragma unroll
          for (int e = 0; e < W; ++e) n[c].v[e] += a.v[e];
        }
        stv(lt + c * NSP + o, n[c]);
      }
      if (f.in) {
        const Row<T, NN> xx(sH + TXX * kAH), xz(sH + TXZ * kAH);
        Vec<T> rxz[2 * NN], rzz[2 * NN];
#pragma unroll
        for (int k = 0; k < 2 * NN; ++k) {
          if (k != NN) rxz[k] = ldv(sH + TXZ * kAH + (k - NN) * kAXW);
          rzz[k] = ldv(sH + TZZ * kAH + (k - NN + 1) * kAXW);
        }
        const Fd<T> fd{g.f0, g.f1, g.f2};
#pragma unroll
        for (int e = 0; e < W; ++e) {
          gx.v[e] += vx_x.v[e] * fd.template diff<NN>([&](int m) { return xx(e + m); }) +
                     vx_z.v[e] * fd.template diff<NN>([&](int m) { return m == 1 ? xz(e) : rxz[NN + m - 1].v[e]; });
          gz.v[e] += vz_x.v[e] * fd.template diff<NN>([&](int m) { return xz(e - 1 + m); }) +
                     vz_z.v[e] * fd.template diff<NN>([&](int m) { return rzz[NN + m - 1].v[e]; });
        }
      }
    }
  }
  if (p.valid && f.in) {
    Vec<T> a = ldv(gbase + 6 * PL + oc), b = ldv(gbase + 7 * PL + oc);
#pragma unroll
    for (int e = 0; e < W; ++e) {
      if (f.in >> e & 1u) a.v[e] += gx.v[e];
      if (f.in >> e & 1u) b.v[e] += gz.v[e];
    }
    stv(gbase + 6 * PL + oc, a);
    stv(gbase + 7 * PL + oc, b);
  }
}

// Reverse of the stress update: lambda of the (split) stresses after the step (lts_in -> lts_out with
// PML), lv from the transposes of its velocity differences, dL/d velocity records of step it - 1, and
// the C gradients.
template <typename T, int NN, bool PML>
__global__ void __launch_bounds__(kAdjThreads<T>, sizeof(T) == 4 ? 2 : 1)
    adj_v_step(Geo<T> g, int it, const T* __restrict__ cf, const T* __restrict__ lt, const T* __restrict__ lts_in,
               T* __restrict__ lts_out, T* lv, const T* __restrict__ v_hist, const T* __restrict__ grec, T* gpart,
               int eg) {
  extern __shared__ __align__(16) unsigned char el_smem[];
  constexpr int W = kVW;
  const AdjTile<T, NN> p(g.L);
  const int64_t PL = g.L.plane, NSP = (int64_t)g.ns * PL;
  const int64_t oc = g.L.off(p.i, p.j), oh = g.L.off(p.hi, p.hj);
  EL_SHOT_GROUP
  const AdjFactors<T, PML> f(g, cf, p.i, p.j), fh(g, cf, p.halo ? p.hi : -1, p.hj);
  Vec<T> c[6] = {}, hc[6] = {};
  if (f.in) {
#pragma unroll
    for (int k = 0; k < 6; ++k) c[k] = ldv(cf + (C11 + k) * PL + oc);
  }
  if (fh.in) {
#pragma unroll
    for (int k = 0; k < 6; ++k) hc[k] = ldv(cf + (C11 + k) * PL + oh);
  }
  constexpr int k11 = 0, k13 = 1, k15 = 2, k33 = 3, k35 = 4, k55 = 5;
  static_assert(C13 == C11 + 1 && C15 == C11 + 2 && C33 == C11 + 3 && C35 == C11 + 4 && C55 == C11 + 5, "order of C");
  Vec<T> gc[6] = {};
  auto buffer = [&](int s) { return reinterpret_cast<T*>(el_smem) + ((s - s_beg) & 1) * kAdjVBuf; };
  const bool any_split = PML && __syncthreads_or(f.split() || fh.split());
  const bool any_unit = !PML || __syncthreads_or(f.unit);
  auto stage_shot = [&](int s) {
    T* b = buffer(s);
    const int64_t so = (int64_t)s * PL;
    if (any_split) {
      stage<3, kAR, kAXW, 0, 4>(g, b, lts_in + so, 2 * NSP, p.i0, p.j0);
      stage<3, kAR + 6, kVecX, 3, 0>(g, b + 4 * kAX, lts_in + NSP + so, 2 * NSP, p.i0, p.j0);
    }
    b += 4 * kAX + 4 * kAZ;
    stage_full<3>(g, b, lt + so, NSP, p.i0, p.j0);
    if (any_unit) stage<2, kAR, kVecX, 0, 0>(g, b + 5 * kAH, (const T*)lv + so, NSP, p.i0, p.j0);
  };
  auto stage_history = [&](int s) {
    stage_full<2>(g, buffer(s) + 4 * kAX + 4 * kAZ + 3 * kAH, v_hist + (int64_t)s * PL, NSP, p.i0, p.j0);
  };
  T* sI = reinterpret_cast<T*>(el_smem) + 2 * kAdjVBuf;
  Inject<T, 2> inj(g, grec, 3, it - 1);
  if (inj.any()) {
    for (int t = threadIdx.x; t < 2 * kAI; t += kAdjThreads<T>) sI[t] = T(0);
    inj.fetch(g, s_beg);
  }
  stage_history(s_beg);
  griddep_wait();  // launched with programmatic serialisation
  griddep_launch_dependents();
  stage_shot(s_beg);
  for (int s = s_beg; s < s_end; ++s) {
    T* sX = buffer(s);
    T* sZ = sX + 4 * kAX;
    const T* sL = sZ + 4 * kAZ;
    const T* sH = sL + 3 * kAH + p.ph;
    const T* sO = sL + 5 * kAH + p.pi;
    cp_async_wait_all();
    __syncthreads();  // the copies of all threads; the other buffer's readers
    if (s + 1 < s_end) {
      stage_shot(s + 1);
      stage_history(s + 1);
    }
    const int64_t so = (int64_t)s * PL, o = so + oc;
    Vec<T> lx[3] = {}, lz[3] = {};  // lambda of txx, tzz, txz after the step times k: x parts, z parts
    if (f.in) {
      Vec<T> l[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) l[k] = ldv(sL + k * kAH + p.ph);
      if (PML && g.fsurf && p.i <= g.h) {
#pragma unroll
        for (int e = 0; e < W; ++e)
          tfs_adjoint(g, sL + TZZ * kAH + p.ph + e, sL + TXZ * kAH + p.ph + e, p.i, kAXW, l[TZZ].v[e], l[TXZ].v[e]);
      }
#pragma unroll
      for (int k = 0; k < 3; ++k) lx[k] = lz[k] = l[k];
      if (f.split()) {
        Vec<T> sp[6];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          sp[2 * k] = ldv(sX + k * kAX + p.px);
          sp[2 * k + 1] = ldv(sZ + k * kAZ + p.pz);
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          Vec<T>&sx = sp[2 * k], &sz = sp[2 * k + 1];
#pragma unroll
          for (int e = 0; e < W; ++e) {
            lx[k].v[e] = f.sx[e] * sx.v[e] + l[k].v[e];
            lz[k].v[e] = f.sz[e] * sz.v[e] + l[k].v[e];
            const bool u = f.unit >> e & 1u;
            sx.v[e] = u ? T(0) : lx[k].v[e];
            sz.v[e] = u ? T(0) : lz[k].v[e];
          }
          stv(lts_out + (2 * k) * NSP + o, sx);
          stv(lts_out + (2 * k + 1) * NSP + o, sz);
        }
      }
#pragma unroll
      for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int e = 0; e < W; ++e) {
          lx[k].v[e] = f.in >> e & 1u ? lx[k].v[e] * f.kx[e] : T(0);
          lz[k].v[e] = f.in >> e & 1u ? lz[k].v[e] * f.kz[e] : T(0);
        }
    }
    // sources of the x differences (of vx backward, forward; of vz backward, forward) and of the z ones
    auto put_x = [&](const Vec<T>* C, const Vec<T>* l, T* at) {
      Vec<T> q[4];
#pragma unroll
      for (int e = 0; e < W; ++e) {
        q[0].v[e] = C[k11].v[e] * l[TXX].v[e] + C[k13].v[e] * l[TZZ].v[e];
        q[1].v[e] = C[k15].v[e] * l[TXZ].v[e];
        q[2].v[e] = C[k15].v[e] * l[TXX].v[e] + C[k35].v[e] * l[TZZ].v[e];
        q[3].v[e] = C[k55].v[e] * l[TXZ].v[e];
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) stv(at + k * kAX, q[k]);
    };
    auto put_z = [&](const Vec<T>* C, const Vec<T>* l, T* at) {
      Vec<T> q[4];
#pragma unroll
      for (int e = 0; e < W; ++e) {
        q[0].v[e] = C[k15].v[e] * l[TXX].v[e] + C[k35].v[e] * l[TZZ].v[e];
        q[1].v[e] = C[k55].v[e] * l[TXZ].v[e];
        q[2].v[e] = C[k13].v[e] * l[TXX].v[e] + C[k33].v[e] * l[TZZ].v[e];
        q[3].v[e] = C[k35].v[e] * l[TXZ].v[e];
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) stv(at + k * kAZ, q[k]);
    };
    put_x(c, lx, sX + p.px);
    put_z(c, lz, sZ + p.pz);
    if (p.halo) {
      Vec<T> l[3] = {};
      if (fh.in) {
#pragma unroll
        for (int k = 0; k < 3; ++k) l[k] = ldv(sL + k * kAH + p.hph);
        if (PML && g.fsurf && p.hi <= g.h) {
#pragma unroll
          for (int e = 0; e < W; ++e)
            tfs_adjoint(g, sL + TZZ * kAH + p.hph + e, sL + TXZ * kAH + p.hph + e, p.hi, kAXW, l[TZZ].v[e], l[TXZ].v[e]);
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          Vec<T> sp{};
          if (fh.split()) sp = ldv((p.hx ? sX + k * kAX : sZ + k * kAZ) + p.hp);
#pragma unroll
          for (int e = 0; e < W; ++e) {
            const T sh = p.hx ? fh.sx[e] : fh.sz[e], kk = p.hx ? fh.kx[e] : fh.kz[e];
            l[k].v[e] = fh.in >> e & 1u ? (sh * sp.v[e] + l[k].v[e]) * kk : T(0);
          }
        }
      }
      if (p.hx)
        put_x(hc, l, sX + p.hp);
      else
        put_z(hc, l, sZ + p.hp);
    }
    if (inj.any()) inj.put(g, s, sI);
    __syncthreads();
    if (s + 1 < s_end) inj.fetch(g, s + 1);
    if (p.valid) {
      Vec<T> n[2];
#pragma unroll
      for (int v = 0; v < 2; ++v) {
        const Row<T, NN> qb(sX + 2 * v * kAX + p.px), qf(sX + (2 * v + 1) * kAX + p.px);
        Vec<T> rb[2 * NN], rf[2 * NN];  // rows i - NN + 1 .. i + NN of the backward, i - NN .. of the forward
#pragma unroll
        for (int k = 0; k < 2 * NN; ++k) {
          rb[k] = ldv(sZ + 2 * v * kAZ + p.pz + (k - NN + 1) * kVecX);
          rf[k] = ldv(sZ + (2 * v + 1) * kAZ + p.pz + (k - NN) * kVecX);
        }
#pragma unroll
        for (int e = 0; e < W; ++e)
          n[v].v[e] = diff_t<NN>(g, [&](int m) { return qb(e + m); }) +
                      diff_t<NN>(g, [&](int m) { return rb[NN + m - 1].v[e]; }) +
                      diff_t<NN>(g, [&](int m) { return qf(e - 1 + m); }) +
                      diff_t<NN>(g, [&](int m) { return rf[NN + m - 1].v[e]; });
        if (f.unit) {
          const Vec<T> old = ldv(sO + v * kAI);
#pragma unroll
          for (int e = 0; e < W; ++e)
            if (f.unit >> e & 1u) n[v].v[e] += old.v[e];
        }
        if (inj.any()) {
          const Vec<T> a = ldv(sI + v * kAI + p.pi);
#pragma unroll
          for (int e = 0; e < W; ++e) n[v].v[e] += a.v[e];
        }
        stv(lv + v * NSP + o, n[v]);
      }
      if (f.in) {
        const Row<T, NN> x(sH + VX * kAH), z(sH + VZ * kAH);
        Vec<T> rx[2 * NN + 1], rz[2 * NN + 1];
#pragma unroll
        for (int k = 0; k <= 2 * NN; ++k)
          if (k != NN) {
            rx[k] = ldv(sH + VX * kAH + (k - NN) * kAXW);
            rz[k] = ldv(sH + VZ * kAH + (k - NN) * kAXW);
          }
        const Fd<T> fd{g.f0, g.f1, g.f2};
#pragma unroll
        for (int e = 0; e < W; ++e) {
          auto zx = [&](int m) { return m == 0 ? x(e) : rx[NN + m].v[e]; };
          auto zz = [&](int m) { return m == 0 ? z(e) : rz[NN + m].v[e]; };
          const T dxb_vx = fd.template diff<NN>([&](int m) { return x(e - 1 + m); });
          const T dxb_vz = fd.template diff<NN>([&](int m) { return z(e - 1 + m); });
          const T dzb_vx = fd.template diff<NN>([&](int m) { return zx(m - 1); });
          const T dzb_vz = fd.template diff<NN>([&](int m) { return zz(m - 1); });
          const T dxf_vx = fd.template diff<NN>([&](int m) { return x(e + m); });
          const T dxf_vz = fd.template diff<NN>([&](int m) { return z(e + m); });
          const T dzf_vx = fd.template diff<NN>(zx);
          const T dzf_vz = fd.template diff<NN>(zz);
          gc[k11].v[e] += lx[TXX].v[e] * dxb_vx;
          gc[k13].v[e] += lz[TXX].v[e] * dzb_vz + lx[TZZ].v[e] * dxb_vx;
          gc[k15].v[e] += lx[TXX].v[e] * dxb_vz + lz[TXX].v[e] * dzb_vx + lx[TXZ].v[e] * dxf_vx;
          gc[k33].v[e] += lz[TZZ].v[e] * dzb_vz;
          gc[k35].v[e] += lx[TZZ].v[e] * dxb_vz + lz[TZZ].v[e] * dzb_vx + lz[TXZ].v[e] * dzf_vz;
          gc[k55].v[e] += lx[TXZ].v[e] * dxf_vz + lz[TXZ].v[e] * dzf_vx;
        }
      }
    }
  }
  if (p.valid && f.in) {
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      Vec<T> a = ldv(gbase + k * PL + oc);
#pragma unroll
      for (int e = 0; e < W; ++e)
        if (f.in >> e & 1u) a.v[e] += gc[k].v[e];
      stv(gbase + k * PL + oc, a);
    }
  }
}

// ABL: stress free-surface adjoint in place, one thread per column.
template <typename T>
__global__ void adj_tfs_abl(Geo<T> g, T* lt) {
  griddep_wait();
  griddep_launch_dependents();
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= g.L.nxp) return;
  const int s = blockIdx.y, h = g.h;
  const int64_t NSP = (int64_t)g.ns * g.L.plane, so = (int64_t)s * g.L.plane;
  T* zz = lt + TZZ * NSP + so;
  T* xz = lt + TXZ * NSP + so;
  const int64_t o3 = g.L.off(h - 3, j), o2 = g.L.off(h - 2, j), o1 = g.L.off(h - 1, j), o0 = g.L.off(h, j);
  xz[o0] -= xz[o3];
  xz[o3] = T(0);
  xz[o1] -= xz[o2];
  xz[o2] = T(0);
  zz[o0] -= zz[o2];
  zz[o2] = T(0);
  zz[o1] = T(0);
}

// Sum the shot groups' gradient partials (8 planes each) into the first group, in group order.
template <typename T>
__global__ void sum_groups(Layout L, int groups, T* part) {
  const int64_t n = (int64_t)L.nzp * L.nxp;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
    const int i = (int)(e / L.nxp), j = (int)(e - (int64_t)i * L.nxp);
    const int64_t o = L.off(i, j);
    for (int q = 0; q < 8; ++q) {
      T acc = part[q * L.plane + o];
      for (int gr = 1; gr < groups; ++gr) acc += part[((int64_t)gr * 8 + q) * L.plane + o];
      part[q * L.plane + o] = acc;
    }
  }
}

template <typename T>
__global__ void pack(Layout L, int h, int w, const T* __restrict__ src, T* __restrict__ dst) {
  int64_t n = (int64_t)h * w;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
    int i = (int)(e / w), j = (int)(e - (int64_t)i * w);
    dst[L.off(i, j)] = src[e];
  }
}

template <typename T>
__global__ void unpack(Layout L, int h, int w, const T* __restrict__ src, T* __restrict__ dst) {
  int64_t n = (int64_t)h * w;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
    int i = (int)(e / w), j = (int)(e - (int64_t)i * w);
    dst[e] = src[L.off(i, j)];
  }
}

}  // namespace el
}  // namespace adfwi

// ----------------------------------------------------------------------------------------
// Plan, workspace and drivers.
// ----------------------------------------------------------------------------------------
using namespace adfwi;

struct adfwi_elastic_plan {
  adfwi_elastic_desc d;
  int nzp, nxp, NN, h, top;
  int nstate;           // state fields per shot: PML 6 split stresses + 4 split velocities + 2 v totals + 3 stress
                        // totals, ABL 3 + 2
  int K, nseg;
  int elem;
  Layout L;
  std::vector<int32_t> tab;
  std::vector<unsigned char> srcm;  // ns x 3 source weights (xx, zz, xz) in the solve's dtype
  PinnedBytes tab_pin, srcm_pin;    // page-locked copies of tab and srcm, the sources of each upload
  int64_t o_srcz, o_srcx, o_rcvz, o_rcvx, o_uz, o_ux, o_ubeg, o_urcv, o_tbeg;
  int ncells;
  std::vector<int> chunk_end;  // last step of each reference checkpoint chunk
};

namespace {

int64_t al256(int64_t x) { return (x + 255) / 256 * 256; }

struct ECarve {
  int64_t coef, st, tt, vtmp, srcm, tab;       // forward
  int64_t snap, snap_scale, hv, ht, lst, lt, lv, lv2, gc;  // gradient
  int64_t total;
};

// Coefficient planes: C11 C13 C15 C33 C35 C55 bx bz + (bcx bcz | damp)
int ncoef(const adfwi_elastic_plan* p) { return p->d.pml ? 10 : 9; }

// Tiles of the reverse kernels (one block each per shot group).
int adj_tiles(const adfwi_elastic_plan* p) {
  return ((p->nzp + el::kAR - 1) / el::kAR) * ((p->nxp + el::kVecX - 1) / el::kVecX);
}
// Shot groups of the reverse kernels: about two waves of two blocks per SM, at most one group per shot.
// More groups split the shots' copies and add gradient planes: 64.4, 65.6 and 71.3 ms for 400 steps of
// 20 shots on a 242 x 480 grid with 600, 900 and 1800 blocks; two and five groups instead of three
// there cost 1 %.
int egroups(const adfwi_elastic_plan* p) {
  const int tiles = adj_tiles(p);
  const int g = std::max(1, std::min(p->d.ns, (600 + tiles - 1) / tiles));
  const int eg = (p->d.ns + g - 1) / g;
  return (p->d.ns + eg - 1) / eg;
}
int eshots_per_group(const adfwi_elastic_plan* p) {
  const int g = egroups(p);
  return (p->d.ns + g - 1) / g;
}

ECarve ecarve(const adfwi_elastic_plan* p, bool grad, int K) {
  ECarve c{};
  const int64_t pl = p->L.plane * p->elem, ns = p->d.ns;
  int64_t o = 0;
  auto take = [&](int64_t b) { int64_t at = o; o += al256(b); return at; };
  c.coef = take(ncoef(p) * pl);
  c.st = take((int64_t)(p->d.pml ? 10 : 0) * ns * pl);  // PML: 6 split stresses + 4 split velocities
  c.tt = take(3 * ns * pl);                               // stress totals
  c.vtmp = take(2 * ns * pl);                             // velocity totals
  c.srcm = take(ns * 3 * p->elem);
  c.tab = take((int64_t)p->tab.size() * 4);
  if (grad) {
    const bool full = K >= p->d.nt;
    const int nseg = (p->d.nt + K - 1) / K;
    const int64_t se = snapshot_value_bytes(p->d.snapshot_precision, p->elem);
    const int64_t nstate = p->nstate;
    c.snap = take(full ? 0 : (int64_t)nseg * nstate * ns * p->L.plane * se);
    c.snap_scale = take(full ? 0 : (int64_t)nseg * nstate * ns * 4);
    c.hv = take((int64_t)K * 2 * ns * pl);  // velocity totals at the start of each step
    c.ht = take((int64_t)K * 3 * ns * pl);  // stress totals after each step's free surface
    // lambda of the split stresses (6) and of the split velocities (4), twice each (a reverse
    // step reads one copy and writes the other)
    c.lst = take((int64_t)(p->d.pml ? 20 : 0) * ns * pl);
    c.lt = take(3 * ns * pl);
    c.lv = take(2 * ns * pl);
    c.lv2 = take((p->d.pml ? 0 : 2) * ns * pl);  // with an absorbing layer lambda of the velocities has two copies
    c.gc = take(8 * pl * egroups(p));
  }
  c.total = o;
  return c;
}

int echoose_K(const adfwi_elastic_plan* p) {
  const int nt = p->d.nt;
  const int64_t budget = p->d.memory_budget;
  if (p->d.snapshot_every > 0) return std::min(p->d.snapshot_every, nt);
  if (budget <= 0) return std::min(nt, std::max(1, (int)std::ceil(std::sqrt(2.4 * nt))));
  if (ecarve(p, true, nt).total <= budget) return nt;
  int kstar = std::min(nt - 1, std::max(1, (int)std::lround(std::sqrt(2.4 * nt))));
  while (kstar > 1 && ecarve(p, true, kstar - 1).total < ecarve(p, true, kstar).total) --kstar;
  while (kstar < nt - 1 && ecarve(p, true, kstar + 1).total < ecarve(p, true, kstar).total) ++kstar;
  if (ecarve(p, true, kstar).total > budget) return kstar;
  int lo = kstar, hi = nt - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) / 2;
    if (ecarve(p, true, mid).total <= budget) lo = mid; else hi = mid - 1;
  }
  return lo;
}

template <typename T>
el::Geo<T> egeo(const adfwi_elastic_plan* p, const unsigned char* ws, const ECarve& c) {
  el::Geo<T> g;
  const adfwi_elastic_desc& d = p->d;
  g.L = p->L;
  g.ns = d.ns;
  g.nt = d.nt;
  g.nr = d.nr;
  g.fsurf = d.free_surface;
  g.h = p->h;
  g.ilo = p->NN;
  g.ihi = p->nzp - p->NN - 1;
  g.jlo = p->NN;
  g.jhi = p->nxp - p->NN - 1;
  g.top = p->top;
  g.nabc = d.nabc;
  g.nz = d.nz;
  g.nx = d.nx;
  g.dt = (T)d.dt;
  g.dx = el::Divisor<T>((T)d.dx);
  g.dz = el::Divisor<T>((T)d.dz);
  g.dt_dx = (T)(d.dt / d.dx);
  g.dt_dz = (T)(d.dt / d.dz);
  g.hdt = (T)(0.5 * d.dt);
  g.f0 = (T)d.fdc[0];
  g.f1 = (T)d.fdc[1];
  g.f2 = (T)(p->NN == 3 ? d.fdc[2] : 0.0);
  const int32_t* tb = reinterpret_cast<const int32_t*>(ws + c.tab);
  g.src_z = tb + p->o_srcz;
  g.src_x = tb + p->o_srcx;
  g.src_m = reinterpret_cast<const T*>(ws + c.srcm);
  g.rcv_z = tb + p->o_rcvz;
  g.rcv_x = tb + p->o_rcvx;
  g.ucell_z = tb + p->o_uz;
  g.ucell_x = tb + p->o_ux;
  g.ucell_beg = tb + p->o_ubeg;
  g.ucell_rcv = tb + p->o_urcv;
  g.tile_beg = tb + p->o_tbeg;
  g.ncells = p->ncells;
  return g;
}

// Blocks of the per-cell kernels (el::kTileThreads threads each): one per 32 x 8 tile.
inline dim3 cells_grid(const adfwi_elastic_plan* p, int ns) {
  const int64_t tiles = (int64_t)((p->nzp + el::kTileZ - 1) / el::kTileZ) * ((p->nxp + el::kTileX - 1) / el::kTileX);
  return dim3((unsigned)tiles, ns);
}

template <typename T>
int esetup(const adfwi_elastic_plan* p, unsigned char* ws, const ECarve& c, const void* const* coef,
           const int32_t* shapes, cudaStream_t st) {
  const int64_t pl = p->L.plane * p->elem;
  ADFWI_CUDA_TRY(cudaMemsetAsync(ws, 0, c.srcm, st));  // coefficient ghosts, state, totals
  ADFWI_CUDA_TRY(cudaMemcpyAsync(ws + c.tab, p->tab_pin.ptr, p->tab.size() * 4, cudaMemcpyHostToDevice, st));
  ADFWI_CUDA_TRY(cudaMemcpyAsync(ws + c.srcm, p->srcm_pin.ptr, p->srcm.size(), cudaMemcpyHostToDevice, st));
  for (int q = 0; q < ncoef(p); ++q) {
    const int h = shapes[2 * q], w = shapes[2 * q + 1];
    if (h < 1 || w < 1 || h > p->nzp || w > p->nxp) {
      set_error("coefficient %d has shape %dx%d, outside the %dx%d grid", q, h, w, p->nzp, p->nxp);
      return kBadArgument;
    }
    const int64_t n = (int64_t)h * w;
    ADFWI_LAUNCH(kAux, st, (el::pack<T><<<(unsigned)std::min<int64_t>((n + 255) / 256, 4096), 256, 0, st>>>(
                               p->L, h, w, static_cast<const T*>(coef[q]),
                               reinterpret_cast<T*>(ws + c.coef + q * pl))));
  }
  ADFWI_CUDA_TRY(cudaGetLastError());
  return kOk;
}

// One forward step. vin, tprev: velocity and stress totals at the start of the step; vout, tt:
// where the new totals go (the same memory when they advance in place). rec: records, or null: the
// velocity records of the step before and the stress records of this one are taken.
// Programmatically serialised launches: each kernel waits for the previous one's data. The stress update
// reads coefficients and previous totals ahead of its wait: `first`, the first step of a loop, follows the
// launches that write those (packing, a snapshot's restoring) and is ordered by the stream.
template <typename T, int NN>
void estep(const adfwi_elastic_plan* p, const el::Geo<T>& g, int it, bool first, const T* cf, const T* wav, T* st, T* tt,
           const T* tprev, T* vin, T* vout, T* rec, cudaStream_t s) {
  const dim3 b(el::kVecThreads);
  const int64_t NSP = (int64_t)p->d.ns * p->L.plane;
  const unsigned tiles = el::vec_tiles<T>(p->L), gy = p->d.ns;
  const unsigned rb = rec != nullptr && p->d.nr > 0 ? (p->d.nr + el::kVecThreads - 1) / el::kVecThreads : 0;
  const dim3 gs(tiles + (it > 0 ? rb : 0), gy), gv(tiles + rb, gy);
  auto stress = p->d.pml ? el::stress_step<T, NN, true> : el::stress_step<T, NN, false>;
  auto vel = p->d.pml ? el::vel_step<T, NN, true> : el::vel_step<T, NN, false>;
  ADFWI_LAUNCH(kElFwdStep, s, (void)launch_kernel(!first, stress, gs, b, 0, s, g, it, cf, vin, st, tt, tprev, wav, rec));
  ADFWI_LAUNCH(kElFwdStep, s, (void)launch_pdl_kernel(vel, gv, b, 0, s, g, it, cf, (const T*)tt,
                                                      p->d.pml ? st + 6 * NSP : nullptr, vout, (const T*)vin, rec));
  if (!p->d.pml && p->d.free_surface) {
    const dim3 gcol((unsigned)((p->nxp + 127) / 128), p->d.ns);
    ADFWI_LAUNCH(kElFwdStep, s, (void)launch_pdl_kernel(el::vel_fs_abl<T>, gcol, dim3(128), 0, s, g, vout));
    ADFWI_LAUNCH(kElFwdStep, s, (void)launch_pdl_kernel(el::damp_v<T>, cells_grid(p, p->d.ns), dim3(el::kTileThreads), 0,
                                                        s, g, cf, vout));
  }
}

// Snapshot helpers: the state of a step start is (PML) 10 split fields in st + 2 velocity
// totals + 3 stress totals (the cells without split fields keep their state in the totals), or
// (ABL) 3 stresses in tt + 2 velocities (nc = 0).
template <typename T>
int esnap(const adfwi_elastic_plan* p, bool store, unsigned char* ws, const ECarve& c, T* a, int64_t na, T* b,
          int64_t nb, T* cc, int64_t nc, int seg, cudaStream_t s) {
  const int64_t pl = p->L.plane;
  const int64_t first = (int64_t)seg * (na + nb + nc);
  T* parts[3] = {a, b, cc};
  const int64_t n[3] = {na, nb, nc};
  int64_t at = first;
  for (int q = 0; q < 3; ++q) {
    if (n[q] == 0) continue;
    const int rc =
        store ? snapshot_store<T>(p->d.snapshot_precision, parts[q], n[q], pl, ws + c.snap, ws + c.snap_scale, at, s)
              : snapshot_load<T>(p->d.snapshot_precision, parts[q], n[q], pl, ws + c.snap, ws + c.snap_scale, at, s);
    if (rc) return rc;
    at += n[q];
  }
  return kOk;
}

template <typename T, int NN>
int eforward(const adfwi_elastic_plan* p, const void* const* coef, const int32_t* shapes, const void* wavelet,
             void* rec, void* fw, bool grad, unsigned char* ws, int64_t ws_bytes, cudaStream_t s) {
  const int K = grad ? p->K : 1;
  ECarve c = ecarve(p, grad, K);
  if (ws_bytes < c.total) {
    set_error("workspace too small: %lld bytes given, %lld needed", (long long)ws_bytes, (long long)c.total);
    return kWorkspaceTooSmall;
  }
  int rc = esetup<T>(p, ws, c, coef, shapes, s);
  if (rc) return rc;
  el::Geo<T> g = egeo<T>(p, ws, c);
  const int64_t NSP = (int64_t)p->d.ns * p->L.plane;
  const T* cf = reinterpret_cast<const T*>(ws + c.coef);
  const T* wav = static_cast<const T*>(wavelet);
  T* stt = reinterpret_cast<T*>(ws + c.st);
  T* tt0 = reinterpret_cast<T*>(ws + c.tt);
  T* v0 = reinterpret_cast<T*>(ws + c.vtmp);
  const bool full = grad && K >= p->d.nt;
  T* hv = grad ? reinterpret_cast<T*>(ws + c.hv) : nullptr;
  T* ht = grad ? reinterpret_cast<T*>(ws + c.ht) : nullptr;
  const int nt = p->d.nt;
  if (fw) ADFWI_CUDA_TRY(cudaMemsetAsync(fw, 0, 5 * (int64_t)p->d.nz * p->d.nx * sizeof(T), s));
  size_t chunk = 0;
  for (int it = 0; it < nt; ++it) {
    if (grad && !full && it % K == 0) {
      if (p->d.pml)
        rc = esnap<T>(p, true, ws, c, stt, 10 * p->d.ns, v0, 2 * p->d.ns, tt0, 3 * p->d.ns, it / K, s);
      else
        rc = esnap<T>(p, true, ws, c, tt0, 3 * p->d.ns, v0, 2 * p->d.ns, nullptr, 0, it / K, s);
      if (rc) return rc;
    }
    T* vin = v0;
    T* vout = v0;
    T* tt = tt0;
    const T* tprev = tt0;  // stress totals at the start of the step
    if (full) {
      // the histories double as the state: Hv[it] = v at the start of step it, Ht[it] = T after it
      vin = it == 0 ? v0 : hv + (int64_t)it * 2 * NSP;
      vout = it + 1 < nt ? hv + (int64_t)(it + 1) * 2 * NSP : v0;
      if (it == 0) ADFWI_CUDA_TRY(cudaMemsetAsync(hv, 0, 2 * NSP * sizeof(T), s));
      if (it == 0) vin = hv;
      tt = ht + (int64_t)it * 3 * NSP;
      if (it > 0) tprev = ht + (int64_t)(it - 1) * 3 * NSP;
    }
    estep<T, NN>(p, g, it, it == 0, cf, wav, stt, tt, tprev, vin, vout, static_cast<T*>(rec), s);
    if (rec && p->d.nr > 0 && it + 1 == nt) {
      dim3 gr((unsigned)((p->d.nr + 127) / 128), p->d.ns);
      ADFWI_LAUNCH(kAux, s, (void)launch_pdl_kernel(el::record_v<T>, gr, dim3(128), 0, s, g, it, (const T*)vout,
                                                    static_cast<T*>(rec), p->d.pml != 0));
    }
    if (fw && chunk < p->chunk_end.size() && it == p->chunk_end[chunk]) {
      const int64_t n = (int64_t)p->d.nz * p->d.nx;
      ADFWI_LAUNCH(kAux, s, (el::energy<T><<<(unsigned)((n + 255) / 256), 256, 0, s>>>(g, tt, vout, static_cast<T*>(fw))));
      ++chunk;
    }
  }
  ADFWI_CUDA_TRY(cudaGetLastError());
  return kOk;
}

template <typename T, int NN>
int ebackward(const adfwi_elastic_plan* p, const void* wavelet, const void* grec, void* const* gcoef,
              const int32_t* shapes, unsigned char* ws, int64_t ws_bytes, cudaStream_t s) {
  const int K = p->K;
  ECarve c = ecarve(p, true, K);
  if (ws_bytes < c.total) {
    set_error("workspace too small: %lld bytes given, %lld needed", (long long)ws_bytes, (long long)c.total);
    return kWorkspaceTooSmall;
  }
  el::Geo<T> g = egeo<T>(p, ws, c);
  const int ns = p->d.ns, nt = p->d.nt;
  const int64_t PL = p->L.plane, NSP = (int64_t)ns * PL;
  const bool full = K >= nt;
  const T* cf = reinterpret_cast<const T*>(ws + c.coef);
  const T* wav = static_cast<const T*>(wavelet);
  T* stt = reinterpret_cast<T*>(ws + c.st);
  T* tt0 = reinterpret_cast<T*>(ws + c.tt);
  T* v0 = reinterpret_cast<T*>(ws + c.vtmp);
  T* hv = reinterpret_cast<T*>(ws + c.hv);
  T* ht = reinterpret_cast<T*>(ws + c.ht);
  T* lst = reinterpret_cast<T*>(ws + c.lst);
  T* lt = reinterpret_cast<T*>(ws + c.lt);
  T* lv = reinterpret_cast<T*>(ws + c.lv);
  T* lv2 = reinterpret_cast<T*>(ws + c.lv2);
  T* gcp = reinterpret_cast<T*>(ws + c.gc);
  const T* gr = static_cast<const T*>(grec);
  if (p->d.pml) ADFWI_CUDA_TRY(cudaMemsetAsync(lst, 0, 20 * NSP * sizeof(T), s));
  ADFWI_CUDA_TRY(cudaMemsetAsync(lt, 0, 3 * NSP * sizeof(T), s));
  ADFWI_CUDA_TRY(cudaMemsetAsync(lv, 0, 2 * NSP * sizeof(T), s));
  const int egr = egroups(p), eg = eshots_per_group(p);
  ADFWI_CUDA_TRY(cudaMemsetAsync(gcp, 0, (int64_t)egr * 8 * PL * sizeof(T), s));
  if (!p->d.pml) ADFWI_CUDA_TRY(cudaMemsetAsync(lv2, 0, 2 * NSP * sizeof(T), s));
  const dim3 ga(adj_tiles(p), egr), ba(el::kAdjThreads<T>);
  auto adj_t = p->d.pml ? el::adj_t_step<T, NN, true> : el::adj_t_step<T, NN, false>;
  auto adj_v = p->d.pml ? el::adj_v_step<T, NN, true> : el::adj_v_step<T, NN, false>;
  // shared memory of the reverse kernels (75 and 91 KB, twice that in double precision: above the 48 KB default)
  const int smem_t = el::kAdjT * (int)sizeof(T), smem_v = el::kAdjV * (int)sizeof(T);
  ADFWI_CUDA_TRY(cudaFuncSetAttribute(adj_t, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_t));
  ADFWI_CUDA_TRY(cudaFuncSetAttribute(adj_v, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_v));
  const dim3 gcol((unsigned)((p->nxp + 127) / 128), ns);
  if (gr && p->ncells > 0)
    ADFWI_LAUNCH(kAux, s, (el::adj_inject<T><<<dim3((unsigned)((p->ncells + 127) / 128), ns), 128, 0, s>>>(g, nt - 1, gr, lv)));
  const int nseg = full ? 1 : (nt + K - 1) / K;
  int flip = 0;  // which copy of the split velocities' lambda the next reverse step reads
  for (int seg = nseg - 1; seg >= 0; --seg) {
    const int t0 = full ? 0 : seg * K;
    const int t1 = full ? nt : std::min(nt, t0 + K);
    if (!full) {
      // restore the state at t0 (v totals straight into Hv[0]) and recompute the segment
      int rc = p->d.pml ? esnap<T>(p, false, ws, c, stt, 10 * ns, hv, 2 * ns, tt0, 3 * ns, seg, s)
                        : esnap<T>(p, false, ws, c, tt0, 3 * ns, hv, 2 * ns, nullptr, 0, seg, s);
      if (rc) return rc;
      for (int it = t0; it < t1; ++it) {
        const int k = it - t0;
        T* vin = hv + (int64_t)k * 2 * NSP;
        T* vout = k + 1 < K && it + 1 < t1 ? hv + (int64_t)(k + 1) * 2 * NSP : v0;
        T* tt = ht + (int64_t)k * 3 * NSP;
        const T* tprev = k > 0 ? ht + (int64_t)(k - 1) * 3 * NSP : tt0;
        estep<T, NN>(p, g, it, k == 0, cf, wav, stt, tt, tprev, vin, vout, (T*)nullptr, s);
      }
    }
    for (int it = t1 - 1; it >= t0; --it) {
      const int k = it - t0;
      const T* vh = hv + (int64_t)k * 2 * NSP;  // velocity totals at the start of step it
      const T* th = ht + (int64_t)k * 3 * NSP;  // stress totals of step it
      // lambda of the split stresses: planes 0-5 / 6-11 of lst, of the split velocities 12-15 /
      // 16-19; each reverse step reads one copy and writes the other
      const int f = flip;
      flip ^= 1;
      const T* lvs_in = lst + (12 + 4 * f) * NSP;
      T* lvs_out = lst + (16 - 4 * f) * NSP;
      const T* lts_in = lst + (6 * f) * NSP;
      T* lts_out = lst + (6 - 6 * f) * NSP;
      // programmatically serialised launches
      ADFWI_LAUNCH(kElAdjStep, s, (void)launch_pdl_kernel(adj_t, ga, ba, (size_t)smem_t, s, g, it, cf, (const T*)lv, lv2,
                                                          lvs_in, lvs_out, lt, th, gr, gcp, eg));
      if (!p->d.pml) {
        std::swap(lv, lv2);
        if (p->d.free_surface)
          ADFWI_LAUNCH(kElAdjStep, s, (void)launch_pdl_kernel(el::adj_tfs_abl<T>, gcol, dim3(128), 0, s, g, lt));
      }
      ADFWI_LAUNCH(kElAdjStep, s, (void)launch_pdl_kernel(adj_v, ga, ba, (size_t)smem_v, s, g, it, cf, (const T*)lt,
                                                          lts_in, lts_out, lv, vh, gr, gcp, eg));
    }
    ADFWI_CUDA_TRY(cudaGetLastError());
  }
  if (egr > 1) {
    const int64_t n = (int64_t)p->nzp * p->nxp;
    ADFWI_LAUNCH(kAux, s, (el::sum_groups<T><<<(unsigned)std::min<int64_t>((n + 255) / 256, 4096), 256, 0, s>>>(
                              p->L, egr, gcp)));
  }
  // gradients out: C11 C13 C15 C33 C35 C55 bx bz, each cropped to its input shape
  for (int q = 0; q < 8; ++q) {
    if (gcoef[q] == nullptr) continue;
    const int h = shapes[2 * q], w = shapes[2 * q + 1];
    const int64_t n = (int64_t)h * w;
    ADFWI_LAUNCH(kAux, s, (el::unpack<T><<<(unsigned)std::min<int64_t>((n + 255) / 256, 4096), 256, 0, s>>>(
                              p->L, h, w, gcp + q * PL, static_cast<T*>(gcoef[q]))));
  }
  ADFWI_CUDA_TRY(cudaGetLastError());
  return kOk;
}

}  // namespace

extern "C" {

int adfwi_elastic_plan_create(const adfwi_elastic_desc* desc, const int32_t* src_z, const int32_t* src_x,
                              const int32_t* rcv_z, const int32_t* rcv_x, const double* moment_tensor,
                              adfwi_elastic_plan** out) {
  ADFWI_CHECK_ARG(desc && out, "null descriptor or output pointer");
  *out = nullptr;
  const adfwi_elastic_desc& d = *desc;
  ADFWI_CHECK_ARG(d.fd_order == 4 || d.fd_order == 6, "fd_order must be 4 or 6");
  ADFWI_CHECK_ARG(d.nz >= 3 && d.nx >= 3 && d.nabc >= 1, "need nz, nx >= 3 and nabc >= 1");
  ADFWI_CHECK_ARG(d.ns >= 1 && d.nt >= 1 && d.nr >= 0, "need ns >= 1, nt >= 1, nr >= 0");
  ADFWI_CHECK_ARG(d.dtype == ADFWI_F32 || d.dtype == ADFWI_F64, "dtype must be ADFWI_F32 or ADFWI_F64");
  ADFWI_CHECK_ARG(d.checkpoint_segments >= 1, "checkpoint_segments must be >= 1");
  ADFWI_CHECK_ARG(d.snapshot_precision >= 0 && d.snapshot_precision <= 3, "bad snapshot_precision");
  ADFWI_CHECK_ARG(src_z && src_x && moment_tensor && (d.nr == 0 || (rcv_z && rcv_x)), "null geometry array");
  adfwi_elastic_plan* p = new (std::nothrow) adfwi_elastic_plan();
  if (!p) {
    set_error("host allocation failed");
    return kBadArgument;
  }
  p->d = d;
  p->NN = d.fd_order / 2;
  p->h = p->NN + 1;
  const int fs_off = d.fd_order / 2;
  p->nxp = d.nx + 2 * d.nabc;
  p->nzp = d.nz + (d.free_surface ? d.nabc + fs_off : 2 * d.nabc + fs_off);
  p->top = d.free_surface ? fs_off : fs_off + d.nabc;
  p->elem = d.dtype == ADFWI_F64 ? 8 : 4;
  p->nstate = d.pml ? 15 : 5;
  p->L = make_layout(p->nzp, p->nxp, 16, 64, p->elem);
  std::vector<int32_t>& t = p->tab;
  p->o_srcz = t.size();
  for (int s = 0; s < d.ns; ++s) {
    const int z = src_z[s] + p->top, x = src_x[s] + d.nabc;
    if (z < 0 || z >= p->nzp || x < 0 || x >= p->nxp) {
      set_error("source %d at (z=%d, x=%d) lies outside the model", s, src_z[s], src_x[s]);
      delete p;
      return kBadGeometry;
    }
    t.push_back(z);
  }
  p->o_srcx = t.size();
  for (int s = 0; s < d.ns; ++s) t.push_back(src_x[s] + d.nabc);
  // source weights: PML adds -MT/2 * w to both split parts, ABL adds -1/3 * MT * w
  p->srcm.resize((size_t)3 * d.ns * p->elem);
  for (int s = 0; s < d.ns; ++s) {
    const double* m = moment_tensor + 9 * s;
    const int idx[3] = {0, 8, 2};  // MT[0,0], MT[2,2], MT[0,2]
    for (int k = 0; k < 3; ++k) {
      unsigned char* dst = p->srcm.data() + (size_t)(3 * s + k) * p->elem;
      if (d.dtype == ADFWI_F32) {
        const float mv = (float)m[idx[k]];
        const float w = d.pml ? -(mv / 2.0f) : (float)(-1.0 / 3.0) * mv;
        memcpy(dst, &w, sizeof(w));
      } else {
        const double w = d.pml ? -(m[idx[k]] / 2.0) : (-1.0 / 3.0) * m[idx[k]];
        memcpy(dst, &w, sizeof(w));
      }
    }
  }
  p->o_rcvz = t.size();
  for (int r = 0; r < d.nr; ++r) {
    const int z = rcv_z[r] + p->top, x = rcv_x[r] + d.nabc;
    if (z < 0 || z >= p->nzp || x < 0 || x >= p->nxp) {
      set_error("receiver %d at (z=%d, x=%d) lies outside the model", r, rcv_z[r], rcv_x[r]);
      delete p;
      return kBadGeometry;
    }
    t.push_back(z);
  }
  p->o_rcvx = t.size();
  for (int r = 0; r < d.nr; ++r) t.push_back(rcv_x[r] + d.nabc);
  // unique receiver cells
  // in the order of the reverse kernels' tiles
  struct Cell {
    int tile, z, x, r;
    bool same(const Cell& o) const { return z == o.z && x == o.x; }
    bool operator<(const Cell& o) const { return tile != o.tile ? tile < o.tile : z != o.z ? z < o.z : x < o.x; }
  };
  const int tiles_x = (p->nxp + el::kVecX - 1) / el::kVecX, tiles = adj_tiles(p);
  std::vector<Cell> cells(d.nr);
  for (int r = 0; r < d.nr; ++r) {
    const int z = rcv_z[r] + p->top, x = rcv_x[r] + d.nabc;
    cells[r] = {z / el::kAR * tiles_x + x / el::kVecX, z, x, r};
  }
  std::stable_sort(cells.begin(), cells.end());
  std::vector<int32_t> uz, ux, ubeg, urcv, tbeg(tiles + 1, 0);
  for (int q = 0; q < d.nr; ++q) {
    if (q == 0 || !cells[q].same(cells[q - 1])) {
      uz.push_back(cells[q].z);
      ux.push_back(cells[q].x);
      ubeg.push_back((int32_t)urcv.size());
      ++tbeg[cells[q].tile + 1];
    }
    urcv.push_back(cells[q].r);
  }
  for (int t = 0; t < tiles; ++t) tbeg[t + 1] += tbeg[t];
  ubeg.push_back((int32_t)urcv.size());
  p->ncells = (int)uz.size();
  p->o_uz = t.size();
  t.insert(t.end(), uz.begin(), uz.end());
  p->o_ux = t.size();
  t.insert(t.end(), ux.begin(), ux.end());
  p->o_ubeg = t.size();
  t.insert(t.end(), ubeg.begin(), ubeg.end());
  p->o_urcv = t.size();
  t.insert(t.end(), urcv.begin(), urcv.end());
  p->o_tbeg = t.size();
  t.insert(t.end(), tbeg.begin(), tbeg.end());
  if (t.empty()) t.push_back(0);
  // torch.chunk(wavelet, checkpoint_segments): the energy maps keep the last step of each chunk
  const int chunk = (d.nt + d.checkpoint_segments - 1) / d.checkpoint_segments;
  for (int e = chunk - 1; e < d.nt; e += chunk) p->chunk_end.push_back(e);
  if (p->chunk_end.empty() || p->chunk_end.back() != d.nt - 1) p->chunk_end.push_back(d.nt - 1);
  if (!p->tab_pin.assign(p->tab.data(), p->tab.size() * 4) || !p->srcm_pin.assign(p->srcm.data(), p->srcm.size())) {
    delete p;
    return kCudaError;
  }
  p->K = echoose_K(p);
  p->nseg = (d.nt + p->K - 1) / p->K;
  *out = p;
  return kOk;
}

void adfwi_elastic_plan_destroy(adfwi_elastic_plan* p) { delete p; }

int adfwi_elastic_workspace_bytes(const adfwi_elastic_plan* p, int32_t with_gradient, int64_t* bytes) {
  ADFWI_CHECK_ARG(p && bytes, "null plan or output pointer");
  *bytes = ecarve(p, with_gradient != 0, with_gradient ? p->K : 1).total;
  return kOk;
}

int adfwi_elastic_snapshot_every(const adfwi_elastic_plan* p, int32_t* steps) {
  ADFWI_CHECK_ARG(p && steps, "null plan or output pointer");
  *steps = p->K;
  return kOk;
}

int adfwi_elastic_forward(const adfwi_elastic_plan* p, const void* const* coef, const int32_t* shapes,
                          const void* wavelet, void* rec, void* fw, int32_t with_gradient, void* workspace,
                          int64_t workspace_bytes, void* stream) {
  ADFWI_CHECK_ARG(p && coef && shapes && wavelet && workspace, "null argument");
  for (int q = 0; q < ncoef(p); ++q) ADFWI_CHECK_ARG(coef[q] != nullptr, "coefficient %d is null", q);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  unsigned char* ws = static_cast<unsigned char*>(workspace);
  const bool g = with_gradient != 0;
  if (p->d.dtype == ADFWI_F64)
    return p->NN == 2 ? eforward<double, 2>(p, coef, shapes, wavelet, rec, fw, g, ws, workspace_bytes, s)
                      : eforward<double, 3>(p, coef, shapes, wavelet, rec, fw, g, ws, workspace_bytes, s);
  return p->NN == 2 ? eforward<float, 2>(p, coef, shapes, wavelet, rec, fw, g, ws, workspace_bytes, s)
                    : eforward<float, 3>(p, coef, shapes, wavelet, rec, fw, g, ws, workspace_bytes, s);
}

int adfwi_elastic_backward(const adfwi_elastic_plan* p, const void* wavelet, const void* grad_rec,
                           void* const* grad_coef, const int32_t* shapes, void* workspace, int64_t workspace_bytes,
                           void* stream) {
  ADFWI_CHECK_ARG(p && wavelet && grad_coef && shapes && workspace, "null argument");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  unsigned char* ws = static_cast<unsigned char*>(workspace);
  if (p->d.dtype == ADFWI_F64)
    return p->NN == 2 ? ebackward<double, 2>(p, wavelet, grad_rec, grad_coef, shapes, ws, workspace_bytes, s)
                      : ebackward<double, 3>(p, wavelet, grad_rec, grad_coef, shapes, ws, workspace_bytes, s);
  return p->NN == 2 ? ebackward<float, 2>(p, wavelet, grad_rec, grad_coef, shapes, ws, workspace_bytes, s)
                    : ebackward<float, 3>(p, wavelet, grad_rec, grad_coef, shapes, ws, workspace_bytes, s);
}

}  // extern "C"
