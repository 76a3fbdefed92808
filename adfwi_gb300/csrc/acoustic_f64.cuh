// Acoustic time step and its reverse in double precision, one launch each (acoustic_kernels.py:115-169
// and its transposes): p on the tile and the halo that u and w read, through shared memory; lambda_p
// likewise.
//
// What bounds them is double-precision arithmetic, two lanes per clock and SM: 28 operations a cell
// forward and 37 in reverse (35 and 46 with the halo), and the launch boundary. So the work is cut
// finely: a block of 128 threads takes 8 rows of 32 columns of one shot group, two columns per
// thread, 570 blocks for five shots of 121 x 193 cells, where tiles of 16 x 64 cells with two shots each
// kept 96 of the 152 SMs busy. 300 forward and reverse steps of those shots: 29.0 -> 10.8 ms (14.8 with
// p and u, w in two launches, which forms nothing twice but waits for its loads twice).
//
// Launches are programmatically serialised, but for the first step of a solve, which follows the kernel that
// writes the coefficients: a kernel reads coefficients and dL/d records ahead of the end of the launch
// before it. The records of a step are taken by extra blocks of the
// next, which reads them.
#pragma once
#include "acoustic_geo.cuh"
#include "common.cuh"

namespace adfwi {
namespace ac3 {

using ac::radd;
using ac::rmul;
using ac::rsub;

constexpr int kX = 32, kThreads = 128, kLanes = kX / 2, kZ = kThreads / kLanes;

// Padded rows and columns of the receivers and of the unique receiver cells (in the order of
// Geo's tcell_rbeg); the unique cells' indices in the order of this file's tiles.
struct Cells {
  const int *rcv_z, *rcv_x;
  const int *cell_z, *cell_x;
  const int* tile_beg;
  const int* tile_cell;
  int ncells;
};

inline int tiles(const Layout& L, int zbeg) { return ((L.nxp + kX - 1) / kX) * ((L.nzp - zbeg + kZ - 1) / kZ); }

struct Pos {
  int i0, j0, i, j;  // the block's tile, this thread's first cell
  bool ok;
  __device__ __forceinline__ explicit Pos(const ac::Geo<double>& g) {
    const int tx = (g.L.nxp + kX - 1) / kX, ti = (int)blockIdx.x / tx;
    i0 = g.zbeg + ti * kZ;
    j0 = ((int)blockIdx.x - ti * tx) * kX;
    i = i0 + (int)threadIdx.x / kLanes;
    j = j0 + (int)threadIdx.x % kLanes * 2;
    ok = i < g.L.nzp && j < g.L.nxp;
  }
};
__device__ __forceinline__ double2 ld(const double* p) { return *reinterpret_cast<const double2*>(p); }
__device__ __forceinline__ void st(double* p, double x, double y) { *reinterpret_cast<double2*>(p) = make_double2(x, y); }
// columns j-2 .. j+3 of a row, j at p
__device__ __forceinline__ void ld6(const double* p, double (&r)[6]) {
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const double2 v = ld(p - 2 + 2 * k);
    r[2 * k] = v.x;
    r[2 * k + 1] = v.y;
  }
}
__device__ __forceinline__ void ld2(const double* p, double (&r)[2]) {
  const double2 v = ld(p);
  r[0] = v.x;
  r[1] = v.y;
}

// Records of step `it` at the receivers from the fields after it, by blocks from `first` on.
__device__ __forceinline__ void record(const ac::Geo<double>& g, const Cells& c, int first, int it, const double* p,
                                       const double* u, const double* w, double* rp, double* ru, double* rw) {
  const int r = ((int)blockIdx.x - first) * kThreads + (int)threadIdx.x;
  if (r >= g.nr) return;
  const int64_t oc = g.L.off(c.rcv_z[r], c.rcv_x[r]);
  for (int s = g.grp_beg[blockIdx.y]; s < g.grp_beg[blockIdx.y + 1]; ++s) {
    const int64_t o = (int64_t)s * g.L.plane + oc, e = ((int64_t)s * g.nt + it) * g.nr + r;
    rp[e] = p[o];
    ru[e] = u[o];
    rw[e] = w[o];
  }
}
// The records of the last step (the next step would have taken them).
__global__ void record_last(ac::Geo<double> g, Cells cells, int it, const double* p, const double* u, const double* w,
                            double* rp, double* ru, double* rw) {
  griddep_wait();
  griddep_launch_dependents();
  record(g, cells, 0, it, p, u, w, rp, ru, rw);
}

// The tile with its halo in shared memory: rows i0 - 1 .. i0 + kZ + 1, columns j0 - 2 .. j0 + kX + 1, in
// tasks of two columns, at most two per thread.
constexpr int kHX = kX + 4, kHZ = kZ + 3, kHV = kHX / 2, kTasks = kHV * kHZ;
static_assert(kTasks <= 2 * kThreads, "two halo tasks per thread");
struct Task {
  int i, j, at;       // first cell and its place in the halo plane (at < 0: no task)
  bool inside, tile;  // on the tiled rows of the grid; in the tile
  __device__ __forceinline__ Task(const ac::Geo<double>& g, int i0, int j0, int t) {
    const int r = t / kHV, c = t % kHV * 2;
    at = t < kTasks ? r * kHX + c : -1;
    i = i0 - 1 + r;
    j = j0 - 2 + c;
    inside = at >= 0 && i >= g.zbeg && i < g.L.nzp && j + 1 >= 0 && j < g.L.nxp;
    tile = inside && r >= 1 && r <= kZ && c >= 2 && c < kX + 2;
  }
};

// One step: p (d1: with its divergence, if kept), u and w from p0, u0, w0; illumination sums acc0 of p and
// acc1 of u (null: none); extra blocks: the records of step it - 1.
__global__ void __launch_bounds__(kThreads)
    fwd_step(ac::Geo<double> g, Cells cells, int ntiles, int it, const double* __restrict__ cf0, int64_t cfs,
             const double* __restrict__ p0, const double* __restrict__ u0, const double* __restrict__ w0, double* p1,
             double* u1, double* w1, double* d1, const double* __restrict__ wav, double* acc0, double* acc1,
             double* rec_p, double* rec_u, double* rec_w) {
  if ((int)blockIdx.x >= ntiles) {
    griddep_wait();
    griddep_launch_dependents();
    record(g, cells, ntiles, it - 1, p0, u0, w0, rec_p, rec_u, rec_w);
    return;
  }
  __shared__ __align__(16) double sp[kHX * kHZ];
  const Pos q(g);
  const Layout L = g.L;
  const int64_t PL = L.plane, P = L.pitch, oc = L.off(q.i, q.j);
  const double* cf = cf0 + g.grp_model[blockIdx.y] * cfs;
  const int s_beg = g.grp_beg[blockIdx.y], s_end = g.grp_beg[blockIdx.y + 1];
  const Task task[2] = {Task(g, q.i0, q.j0, threadIdx.x), Task(g, q.i0, q.j0, threadIdx.x + kThreads)};
  // p[fs-1] = -p[fs+1] (acoustic_kernels.py:135-136): row fs-1 is evaluated at row fs+1
  int64_t ot[2];
  bool mirror[2];
  double a1[2][2] = {}, b1[2][2] = {};
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    mirror[k] = g.fsurf && task[k].i == g.fs - 1;
    ot[k] = L.off(task[k].i + (mirror[k] ? 2 : 0), task[k].j);
    if (task[k].inside) {
      ld2(cf + ac::kA1M * PL + ot[k], a1[k]);
      ld2(cf + ac::kB1 * PL + ot[k], b1[k]);
    }
  }
  // w[fs-1] = w[fs] (acoustic_kernels.py:163-164): row fs-1 is evaluated at row fs
  const int down = g.fsurf && q.i == g.fs - 1 ? 1 : 0;
  double a2u[2] = {}, a2w[2] = {}, b2[2] = {}, b3[2] = {}, sum0[2] = {}, sum1[2] = {};
  bool win[2] = {};
  if (q.ok) {
    ld2(cf + ac::kA2U * PL + oc, a2u);
    ld2(cf + ac::kB2 * PL + oc, b2);
    ld2(cf + ac::kA2W * PL + oc + down * P, a2w);
    ld2(cf + ac::kB3 * PL + oc + down * P, b3);
    for (int e = 0; e < 2; ++e) win[e] = acc0 != nullptr && q.j + e < L.nxp && ac::in_window(g, q.i, q.j + e);
  }
  griddep_wait();
  griddep_launch_dependents();
  for (int s = s_beg; s < s_end; ++s) {
    const int64_t so = s * PL, o = so + oc;
    double uo[2], wo[2];
    if (q.ok) {
      ld2(u0 + o, uo);
      ld2(w0 + o + down * P, wo);
    }
    const int sz = g.src_z[s], sx = g.src_x[s];
    if (s > s_beg) __syncthreads();  // the shot before has read the halo plane
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      if (task[k].at < 0) continue;
      double v[2] = {0.0, 0.0};
      if (task[k].inside) {
        const int64_t t = so + ot[k];
        double u[6], w[4][2], pp[2], dv[2];
        ld6(u0 + t, u);
#pragma unroll
        for (int m = 0; m < 4; ++m) ld2(w0 + t + (m - 2) * P, w[m]);
        ld2(p0 + t, pp);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          // divergence in the reference's operation order (acoustic_kernels.py:118-127)
          const double t1 = rsub(radd(rsub(u[2 + e], u[1 + e]), w[2][e]), w[1][e]);
          const double t2 = rsub(radd(rsub(u[3 + e], u[e]), w[3][e]), w[0][e]);
          dv[e] = radd(rmul(g.c1, t1), rmul(g.c2, t2));
          v[e] = rsub(rmul(b1[k][e], pp[e]), rmul(a1[k][e], dv[e]));
        }
        const int sc = task[k].i + (mirror[k] ? 2 : 0) == sz ? sx - task[k].j : -1;
        if (sc == 0 || sc == 1) {
          const double sval = rmul(g.dt, wav[(int64_t)s * g.nt + it]);
          if (sc == 0) v[0] = radd(v[0], sval);
          if (sc == 1) v[1] = radd(v[1], sval);
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          if (mirror[k]) v[e] = -v[e];
          if (task[k].j + e < 0 || task[k].j + e >= L.nxp) v[e] = 0.0;
        }
        if (task[k].tile) {
          const int64_t c = so + L.off(task[k].i, task[k].j);
          st(p1 + c, v[0], v[1]);
          if (d1 != nullptr)
            st(d1 + c, ac::in_p(g, task[k].i, task[k].j) ? dv[0] : 0.0,
               ac::in_p(g, task[k].i, task[k].j + 1) ? dv[1] : 0.0);
        }
      }
      st(sp + task[k].at, v[0], v[1]);
    }
    __syncthreads();
    if (!q.ok) continue;
    const double* h = sp + (q.i - q.i0 + 1) * kHX + q.j - q.j0 + 2;
    double x[6], zm[2], z0[2], z1[2], z2[2], un[2], wn[2];
    ld6(h, x);
    const double* hw = h + down * kHX;
    ld2(hw - kHX, zm);
    ld2(hw, z0);
    ld2(hw + kHX, z1);
    ld2(hw + 2 * kHX, z2);
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const double dpx = radd(rmul(g.c1, rsub(x[3 + e], x[2 + e])), rmul(g.c2, rsub(x[4 + e], x[1 + e])));
      un[e] = rsub(rmul(b2[e], uo[e]), rmul(a2u[e], dpx));
      const double dpz = radd(rmul(g.c1, rsub(z1[e], z0[e])), rmul(g.c2, rsub(z2[e], zm[e])));
      wn[e] = rsub(rmul(b3[e], wo[e]), rmul(a2w[e], dpz));
      if (win[e]) {
        sum0[e] += x[2 + e] * x[2 + e];
        sum1[e] += un[e] * un[e];
      }
    }
    st(u1 + o, un[0], un[1]);
    st(w1 + o, wn[0], wn[1]);
  }
  for (int e = 0; e < 2; ++e)
    if (win[e]) {
      acc0[blockIdx.y * PL + oc + e] += sum0[e];
      if (acc1 != nullptr) acc1[blockIdx.y * PL + oc + e] += sum1[e];
    }
}

// One reverse step: lambda of p, u and w before the step (l0 -> l1), dL/d alpha1 (acc0) and dL/d alpha2
// (acc1) from the step's divergence dh and p after it ph, and the dL/d p-records of step it - 1.
__global__ void __launch_bounds__(kThreads)
    adj_step(ac::Geo<double> g, Cells cells, int it, const double* __restrict__ cf0, int64_t cfs,
             const double* __restrict__ lp0, const double* __restrict__ lu0, const double* __restrict__ lw0, double* lp1,
             double* lu1, double* lw1, const double* __restrict__ ph, const double* __restrict__ dh, double* acc0,
             double* acc1, const double* __restrict__ gp) {
  __shared__ __align__(16) double sq[kHX * kHZ];
  __shared__ __align__(16) double si[kZ * kX];  // dL/d p-records of the tile's cells
  const Pos q(g);
  const Layout L = g.L;
  const int64_t PL = L.plane, P = L.pitch, oc = L.off(q.i, q.j);
  const double* cf = cf0 + g.grp_model[blockIdx.y] * cfs;
  const int s_beg = g.grp_beg[blockIdx.y], s_end = g.grp_beg[blockIdx.y + 1];
  const Task task[2] = {Task(g, q.i0, q.j0, threadIdx.x), Task(g, q.i0, q.j0, threadIdx.x + kThreads)};
  const int cb = cells.tile_beg[blockIdx.x], ce = gp != nullptr && it >= 1 ? cells.tile_beg[blockIdx.x + 1] : cb;
  double b2[2] = {}, b3[2] = {}, sum1[2] = {}, sum0[2][2] = {};
  if (q.ok) {
    ld2(cf + ac::kB2 * PL + oc, b2);
    ld2(cf + ac::kB3 * PL + oc, b3);
  }
  const double gmul = ce > cb ? ac::fused_scale(g) : 1.0;
  for (int s = s_beg; s < s_end; ++s) {
    const int64_t so = s * PL, o = so + oc;
    if (ce > cb) {
      if (s > s_beg) __syncthreads();
      st(si + 2 * threadIdx.x, 0.0, 0.0);
      __syncthreads();
      for (int k = cb + (int)threadIdx.x; k < ce; k += kThreads) {
        const int c = cells.tile_cell[k];
        double ap = 0.0;
        for (int m = g.tcell_rbeg[c]; m < g.tcell_rbeg[c + 1]; ++m)
          ap += ac::grad_rec_p(g, gp, s, it - 1, g.cell_rcv[m], gmul);
        si[(cells.cell_z[c] - q.i0) * kX + cells.cell_x[c] - q.j0] = ap;
      }
    }
    if (s == s_beg) {
      griddep_wait();  // (the launch before a segment's first reverse step writes ph)
      griddep_launch_dependents();
    }
    // the differences of p after the step, whose products with lambda are dL/d alpha2
    double dpx[2] = {}, dpz[2] = {};
    if (q.ok) {
      double x[6], zm[2], z1[2], z2[2];
      ld6(ph + o, x);
      ld2(ph + o - P, zm);
      ld2(ph + o + P, z1);
      ld2(ph + o + 2 * P, z2);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        dpx[e] = ac::in_u(g, q.i, q.j + e) ? g.c1 * (x[3 + e] - x[2 + e]) + g.c2 * (x[4 + e] - x[1 + e]) : 0.0;
        dpz[e] = ac::in_w(g, q.i, q.j + e) ? g.c1 * (z1[e] - x[2 + e]) + g.c2 * (z2[e] - zm[e]) : 0.0;
      }
    }
    double l[2], m[2];
    if (q.ok) {
      ld2(lu0 + o, l);
      ld2(lw0 + o, m);
    }
    if (ce > cb || s > s_beg) __syncthreads();  // the records; the shot before has read the halo plane
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      if (task[k].at < 0) continue;
      double v[2] = {0.0, 0.0}, a1[2] = {0.0, 0.0};
      // the mirrored row fs-1 carries no sensitivity
      if (task[k].inside) {
        const int64_t c = L.off(task[k].i, task[k].j), t = so + c;
        double b1[2];
        ld2(cf + ac::kB1 * PL + c, b1);
        if (!(g.fsurf && task[k].i == g.fs - 1)) {
          double u[6], w[4][2], au[6], aw[4][2], lp[2], mir[2] = {0.0, 0.0};
          const bool below = g.fsurf && task[k].i == g.fs + 1;
          ld2(cf + ac::kA1M * PL + c, a1);
          ld6(cf + ac::kA2U * PL + c, au);
          ld6(lu0 + t, u);
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            ld2(cf + ac::kA2W * PL + c + (r - 2) * P, aw[r]);
            ld2(lw0 + t + (r - 2) * P, w[r]);
          }
          ld2(lp0 + t, lp);
          if (below) ld2(lp0 + t - 2 * P, mir);
#pragma unroll
          for (int r = 0; r < 5; ++r) u[r] *= -au[r];
#pragma unroll
          for (int e = 0; e < 2; ++e) {
#pragma unroll
            for (int r = 0; r < 4; ++r) w[r][e] *= -aw[r][e];
            v[e] = lp[e] + g.c1 * (u[1 + e] - u[2 + e]) + g.c2 * (u[e] - u[3 + e]) + g.c1 * (w[1][e] - w[2][e]) +
                   g.c2 * (w[0][e] - w[3][e]);
            // adjoint of p[fs-1] = -p[fs+1]: of what lambda_p[fs-1] gathers, only row fs of w is not zero
            if (below) v[e] -= mir[e] - g.c2 * w[1][e];
            if (task[k].j + e < 0 || task[k].j + e >= L.nxp) v[e] = 0.0;
          }
        }
        if (task[k].tile) {
          double d[2], n[2] = {b1[0] * v[0], b1[1] * v[1]};
          ld2(dh + t, d);
          sum0[k][0] -= v[0] * d[0];
          sum0[k][1] -= v[1] * d[1];
          if (ce > cb) {
            const double* r = si + (task[k].i - q.i0) * kX + task[k].j - q.j0;
            n[0] += r[0];
            n[1] += r[1];
          }
          st(lp1 + t, n[0], n[1]);
        }
      }
      st(sq + task[k].at, -a1[0] * v[0], -a1[1] * v[1]);
    }
    __syncthreads();
    if (!q.ok) continue;
    const double* h = sq + (q.i - q.i0 + 1) * kHX + q.j - q.j0 + 2;
    double x[6], zm[2], z1[2], z2[2];
    ld6(h, x);
    ld2(h - kHX, zm);
    ld2(h + kHX, z1);
    ld2(h + 2 * kHX, z2);
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      sum1[e] -= l[e] * dpx[e];
      sum1[e] -= m[e] * dpz[e];
      l[e] = b2[e] * l[e] + g.c1 * (x[2 + e] - x[3 + e]) + g.c2 * (x[1 + e] - x[4 + e]);
      m[e] = b3[e] * m[e] + g.c1 * (x[2 + e] - z1[e]) + g.c2 * (zm[e] - z2[e]);
    }
    if (g.fsurf && q.i == g.fs - 1) m[0] = m[1] = 0.0;
    if (g.fsurf && q.i == g.fs) {  // adjoint of w[fs-1] = w[fs] (rows fs-2 .. of the halo: the tiles begin at fs-1)
      double up[2], ub[2], z[2];
      ld2(lw0 + o - P, up);
      ld2(cf + ac::kB3 * PL + oc - P, ub);
      ld2(h - 2 * kHX, z);
#pragma unroll
      for (int e = 0; e < 2; ++e) m[e] += ub[e] * up[e] + g.c1 * (zm[e] - x[2 + e]) + g.c2 * (z[e] - z1[e]);
    }
    if (q.j + 1 >= L.nxp) l[1] = m[1] = 0.0;
    st(lu1 + o, l[0], l[1]);
    st(lw1 + o, m[0], m[1]);
  }
#pragma unroll
  for (int k = 0; k < 2; ++k)
    if (task[k].tile) {
      double* a = acc0 + blockIdx.y * PL + L.off(task[k].i, task[k].j);
      const double2 t = ld(a);
      st(a, t.x + sum0[k][0], t.y + sum0[k][1]);
    }
  if (q.ok) {
    double* a = acc1 + blockIdx.y * PL + oc;
    const double2 t = ld(a);
    st(a, t.x + sum1[0], t.y + sum1[1]);
  }
}

// dL/d u- and w-records of step it into lambda_u and lambda_w, with the adjoint of w[fs-1] = w[fs]: at the
// receiver cells of row fs-1 (mirrored) or at all others. Two cells of a column can meet on row fs, so the
// two kinds take a launch each: the sums have one order.
__global__ void adj_inject_uw(ac::Geo<double> g, Cells cells, int it, bool mirrored, const double* gu, const double* gw,
                              double* lu, double* lw) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= cells.ncells) return;
  const int s = blockIdx.y, i = cells.cell_z[k], j = cells.cell_x[k];
  if ((g.fsurf && i == g.fs - 1) != mirrored) return;
  double au = 0.0, aw = 0.0;
  for (int m = g.tcell_rbeg[k]; m < g.tcell_rbeg[k + 1]; ++m) {
    const int64_t e = ((int64_t)s * g.nt + it) * g.nr + g.cell_rcv[m];
    if (gu) au += gu[e];
    if (gw) aw += gw[e];
  }
  const int64_t so = s * g.L.plane;
  lu[so + g.L.off(i, j)] += au;
  lw[so + g.L.off(mirrored ? g.fs : i, j)] += aw;
}

}  // namespace ac3
}  // namespace adfwi
