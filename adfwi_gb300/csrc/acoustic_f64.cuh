// Acoustic time step and its reverse in double precision, two launches each: p, then u and w; lambda_p,
// then lambda_u and lambda_w (acoustic_kernels.py:115-169 and its transposes).
//
// What bounds them is double-precision arithmetic, two lanes per clock and SM: 28 operations a cell
// forward and 37 in reverse, 5.6 and 7.4 us for five shots of 121 x 193 cells. So no value is formed
// twice by neighbouring tiles (which costs the fused step of one launch a quarter more operations on
// its halos), and the work is cut finely: a block of 128 threads takes 8 rows of 32 columns of one
// shot group, two columns per thread, 560 blocks there, where tiles of 16 x 64 cells with two shots
// each kept 96 of the 152 SMs busy. 300 forward and reverse steps of those shots: 29.0 -> 14.8 ms; a
// launch takes 12 us, 3 of them arithmetic, the rest the launch boundary and one round of loads.
//
// Launches are programmatically serialised: a kernel reads what the launch before it does not write
// ahead of that launch's end. The records of a step are taken by extra blocks of the first launch that
// only reads the field (p: the second launch of the step; u and w: the first of the next), and the
// dL/d p-records are added by extra blocks of the reverse step's second launch.
#pragma once
#include "acoustic_geo.cuh"
#include "common.cuh"

namespace adfwi {
namespace ac3 {

using ac::radd;
using ac::rmul;
using ac::rsub;

constexpr int kX = 32, kThreads = 128, kLanes = kX / 2, kZ = kThreads / kLanes;

// Padded cells (i << 16 | j) of the receivers and of the unique receiver cells (in the order of
// Geo's tcell_rbeg).
struct Cells {
  const int* rcv;
  const int* cell;
  int ncells;
};

inline int tiles(const Layout& L, int zbeg) { return ((L.nxp + kX - 1) / kX) * ((L.nzp - zbeg + kZ - 1) / kZ); }

struct Pos {
  int i, j;
  bool ok;
  __device__ __forceinline__ explicit Pos(const ac::Geo<double>& g) {
    const int tx = (g.L.nxp + kX - 1) / kX, ti = (int)blockIdx.x / tx;
    i = g.zbeg + ti * kZ + (int)threadIdx.x / kLanes;
    j = ((int)blockIdx.x - ti * tx) * kX + (int)threadIdx.x % kLanes * 2;
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

// Records of step `it` at receiver q of this block's shots: `n` fields from f0, f1.
__device__ __forceinline__ void record(const ac::Geo<double>& g, const Cells& c, int first, int it, int n, const double* f0,
                                       const double* f1, double* r0, double* r1) {
  const int r = ((int)blockIdx.x - first) * kThreads + (int)threadIdx.x;
  if (r >= g.nr) return;
  const int64_t oc = g.L.off(c.rcv[r] >> 16, c.rcv[r] & 0xffff);
  for (int s = g.grp_beg[blockIdx.y]; s < g.grp_beg[blockIdx.y + 1]; ++s) {
    const int64_t o = (int64_t)s * g.L.plane + oc, e = ((int64_t)s * g.nt + it) * g.nr + r;
    r0[e] = f0[o];
    if (n == 2) r1[e] = f1[o];
  }
}

// p and the divergence of step it (d1 null: not kept) from p0, u0, w0; illumination sums of p; extra
// blocks: the records of u and w of step it - 1.
__global__ void __launch_bounds__(kThreads)
    p_step(ac::Geo<double> g, Cells cells, int ntiles, int it, const double* __restrict__ cf0, int64_t cfs,
           const double* p0, const double* __restrict__ u0, const double* __restrict__ w0, double* p1, double* d1,
           const double* __restrict__ wav, double* acc, double* rec_u, double* rec_w) {
  if ((int)blockIdx.x >= ntiles) {
    griddep_wait();
    griddep_launch_dependents();
    record(g, cells, ntiles, it - 1, 2, u0, w0, rec_u, rec_w);
    return;
  }
  const Pos q(g);
  const Layout L = g.L;
  const int64_t PL = L.plane, P = L.pitch, oc = L.off(q.i, q.j);
  const double* cf = cf0 + g.grp_model[blockIdx.y] * cfs;
  const int s_beg = g.grp_beg[blockIdx.y], s_end = g.grp_beg[blockIdx.y + 1];
  double a1[2] = {}, b1[2] = {}, sum[2] = {}, pp[2] = {};
  if (q.ok) {
    ld2(cf + ac::kA1M * PL + oc, a1);
    ld2(cf + ac::kB1 * PL + oc, b1);
    ld2(p0 + s_beg * PL + oc, pp);
  }
  griddep_wait();
  griddep_launch_dependents();
  if (!q.ok) return;
  const bool mirror = g.fsurf && q.i == g.fs - 1;  // p[fs-1] = -p[fs+1], written by row fs+1
  bool win[2];
  for (int e = 0; e < 2; ++e) win[e] = acc != nullptr && q.j + e < L.nxp && ac::in_window(g, q.i, q.j + e);
  for (int s = s_beg; s < s_end; ++s) {
    const int64_t o = s * PL + oc;
    if (s > s_beg) ld2(p0 + o, pp);
    double u[6], w[4][2], dv[2], v[2];
    ld6(u0 + o, u);
#pragma unroll
    for (int k = 0; k < 4; ++k) ld2(w0 + o + (k - 2) * P, w[k]);
    const int sc = q.i == g.src_z[s] ? g.src_x[s] - q.j : -1;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      // divergence in the reference's operation order (acoustic_kernels.py:118-127)
      const double t1 = rsub(radd(rsub(u[2 + e], u[1 + e]), w[2][e]), w[1][e]);
      const double t2 = rsub(radd(rsub(u[3 + e], u[e]), w[3][e]), w[0][e]);
      dv[e] = radd(rmul(g.c1, t1), rmul(g.c2, t2));
      v[e] = rsub(rmul(b1[e], pp[e]), rmul(a1[e], dv[e]));
    }
    if (sc == 0 || sc == 1) {
      const double sval = rmul(g.dt, wav[(int64_t)s * g.nt + it]);
      v[0] = sc == 0 ? radd(v[0], sval) : v[0];
      v[1] = sc == 1 ? radd(v[1], sval) : v[1];
    }
    if (!mirror) st(p1 + o, v[0], v[1]);
    if (g.fsurf && q.i == g.fs + 1) st(p1 + o - 2 * P, -v[0], -v[1]);
    if (d1 != nullptr)
      st(d1 + o, ac::in_p(g, q.i, q.j) ? dv[0] : 0.0, ac::in_p(g, q.i, q.j + 1) ? dv[1] : 0.0);
#pragma unroll
    for (int e = 0; e < 2; ++e)
      if (win[e]) sum[e] += v[e] * v[e];
  }
  if (win[0] || win[1]) {
    double* a = acc + blockIdx.y * PL + oc;
    for (int e = 0; e < 2; ++e)
      if (win[e]) a[e] += sum[e];
  }
}

// u and w of a step from p1 (after the step), u0, w0; illumination sums of u; extra blocks: the records
// of p of step it.
__global__ void __launch_bounds__(kThreads)
    uw_step(ac::Geo<double> g, Cells cells, int ntiles, int it, const double* __restrict__ cf0, int64_t cfs,
            const double* __restrict__ p1, const double* u0, const double* w0, double* u1, double* w1, double* acc,
            double* rec_p) {
  if ((int)blockIdx.x >= ntiles) {
    griddep_wait();
    griddep_launch_dependents();
    record(g, cells, ntiles, it, 1, p1, nullptr, rec_p, nullptr);
    return;
  }
  const Pos q(g);
  const Layout L = g.L;
  const int64_t PL = L.plane, P = L.pitch, oc = L.off(q.i, q.j);
  const double* cf = cf0 + g.grp_model[blockIdx.y] * cfs;
  const int s_beg = g.grp_beg[blockIdx.y], s_end = g.grp_beg[blockIdx.y + 1];
  double a2u[2] = {}, a2w[2] = {}, b2[2] = {}, b3[2] = {}, sum[2] = {}, uo[2] = {}, wo[2] = {};
  if (q.ok) {
    ld2(cf + ac::kA2U * PL + oc, a2u);
    ld2(cf + ac::kB2 * PL + oc, b2);
    ld2(cf + ac::kA2W * PL + oc, a2w);
    ld2(cf + ac::kB3 * PL + oc, b3);
    ld2(u0 + s_beg * PL + oc, uo);
    ld2(w0 + s_beg * PL + oc, wo);
  }
  griddep_wait();
  griddep_launch_dependents();
  if (!q.ok) return;
  bool win[2];
  for (int e = 0; e < 2; ++e) win[e] = acc != nullptr && q.j + e < L.nxp && ac::in_window(g, q.i, q.j + e);
  for (int s = s_beg; s < s_end; ++s) {
    const int64_t o = s * PL + oc;
    if (s > s_beg) {
      ld2(u0 + o, uo);
      ld2(w0 + o, wo);
    }
    double x[6], zm[2], z1[2], z2[2], un[2], wn[2];
    ld6(p1 + o, x);
    ld2(p1 + o - P, zm);
    ld2(p1 + o + P, z1);
    ld2(p1 + o + 2 * P, z2);
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const double dpx = radd(rmul(g.c1, rsub(x[3 + e], x[2 + e])), rmul(g.c2, rsub(x[4 + e], x[1 + e])));
      un[e] = rsub(rmul(b2[e], uo[e]), rmul(a2u[e], dpx));
      const double dpz = radd(rmul(g.c1, rsub(z1[e], x[2 + e])), rmul(g.c2, rsub(z2[e], zm[e])));
      wn[e] = rsub(rmul(b3[e], wo[e]), rmul(a2w[e], dpz));
      if (win[e]) sum[e] += un[e] * un[e];
    }
    st(u1 + o, un[0], un[1]);
    if (!(g.fsurf && q.i == g.fs - 1)) st(w1 + o, wn[0], wn[1]);
    if (g.fsurf && q.i == g.fs) st(w1 + o - P, wn[0], wn[1]);  // w[fs-1] = w[fs] (acoustic_kernels.py:163-164)
  }
  if (win[0] || win[1]) {
    double* a = acc + blockIdx.y * PL + oc;
    for (int e = 0; e < 2; ++e)
      if (win[e]) a[e] += sum[e];
  }
}

// The records of u and w of the last step (the next step's p update would have taken them).
__global__ void record_uw(ac::Geo<double> g, Cells cells, int it, const double* u, const double* w, double* rec_u,
                          double* rec_w) {
  griddep_wait();
  griddep_launch_dependents();
  record(g, cells, 0, it, 2, u, w, rec_u, rec_w);
}

// Reverse of the p update: lambda_p after the transposes of the u and w updates' pressure differences,
// times 1 - damp dt (lp0 -> lp1), q = -alpha1 lambda_p, and dL/d alpha1 (dh: the step's divergence).
__global__ void __launch_bounds__(kThreads)
    adj_p_step(ac::Geo<double> g, const double* __restrict__ cf0, int64_t cfs, const double* __restrict__ lp0,
               const double* __restrict__ lu, const double* __restrict__ lw, double* __restrict__ lp1,
               double* __restrict__ qp, const double* __restrict__ dh, double* acc) {
  const Pos q(g);
  const Layout L = g.L;
  const int64_t PL = L.plane, P = L.pitch, oc = L.off(q.i, q.j);
  const double* cf = cf0 + g.grp_model[blockIdx.y] * cfs;
  const int s_beg = g.grp_beg[blockIdx.y], s_end = g.grp_beg[blockIdx.y + 1];
  double a1[2] = {}, b1[2] = {}, au[6] = {}, aw[4][2] = {}, d[2] = {}, sum[2] = {};
  if (q.ok) {
    ld2(cf + ac::kA1M * PL + oc, a1);
    ld2(cf + ac::kB1 * PL + oc, b1);
    ld6(cf + ac::kA2U * PL + oc, au);
#pragma unroll
    for (int k = 0; k < 4; ++k) ld2(cf + ac::kA2W * PL + oc + (k - 2) * P, aw[k]);
    ld2(dh + s_beg * PL + oc, d);
  }
  griddep_wait();
  griddep_launch_dependents();
  if (!q.ok) return;
  for (int s = s_beg; s < s_end; ++s) {
    const int64_t o = s * PL + oc;
    if (s > s_beg) ld2(dh + o, d);
    double u[6], w[4][2], l[2], v[2];
    ld2(lp0 + o, l);
    ld6(lu + o, u);
#pragma unroll
    for (int k = 0; k < 4; ++k) ld2(lw + o + (k - 2) * P, w[k]);
    double m[2] = {0.0, 0.0};
    const bool below = g.fsurf && q.i == g.fs + 1;
    if (below) ld2(lp0 + o - 2 * P, m);
#pragma unroll
    for (int k = 0; k < 5; ++k) u[k] *= -au[k];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
#pragma unroll
      for (int k = 0; k < 4; ++k) w[k][e] *= -aw[k][e];
      v[e] = l[e] + g.c1 * (u[1 + e] - u[2 + e]) + g.c2 * (u[e] - u[3 + e]) + g.c1 * (w[1][e] - w[2][e]) +
             g.c2 * (w[0][e] - w[3][e]);
      // adjoint of p[fs-1] = -p[fs+1]: of what lambda_p[fs-1] gathers, only row fs of w is not zero
      if (below) v[e] -= m[e] - g.c2 * w[1][e];
      if ((g.fsurf && q.i == g.fs - 1) || q.j + e >= L.nxp) v[e] = 0.0;
      sum[e] -= v[e] * d[e];
    }
    st(lp1 + o, b1[0] * v[0], b1[1] * v[1]);
    st(qp + o, -a1[0] * v[0], -a1[1] * v[1]);
  }
  double* a = acc + blockIdx.y * PL + oc;
  const double2 t = ld(a);
  st(a, t.x + sum[0], t.y + sum[1]);
}

// Reverse of the u and w updates: lambda_u and lambda_w in place from the transposes of the p update's
// differences (q), dL/d alpha2 (ph: p after the step); extra blocks: the dL/d p-records of step it - 1
// into lp.
__global__ void __launch_bounds__(kThreads)
    adj_uw_step(ac::Geo<double> g, Cells cells, int ntiles, int it, const double* __restrict__ cf0, int64_t cfs,
                const double* __restrict__ qp, double* lu, double* lw, const double* __restrict__ ph, double* acc,
                const double* __restrict__ gp, double* lp) {
  if ((int)blockIdx.x >= ntiles) {
    const int k = ((int)blockIdx.x - ntiles) * kThreads + (int)threadIdx.x;
    const double gmul = ac::fused_scale(g);
    griddep_wait();
    griddep_launch_dependents();
    if (k >= cells.ncells) return;
    const int zx = cells.cell[k];
    for (int s = g.grp_beg[blockIdx.y]; s < g.grp_beg[blockIdx.y + 1]; ++s) {
      double ap = 0.0;
      for (int m = g.tcell_rbeg[k]; m < g.tcell_rbeg[k + 1]; ++m)
        ap += ac::grad_rec_p(g, gp, s, it - 1, g.cell_rcv[m], gmul);
      lp[s * g.L.plane + g.L.off(zx >> 16, zx & 0xffff)] += ap;
    }
    return;
  }
  const Pos q(g);
  const Layout L = g.L;
  const int64_t PL = L.plane, P = L.pitch, oc = L.off(q.i, q.j);
  const double* cf = cf0 + g.grp_model[blockIdx.y] * cfs;
  const int s_beg = g.grp_beg[blockIdx.y], s_end = g.grp_beg[blockIdx.y + 1];
  double b2[2] = {}, b3[2] = {}, sum[2] = {}, l[2] = {}, m[2] = {};
  if (q.ok) {
    ld2(cf + ac::kB2 * PL + oc, b2);
    ld2(cf + ac::kB3 * PL + oc, b3);
    ld2(lu + s_beg * PL + oc, l);
    ld2(lw + s_beg * PL + oc, m);
  }
  griddep_wait();
  griddep_launch_dependents();
  if (!q.ok) return;
  for (int s = s_beg; s < s_end; ++s) {
    const int64_t o = s * PL + oc;
    if (s > s_beg) {
      ld2(lu + o, l);
      ld2(lw + o, m);
    }
    {
      // the differences of p whose products with the old lambda are dL/d alpha2
      double x[6], zm[2], z1[2], z2[2];
      ld6(ph + o, x);
      ld2(ph + o - P, zm);
      ld2(ph + o + P, z1);
      ld2(ph + o + 2 * P, z2);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        if (ac::in_u(g, q.i, q.j + e)) sum[e] -= l[e] * (g.c1 * (x[3 + e] - x[2 + e]) + g.c2 * (x[4 + e] - x[1 + e]));
        if (ac::in_w(g, q.i, q.j + e)) sum[e] -= m[e] * (g.c1 * (z1[e] - x[2 + e]) + g.c2 * (z2[e] - zm[e]));
      }
    }
    double x[6], zm[2], z1[2], z2[2];
    ld6(qp + o, x);
    ld2(qp + o - P, zm);
    ld2(qp + o + P, z1);
    ld2(qp + o + 2 * P, z2);
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      l[e] = b2[e] * l[e] + g.c1 * (x[2 + e] - x[3 + e]) + g.c2 * (x[1 + e] - x[4 + e]);
      m[e] = b3[e] * m[e] + g.c1 * (x[2 + e] - z1[e]) + g.c2 * (zm[e] - z2[e]);
      if (q.j + e >= L.nxp) l[e] = m[e] = 0.0;
    }
    st(lu + o, l[0], l[1]);
    if (g.fsurf && q.i == g.fs - 1) continue;  // row fs writes this row of lambda_w
    if (g.fsurf && q.i == g.fs) {  // adjoint of w[fs-1] = w[fs]
      double up[2], ub[2], z[2];
      ld2(lw + o - P, up);
      ld2(cf + ac::kB3 * PL + oc - P, ub);
      ld2(qp + o - 2 * P, z);
#pragma unroll
      for (int e = 0; e < 2; ++e)
        if (q.j + e < L.nxp) m[e] += ub[e] * up[e] + g.c1 * (zm[e] - x[2 + e]) + g.c2 * (z[e] - z1[e]);
      st(lw + o - P, 0.0, 0.0);
    }
    st(lw + o, m[0], m[1]);
  }
  double* a = acc + blockIdx.y * PL + oc;
  const double2 t = ld(a);
  st(a, t.x + sum[0], t.y + sum[1]);
}

// dL/d u- and w-records of step it into lambda_u and lambda_w, with the adjoint of w[fs-1] = w[fs].
__global__ void adj_inject_uw(ac::Geo<double> g, Cells cells, int it, const double* gu, const double* gw, double* lu,
                              double* lw) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= cells.ncells) return;
  const int s = blockIdx.y, zx = cells.cell[k], i = zx >> 16, j = zx & 0xffff;
  double au = 0.0, aw = 0.0;
  for (int m = g.tcell_rbeg[k]; m < g.tcell_rbeg[k + 1]; ++m) {
    const int64_t e = ((int64_t)s * g.nt + it) * g.nr + g.cell_rcv[m];
    if (gu) au += gu[e];
    if (gw) aw += gw[e];
  }
  const int64_t so = s * g.L.plane;
  lu[so + g.L.off(i, j)] += au;
  // two receiver cells can meet on row fs
  atomicAdd(lw + so + g.L.off(g.fsurf && i == g.fs - 1 ? g.fs : i, j), aw);
}

}  // namespace ac3
}  // namespace adfwi
