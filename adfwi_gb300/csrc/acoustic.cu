// Acoustic (p, u, w) 4th-order staggered-grid propagator for sm_103a: forward step,
// exact discrete adjoint step, checkpoint / recompute driver and the C ABI.
//
// Reference algorithm (paths inside liufeng2317/ADFWI):
//   ADFWI/propagator/acoustic_kernels.py:113-174  one time step (p update, source, free-surface
//                                                 mirror, u and w updates, w mirror, receivers,
//                                                 illumination sums)
//   ADFWI/propagator/acoustic_kernels.py:252-265  alpha / kappa coefficient definitions
//   ADFWI/propagator/acoustic_kernels.py:268-301  chunked time loop and the record dict
//
// Float32 solves run on the resident time loop (acoustic_res.cuh) wherever a shot's state fits the
// shared memory of the blocks that work on it; the per-step kernels below take the rest: FP64,
// boundary saving, grids too large, receivers on the mirrored row above a free surface, and
// adjoints driven by dL/d u- or w-records.
//
// Per-step kernels: one launch advances one time step of all shots (acoustic_tma.cuh,
// acoustic_vec.cuh): persistent, warp-specialised blocks stream (tile, shot) items through a TMA / mbarrier
// pipeline; per item the consumers compute the new pressure on a 16 x 64 tile plus its halo
// (1 row / column before, 2 after) and then the new u and w on the tile, four adjacent
// columns per thread, so p, u and w each cross HBM once per step (ping-pong buffers keep the
// Jacobi semantics of the reference's slice assignments). The forward arithmetic uses explicitly rounded operations (no FMA
// contraction) in the reference's evaluation order, so float32 records reproduce the
// reference's PyTorch CPU results bit for bit. The adjoint step is the exact transpose of
// the forward step, in reverse operation order.
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <cmath>
#include <mutex>
#include <new>
#include <vector>

#include "../../include/adfwi_gb300.h"
#include "acoustic_geo.cuh"
#include "common.cuh"
#include "frames.cuh"
#include "l2.cuh"
#include "snapshot.cuh"
#include "tma.cuh"

namespace adfwi {
namespace ac {

// Seed of the reverse pass: lambda = injection of the records of the last step.
template <typename T>
__global__ void adj_seed(Geo<T> g, int ntiles, int tz, int tx, const T* __restrict__ gr_p, const T* __restrict__ gr_u,
                         const T* __restrict__ gr_w, T* lp, T* lu, T* lw) {
  const int sh = blockIdx.y;
  const int64_t rowbase = ((int64_t)sh * g.nt + (g.nt - 1)) * g.nr;
  const int ncell = g.tile_cell_beg[ntiles];
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < ncell; q += gridDim.x * blockDim.x) {
    int tile = 0;
    {  // locate the tile of unique cell q (binary search on tile_cell_beg)
      int lo = 0, hi = ntiles;
      while (hi - lo > 1) {
        int mid = (lo + hi) >> 1;
        if (g.tile_cell_beg[mid] <= q) lo = mid; else hi = mid;
      }
      tile = lo;
    }
    int cell = g.tcell_cell[q];
    int i = g.zbeg + (tile / g.tiles_x) * tz + (cell >> 16);
    int j = (tile % g.tiles_x) * tx + (cell & 0xffff);
    T ap = T(0), au = T(0), aw = T(0);
    const T gmul = fused_scale(g);
    for (int m = g.tcell_rbeg[q]; m < g.tcell_rbeg[q + 1]; ++m) {
      int64_t o = rowbase + g.cell_rcv[m];
      if (gr_p) ap += grad_rec_p(g, gr_p, sh, g.nt - 1, g.cell_rcv[m], gmul);
      if (gr_u) au += gr_u[o];
      if (gr_w) aw += gr_w[o];
    }
    int64_t o = (int64_t)sh * g.L.plane + g.L.off(i, j);
    lp[o] += ap;
    lu[o] += au;
    lw[o] += aw;
  }
}

// The adjoint of w[fs-1] = w[fs] (acoustic_kernels.py:163-164), which closes the last step, on the seed: the
// reverse steps fold what they inject themselves.
template <typename T>
__global__ void fold_mirrored_w(Geo<T> g, T* lw) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= g.L.nxp) return;
  T* up = lw + (int64_t)blockIdx.y * g.L.plane + g.L.off(g.fs - 1, j);
  up[g.L.pitch] += *up;
  *up = T(0);
}

// Copy a dense (h, w) array into a pitched plane at cell (0, 0) (ghosts untouched).
template <typename T>
__global__ void pack_plane(Layout L, int h, int w, const T* __restrict__ src, T* __restrict__ dst) {
  int64_t n = (int64_t)h * w;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
    int i = (int)(e / w), j = (int)(e - (int64_t)i * w);
    dst[L.off(i, j)] = src[e];
  }
}

// dst(h, w) = sum over `groups` partial planes of the window starting at (oi, oj).
template <typename T>
__global__ void reduce_planes(Layout L, int groups, int oi, int oj, int h, int w, const T* __restrict__ src,
                              T* __restrict__ dst) {
  int64_t n = (int64_t)h * w;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
    int i = (int)(e / w), j = (int)(e - (int64_t)i * w);
    T acc = T(0);
    for (int q = 0; q < groups; ++q) acc += src[(int64_t)q * L.plane + L.off(oi + i, oj + j)];
    dst[e] = acc;
  }
}

// forward_wavefield_{p,u,w} of the reference (acoustic_kernels.py:172-174, 285-288):
// fw_p = P, fw_u = P + U(last chunk), fw_w = fw_p + (U(last chunk) + sum_s w(last step)^2).
template <typename T>
__global__ void illum_finalize(Layout L, int groups, int ns, int nabc, int nz, int nx, const T* __restrict__ ip,
                               const T* __restrict__ iu, const T* __restrict__ wlast, T* fw_p, T* fw_u,
                               T* fw_w) {
  int64_t n = (int64_t)nz * nx;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
    int i = (int)(e / nx) + nabc, j = (int)(e % nx) + nabc;
    T P = T(0), U = T(0), W = T(0);
    for (int q = 0; q < groups; ++q) {
      P += ip[(int64_t)q * L.plane + L.off(i, j)];
      U += iu[(int64_t)q * L.plane + L.off(i, j)];
    }
    for (int s = 0; s < ns; ++s) {
      T v = wlast[(int64_t)s * L.plane + L.off(i, j)];
      W += v * v;
    }
    if (fw_p) fw_p[e] = P;
    if (fw_u) fw_u[e] = P + U;
    if (fw_w) fw_w[e] = P + (U + W);
  }
}

template <typename T>
__global__ void mask_coefficients(Geo<T> g, T* cf) {
  const Layout L = g.L;
  const int64_t n = (int64_t)L.nzp * L.nxp;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
    const int i = (int)(e / L.nxp), j = (int)(e - (int64_t)i * L.nxp);
    const int64_t o = L.off(i, j);
    const T* d = cf + kDamp * L.plane;
    const T a1 = cf[kA1 * L.plane + o], a2 = cf[kA2 * L.plane + o];
    const bool pin = in_p(g, i, j), uin = in_u(g, i, j), win = in_w(g, i, j);
    cf[kA1M * L.plane + o] = pin ? a1 : T(0);
    cf[kB1 * L.plane + o] = pin ? rsub(T(1), rmul(d[o], g.dt)) : T(1);
    cf[kA2U * L.plane + o] = uin ? a2 : T(0);
    cf[kB2 * L.plane + o] = uin ? rsub(T(1), rmul(rmul(T(0.5), radd(d[o], d[o + 1])), g.dt)) : T(1);
    cf[kA2W * L.plane + o] = win ? a2 : T(0);
    cf[kB3 * L.plane + o] = win ? rsub(T(1), rmul(rmul(T(0.5), radd(d[o], d[o + L.pitch])), g.dt)) : T(1);
  }
}

}  // namespace ac

namespace res {

// Gradient of one model from its shots' sums: dst = - (sum over the shots) / alpha on rows from
// z0 (zero above); a cell whose alpha is zero was summed without the scale.
__global__ void reduce_scaled(Layout L, int z0, int shots, const float* __restrict__ alpha,
                              const float* __restrict__ src, float* __restrict__ dst) {
  const int64_t n = (int64_t)L.nzp * L.nxp;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
    const int i = (int)(e / L.nxp), j = (int)(e - (int64_t)i * L.nxp);
    const int64_t o = L.off(i, j);
    float acc = 0.0f;
    if (i >= z0)
      for (int s = 0; s < shots; ++s) acc += src[(int64_t)s * L.plane + o];
    const float al = alpha[o];
    dst[e] = -acc / (al == 0.0f ? 1.0f : al);
  }
}

// The divergence histories written by time_loop hold the stencil's value on every row and column;
// the per-step adjoint wants zeroes outside the p region: rows above fs + 1 and the last two, the
// first and last two columns.
__global__ void zero_outside_p(const __grid_constant__ ac::Geo<float> g, int64_t planes, float* hd) {
  const Layout L = g.L;
  const int top = g.fs + 1 - g.zbeg, n = (top + 2) * L.nxp + 4 * (L.nzp - 2 - g.fs - 1);
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < planes * n; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t pl = e / n;
    int k = (int)(e - pl * n), i, j;
    if (k < (top + 2) * L.nxp) {
      i = k / L.nxp;
      j = k - i * L.nxp;
      i = i < top ? g.zbeg + i : L.nzp - 2 + (i - top);
    } else {
      k -= (top + 2) * L.nxp;
      i = g.fs + 1 + k / 4;
      j = k % 4 < 2 ? k % 4 : L.nxp - 4 + k % 4;
    }
    hd[pl * L.plane + L.off(i, j)] = 0.0f;
  }
}

}  // namespace res
}  // namespace adfwi

#include "acoustic_tma.cuh"
#include "acoustic_vec.cuh"
#include "acoustic_f64.cuh"
#include "acoustic_res.h"
#include "bsave.cuh"

// ----------------------------------------------------------------------------------------
// Plan, workspace and drivers.
// ----------------------------------------------------------------------------------------
using namespace adfwi;

// Tiling of the grid for one kernel generation, with its receiver tables (offsets into tab).
struct Tiling {
  int tz, tx;
  int tiles_x, tiles_z, ntiles;
  int G, ngroups;  // shots per unit / units per tile
  int blocks;      // launch width of the adjoint step (persistent kernel)
  int fwd_blocks;  // launch width of the forward step (persistent kernel)
  int64_t o_trb, o_trc, o_tri, o_tcb, o_tcc, o_tcr, o_cr, o_gb, o_gm;
  int ncells;
};

// Launch configuration of the resident time loop (acoustic_res.cuh). G = 0: not taken.
struct Resident {
  int glb = 0;                     // strips exchange rows through global memory (else a cluster)
  int G = 0, S = 0, R = 0, RB = 0, MT = 0, TR = 0, T = 0, CG = 0;
  int oS = 0, oA1 = 0, oA2 = 0, oPH = 0, oDH = 0, oBox = 0, oInj = 0, injw = 0, injg = 0, oRow = 0, oT = 0, words = 0;
  int64_t o_sl = 0, o_sb = 0, o_tp = 0, o_ti = 0, o_rb = 0, o_rv = 0;  // tab: strips' receiver cells
};

struct adfwi_acoustic_plan {
  adfwi_acoustic_desc d;
  int nzp, nxp, fs, zbeg;
  bool rcv_above = false;  // receivers on the mirrored row above a free surface
  Tiling t2;             // 16 x 64 tiles of the pipelined forward and adjoint steps
  Resident rf, ra;       // the resident time loop, forward and adjoint, where the grid allows it
  int64_t o_sm = 0;      // tab: the model of each shot
  // tab (FP64): padded rows and columns of the receivers and of the unique receiver cells; the latter by tile
  int64_t o_rz = 0, o_rx = 0, o_cz = 0, o_cx = 0, o_ftb = 0, o_ftc = 0;
  int K, nseg;           // snapshot interval and number of segments (gradient mode)
  int last_chunk_start;  // first step of the reference's last checkpoint chunk
  int elem;              // bytes per element
  bool deep = false;     // deep-ring variants of the step kernels (FP32 only)
  bool bsave = false;    // gradient by boundary saving (snapshot_every = ADFWI_SNAP_EVERY_BOUNDARY)
  int nframe = 0;        // frame cells of a plane (boundary saving)
  int64_t o_fidx = 0, o_foff = 0;  // tab offsets: frame index of every cell (-1: interior), frame offsets
  ac::BsBox bbox{0, -1, 0, -1};     // the interior the reverse pass rebuilds
  int nm;                // models of a batched plan (1 otherwise)
  std::vector<int> model_shot_beg;  // nm+1 offsets: the shots of each model
  std::vector<int> model_grp_beg;   // nm+1 offsets: the shot groups of each model
  Layout L;
  std::vector<int32_t> tab;  // geometry tables, uploaded into the workspace
  PinnedBytes tab_pin;       // page-locked copy of tab, the source of each upload
  int64_t o_srcz, o_srcx;
};

namespace {

struct Carve {
  int64_t coef, fa, fb, ilp, ilu, tab, flag, box;  // forward (box: the strips' inboxes)
  int64_t snap, snap_scale, bsv, hp, hd, la, lb, abox, g1, g2;  // gradient extras (abox: the adjoint's inboxes)
  int64_t mst, mpk, mnorm, mfac;                     // fused misfit: trace stats, gather peaks, norms, factors
  int64_t total;
};

int64_t align256(int64_t x) { return (x + 255) / 256 * 256; }

int64_t res_box_bytes(const Resident& r);

// A gradient plan in boundary-saving mode (with a single step there is nothing to rebuild: the
// history of that step is kept).
bool boundary_saving(const adfwi_acoustic_plan* p) { return p->bsave && p->d.nt > 1; }

// (box: with the inboxes of the resident loop's strips. They lie in planes that the loop leaves unused,
// the third of each shot in fb and the per-step kernels' illumination sums after it, in lb and the
// per-step gradient sums after it, where they fit: so that a plan's snapshot interval under a memory
// budget, which decides what quantised snapshots round, does not depend on them)
Carve carve(const adfwi_acoustic_plan* p, bool grad, int K, bool box = true) {
  Carve c{};
  const int64_t pl = p->L.plane * p->elem;
  const int64_t ns = p->d.ns;
  int64_t o = 0;
  auto take = [&](int64_t bytes) { int64_t at = o; o += align256(bytes); return at; };
  c.coef = take((int64_t)p->nm * ac::kNumCoef * pl);
  c.fa = take(3 * ns * pl);
  c.fb = take(3 * ns * pl);
  c.ilp = take((int64_t)p->t2.ngroups * pl);
  c.ilu = take((int64_t)p->t2.ngroups * pl);
  c.tab = take((int64_t)p->tab.size() * 4);
  c.flag = take(256);
  c.box = c.fb + 2 * ns * pl;
  if (box && res_box_bytes(p->rf) > c.tab - c.box) c.box = take(res_box_bytes(p->rf));
  if (grad) {
    const int nseg = (p->d.nt + K - 1) / K;
    const bool bs = boundary_saving(p);
    const bool full = !bs && K >= p->d.nt;
    const int64_t snap_elem = snapshot_value_bytes(p->d.snapshot_precision, p->elem);
    c.snap = take(full || bs ? 0 : (int64_t)nseg * 3 * ns * p->L.plane * snap_elem);
    c.snap_scale = take(full || bs ? 0 : (int64_t)nseg * 3 * ns * 4);
    // boundary saving: the frame's p, u, w after each step (slot it: the state before step it)
    c.bsv = take(bs ? (int64_t)p->d.nt * 3 * ns * p->nframe * p->elem : 0);
    c.hp = take((int64_t)K * ns * pl);
    c.hd = take((int64_t)K * ns * pl);
    c.la = take(3 * ns * pl);
    c.lb = take(3 * ns * pl);
    c.g1 = take((int64_t)p->t2.ngroups * pl);
    c.g2 = take((int64_t)p->t2.ngroups * pl);
    c.abox = c.lb + 2 * ns * pl;
    if (res_box_bytes(p->ra) > o - c.abox) c.abox = take(res_box_bytes(p->ra));
    const int64_t traces = (int64_t)ns * std::max(1, p->d.nr);
    const bool f64 = p->elem == 8;
    c.mst = take(traces * (f64 ? (int64_t)sizeof(l2::TraceStats<double>) : (int64_t)sizeof(l2::TraceStats<float>)));
    c.mpk = take(2 * ns * 8);
    c.mnorm = take(traces * 8);
    c.mfac = take(traces * (f64 ? (int64_t)sizeof(l2::TraceFactors<double>) : (int64_t)sizeof(l2::TraceFactors<float>)));
  }
  c.total = o;
  return c;
}

int choose_K(const adfwi_acoustic_plan* p) {
  const int nt = p->d.nt;
  const int64_t budget = p->d.memory_budget;
  if (p->bsave) return 1;  // one slot of divergence history, rebuilt step by step
  if (p->d.snapshot_every > 0) return std::min(p->d.snapshot_every, nt);
  if (budget <= 0) return std::min(nt, std::max(1, (int)std::ceil(std::sqrt(1.5 * nt))));
  // The whole history fits: the forward pass keeps it and no step is recomputed.
  if (carve(p, true, nt).total <= budget) return nt;
  // Otherwise: memory(K) = snapshots (falling with K) + segment history (rising with K) is
  // smallest near K* = sqrt(1.5 nt); take the longest segment beyond K* that still fits
  // (one recomputation pass either way, fewer snapshots).
  int kstar = std::min(nt - 1, std::max(1, (int)std::lround(std::sqrt(1.5 * nt))));
  while (kstar > 1 && carve(p, true, kstar - 1).total < carve(p, true, kstar).total) --kstar;
  while (kstar < nt - 1 && carve(p, true, kstar + 1).total < carve(p, true, kstar).total) ++kstar;
  if (carve(p, true, kstar).total > budget) return kstar;  // does not fit at all: the call reports it
  int lo = kstar, hi = nt - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) / 2;
    if (carve(p, true, mid).total <= budget) lo = mid; else hi = mid - 1;
  }
  return lo;
}

template <typename T>
ac::Geo<T> make_geo(const adfwi_acoustic_plan* p, const unsigned char* ws, const Carve& c, const Tiling& t) {
  ac::Geo<T> g;
  g.L = p->L;
  g.ns = p->d.ns;
  g.nt = p->d.nt;
  g.nr = p->d.nr;
  g.fs = p->fs;
  g.fsurf = p->d.free_surface;
  g.zbeg = p->zbeg;
  g.tiles_x = t.tiles_x;
  g.nabc = p->d.nabc;
  g.nz = p->d.nz;
  g.nx = p->d.nx;
  g.dt = (T)p->d.dt;
  g.c1 = (T)(9.0 / 8.0);
  g.c2 = (T)(-1.0 / 24.0);
  const int32_t* tb = reinterpret_cast<const int32_t*>(ws + c.tab);
  g.src_z = tb + p->o_srcz;
  g.src_x = tb + p->o_srcx;
  g.tile_rcv_beg = tb + t.o_trb;
  g.trcv_cell = tb + t.o_trc;
  g.trcv_id = tb + t.o_tri;
  g.tile_cell_beg = tb + t.o_tcb;
  g.tcell_cell = tb + t.o_tcc;
  g.tcell_rbeg = tb + t.o_tcr;
  g.cell_rcv = tb + t.o_cr;
  g.grp_beg = tb + t.o_gb;
  g.grp_model = tb + t.o_gm;
  g.fz_obs = nullptr;
  g.fz_tr = nullptr;
  g.fz_gmul = nullptr;
  g.fz_norm_obs = 0;
  return g;
}

int grid_blocks(int64_t n) { return (int)std::min<int64_t>(std::max<int64_t>((n + 255) / 256, 1), 152 * 16); }

template <typename T>
int setup_common(const adfwi_acoustic_plan* p, unsigned char* ws, const Carve& c, const void* alpha1,
                 const void* alpha2, const void* damp, bool clear_fields, cudaStream_t st) {
  const int64_t pl = p->L.plane * p->elem;
  // Zero coefficient planes (ghosts) and, where they are read before they are written, field
  // buffers and illumination partials.
  ADFWI_CUDA_TRY(cudaMemsetAsync(ws + c.coef, 0, (clear_fields ? c.tab : c.fa) - c.coef, st));
  ADFWI_CUDA_TRY(cudaMemsetAsync(ws + c.flag, 0, 256, st));
  ADFWI_CUDA_TRY(cudaMemcpyAsync(ws + c.tab, p->tab_pin.ptr, p->tab.size() * 4, cudaMemcpyHostToDevice, st));
  const int64_t n = (int64_t)p->nzp * p->nxp;
  const void* src[3] = {alpha1, alpha2, damp};
  ac::Geo<T> g = make_geo<T>(p, ws, c, p->t2);
  for (int m = 0; m < p->nm; ++m) {  // model m's (nzp, nxp) planes into its coefficient block
    T* cf = reinterpret_cast<T*>(ws + c.coef + (int64_t)m * ac::kNumCoef * pl);
    for (int q = 0; q < 3; ++q) {
      ADFWI_LAUNCH(kAux, st, (ac::pack_plane<T><<<grid_blocks(n), 256, 0, st>>>(
                                  p->L, p->nzp, p->nxp, static_cast<const T*>(src[q]) + (int64_t)m * n,
                                  reinterpret_cast<T*>(reinterpret_cast<unsigned char*>(cf) + q * pl))));
    }
    ADFWI_LAUNCH(kAux, st, (ac::mask_coefficients<T><<<grid_blocks(n), 256, 0, st>>>(g, cf)));
  }
  ADFWI_CUDA_TRY(cudaGetLastError());
  return kOk;
}

// Stages of the TMA ring of each variant of the FP32 step kernels (deep: those compiled for VDEEP
// blocks per SM).
int vec_adj_stages(bool deep) { return (deep ? ac2::VDEEP : ac2::VAMINB) >= 3 ? 2 : 3; }
int vec_stages(bool deep) { return (deep ? ac2::VDEEP : ac2::VMINB) >= 3 ? 3 : 4; }
using StepKernel = void (*)(ac2::Maps, ac::Geo<float>, ac2::StepArgs<float>);
StepKernel fwd_kernel(bool deep) {
  return deep ? ac2::fwd_step_vec<float, ac2::VDEEP> : ac2::fwd_step_vec<float, ac2::VMINB>;
}
StepKernel adj_kernel(bool deep) {
  return deep ? ac2::adj_step_vec<float, ac2::VDEEP> : ac2::adj_step_vec<float, ac2::VAMINB>;
}

// Launch of a persistent step kernel with programmatic stream serialisation (the kernel
// calls griddepcontrol.wait before touching data of the previous launch).
cudaError_t launch_pdl(StepKernel kernel, int blocks, int smem, cudaStream_t st, const ac2::Maps& maps,
                       const ac::Geo<float>& g, const ac2::StepArgs<float>& a) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)blocks);
  cfg.blockDim = dim3(ac2::VTHREADS);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, maps, g, a);
}

ac2::StepArgs<float> step_args(const adfwi_acoustic_plan* p, int it, const float* cf, int* flag) {
  ac2::StepArgs<float> a;
  memset(&a, 0, sizeof(a));
  a.it = it;
  a.G = p->t2.G;
  a.ngroups = p->t2.ngroups;
  a.ntiles = p->t2.ntiles;
  a.cf = cf;
  a.cf_stride = (int64_t)ac::kNumCoef * p->L.plane;
  a.flag = flag;
  return a;
}

int launch_fwd(const adfwi_acoustic_plan* p, const ac::Geo<float>& g, int it, int accum_u, const float* cf,
               const float* wav, const float* p0, const float* u0, const float* w0, float* p1, float* u1, float* w1, float* d1, float* rp, float* ru,
               float* rw, float* ilp, float* ilu, int* flag, cudaStream_t st) {
  const int64_t ns = p->d.ns;
  ac2::Maps maps;
  int rc = make_plane_map(&maps.a, u0, sizeof(float), p->L, ns, ac2::BOXX, ac2::EZ);
  if (!rc) rc = make_plane_map(&maps.b, w0, sizeof(float), p->L, ns, ac2::BOXX, ac2::WZ);
  if (!rc) rc = make_plane_map(&maps.c, p0, sizeof(float), p->L, ns, ac2::BOXX, ac2::EZ);
  if (rc) return rc;
  ac2::StepArgs<float> a = step_args(p, it, cf, flag);
  a.accum_u = accum_u;
  a.stages = vec_stages(p->deep);
  a.wav = wav;
  a.o0 = p1;
  a.o1 = u1;
  a.o2 = w1;
  a.d1 = d1;
  a.rec_p = rp;
  a.rec_u = ru;
  a.rec_w = rw;
  a.acc0 = ilp;
  a.acc1 = ilu;
  const int smem = ac2::VecFwdLayout<float>::bytes(a.stages);
  ADFWI_LAUNCH(kAcFwdStep, st,
               ADFWI_CUDA_TRY(launch_pdl(fwd_kernel(p->deep), p->t2.fwd_blocks, smem, st, maps, g, a)));
  return kOk;
}

int launch_adj(const adfwi_acoustic_plan* p, const ac::Geo<float>& g, int it, const float* cf, const float* lp0, const float* lu0,
               const float* lw0, float* lp1, float* lu1, float* lw1, const float* ph, const float* dh, const float* gp, const float* gu, const float* gw,
               float* g1, float* g2, int* flag, cudaStream_t st) {
  const int64_t ns = p->d.ns;
  ac2::Maps maps;
  int rc = make_plane_map(&maps.a, lu0, sizeof(float), p->L, ns, ac2::BOXX, ac2::EZ);
  if (!rc) rc = make_plane_map(&maps.b, lw0, sizeof(float), p->L, ns, ac2::BOXX, ac2::WZ);
  if (!rc) rc = make_plane_map(&maps.c, lp0, sizeof(float), p->L, ns, ac2::BOXX, ac2::EZ);
  if (!rc) rc = make_plane_map(&maps.d, ph, sizeof(float), p->L, ns, ac2::BOXX, ac2::EZ);
  if (!rc) rc = make_plane_map(&maps.e, dh, sizeof(float), p->L, ns, ac2::BOXX, ac2::EZ);
  if (rc) return rc;
  ac2::StepArgs<float> a = step_args(p, it, cf, flag);
  a.stages = vec_adj_stages(p->deep);
  a.o0 = lp1;
  a.o1 = lu1;
  a.o2 = lw1;
  a.rec_p = gp;
  a.rec_u = gu;
  a.rec_w = gw;
  a.acc0 = g1;
  a.acc1 = g2;
  const int smem = ac2::VecAdjLayout<float>::bytes(a.stages);
  ADFWI_LAUNCH(kAcAdjStep, st,
               ADFWI_CUDA_TRY(launch_pdl(adj_kernel(p->deep), p->t2.blocks, smem, st, maps, g, a)));
  return kOk;
}

// The double-precision steps (acoustic_f64.cuh): the same arguments.
ac3::Cells f64_cells(const adfwi_acoustic_plan* p, const ac::Geo<double>& g) {
  const int32_t* tb = g.src_z - p->o_srcz;
  return {tb + p->o_rz, tb + p->o_rx, tb + p->o_cz, tb + p->o_cx, tb + p->o_ftb, tb + p->o_ftc, p->t2.ncells};
}
unsigned f64_blocks(int64_t n) { return (unsigned)((n + ac3::kThreads - 1) / ac3::kThreads); }

int launch_fwd(const adfwi_acoustic_plan* p, const ac::Geo<double>& g, int it, int accum_u, const double* cf,
               const double* wav, const double* p0, const double* u0, const double* w0, double* p1, double* u1,
               double* w1, double* d1, double* rp, double* ru, double* rw, double* ilp, double* ilu, int*,
               cudaStream_t st) {
  const ac3::Cells cells = f64_cells(p, g);
  const int64_t cfs = (int64_t)ac::kNumCoef * p->L.plane;
  const unsigned nt = ac3::tiles(p->L, p->zbeg), gy = p->t2.ngroups;
  const unsigned rb = rp != nullptr && p->d.nr > 0 ? f64_blocks(p->d.nr) : 0;
  const dim3 b(ac3::kThreads);
  // (the step reads coefficients ahead of its wait: the first one of a solve follows the kernel that writes them)
  ADFWI_LAUNCH(kAcFwdStep, st,
               ADFWI_CUDA_TRY(launch_kernel(it > 0, ac3::fwd_step, dim3(nt + (it > 0 ? rb : 0), gy), b, 0, st, g, cells,
                                            (int)nt, it, cf, cfs, p0, u0, w0, p1, u1, w1, d1, wav, ilp,
                                            accum_u ? ilu : nullptr, rp, ru, rw)));
  if (rb && it + 1 == p->d.nt)
    ADFWI_LAUNCH(kAux, st, ADFWI_CUDA_TRY(launch_pdl_kernel(ac3::record_last, dim3(rb, gy), b, 0, st, g, cells, it,
                                                            (const double*)p1, (const double*)u1, (const double*)w1, rp,
                                                            ru, rw)));
  return kOk;
}

int launch_adj(const adfwi_acoustic_plan* p, const ac::Geo<double>& g, int it, const double* cf, const double* lp0,
               const double* lu0, const double* lw0, double* lp1, double* lu1, double* lw1, const double* ph,
               const double* dh, const double* gp, const double* gu, const double* gw, double* g1, double* g2, int*,
               cudaStream_t st) {
  const ac3::Cells cells = f64_cells(p, g);
  const int64_t cfs = (int64_t)ac::kNumCoef * p->L.plane;
  const unsigned nt = ac3::tiles(p->L, p->zbeg), gy = p->t2.ngroups;
  const dim3 b(ac3::kThreads);
  ADFWI_LAUNCH(kAcAdjStep, st,
               ADFWI_CUDA_TRY(launch_pdl_kernel(ac3::adj_step, dim3(nt, gy), b, 0, st, g, cells, it, cf, cfs, lp0, lu0, lw0,
                                                lp1, lu1, lw1, ph, dh, g1, g2, gp)));
  if ((gu || gw) && it >= 1 && cells.ncells > 0) {
    for (int mirrored = 0; mirrored <= (p->rcv_above ? 1 : 0); ++mirrored)
      ADFWI_LAUNCH(kAux, st, (ac3::adj_inject_uw<<<dim3(f64_blocks(cells.ncells), p->d.ns), b, 0, st>>>(
                                 g, cells, it - 1, mirrored != 0, gu, gw, lu1, lw1)));
    ADFWI_CUDA_TRY(cudaGetLastError());
  }
  return kOk;
}

// The opt-in above 48 KB of dynamic shared memory is a property of the kernel in one device's
// context, so it is set once per device ordinal, under a mutex: the
// serving workers call solves from several threads, and a process may drive more than one GPU.
std::mutex g_smem_mu;
std::vector<unsigned char> g_smem_done;  // per device

int set_smem_limits() {
  int dev = 0;
  ADFWI_CUDA_TRY(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(g_smem_mu);
  if ((int)g_smem_done.size() <= dev) g_smem_done.resize(dev + 1, 0);
  if (!g_smem_done[dev]) {
    for (int deep = 0; deep < 2; ++deep) {
      ADFWI_CUDA_TRY(cudaFuncSetAttribute(fwd_kernel(deep), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          ac2::VecFwdLayout<float>::bytes(vec_stages(deep))));
      ADFWI_CUDA_TRY(cudaFuncSetAttribute(adj_kernel(deep), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          ac2::VecAdjLayout<float>::bytes(vec_adj_stages(deep))));
    }
    g_smem_done[dev] = 1;
  }
  return kOk;
}

// ---------------------------------------------------------------- resident time loop (host)
using res::ResKernel;
ResKernel res_kernel(const Resident& r, bool adj, bool sums) {
  return adj ? res::adjoint_kernel(r.RB, r.MT, r.glb) : res::forward_kernel(r.RB, r.MT, sums, r.glb);
}

// Shared memory above 48 KB and clusters of more than 8 blocks are properties of the kernel in one
// device's context: opted into once per (device, kernel), to the most that any configuration
// takes, since solves run from several threads.
std::mutex g_res_mu;
std::vector<std::pair<int, ResKernel>> g_res_done;
cudaError_t res_prepare(ResKernel k) {
  int dev = 0, most = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lk(g_res_mu);
  for (const auto& d : g_res_done)
    if (d.first == dev && d.second == k) return cudaSuccess;
  e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e == cudaSuccess) g_res_done.push_back({dev, k});
  return e;
}

// A cluster per shot, or a cooperative launch (strips that wait for one another through global
// memory are resident together).
void res_config(cudaLaunchConfig_t* cfg, cudaLaunchAttribute* attr, const Resident& r, cudaStream_t st) {
  *cfg = cudaLaunchConfig_t{};
  cfg->gridDim = dim3((unsigned)(r.G * r.S));
  cfg->blockDim = dim3((unsigned)r.T);
  cfg->dynamicSmemBytes = (size_t)r.words * 4;
  cfg->stream = st;
  if (r.glb) {
    attr->id = cudaLaunchAttributeCooperative;
    attr->val.cooperative = 1;
  } else {
    attr->id = cudaLaunchAttributeClusterDimension;
    attr->val.clusterDim.x = (unsigned)r.G;
    attr->val.clusterDim.y = attr->val.clusterDim.z = 1;
  }
  cfg->attrs = attr;
  cfg->numAttrs = 1;
}

int64_t res_box_bytes(const Resident& r) {
  return r.glb ? (int64_t)2 * r.G * r.S * res::kBoxRows * r.CG * 32 : 0;
}

res::ResArgs res_args(const adfwi_acoustic_plan* p, const Resident& r, unsigned char* ws, const Carve& c) {
  res::ResArgs a;
  memset(&a, 0, sizeof(a));
  a.G = r.G;
  a.S = r.S;
  a.z0 = p->d.free_surface ? p->fs : 0;
  a.NR = p->nzp - a.z0;
  a.TR = r.TR;
  a.CG = r.CG;
  a.oS = r.oS;
  a.oA1 = r.oA1;
  a.oA2 = r.oA2;
  a.oPH = r.oPH;
  a.oDH = r.oDH;
  a.oBox = r.oBox;
  a.oInj = r.oInj;
  a.injw = r.injw;
  a.injg = r.injg;
  a.oRow = r.oRow;
  a.oT = r.oT;
  a.cf = reinterpret_cast<const float*>(ws + c.coef);
  a.cf_stride = (int64_t)ac::kNumCoef * p->L.plane;
  const int32_t* tb = reinterpret_cast<const int32_t*>(ws + c.tab);
  a.shot_model = tb + p->o_sm;
  a.row_slot = tb + r.o_sl;
  a.strip_beg = tb + r.o_sb;
  a.tpos = tb + r.o_tp;
  a.trid = tb + r.o_ti;
  a.srbeg = tb + r.o_rb;
  a.srcv = tb + r.o_rv;
  a.box = reinterpret_cast<unsigned long long*>(ws + (&r == &p->ra ? c.abox : c.box));
  a.flag = reinterpret_cast<int*>(ws + c.flag);
  a.nz = 0x8000000080000000ull;
  return a;
}

// Steps t0 .. t1-1 (the adjoint downwards) in launches of at most about a tenth of a second (6 us
// per step and wave of shots): blocks that wait for their neighbours are then never held up for
// long by another stream's launch. Between launches the state and the sums are in s1, acc0 and
// acc1; a launch's split changes no result.
int res_launch(const adfwi_acoustic_plan* p, const Resident& r, bool adj, bool sums, const ac::Geo<float>& g,
               res::ResArgs a, int t0, int t1, cudaStream_t st) {
  ResKernel k = res_kernel(r, adj, sums);
  ADFWI_CUDA_TRY(res_prepare(k));
  const int waves = r.glb ? (p->d.ns + r.S - 1) / r.S : (p->d.ns * r.G + 151) / 152;
  const int most = std::max(64, 16000 / waves);
  for (int done = 0; done < t1 - t0; done += most) {
    const int n = std::min(most, t1 - t0 - done);
    a.t0 = adj ? t1 - done - n : t0 + done;
    a.t1 = a.t0 + n;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[1];
    res_config(&cfg, attr, r, st);
    if (r.glb) ADFWI_CUDA_TRY(cudaMemsetAsync(a.box, 0, res_box_bytes(r), st));
    ADFWI_LAUNCH(adj ? kAcAdjStep : kAcFwdStep, st, ADFWI_CUDA_TRY(cudaLaunchKernelEx(&cfg, k, g, a)));
    a.s0 = a.s1;
    a.first = 0;
  }
  return kOk;
}

// The forward solve on the resident time loop: one launch, or one per snapshot interval. The
// state lives in fa between launches and the per-shot illumination sums in fb (3 ns planes each;
// the per-step kernels' ping-pong buffers).
int forward_resident(const adfwi_acoustic_plan* p, unsigned char* ws, const Carve& c, const float* wav, float* rec_p,
                     float* rec_u, float* rec_w, bool grad, int K, cudaStream_t st) {
  const int nt = p->d.nt, ns = p->d.ns;
  const int64_t pl = p->L.plane;
  const bool full = grad && K >= nt;
  const ac::Geo<float> g = make_geo<float>(p, ws, c, p->t2);
  res::ResArgs a = res_args(p, p->rf, ws, c);
  float* fa = reinterpret_cast<float*>(ws + c.fa);
  float* fb = reinterpret_cast<float*>(ws + c.fb);
  a.wav = wav;
  a.rec_p = rec_p;
  a.rec_u = rec_u;
  a.rec_w = rec_w;
  a.accum_u = p->last_chunk_start;
  a.acc0 = fb;
  a.acc1 = fb + ns * pl;
  a.s1 = fa;
  if (full) {
    a.hp = reinterpret_cast<float*>(ws + c.hp);
    a.hd = reinterpret_cast<float*>(ws + c.hd);
  }
  const int step = grad && !full ? K : nt;
  for (int t0 = 0; t0 < nt; t0 += step) {
    if (grad && !full) {
      const int rc = snapshot_store<float>(p->d.snapshot_precision, fa, 3 * (int64_t)ns, pl, ws + c.snap,
                                           ws + c.snap_scale, (int64_t)(t0 / K) * 3 * ns, st);
      if (rc) return rc;
    }
    a.s0 = t0 == 0 ? nullptr : fa;
    a.first = t0 == 0;
    const int rc = res_launch(p, p->rf, false, true, g, a, t0, std::min(nt, t0 + step), st);
    if (rc) return rc;
  }
  return kOk;
}

// Steps t0 .. t1-1 again from the state in fa, keeping their histories (slot 0 is step t0).
int recompute_resident(const adfwi_acoustic_plan* p, unsigned char* ws, const Carve& c, const float* wav, int t0, int t1,
                       cudaStream_t st) {
  const ac::Geo<float> g = make_geo<float>(p, ws, c, p->t2);
  res::ResArgs a = res_args(p, p->rf, ws, c);
  a.wav = wav;
  a.s0 = a.s1 = reinterpret_cast<float*>(ws + c.fa);
  a.hp = reinterpret_cast<float*>(ws + c.hp);
  a.hd = reinterpret_cast<float*>(ws + c.hd);
  a.h0 = t0;
  return res_launch(p, p->rf, false, false, g, a, t0, t1, st);
}

// What the per-step adjoint expects of the divergence history of a resident forward.
int mask_divergence(const ac::Geo<float>& g, int64_t planes, float* hd, cudaStream_t st) {
  ADFWI_LAUNCH(kAux, st, (res::zero_outside_p<<<152 * 8, 256, 0, st>>>(g, planes, hd)));
  ADFWI_CUDA_TRY(cudaGetLastError());
  return kOk;
}

// Reverse steps t1-1 .. t0 on the histories of a segment that begins at step h0. grec_p: dL/d
// p-records of rnt steps per shot from step r0. The adjoint state lives in la between launches
// and the per-shot gradient sums in lb (3 ns planes each).
int adjoint_resident(const adfwi_acoustic_plan* p, unsigned char* ws, const Carve& c, const float* grec_p, int r0, int rnt,
                     int t0, int t1, int h0, bool first, cudaStream_t st) {
  const ac::Geo<float> g = make_geo<float>(p, ws, c, p->t2);
  res::ResArgs a = res_args(p, p->ra, ws, c);
  float* la = reinterpret_cast<float*>(ws + c.la);
  float* lb = reinterpret_cast<float*>(ws + c.lb);
  a.s0 = first ? nullptr : la;
  a.s1 = la;
  a.first = first;
  a.hp = reinterpret_cast<float*>(ws + c.hp);
  a.hd = reinterpret_cast<float*>(ws + c.hd);
  a.rec_p = const_cast<float*>(grec_p);
  a.r0 = r0;
  a.rnt = rnt;
  a.acc0 = lb;
  a.acc1 = lb + p->d.ns * p->L.plane;
  a.h0 = h0;
  return res_launch(p, p->ra, true, true, g, a, t0, t1, st);
}

template <typename T>
int forward_impl(const adfwi_acoustic_plan* p, const void* alpha1, const void* alpha2, const void* damp,
                 const void* wavelet, void* rec_p, void* rec_u, void* rec_w, void* fw_p, void* fw_u,
                 void* fw_w, bool grad, unsigned char* ws, int64_t ws_bytes, cudaStream_t st, bool box = true) {
  int rc = sizeof(T) == 4 ? set_smem_limits() : kOk;
  if (rc) return rc;
  const int K = grad ? p->K : 1;
  Carve c = carve(p, grad, K, box);
  if (ws_bytes < c.total) {
    set_error("workspace too small: %lld bytes given, %lld needed", (long long)ws_bytes, (long long)c.total);
    return kWorkspaceTooSmall;
  }
  const bool bs = grad && boundary_saving(p);
  const bool full = grad && !bs && K >= p->d.nt;
  bool resident = false;
  if constexpr (sizeof(T) == 4) resident = p->rf.G > 0 && (box || !p->rf.glb);
  // (the resident loop starts from zeroes of its own; the first snapshot is the zero state)
  rc = setup_common<T>(p, ws, c, alpha1, alpha2, damp, !resident || (grad && !full), st);
  if (rc) return rc;
  ac::Geo<T> g = make_geo<T>(p, ws, c, p->t2);
  const int64_t pl = p->L.plane;
  const int64_t ns = p->d.ns;
  const T* cf = reinterpret_cast<const T*>(ws + c.coef);
  T* fa = reinterpret_cast<T*>(ws + c.fa);
  T* fb = reinterpret_cast<T*>(ws + c.fb);
  T* ilp = reinterpret_cast<T*>(ws + c.ilp);
  T* ilu = reinterpret_cast<T*>(ws + c.ilu);
  int* flag = reinterpret_cast<int*>(ws + c.flag);
  const T* wav = static_cast<const T*>(wavelet);
  T* hp = grad ? reinterpret_cast<T*>(ws + c.hp) : nullptr;
  T* hd = grad ? reinterpret_cast<T*>(ws + c.hd) : nullptr;
  if (full && !resident) {
    // the pressure history is read with its halo (as the next step's input and by the adjoint)
    rc = zero_frames<T>(hp, (int64_t)K * ns, p->L, st);
    if (rc) return rc;
  }
  T* cur = fa;
  T* nxt = fb;
  const int64_t bslot = (int64_t)3 * ns * p->nframe;  // elements of one boundary-saving slot
  if constexpr (sizeof(T) == 4) {
    if (resident) {
      rc = forward_resident(p, ws, c, wav, static_cast<T*>(rec_p), static_cast<T*>(rec_u), static_cast<T*>(rec_w),
                            grad, K, st);
      if (rc) return rc;
      ilp = fb;  // one partial plane per shot
      ilu = fb + ns * pl;
    }
  }
  for (int it = resident ? p->d.nt : 0; it < p->d.nt; ++it) {
    if (grad && !full && !bs && it % K == 0) {
      rc = snapshot_store<T>(p->d.snapshot_precision, cur, 3 * ns, pl, ws + c.snap, ws + c.snap_scale,
                             (int64_t)(it / K) * 3 * ns, st);
      if (rc) return rc;
    }
    const T* p0 = cur;
    T* p1 = nxt;
    T* d1 = nullptr;
    if (full) {
      // the whole pressure history doubles as the pressure ping-pong buffer
      p0 = it == 0 ? cur : hp + (int64_t)(it - 1) * ns * pl;
      p1 = hp + (int64_t)it * ns * pl;
      d1 = hd + (int64_t)it * ns * pl;
    }
    rc = launch_fwd(p, g, it, it >= p->last_chunk_start ? 1 : 0, cf, wav, p0, cur + ns * pl, cur + 2 * ns * pl,
                       p1, nxt + ns * pl, nxt + 2 * ns * pl, d1, static_cast<T*>(rec_p), static_cast<T*>(rec_u),
                       static_cast<T*>(rec_w), ilp, ilu, flag, st);
    if (rc) return rc;
    if (bs && it + 1 < p->d.nt) {
      const dim3 gs((unsigned)((p->nframe + 255) / 256), (unsigned)ns);
      const int* foff = reinterpret_cast<const int*>(ws + c.tab) + p->o_foff;
      ADFWI_LAUNCH(kAux, st, (ac::bs_save<T><<<gs, 256, 0, st>>>(p->L, (int)ns, p->nframe, foff, nxt,
                                                                  reinterpret_cast<T*>(ws + c.bsv) +
                                                                      (it + 1) * bslot)));
    }
    std::swap(cur, nxt);
  }
  ADFWI_CUDA_TRY(cudaGetLastError());
  if (fw_p || fw_u || fw_w) {
    const int64_t n = (int64_t)p->d.nz * p->d.nx;
    auto at = [&](void* f, int m) { return f ? static_cast<T*>(f) + (int64_t)m * n : nullptr; };
    for (int m = 0; m < p->nm; ++m) {  // model m: its groups' partial planes and its shots' last w
      const int s0 = p->model_shot_beg[m], g0 = resident ? s0 : p->model_grp_beg[m];
      const int ng = (resident ? p->model_shot_beg[m + 1] : p->model_grp_beg[m + 1]) - g0;
      ADFWI_LAUNCH(kAux, st, (ac::illum_finalize<T><<<grid_blocks(n), 256, 0, st>>>(
                                  p->L, ng, p->model_shot_beg[m + 1] - s0, p->d.nabc,
                                  p->d.nz, p->d.nx, ilp + (int64_t)g0 * pl, ilu + (int64_t)g0 * pl,
                                  cur + 2 * ns * pl + (int64_t)s0 * pl, at(fw_p, m), at(fw_u, m), at(fw_w, m))));
    }
    ADFWI_CUDA_TRY(cudaGetLastError());
  }
  return kOk;
}

// The normalised L2 misfit fused into the adjoint: the dL/d p-records are formed from the
// records (passed as the p-record gradient) and the observed data with the factors that
// l2_loss_impl left in the workspace, scaled by *gmul.
struct FusedL2 {
  const void* obs;
  const double* gmul;
  int norm_obs;
};

template <typename T>
int backward_impl(const adfwi_acoustic_plan* p, const void* wavelet, const void* grp, const void* gru,
                  const void* grw, void* ga1, void* ga2, unsigned char* ws, int64_t ws_bytes, cudaStream_t st,
                  const FusedL2* fz = nullptr) {
  int rc = sizeof(T) == 4 ? set_smem_limits() : kOk;
  if (rc) return rc;
  const int K = p->K;
  Carve c = carve(p, true, K);
  if (ws_bytes < c.total) {
    set_error("workspace too small: %lld bytes given, %lld needed", (long long)ws_bytes, (long long)c.total);
    return kWorkspaceTooSmall;
  }
  ac::Geo<T> g2 = make_geo<T>(p, ws, c, p->t2);
  if (fz != nullptr) {
    g2.fz_obs = static_cast<const T*>(fz->obs);
    g2.fz_tr = reinterpret_cast<const l2::TraceFactors<T>*>(ws + c.mfac);
    g2.fz_gmul = fz->gmul;
    g2.fz_norm_obs = fz->norm_obs;
  }
  const int64_t pl = p->L.plane;
  const int64_t ns = p->d.ns;
  const int nt = p->d.nt;
  const bool full = K >= nt;
  const T* cf = reinterpret_cast<const T*>(ws + c.coef);
  T* fa = reinterpret_cast<T*>(ws + c.fa);
  T* fb = reinterpret_cast<T*>(ws + c.fb);
  T* hp = reinterpret_cast<T*>(ws + c.hp);
  T* hd = reinterpret_cast<T*>(ws + c.hd);
  T* la = reinterpret_cast<T*>(ws + c.la);
  T* lb = reinterpret_cast<T*>(ws + c.lb);
  T* g1p = reinterpret_cast<T*>(ws + c.g1);
  T* g2p = reinterpret_cast<T*>(ws + c.g2);
  int* flag = reinterpret_cast<int*>(ws + c.flag);
  const T* wav = static_cast<const T*>(wavelet);
  const T* gp = static_cast<const T*>(grp);
  const T* gu = static_cast<const T*>(gru);
  const T* gw = static_cast<const T*>(grw);

  ADFWI_CUDA_TRY(cudaMemsetAsync(la, 0, 3 * ns * pl * sizeof(T), st));
  if constexpr (sizeof(T) == 4) {
    // the resident adjoint takes dL/d p-records; dL/d u- and w-records go through the per-step
    // kernels. A fused misfit's records are formed a stretch of steps at a time in fb, which the
    // adjoint does not use.
    const int64_t stretch = fz == nullptr ? nt : 3 * pl / p->d.nr;
    if (p->ra.G > 0 && gu == nullptr && gw == nullptr && stretch > 0) {
      const int nseg = full ? 1 : (nt + K - 1) / K;
      for (int seg = nseg - 1; seg >= 0; --seg) {
        const int t0 = seg * K, t1 = std::min(nt, t0 + K);
        if (!full) {
          rc = snapshot_load<T>(p->d.snapshot_precision, fa, 3 * ns, pl, ws + c.snap, ws + c.snap_scale,
                                (int64_t)seg * 3 * ns, st);
          if (!rc) rc = recompute_resident(p, ws, c, wav, t0, t1, st);
          if (rc) return rc;
        }
        for (int e1 = t1; e1 > t0;) {
          const int e0 = (int)std::max<int64_t>(t0, e1 - stretch);
          if (fz != nullptr)
            ADFWI_LAUNCH(kAux, st, (l2::sources<T><<<l2::grid((int)ns, p->d.nr), l2::block(), 0, st>>>(
                                       (int)ns, nt, p->d.nr, e0, e1, fz->norm_obs, gp, static_cast<const T*>(fz->obs),
                                       g2.fz_tr, fz->gmul, fb)));
          rc = adjoint_resident(p, ws, c, fz != nullptr ? fb : gp, fz != nullptr ? e0 : 0, fz != nullptr ? e1 - e0 : nt,
                                e0, e1, t0, e1 == nt, st);
          if (rc) return rc;
          e1 = e0;
        }
      }
      const int64_t n = (int64_t)p->nzp * p->nxp;
      for (int m = 0; m < p->nm; ++m) {  // model m's gradients: the sums over its shots
        const int s0 = p->model_shot_beg[m], nm = p->model_shot_beg[m + 1] - s0;
        const T* cm = cf + (int64_t)m * ac::kNumCoef * pl;
        ADFWI_LAUNCH(kAux, st, (res::reduce_scaled<<<grid_blocks(n), 256, 0, st>>>(
                                    p->L, p->d.free_surface ? p->fs : 0, nm, cm + ac::kA1 * pl, lb + (int64_t)s0 * pl,
                                    static_cast<T*>(ga1) + m * n)));
        ADFWI_LAUNCH(kAux, st, (res::reduce_scaled<<<grid_blocks(n), 256, 0, st>>>(
                                    p->L, p->d.free_surface ? p->fs : 0, nm, cm + ac::kA2 * pl, lb + (ns + s0) * pl,
                                    static_cast<T*>(ga2) + m * n)));
      }
      ADFWI_CUDA_TRY(cudaGetLastError());
      return kOk;
    }
  }
  ADFWI_CUDA_TRY(cudaMemsetAsync(lb, 0, 3 * ns * pl * sizeof(T), st));
  ADFWI_CUDA_TRY(cudaMemsetAsync(g1p, 0, (size_t)p->t2.ngroups * pl * sizeof(T), st));
  ADFWI_CUDA_TRY(cudaMemsetAsync(g2p, 0, (size_t)p->t2.ngroups * pl * sizeof(T), st));
  if (!full || p->rf.G > 0) {
    // the recomputed pressure history is read with its halo by the next step and the adjoint (the
    // resident forward leaves the frames of a whole history as they were)
    rc = zero_frames<T>(hp, (int64_t)K * ns, p->L, st);
    if constexpr (sizeof(T) == 4) {
      if (!rc && full && p->rf.G > 0) rc = mask_divergence(g2, (int64_t)nt * ns, hd, st);
    }
    if (rc) return rc;
  }
  if (gp || gu || gw) {
    dim3 sg(std::max(1, std::min(64, (p->t2.ncells + 127) / 128)), p->d.ns);
    ADFWI_LAUNCH(kAux, st, (ac::adj_seed<T><<<sg, 128, 0, st>>>(g2, p->t2.ntiles, ac2::TZ, ac2::TX, gp, gu, gw, la,
                                                                   la + ns * pl, la + 2 * ns * pl)));
    if (gw && p->rcv_above)
      ADFWI_LAUNCH(kAux, st, (ac::fold_mirrored_w<T><<<dim3((p->nxp + 127) / 128, p->d.ns), 128, 0, st>>>(
                                 g2, la + 2 * ns * pl)));
  }
  T* lcur = la;
  T* lnxt = lb;
  // reverse step it on p after it and its divergence
  auto reverse = [&](int it, const T* ph, const T* dh) {
    const int e = launch_adj(p, g2, it, cf, lcur, lcur + ns * pl, lcur + 2 * ns * pl, lnxt, lnxt + ns * pl,
                             lnxt + 2 * ns * pl, ph, dh, gp, gu, gw, g1p, g2p, flag, st);
    std::swap(lcur, lnxt);
    return e;
  };
  if (boundary_saving(p)) {
    // The forward left its last state in fa (nt even) or fb; rebuild the states backwards, the
    // pressure ping-ponging between the two buffers' p planes, u and w in place.
    T* sbuf = nt % 2 == 0 ? fa : fb;
    T* pcur = sbuf;
    T* poth = sbuf == fa ? fb : fa;
    T* u = sbuf + ns * pl;
    T* w = sbuf + 2 * ns * pl;
    const int* fidx = reinterpret_cast<const int*>(ws + c.tab) + p->o_fidx;
    const T* bsv = reinterpret_cast<const T*>(ws + c.bsv);
    const int64_t bslot = (int64_t)3 * ns * p->nframe;
    const dim3 gb(32, 8), gr((unsigned)((p->nxp + 31) / 32), (unsigned)((p->nzp + 7) / 8), (unsigned)ns);
    for (int it = nt - 1; it >= 0; --it) {
      const T* slot = it > 0 ? bsv + it * bslot : nullptr;
      ADFWI_LAUNCH(kAux, st, (ac::bs_reverse_uw<T><<<gr, gb, 0, st>>>(g2, p->bbox, fidx, cf, pcur, u, w, slot,
                                                                      p->nframe)));
      ADFWI_LAUNCH(kAux, st, (ac::bs_reverse_p<T><<<gr, gb, 0, st>>>(g2, p->bbox, it, fidx, cf, pcur, u, w, poth, hd,
                                                                     slot, p->nframe, wav)));
      rc = reverse(it, pcur, hd);
      if (rc) return rc;
      std::swap(pcur, poth);
    }
    ADFWI_CUDA_TRY(cudaGetLastError());
  }
  const int nseg = boundary_saving(p) ? 0 : (full ? 1 : (nt + K - 1) / K);
  for (int seg = nseg - 1; seg >= 0; --seg) {
    const int t0 = full ? 0 : seg * K;
    const int t1 = full ? nt : std::min(nt, t0 + K);
    if (!full) {
      // Recompute the segment from its snapshot, keeping p and the divergence of every step.
      rc = snapshot_load<T>(p->d.snapshot_precision, fa, 3 * ns, pl, ws + c.snap, ws + c.snap_scale,
                            (int64_t)seg * 3 * ns, st);
      if (rc) return rc;
      T* cur = fa;
      T* nxt = fb;
      bool resident = false;
      if constexpr (sizeof(T) == 4) {
        resident = p->rf.G > 0;
        if (resident) rc = recompute_resident(p, ws, c, wav, t0, t1, st);
        if (!rc && resident) rc = mask_divergence(g2, (int64_t)(t1 - t0) * ns, hd, st);
        if (rc) return rc;
      }
      for (int it = resident ? t1 : t0; it < t1; ++it) {
        const T* p0 = it == t0 ? fa : hp + (int64_t)(it - 1 - t0) * ns * pl;
        rc = launch_fwd(p, g2, it, 0, cf, wav, p0, cur + ns * pl, cur + 2 * ns * pl,
                           hp + (int64_t)(it - t0) * ns * pl, nxt + ns * pl, nxt + 2 * ns * pl,
                           hd + (int64_t)(it - t0) * ns * pl, nullptr, nullptr, nullptr, nullptr, nullptr, flag, st);
        if (rc) return rc;
        std::swap(cur, nxt);
      }
    }
    for (int it = t1 - 1; it >= t0; --it) {
      rc = reverse(it, hp + (int64_t)(it - t0) * ns * pl, hd + (int64_t)(it - t0) * ns * pl);
      if (rc) return rc;
    }
    ADFWI_CUDA_TRY(cudaGetLastError());
  }
  const int64_t n = (int64_t)p->nzp * p->nxp;
  for (int m = 0; m < p->nm; ++m) {  // model m's gradients: the sum over its groups' partial planes
    const int g0 = p->model_grp_beg[m], ng = p->model_grp_beg[m + 1] - g0;
    ADFWI_LAUNCH(kAux, st, (ac::reduce_planes<T><<<grid_blocks(n), 256, 0, st>>>(
                                p->L, ng, 0, 0, p->nzp, p->nxp, g1p + (int64_t)g0 * pl, static_cast<T*>(ga1) + m * n)));
    ADFWI_LAUNCH(kAux, st, (ac::reduce_planes<T><<<grid_blocks(n), 256, 0, st>>>(
                                p->L, ng, 0, 0, p->nzp, p->nxp, g2p + (int64_t)g0 * pl, static_cast<T*>(ga2) + m * n)));
  }
  ADFWI_CUDA_TRY(cudaGetLastError());
  return kOk;
}

// Normalised L2 misfit of the records `syn` against `obs` (the misfit of adfwi_l2_misfit) into
// the gradient workspace's factor arrays, and each model's loss: the sum of its traces' norms.
template <typename T>
int l2_loss_impl(const adfwi_acoustic_plan* p, const void* syn, const void* obs, double silent_rel, int flags,
                 double* loss, unsigned char* ws, int64_t ws_bytes, cudaStream_t st) {
  const Carve c = carve(p, true, p->K);
  if (ws_bytes < c.total) {
    set_error("workspace too small: %lld bytes given, %lld needed", (long long)ws_bytes, (long long)c.total);
    return kWorkspaceTooSmall;
  }
  const int ns = p->d.ns, nt = p->d.nt, nr = p->d.nr;
  auto* stats = reinterpret_cast<l2::TraceStats<T>*>(ws + c.mst);
  auto* gsyn = reinterpret_cast<l2::PeakWord<T>*>(ws + c.mpk);
  auto* gobs = gsyn + ns;
  auto* norms = reinterpret_cast<double*>(ws + c.mnorm);
  auto* fac = reinterpret_cast<l2::TraceFactors<T>*>(ws + c.mfac);
  ADFWI_CUDA_TRY(cudaMemsetAsync(ws + c.mpk, 0, 2 * (size_t)ns * 8, st));  // peaks start at +0
  const dim3 grid = l2::grid(ns, nr);
  const T* sy = static_cast<const T*>(syn);
  const T* ob = static_cast<const T*>(obs);
  ADFWI_LAUNCH(kAux, st, (l2::peaks<T><<<grid, l2::block(), 0, st>>>(ns, nt, nr, sy, ob, stats, gsyn, gobs)));
  ADFWI_LAUNCH(kAux, st, (l2::factors<T><<<grid, l2::block(), 0, st>>>(ns, nt, nr, p->d.dt, silent_rel, flags & 1, sy,
                                                                         ob, stats, gsyn, gobs, fac, norms)));
  for (int m = 0; m < p->nm; ++m) {
    const int s0 = p->model_shot_beg[m], s1 = p->model_shot_beg[m + 1];
    ADFWI_LAUNCH(kAux, st, (l2::sum_norms<<<1, l2::kThreads, 0, st>>>((int64_t)(s1 - s0) * nr,
                                                                       norms + (int64_t)s0 * nr, loss + m)));
  }
  ADFWI_CUDA_TRY(cudaGetLastError());
  return kOk;
}

// The misfit's adjoint source of every record sample into adj (ns, nt, nr), times *gmul, from
// the factors l2_loss_impl left in the workspace.
template <typename T>
int l2_sources_impl(const adfwi_acoustic_plan* p, const void* syn, const void* obs, int flags, const double* gmul,
                    void* adj, unsigned char* ws, int64_t ws_bytes, cudaStream_t st) {
  const Carve c = carve(p, true, p->K);
  if (ws_bytes < c.total) {
    set_error("workspace too small: %lld bytes given, %lld needed", (long long)ws_bytes, (long long)c.total);
    return kWorkspaceTooSmall;
  }
  const int ns = p->d.ns, nt = p->d.nt, nr = p->d.nr;
  const auto* fac = reinterpret_cast<const l2::TraceFactors<T>*>(ws + c.mfac);
  ADFWI_LAUNCH(kAux, st, (l2::sources<T><<<l2::grid(ns, nr), l2::block(), 0, st>>>(
                             ns, nt, nr, 0, nt, flags & 1, static_cast<const T*>(syn), static_cast<const T*>(obs), fac, gmul,
                             static_cast<T*>(adj))));
  ADFWI_CUDA_TRY(cudaGetLastError());
  return kOk;
}

// Resident blocks of a persistent step kernel on the current device (`fallback` per SM x 152
// without a GPU).
template <typename K>
int resident_blocks(K kernel, int threads, int smem, int fallback) {
  int dev = 0, sms = 0, occ = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
    cudaGetLastError();
    return 152 * fallback;
  }
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, threads, smem) != cudaSuccess || occ < 1) {
    cudaGetLastError();
    return 152 * fallback;
  }
  return sms * occ;
}

int resident_adj_blocks(bool deep) {
  return resident_blocks(adj_kernel(deep), ac2::VTHREADS, ac2::VecAdjLayout<float>::bytes(vec_adj_stages(deep)),
                         deep ? ac2::VDEEP : ac2::VAMINB);
}
int resident_fwd_blocks(bool deep) {
  return resident_blocks(fwd_kernel(deep), ac2::VTHREADS, ac2::VecFwdLayout<float>::bytes(vec_stages(deep)),
                         deep ? ac2::VDEEP : ac2::VMINB);
}

// Padded grids at least this wide run the deep-ring variants (one more stage, 2 blocks per SM), where
// the per-step kernels are taken at all (boundary saving, dL/d u- and w-records, grids that do not fit
// on the chip). An empirical rule from per-launch times of both rings (FP32, full history; forward / adjoint
// in us, shallow -> deep): 600 x 1600 padded with 4 / 8 / 16 shots 44.1 -> 41.6 / 77.2 -> 69.1,
// 86.0 -> 73.5 / 130.8 -> 118.0, 161.8 -> 165.8 / 227.6 -> 217.1; every narrower grid measured
// (300 x 700 with 10 / 30 / 60 shots, 400 x 1000 with 8 / 16 / 30, 200 x 400 with 16 / 64,
// up to 144 MB of fields per time level) ran 4-42 % slower with the deep ring. The wide grid's
// kernels read 27 B per cell-update from DRAM against 13.5 B on the 300 x 700 grid (L2 hit
// rate 19 % against 30 %), so they wait longer per stage and profit from the extra stage.
constexpr int kDeepRingCols = 1400;

// Shots per unit for the persistent TMA kernels: balance the units over the resident blocks
// (the block with the most units sets the time) against the per-unit costs (the coefficient
// loads, and the load and flush of the partial accumulator planes), weighted as 1.5 items: the
// weight that reproduces the measured optimum of a sweep of 1, 2, 4 and 8 shots per unit on the
// 600 x 1600 grid with 8 and 32 shots.
int pick_unit_shots(const std::vector<int>& model_shot_beg, int ntiles, int blocks_fwd, int blocks_adj) {
  const int nm = (int)model_shot_beg.size() - 1;
  int maxns = 1;
  for (int m = 0; m < nm; ++m) maxns = std::max(maxns, model_shot_beg[m + 1] - model_shot_beg[m]);
  int best = 1;
  double best_cost = 1e30;
  for (int G = 1; G <= maxns; ++G) {
    int groups = 0;
    for (int m = 0; m < nm; ++m) groups += (model_shot_beg[m + 1] - model_shot_beg[m] + G - 1) / G;
    const long long units = (long long)ntiles * groups;
    const long long pf = (units + blocks_fwd - 1) / blocks_fwd;
    const long long pa = (units + blocks_adj - 1) / blocks_adj;
    const double cost = (double)(pf + 2 * pa) * (G + 1.5);  // the adjoint step takes about twice as long
    if (cost < best_cost - 1e-9) {
      best_cost = cost;
      best = G;
    }
  }
  return best;
}

// Tile the grid and build the receiver tables of that tiling (appended to p->tab).
void build_tiling(adfwi_acoustic_plan* p, Tiling* tl, int tz, int tx, const std::vector<int>& Gm, const int32_t* rcv_z,
                  const int32_t* rcv_x) {
  const adfwi_acoustic_desc& d = p->d;
  std::vector<int32_t>& t = p->tab;
  tl->tz = tz;
  tl->tx = tx;
  tl->tiles_x = (p->nxp + tx - 1) / tx;
  tl->tiles_z = (p->nzp - p->zbeg + tz - 1) / tz;
  tl->ntiles = tl->tiles_x * tl->tiles_z;
  tl->G = 1;
  tl->blocks = 0;
  // shot groups of at most Gm[m] shots of model m, never across two models
  std::vector<int32_t> gb(1, 0), gm;
  p->model_grp_beg.assign(1, 0);
  for (int m = 0; m < p->nm; ++m) {
    const int G = std::max(1, Gm[m]);
    tl->G = std::max(tl->G, G);
    for (int s = p->model_shot_beg[m]; s < p->model_shot_beg[m + 1]; s += G) {
      gb.push_back(std::min(s + G, p->model_shot_beg[m + 1]));
      gm.push_back(m);
    }
    p->model_grp_beg.push_back((int)gm.size());
  }
  tl->ngroups = (int)gm.size();
  tl->o_gb = t.size();
  t.insert(t.end(), gb.begin(), gb.end());
  tl->o_gm = t.size();
  t.insert(t.end(), gm.begin(), gm.end());
  struct R {
    int tile, cell, id;
  };
  std::vector<R> rs(d.nr);
  for (int r = 0; r < d.nr; ++r) {
    int z = rcv_z[r] + d.nabc - p->zbeg, x = rcv_x[r] + d.nabc;
    rs[r].tile = (z / tz) * tl->tiles_x + x / tx;
    rs[r].cell = ((z % tz) << 16) | (x % tx);
    rs[r].id = r;
  }
  std::stable_sort(rs.begin(), rs.end(), [](const R& a, const R& b) {
    return a.tile != b.tile ? a.tile < b.tile : a.cell < b.cell;
  });
  tl->o_trb = t.size();
  {
    std::vector<int32_t> beg(tl->ntiles + 1, 0);
    for (const R& r : rs) beg[r.tile + 1]++;
    for (int q = 0; q < tl->ntiles; ++q) beg[q + 1] += beg[q];
    t.insert(t.end(), beg.begin(), beg.end());
  }
  tl->o_trc = t.size();
  for (const R& r : rs) t.push_back(r.cell);
  tl->o_tri = t.size();
  for (const R& r : rs) t.push_back(r.id);
  std::vector<int32_t> tcb(tl->ntiles + 1, 0), tcc, tcr, cr;
  for (size_t q = 0; q < rs.size(); ++q) {
    bool fresh = q == 0 || rs[q].tile != rs[q - 1].tile || rs[q].cell != rs[q - 1].cell;
    if (fresh) {
      tcb[rs[q].tile + 1]++;
      tcc.push_back(rs[q].cell);
      tcr.push_back((int32_t)cr.size());
    }
    cr.push_back(rs[q].id);
  }
  tcr.push_back((int32_t)cr.size());
  for (int q = 0; q < tl->ntiles; ++q) tcb[q + 1] += tcb[q];
  tl->ncells = (int)tcc.size();
  tl->o_tcb = t.size();
  t.insert(t.end(), tcb.begin(), tcb.end());
  tl->o_tcc = t.size();
  t.insert(t.end(), tcc.begin(), tcc.end());
  tl->o_tcr = t.size();
  t.insert(t.end(), tcr.begin(), tcr.end());
  tl->o_cr = t.size();
  t.insert(t.end(), cr.begin(), cr.end());
}

// Shots per group of the double-precision steps: one while that gives at most 16 blocks of 128 threads
// per SM (more blocks than are resident), then as many as keep to that. A group has one partial plane
// per sum, so where memory is short (the allocation-free forward's scratch, a budget below the whole
// history) groups stay as large as one block per SM of 16 x 64 tiles would make them. Short is what the whole
// batch takes: there a model's shots may be grouped otherwise than in a plan of its own, and its FP64
// sums rounded in another order.
int f64_group_shots(const adfwi_acoustic_plan* p, const std::vector<int>& alone, int ntiles, int64_t scratch) {
  const int ns = alone[1], tight = pick_unit_shots(alone, ntiles, 152, 152);
  const int fine = std::max(1, (int)((int64_t)ns * ac3::tiles(p->L, p->zbeg) / (152 * 16)));
  auto bytes = [&](int G, int64_t fields) {
    const int64_t groups = (int64_t)p->nm * ((ns + G - 1) / G);
    return (ac::kNumCoef * (int64_t)p->nm + fields * p->d.ns + (fields > 6 ? 4 : 2) * groups) * p->L.plane * 8 + (1 << 20);
  };
  if (bytes(fine, 6) > scratch && bytes(tight, 6) <= scratch + (2 << 20)) return tight;
  if (p->d.memory_budget > 0 && bytes(fine, 12 + 2 * (int64_t)p->d.nt) > p->d.memory_budget / 50 * 49) return tight;
  return fine;
}

// Shared memory of a configuration, in words.
// (most, most_rows: receiver cells, and rows holding any, of the strip that has the most)
void res_layout(Resident* r, bool adj, int kept, bool tables, int most, int most_rows) {
  const int w4 = 4 * r->CG, R = r->R, sb = res::kGrp * (r->CG + 1);
  int o = res::kHeadWords;
  r->oS = o;
  o += (R + 4) * sb + res::kGrp;
  r->oA1 = kept >= 1 ? o : 0;
  if (kept >= 1) o += R * w4;
  r->oA2 = kept >= 2 ? o : 0;
  if (kept >= 2) o += R * w4;
  r->oPH = r->oDH = 0;
  if (adj) {
    r->oPH = o;
    o += (R + 3) * w4 + 4;
    r->oDH = o;
    o += R * w4;
  }
  r->oBox = o;
  if (!r->glb && r->G > 1) o += res::kBoxRows * r->CG * 8;
  // dL/d records of the step and of the next: one row lies in the unused U slots of rows R and R+1
  r->injg = most_rows <= 1 ? res::kGrp : 4;
  r->injw = most_rows <= 1 ? sb : most_rows * w4;
  r->oInj = most_rows <= 1 ? r->oS + (R + 2) * sb + res::kGrp : o;
  if (adj && most_rows > 1) o += 2 * r->injw;
  r->oRow = o;
  if (adj) o += R;
  r->oT = tables ? o : 0;
  r->words = o + (tables ? 2 * most : 0);
}

// Blocks of a variant that an SM holds: MT threads of 65536 / MT registers, and the shared memory.
int res_per_sm(const Resident& r) {
  const int regs = 65536 / r.MT / 8 * 8;
  return std::min(65536 / (regs * r.T), 233472 / (r.words * 4 + 1024));
}

// Clusters of C blocks that are resident at a time when an SM holds n such blocks: asked of the
// runtime once per (device, C, n), since it depends on how the SMs are grouped.
std::mutex g_cluster_mu;
std::vector<std::vector<int>> g_clusters;  // per device: C x n, -1 unknown
int resident_clusters(const Resident& r, int n, int dev, ResKernel k) {
  constexpr int kN = 32;
  n = std::min(n, kN - 1);
  std::lock_guard<std::mutex> lk(g_cluster_mu);
  if ((int)g_clusters.size() <= dev) g_clusters.resize(dev + 1);
  std::vector<int>& t = g_clusters[dev];
  if (t.empty()) t.assign((res::kMaxCluster + 1) * kN, -1);
  int& v = t[r.G * kN + n];
  if (v < 0) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[1];
    res_config(&cfg, attr, r, nullptr);
    if (res_prepare(k) != cudaSuccess || cudaOccupancyMaxActiveClusters(&v, k, &cfg) != cudaSuccess) {
      cudaGetLastError();
      v = 0;
    }
  }
  return v;
}

// The configuration with the least estimated time per step of all shots: waves of shots x (what
// the exchange between strips costs + the 128-cell units of an SM x the variant's time per unit).
// In us, from sweeps of G and of the variants with per-launch times (300 x 700 padded with 10 and
// 30 shots, 148 x 260 with 40, 200 x 200 with 10, 600 x 1600 with 8):
//   exchange: 1.6 through global memory, 0.7 in a cluster (whose shared memory is next door, but
//     only 7 clusters of 16 blocks, 13 of 10 or 23 of 6 fit the GPU at a time), 0.3 without one;
//   0.6 more in blocks of less than two warps, and in the forward loop with strips of at most 5 rows,
//     whose few threads wait for both neighbours;
//   per unit, forward / adjoint: 0.065 / 0.09 for 3 rows per thread and 128 registers (0.06 for 2, forward, which
//     strips of equal even height take); the adjoint
//     loses a third at 80 registers (spills), and more rows per thread leave fewer warps; 6 rows take
//     168 registers where 384 threads do (at 128 the adjoint through global memory spills 80 B);
//   several blocks per SM run 15 % slower than one that does the same work; clusters that do not fit
//     at one block per SM double up on some SMs while others idle, however few blocks there are in
//     all (10 shots of 200 x 200: 2.87 us with 15 strips, 2.35 with 10; 20 of 96 x 232: 3.9 with 7, 2.4
//     with 6; 30 of 100 x 120: 2.7 with 5, 2.1 with 9): forward 0.9, adjoint 0.75 of their number.
// For example 300 x 700 with 30 shots, us per step: forward 29.2 with 25 strips of 12 rows and
// 3 rows per thread (35.4 with 6, 43.5 with 38 strips of 8), adjoint 37.2 with 25 strips and 6
// rows per thread (40.2 at 128 registers; 45.8 with 4 rows, 46.9 with 3, 52.6 with 50 strips of 6).
Resident res_choose(const adfwi_acoustic_plan* p, bool adj, const std::vector<std::pair<int64_t, int>>& rc, int max_smem,
                    int sms, int dev) {
  const int z0 = p->d.free_surface ? p->fs : 0;
  const int NR = p->nzp - z0, CG = (p->nxp + 3) / 4, ns = p->d.ns;
  std::vector<int> cells(NR + 1, 0);  // receiver cells of the rows before each row
  for (size_t q = 0; q < rc.size(); ++q)
    if (q == 0 || rc[q].first != rc[q - 1].first) cells[(rc[q].first >> 32) + 1]++;
  std::vector<int> held(NR + 1, 0);   // rows before each row that hold any
  for (int r = 0; r < NR; ++r) {
    held[r + 1] = held[r] + (cells[r + 1] > 0);
    cells[r + 1] += cells[r];
  }
  Resident best;
  double best_cost = 1e30;
  for (int glb = 0; glb < 2; ++glb) {
    for (int G = glb ? 2 : 1; G <= (glb ? 2 * sms : res::kMaxCluster); ++G) {
      const int least = NR / G;
      if (least < 4) break;
      int most = 0, most_rows = 0;
      for (int k = 0; k < G; ++k) {
        const int b = (int)((int64_t)k * NR / G), e = (int)((int64_t)(k + 1) * NR / G);
        most = std::max(most, cells[e] - cells[b]);
        most_rows = std::max(most_rows, held[e] - held[b]);
      }
      Resident r;
      r.glb = glb;
      r.G = G;
      r.R = (NR + G - 1) / G;
      r.CG = CG;
      for (const int* v : res::kVariants) {
        r.RB = v[0];
        r.MT = v[1];
        r.TR = (r.R + r.RB - 1) / r.RB;
        if (adj ? r.RB == 2 : r.MT == 384) continue;
        if (least / r.TR < 2) continue;  // the boundary threads own both rows that cross
        r.T = (r.TR * CG + 31) / 32 * 32;
        if (r.T > r.MT) continue;
        for (int kept = 2; kept >= -1; --kept) {  // alpha1, alpha2 kept; -1: not even the receiver tables
          res_layout(&r, adj, std::max(0, kept), kept >= 0, most, most_rows);
          if (r.words * 4 > max_smem) continue;
          const int n = res_per_sm(r);
          if (n < 1) continue;
          r.S = 1;
          const int cap = glb ? n * sms / G : resident_clusters(r, n, dev, res_kernel(r, adj, true));
          if (cap < 1) continue;
          r.S = glb ? std::min(ns, cap) : ns;
          const int waves = (ns + cap - 1) / cap;
          const int act = std::min(ns, cap);
          double load = (double)act * G / sms;
          load = load > 1.0 ? 1.15 * load : 1.0;
          if (!glb && G > 1) {  // clusters at one block per SM, and how many share an SM beyond that
            Resident one = r;
            one.words = max_smem / 4;
            const int alone = std::max(1, resident_clusters(one, 1, dev, res_kernel(r, adj, true)));
            load = std::max(std::max(1.0, load), (act > alone ? adj ? 0.75 : 0.9 : 0.0) * ((act + alone - 1) / alone));
          }
          const double per_unit = adj ? (r.RB == 3 ? (r.MT == 512 ? 0.09 : 0.12) : r.RB == 4 ? (r.MT == 512 ? 0.105 : 0.115) : r.MT == 384 ? 0.095 : 0.1)
                                      : (r.RB == 2 ? 0.06 : r.RB == 3 ? 0.065 : r.RB == 4 ? (r.MT == 512 ? 0.09 : 0.076) : 0.084);
          const double fixed = (glb ? 1.6 : G > 1 ? 0.7 : 0.3) + (r.T < 64 || (!adj && r.R <= 5) ? 0.6 : 0.0);
          const double cost = waves * (fixed + per_unit * r.R * CG / 32.0 * load) * (1.0 - 0.01 * kept);
          if (cost < best_cost) {
            best_cost = cost;
            best = r;
          }
          break;
        }
      }
    }
  }
  if (best.G > 0 && best.glb) {  // what the runtime says of the chosen one decides
    int occ = 0;
    ResKernel k = res_kernel(best, adj, true);
    if (res_prepare(k) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k, best.T, (size_t)best.words * 4) != cudaSuccess)
      cudaGetLastError();
    best.S = std::min(ns, occ * sms / best.G);
    if (best.S < 1) best = Resident();
  }
  return best;
}

// Configurations of the resident time loop for this plan's grid and shots, and their tables
// (appended to p->tab). They stay empty where the state does not fit.
void plan_resident(adfwi_acoustic_plan* p, const int32_t* rcv_z, const int32_t* rcv_x) {
  const adfwi_acoustic_desc& d = p->d;
  if (p->elem != 4 || p->bsave) return;
  int dev = 0, max_smem = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
    cudaGetLastError();
    return;  // no device: plans made for their sizes only
  }
  // receivers in (row, column) order; receivers on the mirrored row above a free surface stay with
  // the per-step kernels (their dL/d records fold into the interior)
  const int z0 = d.free_surface ? p->fs : 0;
  std::vector<std::pair<int64_t, int>> rc(d.nr);
  bool above = false;
  for (int r = 0; r < d.nr; ++r) {
    const int z = rcv_z[r] + d.nabc - z0, x = rcv_x[r] + d.nabc;
    rc[r] = {((int64_t)z << 32) | x, r};
    above = above || z < 0;
  }
  if (above) return;
  std::stable_sort(rc.begin(), rc.end(), [](const std::pair<int64_t, int>& a, const std::pair<int64_t, int>& b) {
    return a.first < b.first;
  });
  p->rf = res_choose(p, false, rc, max_smem, sms, dev);
  if (p->rf.G > 0) p->ra = res_choose(p, true, rc, max_smem, sms, dev);
  std::vector<int32_t>& t = p->tab;
  p->o_sm = t.size();
  for (int m = 0; m < p->nm; ++m)
    for (int s = p->model_shot_beg[m]; s < p->model_shot_beg[m + 1]; ++s) t.push_back(m);
  const int64_t NR = p->nzp - z0;
  for (Resident* r : {&p->rf, &p->ra}) {
    if (r->G == 0) continue;
    std::vector<int32_t> beg(r->G + 1, 0), slot(NR, 0), pos, rid, rbeg, rcv;
    const int sb = res::kGrp * (r->CG + 1);
    int strip = 0, last = -1, nslot = 0;
    for (size_t q = 0; q < rc.size(); ++q) {
      const int z = (int)(rc[q].first >> 32), x = (int)(rc[q].first & 0xffffffff);
      while (z >= (int)((int64_t)(strip + 1) * NR / r->G)) ++strip, nslot = 0;
      if (z != last) slot[z] = ++nslot;
      last = z;
      if (q == 0 || rc[q].first != rc[q - 1].first) {
        beg[strip + 1]++;
        const int row = z - (int)((int64_t)strip * NR / r->G);
        pos.push_back(r == &p->ra ? ((slot[z] - 1) * r->CG + x / 4) * r->injg + x % 4 : row * sb + res::kGrp * (x / 4) + x % 4);
        rid.push_back(rc[q].second);
        rbeg.push_back((int32_t)rcv.size());
      } else {
        rid.back() = -(int32_t)rid.size();  // -1 - cell: several receivers
      }
      rcv.push_back(rc[q].second);
    }
    rbeg.push_back((int32_t)rcv.size());
    for (int q = 0; q < r->G; ++q) beg[q + 1] += beg[q];
    r->o_sl = t.size();
    t.insert(t.end(), slot.begin(), slot.end());
    r->o_sb = t.size();
    t.insert(t.end(), beg.begin(), beg.end());
    r->o_tp = t.size();
    t.insert(t.end(), pos.begin(), pos.end());
    r->o_ti = t.size();
    t.insert(t.end(), rid.begin(), rid.end());
    r->o_rb = t.size();
    t.insert(t.end(), rbeg.begin(), rbeg.end());
    r->o_rv = t.size();
    t.insert(t.end(), rcv.begin(), rcv.end());
  }
}

// ----------------------------------------------------------------------------------------
// Forward solve for callers that cannot allocate device memory.
//
// Its scratch (staged coefficients, wavefield ping-pong buffers, illumination partials and
// geometry tables) lives in one file-scope __device__ array of kStaticScratchBytes, which
// every GPU that loads this library reserves until the process exits. Host code never
// passes the symbol itself to a kernel (on the host it only names a stand-in object):
// the device address is looked up once per device with cudaGetSymbolAddress, on that
// device, by the first call made there.
// ----------------------------------------------------------------------------------------
constexpr int64_t kStaticScratchBytes = int64_t(64) << 20;  // 64 MiB
__device__ __align__(256) unsigned char g_static_scratch[kStaticScratchBytes];
std::mutex g_static_mu;
std::vector<void*> g_static_addr;  // device address of g_static_scratch, per device ordinal

int static_scratch_address(void** out) {
  int dev = 0;
  ADFWI_CUDA_TRY(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(g_static_mu);
  if ((int)g_static_addr.size() <= dev) g_static_addr.resize(dev + 1, nullptr);
  if (g_static_addr[dev] == nullptr) {
    void* addr = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&addr, g_static_scratch);
    if (e != cudaSuccess || addr == nullptr) {
      set_error("cudaGetSymbolAddress(static scratch) failed on device %d: %s", dev, cudaGetErrorString(e));
      return kCudaError;
    }
    g_static_addr[dev] = addr;
  }
  *out = g_static_addr[dev];
  return kOk;
}

}  // namespace

extern "C" {

int adfwi_acoustic_forward_noalloc(const adfwi_acoustic_plan* p, const void* alpha1, const void* alpha2,
                                   const void* damp, const void* wavelet, void* rec_p, void* rec_u, void* rec_w,
                                   void* fw_p, void* fw_u, void* fw_w, void* stream) {
  ADFWI_CHECK_ARG(p && alpha1 && alpha2 && damp && wavelet, "null argument");
  ADFWI_CHECK_ARG((rec_p && rec_u && rec_w) || (!rec_p && !rec_u && !rec_w), "records: give all three or none");
  ADFWI_CHECK_ARG(p->d.nr > 0 || rec_p == nullptr, "records requested without receivers");
  // strips that exchange rows through global memory need inboxes: without the room for them the
  // per-step kernels solve (the same records)
  const bool box = carve(p, false, 1).total <= kStaticScratchBytes;
  const int64_t need = carve(p, false, 1, box).total;
  if (need > kStaticScratchBytes) {
    set_error("adfwi_acoustic_forward_noalloc: this solve needs %lld bytes of scratch but the static scratch "
              "array holds %lld bytes (64 MiB); use adfwi_acoustic_forward with a caller-provided workspace",
              (long long)need, (long long)kStaticScratchBytes);
    return kWorkspaceTooSmall;
  }
  void* ws = nullptr;
  int rc = static_scratch_address(&ws);
  if (rc) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  unsigned char* w = static_cast<unsigned char*>(ws);
  // forward_impl clears every scratch region it accumulates into (coefficient ghosts, field
  // buffers, illumination partials) before the first step, so a previous call's leftovers
  // in the shared array do not leak into this one.
  if (p->d.dtype == ADFWI_F64)
    return forward_impl<double>(p, alpha1, alpha2, damp, wavelet, rec_p, rec_u, rec_w, fw_p, fw_u, fw_w, false, w,
                                kStaticScratchBytes, st, box);
  return forward_impl<float>(p, alpha1, alpha2, damp, wavelet, rec_p, rec_u, rec_w, fw_p, fw_u, fw_w, false, w,
                             kStaticScratchBytes, st, box);
}

int adfwi_acoustic_noalloc_status(const adfwi_acoustic_plan* p, int32_t* status, void* stream) {
  ADFWI_CHECK_ARG(p && status, "null argument");
  const Carve c = carve(p, false, 1, false);
  ADFWI_CHECK_ARG(c.total <= kStaticScratchBytes, "this plan's forward does not fit the static scratch array");
  void* ws = nullptr;
  int rc = static_scratch_address(&ws);
  if (rc) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  int32_t v = 0;
  ADFWI_CUDA_TRY(cudaMemcpyAsync(&v, static_cast<const unsigned char*>(ws) + c.flag, sizeof(v),
                                 cudaMemcpyDeviceToHost, st));
  ADFWI_CUDA_TRY(cudaStreamSynchronize(st));
  *status = v;
  return kOk;
}

}  // extern "C"

namespace {

int plan_create_impl(const adfwi_acoustic_desc* desc, const int32_t* src_z, const int32_t* src_x,
                     const int32_t* rcv_z, const int32_t* rcv_x, int32_t nmodels, const int32_t* shot_model,
                     adfwi_acoustic_plan** out) {
  ADFWI_CHECK_ARG(desc && out, "null descriptor or output pointer");
  *out = nullptr;
  const adfwi_acoustic_desc& d = *desc;
  ADFWI_CHECK_ARG(nmodels >= 1, "need nmodels >= 1");
  ADFWI_CHECK_ARG(d.ns >= 1, "need ns >= 1");
  std::vector<int> model_shot_beg(nmodels + 1, 0);
  if (shot_model != nullptr) {
    // shots of one model are consecutive, models in order, every model has a shot
    for (int s = 0; s < d.ns; ++s) {
      ADFWI_CHECK_ARG(shot_model[s] >= 0 && shot_model[s] < nmodels && (s == 0 || shot_model[s] >= shot_model[s - 1]),
                      "shot_model must be non-decreasing in [0, nmodels) (shot %d)", s);
      model_shot_beg[shot_model[s] + 1]++;
    }
    for (int m = 0; m < nmodels; ++m) {
      ADFWI_CHECK_ARG(model_shot_beg[m + 1] > 0, "model %d has no shot", m);
      model_shot_beg[m + 1] += model_shot_beg[m];
    }
  } else {
    ADFWI_CHECK_ARG(nmodels == 1, "shot_model is required for several models");
    model_shot_beg[1] = d.ns;
  }
  ADFWI_CHECK_ARG(d.nz >= 1 && d.nx >= 1 && d.nabc >= 2, "need nz, nx >= 1 and nabc >= 2");
  ADFWI_CHECK_ARG(d.ns >= 1 && d.nt >= 1 && d.nr >= 0, "need ns >= 1, nt >= 1, nr >= 0");
  ADFWI_CHECK_ARG(d.dtype == ADFWI_F32 || d.dtype == ADFWI_F64, "dtype must be ADFWI_F32 or ADFWI_F64");
  ADFWI_CHECK_ARG(d.snapshot_precision >= 0 && d.snapshot_precision <= 3, "bad snapshot_precision");
  ADFWI_CHECK_ARG(d.checkpoint_segments >= 1, "checkpoint_segments must be >= 1");
  ADFWI_CHECK_ARG(d.ring_depth >= 0 && d.ring_depth <= 2, "ring_depth must be 0, 1 or 2");
  ADFWI_CHECK_ARG(d.snapshot_every >= ADFWI_SNAP_EVERY_BOUNDARY,
                  "snapshot_every must be >= 0, or ADFWI_SNAP_EVERY_BOUNDARY for boundary saving");
  ADFWI_CHECK_ARG(d.snapshot_every != ADFWI_SNAP_EVERY_BOUNDARY || nmodels == 1,
                  "boundary saving takes a single-model plan");
  ADFWI_CHECK_ARG(src_z && src_x && (d.nr == 0 || (rcv_z && rcv_x)), "null geometry array");
  adfwi_acoustic_plan* p = new (std::nothrow) adfwi_acoustic_plan();
  if (!p) {
    set_error("host allocation failed");
    return kBadArgument;
  }
  p->d = d;
  p->nm = nmodels;
  p->model_shot_beg = model_shot_beg;
  p->nzp = d.nz + 2 * d.nabc;
  p->nxp = d.nx + 2 * d.nabc;
  p->fs = d.free_surface ? d.nabc : 1;
  p->zbeg = d.free_surface ? p->fs - 1 : 0;
  p->elem = d.dtype == ADFWI_F64 ? 8 : 4;
  p->L = make_layout(p->nzp, p->nxp, ac2::TZ, ac2::TX, p->elem);
  p->bsave = d.snapshot_every == ADFWI_SNAP_EVERY_BOUNDARY;
  if (p->bsave) {
    // The interior whose update inverts exactly: the model window, inside every update region,
    // away from the free-surface rows, and one cell short of the frame on the right and at the
    // bottom (the u / w damping averages a cell with its right / lower neighbour). Everything
    // else is the frame that the forward keeps step by step.
    const int i_lo = std::max(d.nabc, p->fs + 1), i_hi = std::min(d.nabc + d.nz - 2, p->nzp - 4);
    const int j_lo = std::max(d.nabc, 2), j_hi = std::min(d.nabc + d.nx - 2, p->nxp - 4);
    p->bbox = ac::BsBox{i_lo, i_hi, j_lo, j_hi};
    std::vector<int32_t>& tb = p->tab;
    p->o_fidx = tb.size();
    tb.resize(tb.size() + (size_t)p->nzp * p->nxp, -1);
    std::vector<int32_t> off;
    for (int i = 0; i < p->nzp; ++i)
      for (int j = 0; j < p->nxp; ++j)
        if (!(i >= i_lo && i <= i_hi && j >= j_lo && j <= j_hi)) {
          tb[p->o_fidx + (size_t)i * p->nxp + j] = (int32_t)off.size();
          off.push_back((int32_t)p->L.off(i, j));
        }
    p->nframe = (int)off.size();
    p->o_foff = tb.size();
    tb.insert(tb.end(), off.begin(), off.end());
  }
  // torch.chunk(wavelet, checkpoint_segments): chunks of ceil(nt / segments) steps.
  const int chunk = (d.nt + d.checkpoint_segments - 1) / d.checkpoint_segments;
  const int nchunks = (d.nt + chunk - 1) / chunk;
  p->last_chunk_start = (nchunks - 1) * chunk;

  // Geometry tables.
  std::vector<int32_t>& t = p->tab;
  p->o_srcz = t.size();
  for (int s = 0; s < d.ns; ++s) {
    int z = src_z[s] + d.nabc, x = src_x[s] + d.nabc;
    if (z < p->zbeg || z >= p->nzp || x < 0 || x >= p->nxp) {
      set_error("source %d at (z=%d, x=%d) lies outside the model", s, src_z[s], src_x[s]);
      delete p;
      return kBadGeometry;
    }
    t.push_back(z);
  }
  p->o_srcx = t.size();
  for (int s = 0; s < d.ns; ++s) t.push_back(src_x[s] + d.nabc);
  for (int r = 0; r < d.nr; ++r) {
    int z = rcv_z[r] + d.nabc, x = rcv_x[r] + d.nabc;
    // u has nxp-1 columns and w has nzp-1 rows (acoustic_kernels.py:241-242, 167-169)
    if (z < p->zbeg || z > p->nzp - 2 || x < 0 || x > p->nxp - 2) {
      set_error("receiver %d at (z=%d, x=%d) lies outside the recordable model", r, rcv_z[r], rcv_x[r]);
      delete p;
      return kBadGeometry;
    }
    p->rcv_above = p->rcv_above || (d.free_surface && z < p->fs);
  }
  // 16 x 64 tiles: units of G shots spread over the resident blocks of the pipelined steps.
  {
    const int ntiles = ((p->nxp + ac2::TX - 1) / ac2::TX) * ((p->nzp - p->zbeg + ac2::TZ - 1) / ac2::TZ);
    // shots per group from the shallow variants' widths whatever the ring, so that the ring
    // changes launch widths and stages only, never the results
    const bool f64 = p->elem == 8;
    const int blocks = f64 ? 1 : resident_adj_blocks(false), fblocks = f64 ? 1 : resident_fwd_blocks(false);
    p->deep = !f64 && (d.ring_depth == 2 || (d.ring_depth == 0 && p->nxp >= kDeepRingCols));
    const int run_blocks = p->deep ? resident_adj_blocks(true) : blocks;
    const int run_fblocks = p->deep ? resident_fwd_blocks(true) : fblocks;
    // shots per group of each model: as a plan of that model alone would choose them, so a
    // model's partial sums (and so its results) do not depend on the other models of a batch
    std::vector<int> Gm(p->nm);
    for (int m = 0; m < p->nm; ++m) {
      const std::vector<int> alone = {0, p->model_shot_beg[m + 1] - p->model_shot_beg[m]};
      if (d.shots_per_block > 0) Gm[m] = d.shots_per_block;
      else if (f64) Gm[m] = f64_group_shots(p, alone, ntiles, kStaticScratchBytes);
      else Gm[m] = pick_unit_shots(alone, ntiles, fblocks, blocks);
    }
    build_tiling(p, &p->t2, ac2::TZ, ac2::TX, Gm, rcv_z, rcv_x);
    p->t2.blocks = std::max(1, std::min(run_blocks, p->t2.ntiles * p->t2.ngroups));
    p->t2.fwd_blocks = std::max(1, std::min(run_fblocks, p->t2.ntiles * p->t2.ngroups));
  }
  if (p->elem == 8) {
    p->o_rz = t.size();
    for (int r = 0; r < d.nr; ++r) t.push_back(rcv_z[r] + d.nabc);
    p->o_rx = t.size();
    for (int r = 0; r < d.nr; ++r) t.push_back(rcv_x[r] + d.nabc);
    auto first_at = [&](int q) { return t[p->t2.o_cr + t[p->t2.o_tcr + q]]; };  // a cell lies where its first receiver does
    p->o_cz = t.size();
    for (int q = 0; q < p->t2.ncells; ++q) t.push_back(rcv_z[first_at(q)] + d.nabc);
    p->o_cx = t.size();
    for (int q = 0; q < p->t2.ncells; ++q) t.push_back(rcv_x[first_at(q)] + d.nabc);
    const int tx = (p->nxp + ac3::kX - 1) / ac3::kX, nt = ac3::tiles(p->L, p->zbeg);
    std::vector<int32_t> beg(nt + 1, 0), order(p->t2.ncells);
    auto tile = [&](int q) { return (t[p->o_cz + q] - p->zbeg) / ac3::kZ * tx + t[p->o_cx + q] / ac3::kX; };
    for (int q = 0; q < p->t2.ncells; ++q) ++beg[tile(q) + 1];
    for (int q = 0; q < nt; ++q) beg[q + 1] += beg[q];
    std::vector<int32_t> at(beg.begin(), beg.end() - 1);
    for (int q = 0; q < p->t2.ncells; ++q) order[at[tile(q)]++] = q;
    p->o_ftb = t.size();
    t.insert(t.end(), beg.begin(), beg.end());
    p->o_ftc = t.size();
    t.insert(t.end(), order.begin(), order.end());
  }
  plan_resident(p, rcv_z, rcv_x);
  if (t.empty()) t.push_back(0);

  if (!p->tab_pin.assign(p->tab.data(), p->tab.size() * 4)) {
    delete p;
    return kCudaError;
  }
  p->K = choose_K(p);
  p->nseg = (d.nt + p->K - 1) / p->K;
  *out = p;
  return kOk;
}

}  // namespace

extern "C" {

int adfwi_acoustic_plan_create(const adfwi_acoustic_desc* desc, const int32_t* src_z, const int32_t* src_x,
                               const int32_t* rcv_z, const int32_t* rcv_x, adfwi_acoustic_plan** out) {
  return plan_create_impl(desc, src_z, src_x, rcv_z, rcv_x, 1, nullptr, out);
}

int adfwi_acoustic_plan_create_batched(const adfwi_acoustic_desc* desc, const int32_t* src_z,
                                       const int32_t* src_x, const int32_t* rcv_z, const int32_t* rcv_x,
                                       int32_t nmodels, const int32_t* shot_model, adfwi_acoustic_plan** out) {
  if (shot_model == nullptr) {
    set_error("adfwi_acoustic_plan_create_batched: null shot_model");
    return kBadArgument;
  }
  return plan_create_impl(desc, src_z, src_x, rcv_z, rcv_x, nmodels, shot_model, out);
}

int32_t adfwi_acoustic_plan_models(const adfwi_acoustic_plan* plan) { return plan ? plan->nm : 0; }

void adfwi_acoustic_plan_destroy(adfwi_acoustic_plan* plan) { delete plan; }

int adfwi_acoustic_status(const adfwi_acoustic_plan* p, const void* workspace, int64_t workspace_bytes,
                          int32_t with_gradient, int32_t* status, void* stream) {
  ADFWI_CHECK_ARG(p && workspace && status, "null argument");
  Carve c = carve(p, with_gradient != 0, with_gradient ? p->K : 1);
  ADFWI_CHECK_ARG(workspace_bytes >= c.total, "workspace smaller than the plan's layout");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  int32_t v = 0;
  ADFWI_CUDA_TRY(cudaMemcpyAsync(&v, static_cast<const unsigned char*>(workspace) + c.flag, sizeof(v),
                                 cudaMemcpyDeviceToHost, st));
  ADFWI_CUDA_TRY(cudaStreamSynchronize(st));
  *status = v;
  return kOk;
}

int adfwi_acoustic_workspace_bytes(const adfwi_acoustic_plan* p, int32_t with_gradient, int64_t* bytes) {
  ADFWI_CHECK_ARG(p && bytes, "null plan or output pointer");
  *bytes = carve(p, with_gradient != 0, with_gradient ? p->K : 1).total;
  return kOk;
}

int adfwi_row_wait_selftest(int64_t limit_ns, int32_t* flag, float* row, void* stream) {
  ADFWI_CHECK_ARG(flag != nullptr && row != nullptr, "null flag or row");
  ADFWI_CHECK_ARG(limit_ns > 0 && limit_ns <= 2000000000ll, "limit_ns must be in (0, 2 s]");
  return res::row_wait_selftest(limit_ns, reinterpret_cast<int*>(flag), row, static_cast<cudaStream_t>(stream));
}

int adfwi_acoustic_snapshot_every(const adfwi_acoustic_plan* p, int32_t* steps) {
  ADFWI_CHECK_ARG(p && steps, "null plan or output pointer");
  *steps = p->bsave ? ADFWI_SNAP_EVERY_BOUNDARY : p->K;
  return kOk;
}

int adfwi_acoustic_forward(const adfwi_acoustic_plan* p, const void* alpha1, const void* alpha2, const void* damp,
                           const void* wavelet, void* rec_p, void* rec_u, void* rec_w, void* fw_p, void* fw_u,
                           void* fw_w, int32_t with_gradient, void* workspace, int64_t workspace_bytes,
                           void* stream) {
  ADFWI_CHECK_ARG(p && alpha1 && alpha2 && damp && wavelet && workspace, "null argument");
  ADFWI_CHECK_ARG((rec_p && rec_u && rec_w) || (!rec_p && !rec_u && !rec_w), "records: give all three or none");
  ADFWI_CHECK_ARG(p->d.nr > 0 || rec_p == nullptr, "records requested without receivers");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  unsigned char* ws = static_cast<unsigned char*>(workspace);
  if (p->d.dtype == ADFWI_F64)
    return forward_impl<double>(p, alpha1, alpha2, damp, wavelet, rec_p, rec_u, rec_w, fw_p, fw_u, fw_w,
                                with_gradient != 0, ws, workspace_bytes, st);
  return forward_impl<float>(p, alpha1, alpha2, damp, wavelet, rec_p, rec_u, rec_w, fw_p, fw_u, fw_w,
                             with_gradient != 0, ws, workspace_bytes, st);
}

int adfwi_acoustic_backward(const adfwi_acoustic_plan* p, const void* alpha1, const void* alpha2, const void* damp,
                            const void* wavelet, const void* grad_rec_p, const void* grad_rec_u,
                            const void* grad_rec_w, void* grad_alpha1, void* grad_alpha2, void* workspace,
                            int64_t workspace_bytes, void* stream) {
  ADFWI_CHECK_ARG(p && alpha1 && alpha2 && damp && wavelet && workspace && grad_alpha1 && grad_alpha2,
                  "null argument");
  (void)alpha1;
  (void)alpha2;
  (void)damp;  // the coefficient planes staged by the forward call are reused from the workspace
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  unsigned char* ws = static_cast<unsigned char*>(workspace);
  if (p->d.dtype == ADFWI_F64)
    return backward_impl<double>(p, wavelet, grad_rec_p, grad_rec_u, grad_rec_w, grad_alpha1, grad_alpha2, ws,
                                 workspace_bytes, st);
  return backward_impl<float>(p, wavelet, grad_rec_p, grad_rec_u, grad_rec_w, grad_alpha1, grad_alpha2, ws,
                              workspace_bytes, st);
}

int adfwi_acoustic_l2_loss(const adfwi_acoustic_plan* p, const void* syn, const void* obs, double silent_rel,
                           int32_t flags, double* loss, void* workspace, int64_t workspace_bytes, void* stream) {
  ADFWI_CHECK_ARG(p && syn && obs && loss && workspace, "null argument");
  ADFWI_CHECK_ARG(p->d.nr > 0, "the plan has no receivers");
  ADFWI_CHECK_ARG(silent_rel >= 0.0, "silent_rel must be non-negative");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  unsigned char* ws = static_cast<unsigned char*>(workspace);
  if (p->d.dtype == ADFWI_F64)
    return l2_loss_impl<double>(p, syn, obs, silent_rel, flags, loss, ws, workspace_bytes, st);
  return l2_loss_impl<float>(p, syn, obs, silent_rel, flags, loss, ws, workspace_bytes, st);
}

int adfwi_acoustic_l2_sources(const adfwi_acoustic_plan* p, const void* syn, const void* obs, int32_t flags,
                              const double* grad_scale, void* adj, void* workspace, int64_t workspace_bytes,
                              void* stream) {
  ADFWI_CHECK_ARG(p && syn && obs && grad_scale && adj && workspace, "null argument");
  ADFWI_CHECK_ARG(p->d.nr > 0, "the plan has no receivers");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  unsigned char* ws = static_cast<unsigned char*>(workspace);
  if (p->d.dtype == ADFWI_F64)
    return l2_sources_impl<double>(p, syn, obs, flags, grad_scale, adj, ws, workspace_bytes, st);
  return l2_sources_impl<float>(p, syn, obs, flags, grad_scale, adj, ws, workspace_bytes, st);
}

int adfwi_acoustic_backward_l2(const adfwi_acoustic_plan* p, const void* wavelet, const void* syn, const void* obs,
                               int32_t flags, const double* grad_scale, void* grad_alpha1, void* grad_alpha2,
                               void* workspace, int64_t workspace_bytes, void* stream) {
  ADFWI_CHECK_ARG(p && wavelet && syn && obs && grad_scale && grad_alpha1 && grad_alpha2 && workspace,
                  "null argument");
  ADFWI_CHECK_ARG(p->d.nr > 0, "the plan has no receivers");
  const FusedL2 fz{obs, grad_scale, flags & 1};
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  unsigned char* ws = static_cast<unsigned char*>(workspace);
  if (p->d.dtype == ADFWI_F64)
    return backward_impl<double>(p, wavelet, syn, nullptr, nullptr, grad_alpha1, grad_alpha2, ws, workspace_bytes, st,
                                 &fz);
  return backward_impl<float>(p, wavelet, syn, nullptr, nullptr, grad_alpha1, grad_alpha2, ws, workspace_bytes, st,
                              &fz);
}

}  // extern "C"
