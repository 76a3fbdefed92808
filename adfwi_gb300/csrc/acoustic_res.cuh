// Resident acoustic time loop: one launch advances many time steps, forward or adjoint, with the
// state of every shot it works on held in shared memory.
//
// The per-step kernels (acoustic_vec.cuh) read and write the whole state through L2 / HBM every
// step and pay a launch for it: 8.3 (forward) and 12.7 ns (adjoint) per thousand cell-updates on
// the 300 x 700 grid, and the launch rate on small ones. Here a shot's rows are cut into G strips
// of R rows, one block each, and a block keeps its strip on the chip for the whole loop. The
// update is in place, so a step is two phases with a block barrier after each:
//   1  p from u (its own rows: u has no vertical neighbours) and w (2 rows above, 1 below);
//   2  u and w from p (1 row above, 2 below).
// The rows that cross between strips go through the neighbour's inbox: in shared memory when the
// shot's blocks are a cluster (small grids), in global memory when they are part of a cooperative
// launch (grids of up to 150 strips); 30 shots of the 300 x 700 grid run as five waves of six
// shots x 25 strips. HBM sees only what has to leave the chip, the histories of a gradient solve
// and the records.
//
// A thread owns four adjacent columns of up to RB consecutive rows for the whole loop: the
// vertical stencils slide a window of rows through registers (one 16-byte shared load per row
// instead of four), and the sums over time of its cells (illumination, or the coefficient
// gradients) stay in registers. Arithmetic is in pairs of floats (f32x2), which halves its
// instructions. The adjoint's histories land in shared memory by bulk copies a phase ahead.
//
// What bounds it is the shared-memory pipe: about 90 wavefronts per 128 cells and step of the 130
// to 190 clocks they take, next to the exchange (1 to 2 us per step, acoustic.cu res_choose).
// Measured per step of all shots, per-step kernels -> here, in us: 300 x 700 with 30 shots forward 52 -> 29,
// adjoint 80 -> 37; 600 x 1600 with 8 shots 79 -> 54, 120 -> 66; 148 x 260 with 40 shots and a free
// surface 18.7 -> 7.3, 35 -> 9.4; 200 x 200 with 10 shots (records only) 9.2 -> 2.4.
// Tried and slower: the state of a thread's cells in registers with shuffles for the horizontal
// neighbours (spills; 4.3 against 3.1 us on 20 rows x 256), all coefficients in shared memory with
// loads lifted across rows (the same or slower), two smaller blocks per SM to hide the exchange
// (36.6 against 29.2 us on 300 x 700).
//
// The forward arithmetic is explicitly rounded in the reference's operation order, as in
// fwd_step_vec: records and histories are bit-identical. The adjoint runs the same recursion:
// with V = alpha1 lambda_p (before the damping factor of the step), U = alpha2 lambda_u and
// W = alpha2 lambda_w the transposed update is
//   V <- b1 V + alpha1 (dL/drec + div(U, W));  U <- b2 U + alpha2 d(V)/dx;  W <- b3 W + alpha2 d(V)/dz,
// with the free surface's mirrored rows exactly as in the forward (p odd, w even), and
//   dL/d alpha1 = - sum V div(u, w) / alpha1,   dL/d alpha2 = - sum (U dp/dx + W dp/dz) / alpha2,
// so no neighbour's coefficient is needed. Cells of an update region whose alpha is zero carry
// the unscaled lambda in the global state planes instead (V, U, W are zero there). No result
// depends on G, R or the variant. Nor does it on how the steps are split into launches, but for the
// gradients of the four columns of a thread that hold such a cell: their sums begin anew in every launch and
// are added up at its end.
#pragma once
#include "acoustic_res.h"
#include "tma.cuh"

namespace adfwi {
namespace res {

__device__ __forceinline__ int at(int c) { return kGrp * (c >> 2) + (c & 3); }  // column c (any sign) from column 0

// ------------------------------------------------------------------ pairs of floats
using f2 = unsigned long long;
__device__ __forceinline__ f2 pk(float a, float b) {
  f2 d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
  return d;
}
__device__ __forceinline__ void upk(f2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ float lo(f2 v) {
  float a, b;
  upk(v, a, b);
  return a;
}
__device__ __forceinline__ float hi(f2 v) {
  float a, b;
  upk(v, a, b);
  return b;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
  f2 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f2 sub2(f2 a, f2 b) {
  f2 d;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
  f2 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
// The product rounded by itself. nz is a pair of -0 that comes with the launch: adding it changes
// no product, not even a zero's sign, and the assembler, which contracts mul.rn.f32x2 with a
// following add, cannot know it.
__device__ __forceinline__ f2 rmul2(f2 a, f2 b, f2 nz) { return fma2(a, b, nz); }
__device__ __forceinline__ void ld4(const float* p, float (&v)[4]) {
  const float4 q = *reinterpret_cast<const float4*>(p);
  v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
}
__device__ __forceinline__ void ldg4(const float* p, float (&v)[4]) {
  const float4 q = __ldg(reinterpret_cast<const float4*>(p));
  v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
}
__device__ __forceinline__ void st4(float* p, const float (&v)[4]) {
  *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void ldq(const float* p, f2 (&v)[2]) {
  const ulonglong2 q = *reinterpret_cast<const ulonglong2*>(p);
  v[0] = q.x;
  v[1] = q.y;
}
__device__ __forceinline__ void ldgq(const float* p, f2 (&v)[2]) {
  const ulonglong2 q = __ldg(reinterpret_cast<const ulonglong2*>(p));
  v[0] = q.x;
  v[1] = q.y;
}
__device__ __forceinline__ void stq(float* p, const f2 (&v)[2]) {
  *reinterpret_cast<ulonglong2*>(p) = make_ulonglong2(v[0], v[1]);
}
// Keeps what is computed from v inside the loop body (hoisted out, a thread's addresses and tests
// of all its rows would take more registers than there are).
__device__ __forceinline__ unsigned opaque(unsigned v) {
  asm volatile("" : "+r"(v));
  return v;
}
__device__ __forceinline__ f2 ldp(const float* p) { return *reinterpret_cast<const f2*>(p); }

// The forward keeps the reference's rounding and order; the adjoint's sums contract to FMA.
// div: c1 ((u0 - um) + w0 - wm) + c2 ((u1 - um2) + w1 - wm2)
template <bool ADJ>
__device__ __forceinline__ f2 div2(f2 nz, f2 c1, f2 c2, f2 u0, f2 um, f2 u1, f2 um2, f2 w0, f2 wm, f2 w1, f2 wm2) {
  const f2 t1 = sub2(add2(sub2(u0, um), w0), wm);
  const f2 t2 = sub2(add2(sub2(u1, um2), w1), wm2);
  return ADJ ? fma2(c1, t1, mul2(c2, t2)) : add2(rmul2(c1, t1, nz), rmul2(c2, t2, nz));
}
template <bool ADJ>
__device__ __forceinline__ f2 diff2(f2 nz, f2 c1, f2 c2, f2 p1, f2 p0, f2 p2, f2 pm) {
  return ADJ ? fma2(c1, sub2(p1, p0), mul2(c2, sub2(p2, pm)))
             : add2(rmul2(c1, sub2(p1, p0), nz), rmul2(c2, sub2(p2, pm), nz));
}
// x - a y (forward), x + a y (adjoint)
template <bool ADJ>
__device__ __forceinline__ f2 step2(f2 nz, f2 x, f2 a, f2 y) {
  return ADJ ? fma2(a, y, x) : sub2(x, rmul2(a, y, nz));
}

// ------------------------------------------------------------------ rows between strips
// A row crosses to the neighbouring strip as 8-byte words of (step tag, value): the word is
// written and read in one access, so the reader polls the values themselves and no fence or
// flag is needed. A word is written again only after its reader has answered (the thread that
// writes a boundary column is the one that reads the neighbour's reply for it), so one copy
// per direction suffices.
__device__ __forceinline__ f2 word(unsigned tag, float v) { return ((f2)tag << 32) | __float_as_uint(v); }
__device__ __forceinline__ uint32_t map_rank(const void* p, int rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(p)), "r"(rank));
  return r;
}
// Store word pairs of a row's four values at `box` (a neighbour's inbox: in global memory, or the
// same shared address of block `rank` of the cluster).
template <bool GLB>
__device__ __forceinline__ void put_row(f2* box, int rank, unsigned tag, const float* row) {
  const float4 v = *reinterpret_cast<const float4*>(row);
  const f2 a = word(tag, v.x), b = word(tag, v.y), c = word(tag, v.z), d = word(tag, v.w);
  if (GLB) {
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(box), "l"(a), "l"(b) : "memory");
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(box + 2), "l"(c), "l"(d) : "memory");
  } else {
    const uint32_t r = map_rank(box, rank);
    asm volatile("st.relaxed.cluster.shared::cluster.v2.b64 [%0], {%1, %2};" ::"r"(r), "l"(a), "l"(b) : "memory");
    asm volatile("st.relaxed.cluster.shared::cluster.v2.b64 [%0], {%1, %2};" ::"r"(r + 16), "l"(c), "l"(d) : "memory");
  }
}
// Wait for the row's words of step `tag` and put the values at dst. A wait that runs out of time
// raises the device flag and the block's `dead` mark: from then on nothing waits, and every
// block runs to its end.
template <bool GLB>
__device__ __forceinline__ void take_row(const f2* box, unsigned tag, float* dst, int* flag, volatile int* dead,
                                         unsigned long long limit_ns = kWaitNs) {
  f2 a, b, c, d;
  unsigned long long t0 = 0;
  for (unsigned n = 0;; ++n) {
    if (GLB) {
      asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(box) : "memory");
      asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(c), "=l"(d) : "l"(box + 2) : "memory");
    } else {
      asm volatile("ld.relaxed.cluster.shared::cta.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "r"(smem_u32(box)) : "memory");
      asm volatile("ld.relaxed.cluster.shared::cta.v2.b64 {%0, %1}, [%2];" : "=l"(c), "=l"(d) : "r"(smem_u32(box + 2)) : "memory");
    }
    if ((unsigned)(a >> 32) == tag && (unsigned)(b >> 32) == tag && (unsigned)(c >> 32) == tag && (unsigned)(d >> 32) == tag)
      break;
    if ((n & 63) == 63) {
      if (*dead) break;
      const unsigned long long t = global_ns();
      if (t0 == 0) t0 = t;
      if (t - t0 > limit_ns || *(volatile int*)flag != 0) {
        raise_flag(flag, kErrWaitTimeout);
        *dead = 1;
      }
    }
  }
  *reinterpret_cast<float4*>(dst) = make_float4(lo(a), lo(b), lo(c), lo(d));
}

__device__ __forceinline__ void bulk_row(float* dst, const float* src, unsigned bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

__device__ __forceinline__ bool zero_in(bool in, float alpha) { return in && alpha == 0.0f; }

// Adjoint, cells of the p region whose alpha1 is zero (one row, columns j .. j+3; S: the row's
// group): V is zero there, so lambda_p itself is advanced in the global state plane z and its
// share of the sum is kept in the global plane acc.
static __device__ __noinline__ void zero_alpha_p(const ac::Geo<float>& g, const float* cf, int64_t PL, int64_t o, int i, int j,
                                          const float* S, int SB, const float* dh, const float* inj, float* z, float* acc) {
  const float* W = S + kW;
  for (int c = 0; c < 4; ++c) {
    if (!zero_in(ac::in_p(g, i, j + c), cf[ac::kA1M * PL + o + c])) continue;
    const float x = g.c1 * (S[c] - S[at(c - 1)] + W[c] - W[c - SB]) + g.c2 * (S[at(c + 1)] - S[at(c - 2)] + W[c + SB] - W[c - 2 * SB]);
    const float lam = cf[ac::kB1 * PL + o + c] * z[o + c] + x + (inj != nullptr ? inj[c] : 0.0f);
    z[o + c] = lam;
    acc[o + c] += lam * dh[c];
  }
}
// The same for lambda_u and lambda_w where alpha2 is zero; H: the forward's pressure in the row.
static __device__ __noinline__ void zero_alpha_uw(const ac::Geo<float>& g, const float* cf, int64_t PL, int64_t o, int i, int j,
                                           const float* S, int SB, const float* H, int W4, float* zu, float* zw,
                                           float* acc) {
  const float* P = S + kP;
  for (int c = 0; c < 4; ++c) {
    if (zero_in(ac::in_u(g, i, j + c), cf[ac::kA2U * PL + o + c])) {
      acc[o + c] += zu[o + c] * (g.c1 * (H[c + 1] - H[c]) + g.c2 * (H[c + 2] - H[c - 1]));
      zu[o + c] = cf[ac::kB2 * PL + o + c] * zu[o + c] + g.c1 * (P[at(c + 1)] - P[c]) + g.c2 * (P[at(c + 2)] - P[at(c - 1)]);
    }
    if (zero_in(ac::in_w(g, i, j + c), cf[ac::kA2W * PL + o + c])) {
      acc[o + c] += zw[o + c] * (g.c1 * (H[c + W4] - H[c]) + g.c2 * (H[c + 2 * W4] - H[c - W4]));
      zw[o + c] = cf[ac::kB3 * PL + o + c] * zw[o + c] + g.c1 * (P[c + SB] - P[c]) + g.c2 * (P[c + 2 * SB] - P[c - SB]);
    }
  }
}
// Factors of four cells: 1 (registers as they come) unless the row is damped.
__device__ __forceinline__ void factors(bool damped, const float* p, f2 (&b)[2]) {
  b[0] = b[1] = 0x3f8000003f800000ull;
  asm("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %3, 0;\n\t@p ld.global.nc.v2.b64 {%0, %1}, [%2];\n\t}"
      : "+l"(b[0]), "+l"(b[1])
      : "l"(p), "r"((unsigned)damped));
}

template <int RB, int MT, bool ADJ, bool SUMS, bool GLB>
__global__ void __launch_bounds__(MT, 1) time_loop(const __grid_constant__ ac::Geo<float> g,
                                                   const __grid_constant__ ResArgs a) {
  extern __shared__ __align__(128) float sm[];
  const int tid = threadIdx.x, T = blockDim.x;
  const int slot = blockIdx.x / a.G, rank = blockIdx.x - slot * a.G;
  const int beg = (int)((int64_t)rank * a.NR / a.G), rows = (int)((int64_t)(rank + 1) * a.NR / a.G) - beg;
  const int i0 = a.z0 + beg;
  const int CG = a.CG, W4 = 4 * CG, SB = kGrp * (CG + 1);
  const int64_t PL = g.L.plane, NSP = (int64_t)g.ns * PL;
  float* const S = sm + a.oS + 2 * SB + kGrp;  // row 0, group 0
  uint64_t* const bar = reinterpret_cast<uint64_t*>(sm);  // adjoint: landings of the p / divergence rows
  volatile int* const dead = reinterpret_cast<volatile int*>(sm + 4);
  // receiver cells of the strip: where the cell is (forward: from S; adjoint: in the rows of dL/d
  // records) and its receiver (or -1 - cell when several share it); in shared memory if they fit
  const int cb = a.strip_beg[rank], nc = a.strip_beg[rank + 1] - cb;
  const int *tpos = a.tpos + cb, *trid = a.trid + cb;
  if (a.oT != 0) {
    int* const tab = reinterpret_cast<int*>(sm + a.oT);
    for (int q = tid; q < nc; q += T) {
      tab[q] = tpos[q];
      tab[nc + q] = trid[q];
    }
    tpos = tab;
    trid = tab + nc;
  }
  int* const rslot = reinterpret_cast<int*>(sm + a.oRow);  // adjoint: 1 + the strip row's row of dL/d records
  // this thread's cells: columns j .. j+3 of rows r0 .. r0 + nrow - 1 of the strip
  const int tr = tid / CG, j = 4 * (tid - tr * CG);
  const int r0 = tr < a.TR ? tr * rows / a.TR : 0, nrow = tr < a.TR ? (tr + 1) * rows / a.TR - r0 : 0;
  // roles: 1 / 2 takes rows from and gives rows to the strip above / below; 4 / 8 owns row fs /
  // fs+1 (strip rows 0 and 1 below a free surface; the mirrored row fs-1 is row -1)
  int role = 0;
  if (nrow > 0) {
    if (r0 == 0 && rank > 0) role |= 1;
    if (r0 + nrow == rows && rank + 1 < a.G) role |= 2;
    if (g.fsurf && rank == 0 && r0 == 0) role |= 4;
    if (g.fsurf && rank == 0 && r0 <= 1 && r0 + nrow > 1) role |= 8;
  }
  const unsigned oc = (unsigned)g.L.off(i0 + r0, j);              // the first cell in a plane
  const unsigned lc = (unsigned)(r0 * SB + kGrp * (tid - tr * CG));  // from S
  const f2 c1 = pk(g.c1, g.c1), c2 = pk(g.c2, g.c2);
  const int nsteps = a.t1 - a.t0;
  unsigned land = 0;  // adjoint: parities of the next landings (bit 0: p, bit 1: divergence)
  if (ADJ) {
    if (tid == 0) {
      mbar_init(&bar[0], 1);
      mbar_init(&bar[1], 1);
      fence_barrier_init();
    }
    for (int r = tid; r < rows; r += T) rslot[r] = a.row_slot[beg + r];
  }
  if (tid == 0) *dead = 0;

  int wave = 0;
  for (int sh = slot; sh < g.ns; sh += a.S, ++wave) {
    const int64_t so = (int64_t)sh * PL;
    const unsigned tag0 = (unsigned)wave * (unsigned)nsteps + 1u;
    const float* const cf = a.cf + (int64_t)a.shot_model[sh] * a.cf_stride;
    // this strip's inbox (row slots of CG entries of four words); the neighbours' are one away
    const int64_t per = GLB ? (int64_t)kBoxRows * CG * 4 : 0;
    f2* const box = GLB ? a.box + ((int64_t)(wave & 1) * gridDim.x + blockIdx.x) * per : reinterpret_cast<f2*>(sm + a.oBox);
    __syncthreads();  // the previous shot's planes are no longer read
    for (int q = a.oS + tid; q < a.oRow; q += T) sm[q] = 0.0f;
    __syncthreads();
    if (a.s0 != nullptr) {  // the strip's state with its halo rows
      for (int q = tid; q < (rows + 4) * CG; q += T) {
        const int r = q / CG - 2, b = q - (r + 2) * CG, i = i0 + r;
        if (i < a.z0 || i >= g.L.nzp) continue;
        const int64_t o = g.L.off(i, 4 * b);
        float vp[4], vu[4], vw[4];
        ld4(a.s0 + so + o, vp);
        ld4(a.s0 + NSP + so + o, vu);
        ld4(a.s0 + 2 * NSP + so + o, vw);
        if (ADJ) {  // cells without a scale keep their lambda in the global planes
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            if (cf[ac::kA1M * PL + o + k] == 0.0f) vp[k] = 0.0f;
            if (cf[ac::kA2U * PL + o + k] == 0.0f) vu[k] = 0.0f;
            if (cf[ac::kA2W * PL + o + k] == 0.0f) vw[k] = 0.0f;
          }
        }
        float* d = S + r * SB + kGrp * b;
        if (r >= 0 && r < rows) st4(d, vu);
        st4(d + kW, vw);
        st4(d + kP, vp);
      }
      __syncthreads();
      if (role & 4) *reinterpret_cast<float4*>(S + lc + kW - SB) = *reinterpret_cast<const float4*>(S + lc + kW);  // w[fs-1] = w[fs]
    }
    for (int kept = 0; kept < 2; ++kept) {
      const int to = kept ? a.oA2 : a.oA1, plane = kept ? ac::kA2U : ac::kA1M;
      if (to != 0)
        for (int q = tid; q < rows * CG; q += T) {
          const int r = q / CG, c = 4 * (q - r * CG);
          float v[4];
          ldg4(cf + plane * PL + g.L.off(i0 + r, c), v);
          st4(sm + to + r * W4 + c, v);
        }
    }

    // bits of row q: 6+q damped; 12+q (phase 1) holds receivers (adjoint), (phase 2) the alpha2
    // masks of u and w differ; 24+q region cells with alpha = 0 (adjoint)
    unsigned m1 = 0, m2 = 0;
    int src = -1;  // the source cell, if this thread owns it: 4 row + column
    unsigned src_l = 0, src_o = 0;
    if (!ADJ) {
      const int sr = g.src_z[sh] - i0 - r0, sc = g.src_x[sh] - j;
      if (sr >= 0 && sr < nrow && sc >= 0 && sc < 4) {
        src = 4 * sr + sc;
        src_l = lc + sr * SB + kP + sc;
        src_o = oc + sr * g.L.pitch + sc;
      }
    }
    f2 s0[RB][2], s1[RB][2];
#pragma unroll
    for (int q = 0; q < RB; ++q) {
      s0[q][0] = s0[q][1] = s1[q][0] = s1[q][1] = 0ull;
      if (q >= nrow) continue;
      const int r = r0 + q;
      const int64_t o = oc + (int64_t)q * g.L.pitch;
      bool n1 = false, n2 = false, differ = false, z1 = false, z2 = false;
      for (int c = 0; c < 4; ++c) {
        n1 = n1 || cf[ac::kB1 * PL + o + c] != 1.0f;
        n2 = n2 || cf[ac::kB2 * PL + o + c] != 1.0f || cf[ac::kB3 * PL + o + c] != 1.0f;
        const float au = cf[ac::kA2U * PL + o + c], aw = cf[ac::kA2W * PL + o + c];
        differ = differ || !(au == aw);
        if (ADJ) {
          z1 = z1 || zero_in(ac::in_p(g, i0 + r, j + c), cf[ac::kA1M * PL + o + c]);
          z2 = z2 || zero_in(ac::in_u(g, i0 + r, j + c), au) || zero_in(ac::in_w(g, i0 + r, j + c), aw);
        }
      }
      m1 |= ((unsigned)n1 << 6 | (unsigned)(ADJ && rslot[r] != 0) << 12 | (unsigned)z1 << 24) << q;
      m2 |= ((unsigned)n2 << 6 | (unsigned)differ << 12 | (unsigned)z2 << 24) << q;
      if (SUMS && !a.first) {
        ldq(a.acc0 + so + o, s0[q]);
        ldq(a.acc1 + so + o, s1[q]);
      }
      if (ADJ && (z1 || z2)) {  // these cells' shares are added to the global planes step by step
        if (a.first) {
          stq(a.acc0 + so + o, s0[q]);
          stq(a.acc1 + so + o, s1[q]);
        }
        s0[q][0] = s0[q][1] = s1[q][0] = s1[q][1] = 0ull;
      }
    }
    const int64_t RS = (int64_t)sh * g.nt * g.nr;
    // adjoint: dL/d p-records of step it at the strip's receiver cells into one of two copies of
    // their rows, a step before they are needed
    auto inject = [&](int it, int copy) {
      const float* gr = a.rec_p + ((int64_t)sh * a.rnt + (it - a.r0)) * g.nr;
      for (int q = tid; q < nc; q += T) {
        float* d = sm + a.oInj + copy * a.injw + tpos[q];
        const int id = trid[q];
        if (id >= 0) {
          asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(d)), "l"(gr + id) : "memory");
        } else {
          float v = 0.0f;
          for (int m = a.srbeg[-1 - id]; m < a.srbeg[-id]; ++m) v += gr[a.srcv[m]];
          *d = v;
        }
      }
    };
    auto injected = [] { asm volatile("cp.async.wait_all;" ::: "memory"); };
    // adjoint: the histories' rows of a step into shared memory (one thread)
    auto fetch_p = [&](int it) {
      const float* h = a.hp + (int64_t)(it - a.h0) * NSP + so;
      const int lo_i = max(g.zbeg, i0 - 1), hi_i = min(g.L.nzp, i0 + rows + 2);
      mbar_arrive_expect_tx(&bar[0], (unsigned)(hi_i - lo_i) * CG * 16);
      for (int i = lo_i; i < hi_i; ++i) bulk_row(sm + a.oPH + (i - i0 + 1) * W4, h + g.L.off(i, 0), CG * 16, &bar[0]);
    };
    auto fetch_d = [&](int it) {
      const float* h = a.hd + (int64_t)(it - a.h0) * NSP + so;
      mbar_arrive_expect_tx(&bar[1], (unsigned)rows * CG * 16);
      for (int r = 0; r < rows; ++r) bulk_row(sm + a.oDH + r * W4, h + g.L.off(i0 + r, 0), CG * 16, &bar[1]);
    };
    auto landed = [&](int b) {
      if (!*dead && !mbar_wait(&bar[b], (land >> b) & 1u)) {
        raise_flag(a.flag, kErrWaitTimeout);
        *dead = 1;
      }
      land ^= 1u << b;
    };
    float sval = 0.0f;
    const int first_it = ADJ ? a.t1 - 1 : a.t0;
    if (!ADJ && src >= 0) sval = ac::rmul(g.dt, a.wav[(int64_t)sh * g.nt + first_it]);
    if (ADJ && a.rec_p != nullptr) {
      inject(first_it, 0);
      injected();
    }
    if (ADJ) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the zeroes above, before the copies
    __syncthreads();
    if (ADJ && tid == 0) {
      fetch_d(first_it);
      fetch_p(first_it);
    }
    if (!GLB) {  // every block's inbox is ready
      asm volatile("barrier.cluster.arrive.release;" ::: "memory");
      asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    }

    for (int k = 0; k < nsteps; ++k) {
      const int it = ADJ ? a.t1 - 1 - k : a.t0 + k;
      const int64_t ho = (int64_t)(it - a.h0) * NSP + so;
      float* const hp = a.hp + ho;  // (forward without histories: not used)
      float* const hd = a.hd + ho;
      const bool keep = !ADJ && a.hp != nullptr;
      // -------------------------------------------------------------- phase 1: p
      if (ADJ && a.rec_p != nullptr && k + 1 < nsteps) inject(it - 1, (k + 1) & 1);
      if (ADJ) landed(1);
      if ((role & 3) && k > 0) {
        const unsigned e = opaque((unsigned)j), tag = tag0 + (unsigned)k - 1u;
        float* d = S + kW + 3 * e;
        if (role & 1) {
          take_row<GLB>(box + e, tag, d - 2 * SB, a.flag, dead);
          take_row<GLB>(box + W4 + e, tag, d - SB, a.flag, dead);
        }
        if (role & 2) take_row<GLB>(box + 2 * W4 + e, tag, d + rows * SB, a.flag, dead);
      }
      if (nrow > 0) {
        f2 wa[2], wb[2], wc[2], wd[2];
        const unsigned m = opaque(m1);
        unsigned o = opaque(oc), lk = opaque((unsigned)(r0 * W4 + j));
        float* s = S + opaque(lc);
        ldq(s + kW - 2 * SB, wa);
        ldq(s + kW - SB, wb);
        ldq(s + kW, wc);
#pragma unroll
        for (int q = 0; q < RB; ++q) {
          if (q >= nrow) break;
          f2 uc[2], v[2], a1[2], x[2], dh[2], b1[2];
          factors((m >> (6 + q)) & 1u, cf + ac::kB1 * PL + o, b1);
          if (a.oA1 != 0) ldq(sm + a.oA1 + lk, a1); else ldgq(cf + ac::kA1M * PL + o, a1);
          if (ADJ) ldq(sm + a.oDH + lk, dh);
          float* const sn = s + SB;
          ldq(sn + kW, wd);
          const f2 ul = ldp(s - kGrp + 2);
          ldq(s, uc);
          const float ur = s[kGrp];
          ldq(s + kP, v);
          const f2 n0 = pk(hi(ul), lo(uc[0])), n1 = pk(hi(uc[0]), lo(uc[1])), n2 = pk(hi(uc[1]), ur);
          x[0] = div2<ADJ>(a.nz, c1, c2, uc[0], n0, n1, ul, wc[0], wb[0], wd[0], wa[0]);
          x[1] = div2<ADJ>(a.nz, c1, c2, uc[1], n1, n2, uc[0], wc[1], wb[1], wd[1], wa[1]);
          if (keep) stq(hd + o, x);
          v[0] = step2<ADJ>(a.nz, rmul2(b1[0], v[0], a.nz), a1[0], x[0]);
          v[1] = step2<ADJ>(a.nz, rmul2(b1[1], v[1], a.nz), a1[1], x[1]);
          stq(s + kP, v);
          if (keep) stq(hp + o, v);
          if (ADJ) {
            s0[q][0] = fma2(v[0], dh[0], s0[q][0]);
            s0[q][1] = fma2(v[1], dh[1], s0[q][1]);
          } else if (SUMS) {
            s0[q][0] = fma2(v[0], v[0], s0[q][0]);
            s0[q][1] = fma2(v[1], v[1], s0[q][1]);
          }
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            wa[c] = wb[c];
            wb[c] = wc[c];
            wc[c] = wd[c];
          }
          s = sn;
          lk += W4;
          o += g.L.pitch;
        }
      }
      if (!ADJ && src >= 0) {  // the source; its square's share of the sum goes with it
        const float v = S[src_l], n = ac::radd(v, sval), d = __fmaf_rn(n, n, -__fmul_rn(v, v));
        S[src_l] = n;
        if (keep) hp[src_o] = n;
        if (SUMS) {
          const f2 e = src & 1 ? pk(0.0f, d) : pk(d, 0.0f);
#pragma unroll
          for (int q = 0; q < RB; ++q)
            if (src >> 2 == q) {
              if (src & 2) s0[q][1] = add2(s0[q][1], e); else s0[q][0] = add2(s0[q][0], e);
            }
        }
      }
      if (ADJ && ((m1 >> 12) & 63u)) {  // V += alpha1 dL/drec, with its share of the sum
#pragma unroll
        for (int q = 0; q < RB; ++q)
          if ((m1 >> (12 + q)) & 1u) {
            const int r = r0 + q;
            f2 e[2], a1[2], v[2], dh[2];
            ldq(sm + a.oInj + (k & 1) * a.injw + ((rslot[r] - 1) * CG + (j >> 2)) * a.injg, e);
            ldgq(cf + ac::kA1M * PL + oc + q * g.L.pitch, a1);
            ldq(S + lc + q * SB + kP, v);
            ldq(sm + a.oDH + r * W4 + j, dh);
            v[0] = fma2(a1[0], e[0], v[0]);
            v[1] = fma2(a1[1], e[1], v[1]);
            stq(S + lc + q * SB + kP, v);
            e[0] = mul2(a1[0], e[0]);
            e[1] = mul2(a1[1], e[1]);
            s0[q][0] = fma2(e[0], dh[0], s0[q][0]);
            s0[q][1] = fma2(e[1], dh[1], s0[q][1]);
          }
      }
      if (role) {
        const unsigned e = opaque((unsigned)j), tag = tag0 + (unsigned)k;
        float* d = S + kP + 3 * e;
        if (role & 1) {
          put_row<GLB>(box - per + 4 * W4 + e, rank - 1, tag, d);
          put_row<GLB>(box - per + 5 * W4 + e, rank - 1, tag, d + SB);
        }
        if (role & 2) put_row<GLB>(box + per + 3 * W4 + e, rank + 1, tag, d + (rows - 1) * SB);
        if (role & 8) {  // p[fs-1] = -p[fs+1]
          const float4 v = *reinterpret_cast<const float4*>(d + SB), n = make_float4(-v.x, -v.y, -v.z, -v.w);
          *reinterpret_cast<float4*>(d - SB) = n;
          if (keep) *reinterpret_cast<float4*>(hp + g.L.off(i0 - 1, e)) = n;
        }
      }
      if (ADJ && (m1 >> 24)) {
        for (int q = 0; q < nrow; ++q)
          if ((m1 >> (24 + q)) & 1u) {
            const int r = r0 + q;
            zero_alpha_p(g, cf, PL, oc + (int64_t)q * g.L.pitch, i0 + r, j, S + lc + q * SB, SB, sm + a.oDH + r * W4 + j,
                         rslot[r] ? sm + a.oInj + (k & 1) * a.injw + ((rslot[r] - 1) * CG + (j >> 2)) * a.injg : nullptr, a.s1 + so, a.acc0 + so);
          }
      }
      __syncthreads();
      // -------------------------------------------------------------- phase 2: u, w
      if (ADJ && tid == 0 && k + 1 < nsteps) fetch_d(it - 1);
      if (!ADJ && src >= 0 && k + 1 < nsteps) sval = ac::rmul(g.dt, a.wav[(int64_t)sh * g.nt + it + 1]);
      if (!ADJ && a.rec_p != nullptr) {
        float* rr = a.rec_p + RS + (int64_t)it * g.nr;
        for (int q = tid; q < nc; q += T) {
          const int id = trid[q];
          const float v = S[kP + tpos[q]];
          if (id >= 0) {
            rr[id] = v;
          } else {
            for (int m = a.srbeg[-1 - id]; m < a.srbeg[-id]; ++m) rr[a.srcv[m]] = v;
          }
        }
      }
      if (ADJ) landed(0);
      if (role & 3) {
        const unsigned e = opaque((unsigned)j), tag = tag0 + (unsigned)k;
        float* d = S + kP + 3 * e;
        if (role & 1) take_row<GLB>(box + 3 * W4 + e, tag, d - SB, a.flag, dead);
        if (role & 2) {
          take_row<GLB>(box + 4 * W4 + e, tag, d + rows * SB, a.flag, dead);
          take_row<GLB>(box + 5 * W4 + e, tag, d + (rows + 1) * SB, a.flag, dead);
        }
      }
      if (ADJ && (m2 >> 24)) {
        for (int q = 0; q < nrow; ++q)
          if ((m2 >> (24 + q)) & 1u) {
            const int r = r0 + q;
            zero_alpha_uw(g, cf, PL, oc + (int64_t)q * g.L.pitch, i0 + r, j, S + lc + q * SB, SB,
                          sm + a.oPH + (r + 1) * W4 + j, W4, a.s1 + NSP + so, a.s1 + 2 * NSP + so, a.acc1 + so);
          }
      }
      if (nrow > 0) {
        f2 pa[2], pb[2], pc[2], pd[2];
        const unsigned m = opaque(m2);
        unsigned o = opaque(oc), lk = opaque((unsigned)(r0 * W4 + j));
        float* s = S + opaque(lc);
        ldq(s + kP - SB, pa);
        ldq(s + kP, pb);
        ldq(s + kP + SB, pc);
        const float* H = sm + a.oPH + W4 + lk;  // adjoint: the forward's pressure
        f2 ha[2], hb[2], hc[2], he[2];
        if (ADJ) {
          ldq(H - W4, ha);
          ldq(H, hb);
          ldq(H + W4, hc);
        }
#pragma unroll
        for (int q = 0; q < RB; ++q) {
          if (q >= nrow) break;
          f2 uo[2], wo[2], a2[2], un[2], wn[2], b2[2], b3[2];
          const bool damped = (m >> (6 + q)) & 1u;
          factors(damped, cf + ac::kB2 * PL + o, b2);
          factors(damped, cf + ac::kB3 * PL + o, b3);
          if (a.oA2 != 0) ldq(sm + a.oA2 + lk, a2); else ldgq(cf + ac::kA2U * PL + o, a2);
          ldq(s + kP + 2 * SB, pd);
          if (ADJ) ldq(H + 2 * W4, he);
          ldq(s, uo);
          ldq(s + kW, wo);
          if (ADJ) {
            const float hl = H[-1];
            const f2 hr = ldp(H + 4);
            const f2 n0 = pk(hl, lo(hb[0])), n1 = pk(hi(hb[0]), lo(hb[1])), n2 = pk(hi(hb[1]), lo(hr));
            s1[q][0] = fma2(uo[0], diff2<true>(0ull, c1, c2, n1, hb[0], hb[1], n0), s1[q][0]);
            s1[q][1] = fma2(uo[1], diff2<true>(0ull, c1, c2, n2, hb[1], hr, n1), s1[q][1]);
            s1[q][0] = fma2(wo[0], diff2<true>(0ull, c1, c2, hc[0], hb[0], he[0], ha[0]), s1[q][0]);
            s1[q][1] = fma2(wo[1], diff2<true>(0ull, c1, c2, hc[1], hb[1], he[1], ha[1]), s1[q][1]);
          }
          const float pl = s[kP - kGrp + 3];
          const f2 pr = ldp(s + kP + kGrp);
          const f2 n0 = pk(pl, lo(pb[0])), n1 = pk(hi(pb[0]), lo(pb[1])), n2 = pk(hi(pb[1]), lo(pr));
          un[0] = step2<ADJ>(a.nz, rmul2(b2[0], uo[0], a.nz), a2[0], diff2<ADJ>(a.nz, c1, c2, n1, pb[0], pb[1], n0));
          un[1] = step2<ADJ>(a.nz, rmul2(b2[1], uo[1], a.nz), a2[1], diff2<ADJ>(a.nz, c1, c2, n2, pb[1], pr, n1));
          if ((m >> (12 + q)) & 1u) ldgq(cf + ac::kA2W * PL + o, a2);
          wn[0] = step2<ADJ>(a.nz, rmul2(b3[0], wo[0], a.nz), a2[0], diff2<ADJ>(a.nz, c1, c2, pc[0], pb[0], pd[0], pa[0]));
          wn[1] = step2<ADJ>(a.nz, rmul2(b3[1], wo[1], a.nz), a2[1], diff2<ADJ>(a.nz, c1, c2, pc[1], pb[1], pd[1], pa[1]));
          stq(s, un);
          stq(s + kW, wn);
          if (SUMS && !ADJ && it >= a.accum_u) {
            s1[q][0] = fma2(un[0], un[0], s1[q][0]);
            s1[q][1] = fma2(un[1], un[1], s1[q][1]);
          }
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            pa[c] = pb[c];
            pb[c] = pc[c];
            pc[c] = pd[c];
            if (ADJ) {
              ha[c] = hb[c];
              hb[c] = hc[c];
              hc[c] = he[c];
            }
          }
          s += SB;
          lk += W4;
          o += g.L.pitch;
          if (ADJ) H += W4;
        }
      }
      if (role) {
        const unsigned e = opaque((unsigned)j), tag = tag0 + (unsigned)k;
        float* d = S + kW + 3 * e;
        if (role & 1) put_row<GLB>(box - per + 2 * W4 + e, rank - 1, tag, d);
        if (role & 2) {
          put_row<GLB>(box + per + e, rank + 1, tag, d + (rows - 2) * SB);
          put_row<GLB>(box + per + W4 + e, rank + 1, tag, d + (rows - 1) * SB);
        }
        if (role & 4) *reinterpret_cast<float4*>(d - SB) = *reinterpret_cast<const float4*>(d);  // w[fs-1] = w[fs]
      }
      if (ADJ) injected();
      __syncthreads();
      if (ADJ && tid == 0 && k + 1 < nsteps) fetch_p(it - 1);
      if (!ADJ && a.rec_u != nullptr) {  // u and w stay as they are until phase 2 of the next step
        float* ru = a.rec_u + RS + (int64_t)it * g.nr;
        float* rw = a.rec_w + RS + (int64_t)it * g.nr;
        for (int q = tid; q < nc; q += T) {
          const int id = trid[q];
          const float vu = S[tpos[q]], vw = S[kW + tpos[q]];
          if (id >= 0) {
            ru[id] = vu;
            rw[id] = vw;
          } else {
            for (int m = a.srbeg[-1 - id]; m < a.srbeg[-id]; ++m) {
              ru[a.srcv[m]] = vu;
              rw[a.srcv[m]] = vw;
            }
          }
        }
      }
    }

    // the state and the sums leave the chip
#pragma unroll
    for (int q = 0; q < RB; ++q) {
      if (q >= nrow) continue;
      const int64_t o = so + oc + (int64_t)q * g.L.pitch;
      const bool zero = ADJ && (((m1 | m2) >> (24 + q)) & 1u);
      if (a.s1 != nullptr) {
        float vp[4], vu[4], vw[4];
        const float* s = S + lc + q * SB;
        ld4(s, vu);
        ld4(s + kW, vw);
        ld4(s + kP, vp);
        if (zero) {  // cells without a scale already hold their lambda there
          for (int c = 0; c < 4; ++c) {
            const int64_t oo = oc + (int64_t)q * g.L.pitch + c;
            const int i = i0 + r0 + q;
            if (!zero_in(ac::in_p(g, i, j + c), cf[ac::kA1M * PL + oo])) a.s1[o + c] = vp[c];
            if (!zero_in(ac::in_u(g, i, j + c), cf[ac::kA2U * PL + oo])) a.s1[NSP + o + c] = vu[c];
            if (!zero_in(ac::in_w(g, i, j + c), cf[ac::kA2W * PL + oo])) a.s1[2 * NSP + o + c] = vw[c];
          }
        } else {
          st4(a.s1 + o, vp);
          st4(a.s1 + NSP + o, vu);
          st4(a.s1 + 2 * NSP + o, vw);
        }
      }
      if (SUMS) {
        if (zero) {
          f2 t[2];
          ldq(a.acc0 + o, t);
          s0[q][0] = add2(s0[q][0], t[0]);
          s0[q][1] = add2(s0[q][1], t[1]);
          ldq(a.acc1 + o, t);
          s1[q][0] = add2(s1[q][0], t[0]);
          s1[q][1] = add2(s1[q][1], t[1]);
        }
        stq(a.acc0 + o, s0[q]);
        stq(a.acc1 + o, s1[q]);
      }
    }
  }
  if (!GLB) {  // no block leaves while a neighbour may still write into its inbox
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
  }
}

}  // namespace res
}  // namespace adfwi
