// Resident acoustic time loop, host side: shared-memory layout, arguments and compiled variants
// (the time loop itself is in acoustic_res.cuh, compiled by acoustic_res_fwd.cu and
// acoustic_res_adj.cu).
#pragma once
#include "acoustic_geo.cuh"

namespace adfwi {
namespace res {

constexpr int kMaxCluster = 16;
constexpr int kBoxRows = 6;           // rows that a strip takes from its neighbours: w -2, -1, R; p -1, R, R+1
constexpr int kHeadWords = 16;        // two mbarriers and the block's give-up mark
// Shared-memory layout of the state: the four columns of a thread's group lie together, U, W, P
// (12 words: a stride of 3 x 16 bytes has no bank conflicts), so one address with constant
// offsets reaches everything of a row. Rows are 12 (CG + 1) words apart: the spare group is the
// zero ghost on both sides. Rows -2 .. R+1 exist.
constexpr int kGrp = 12, kW = 4, kP = 8;

struct ResArgs {
  int G, S, NR, z0, TR, CG;  // blocks per shot, shots at a time, rows and the first of them, thread rows, column groups
  int oS, oA1, oA2, oPH, oDH, oBox, oInj, injw, injg, oRow, oT;  // shared memory, in words (oA1, oA2: 0 = not kept)
  int t0, t1;                 // steps t0 .. t1-1 (the adjoint runs them downwards)
  int h0;                     // step of history slot 0
  int accum_u;                // first step whose u^2 is summed
  int first;                  // the sums start at zero (else from acc0 / acc1)
  const float* cf;            // coefficient block of model 0; model m at cf + m * cf_stride
  int64_t cf_stride;
  const int* shot_model;
  const float* wav;
  const float* s0;            // state in: p, u, w blocks of ns planes (null: zero)
  float* s1;                  // state out (null: dropped)
  float* hp;                  // histories (forward: written if not null; adjoint: read)
  float* hd;
  float* rec_p;               // forward: records written; adjoint: dL/d p-records read
  int r0, rnt;                // adjoint: first step and steps per shot of rec_p
  float* rec_u;
  float* rec_w;
  float* acc0;                // sums over time per shot: ns planes each
  float* acc1;
  const int* row_slot;        // adjoint: per row from z0, 1 + the row of dL/d records of its strip (0: no receivers)
  const int* strip_beg;       // G+1 offsets into the unique receiver cells, sorted by (row, column)
  const int* tpos;            // where each cell is: from the strip's first cell (forward), in its rows of dL/d records (adjoint)
  const int* trid;            // its receiver, or -1 - cell
  const int* srbeg;           // ncells+1 offsets into srcv
  const int* srcv;            // receiver ids grouped by cell
  unsigned long long* box;    // inboxes of the strips (global exchange), zeroed before the launch
  int* flag;
  unsigned long long nz;      // a pair of -0 (rmul2)
};

using ResKernel = void (*)(const ac::Geo<float>, const ResArgs);

// Rows per thread and most threads of a block of each compiled variant (2 rows: the
// forward loop only; 384 threads, 168 registers each: the adjoint only).
// (Registers decide: the sums over time take 8 per row beside some 90 of the stencils, and what
// spills goes to L2, the L1 being shared memory.)
constexpr int kVariants[][2] = {{2, 512}, {3, 512}, {3, 768}, {4, 512}, {4, 640}, {6, 384}, {6, 512}};
// The variant's kernel (glb: strips of a cooperative launch instead of a cluster; sums: the
// illumination is summed).
ResKernel forward_kernel(int rb, int mt, bool sums, bool glb);
ResKernel adjoint_kernel(int rb, int mt, bool glb);
int row_wait_selftest(int64_t limit_ns, int* flag, float* row, cudaStream_t st);

}  // namespace res
}  // namespace adfwi
