// The dual Chebyshev-CG of FAST mode on a spatial partition of the
// constraints (dcg.cu; the partition is built on the host by dcg_plan.cpp).
//
// A solve is cut into blocks that own compact sets of constraints (recursive
// bisection of their centroids).  A block keeps the vector A is applied to
// and the velocities u of the vertices its constraints touch in shared
// memory, so both gathers of A x = J W J^T x + alpha~ x are shared-memory
// reads, and only the sums of vertices on the boundary between blocks travel:
// one meeting with its neighbours per application of A.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <utility>
#include <vector>

#include "dcg_plan.h"
#include "jform.cuh"

namespace mgpbd {

// Device arrays of a plan and its per-solve data
struct DcgDev {
  const DBlock* blocks = nullptr;
  const int32_t* perm = nullptr;
  const uint2* ti = nullptr;
  const int32_t* pos_v = nullptr;
  const uint2* pos_info = nullptr;
  const uint32_t* tgt = nullptr;
  const uint2* slice = nullptr;
  const int32_t* row_ent = nullptr;
  const uint16_t* row_idx = nullptr;
  const DWarp* warps = nullptr;
  unsigned char* rows = nullptr;  // kDRow bytes each
  float4* tg = nullptr;           // 3 planes of nc float4 (length constraints: plane 0 only)
  float2* ad = nullptr;           // (nc) alpha~ (as of the solve), 1/diag in plan order
  float* x = nullptr;             // (nc) CG vectors in plan order
  float* xc = nullptr;
  float* r = nullptr;
  float* d = nullptr;
  float* p = nullptr;
  float4* exch = nullptr;         // 2 buffers of n_slots
  int64_t n_slots = 0;
  uint4* partials = nullptr;      // grid: 2 x 3 planes of nblk tagged partials, after exch
  uint32_t* gflag = nullptr;      // 1: some slot-0 gradient is not minus the sum of the others
  int32_t nc = 0, n4 = 0;         // n4: first length constraint (original order)
};

// Gradients, compliances and 1/diag in plan order, once per Newton iteration
void launch_dcg_pack(const JView& j, const DcgDev& d, int64_t n_rows, cudaStream_t s);

// The whole solve; b, x, r and xc as in launch_jcg_persistent (original
// order: x + xc is the solution, r its residual).  iters (nprob): each
// problem's iterations, or null.  per_problem: a problem with b = 0 has
// x = 0 at once (a body whose Newton loop has ended).  estimate: each problem's
// Chebyshev interval [1.02 lmax lo_ratio, 1.02 lmax] comes from Lanczos steps of
// its own first (problem 0's is left in js->cf); otherwise it is that of js->cf.
void launch_dcg(const JView& j, const JcgVecs& v, const DcgPlan& plan, const DcgDev& d,
                JState* js, CgState* st, double tol_abs, double tol_rel, int maxiter, int degree,
                double lo_ratio, bool estimate, bool warm, bool per_problem, int32_t* iters,
                double spin_limit_s, cudaStream_t s, const JcgCtl* ctl = nullptr);

// A mesh of at most this many vertex entries (4 per 4-slot, 2 per length
// constraint) runs on one cluster of 16 blocks, a larger one on the whole
// grid.  A cluster's exchanges go through distributed shared memory, a grid's
// through L2, but it has a tenth of the SMs.  Measured on cubes of n^3 hexes, us
// per CG iteration cluster / grid, length + volume: n = 10 (34k entries) 27 / 34,
// 14 (91k) 35 / 33, 17 (163k) 43 / 35, 20 (263k) 73 / 37; on another box the grid
// took 39 / 40 / 38 / 39 of these.  ARAP: 10 (20k) 23 / 32, 14 (55k) 27 / 30, 17
// (98k) 31 / 32, 18 (117k) 36 / 32, 20 (160k) 42 / 33.
constexpr double kDClusterEntries = 120e3;
// From this many constraints a block on it runs 768 threads, below 512: more
// warps hide more of the shared-memory latency, fewer have less to issue
// besides the constraints.  us per CG iteration at 512 / 768 threads, 600
// constraints a block 39.4 / 41.7, 1600: 45.0 / 46.2, 4700: 70.8 / 67.2.
constexpr double kDWideConstraints = 3000.0;

// Dynamic shared memory a block of the kernel may use on this device (and the
// kernel's attributes set for it): before a plan is built or launched there.
int dcg_smem_limit();
// The most clusters of `size` blocks that are resident at once (0: none).
int dcg_max_clusters(int size, int threads, int smem);

}  // namespace mgpbd
