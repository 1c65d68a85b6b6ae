// Jacobi sweeps on the coarsest multigrid level by one thread-block cluster
// (sweep.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

#include "common.h"
#include "kernels.cuh"

namespace mgpbd {

// How a matrix is spread over the cluster.  blocks == 0: it is not (it does
// not fit into the blocks' shared memory).
struct SweepPlan {
  int32_t blocks = 0, threads = 0, lanes = 0;  // of the cluster, a block, a row
  int32_t rows = 0, steps = 0, nx = 0;  // the most rows, steps and x of a block
  int32_t smem = 0;
  DevBuf<int32_t> dev;    // first row of each block and the end; quads of x it receives
  DevBuf<int32_t> step;   // first step of each task (a warp's rows)
  DevBuf<int32_t> src;    // [step][lane][4]: element of the matrix, -1: padding
  DevBuf<uint16_t> cols;  // and its column, as a byte offset in the block's x
  DevBuf<uint16_t> pos;   // where each block keeps a quad of rows (kSweepNone: nowhere)
};
constexpr uint16_t kSweepNone = 0xffff;
constexpr int64_t kSweepMaxNnz = 1 << 20;  // the values of more exceed 16 blocks' shared memory

// The plan of a matrix of n rows (host structure).
void build_sweep_plan(const std::vector<int32_t>& indptr, const std::vector<int32_t>& indices,
                      int32_t n, SweepPlan& plan, cudaStream_t s);

// What surrounds the sweeps: r (not null): their b is the sum of r over each
// row's members (k_restrict), left in b_out; xf (not null): x of each row is
// added to xf of its members afterwards (k_prolong_add).
struct SweepTransfer {
  const float* r = nullptr;
  float* b_out = nullptr;
  const int32_t *mem_ptr = nullptr, *mem_rows = nullptr;
  float* xf = nullptr;
};

// x = `sweeps` sweeps x += w D^-1 (b - A x) from x = 0, w from w_dev when not
// null; zero_first: the first sweep is written down as w D^-1 b.  A no-op
// once st->done.  A wait longer than spin_limit_s leaves NaN in the x (and xf)
// of the blocks that gave up and 1 in *timed_out (pinned host memory).
void launch_sweeps(const CgState* st, const CsrView& a, const SweepPlan& plan, const float* b, float w,
                   const float* w_dev, int32_t sweeps, bool zero_first, float* x,
                   const SweepTransfer& t, double spin_limit_s, int32_t* timed_out, cudaStream_t s);

}  // namespace mgpbd
