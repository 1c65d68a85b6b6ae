// The coarsest level of the V-cycle takes some 50 Jacobi sweeps over a few
// thousand rows.  As launches of their own they were bound by launch and drain:
// the matrix is 1 to 3 MB, and each sweep depends on the one before it.  Here one
// cluster of 16 blocks makes them all: each block keeps its rows of A in
// shared memory and a copy of the whole of x, and sends its rows of the new x
// to the other blocks' copies with st.async, whose bytes complete on the
// receiver's barrier.  A sweep is then one exchange over distributed shared
// memory.  The restriction before it and the prolongation behind it ride along.
// A V-cycle with 50 sweeps takes 38 us less with 3,100 rows (110,000 nonzeros;
// 208 -> 170 us a CG iteration) and 74 us less with 6,000 (150,000; 350 -> 276).
#include "sweep.cuh"

#include <algorithm>
#include <cmath>

#include "cluster_dev.cuh"

namespace mgpbd {

namespace {

using namespace cdev;

constexpr int kSweepThreads = 1024;
constexpr int kSweepWarps = kSweepThreads / 32;
constexpr int kSweepBlocks = 16;
constexpr int kCutRows = 8;             // rows are handed out in groups of 8
constexpr uint32_t kPollLimit = 1 << 24;  // polls of a barrier before a wait gives up

struct SArgs {
  const CgState* st;
  const int32_t *indptr, *indices;
  const float *data, *dinv;
  const int32_t* cuts;  // blocks + 1 first rows
  const int32_t* qoff;  // first group of each row in its block
  const float* b;
  float* x;
  float w;
  const float* wp;
  SweepTransfer t;
  int32_t* status;
  int32_t n, npad, blocks, rows, quads, sweeps, zero_first;
};

extern __shared__ __align__(16) unsigned char s_mem[];

// G lanes of a warp share a row (32 / G rows a warp); a lane takes every G-th
// group of four elements.  Rows are padded to whole groups, the padding
// multiplies x[npad] = 0.
template <int G>
__global__ void __launch_bounds__(kSweepThreads, 1) k_sweeps(SArgs a) {
  if (a.st && a.st->done) return;
  constexpr int R = 32 / G;
  __shared__ __align__(8) unsigned long long s_bar[2];
  __shared__ int s_fail;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, gl = lane % G;
  uint32_t rank;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const int r0 = a.cuts[rank], nr = a.cuts[rank + 1] - r0;
  const int nx = a.npad + 4;
  float4* val = reinterpret_cast<float4*>(s_mem);
  uint2* idx = reinterpret_cast<uint2*>(val + a.quads);
  float2* bw = reinterpret_cast<float2*>(idx + a.quads);  // b, w / diagonal
  int2* rq = reinterpret_cast<int2*>(bw + a.rows);        // groups of a row
  float* xs = reinterpret_cast<float*>(rq + a.rows);      // x, two copies
  if (tid == 0) {
    s_fail = 0;
    for (int k = 0; k < 2; ++k)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&s_bar[k])) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (int i = tid; i < 2 * nx; i += kSweepThreads) xs[i] = 0.0f;
  const int tasks = nr / R;
  for (int t = wid; t < tasks; t += kSweepWarps) {
    const int row = t * R + lane / G, r = r0 + row;
    const bool in = r < a.n;
    const int k0 = in ? a.indptr[r] : 0, len = in ? a.indptr[r + 1] - k0 : 0;
    const int q0 = in ? a.qoff[r] : 0, nq = (len + 3) >> 2;
    if (gl == 0) rq[row] = make_int2(q0, q0 + nq);
    float* v = reinterpret_cast<float*>(val + q0);
    uint16_t* c = reinterpret_cast<uint16_t*>(idx + q0);
#pragma unroll 4
    for (int e = gl; e < 4 * nq; e += G) {
      const bool el = e < len;
      v[e] = el ? __ldg(a.data + k0 + e) : 0.0f;
      c[e] = static_cast<uint16_t>(el ? __ldg(a.indices + k0 + e) : a.npad);
    }
  }
  const float w = a.wp ? *a.wp : a.w;
  for (int row = tid; row < nr; row += kSweepThreads) {
    const int r = r0 + row;
    float b = 0.0f, wd = 0.0f;
    if (r < a.n) {
      if (a.t.r) {
        const int k1 = a.t.mem_ptr[r + 1];
#pragma unroll 4
        for (int k = a.t.mem_ptr[r]; k < k1; ++k) b += a.t.r[a.t.mem_rows[k]];
        a.t.b_out[r] = b;
      } else {
        b = a.b[r];
      }
      wd = w * a.dinv[r];
    }
    bw[row] = make_float2(b, wd);
  }
  __syncthreads();
  cluster_meet();  // every block's barriers and copies are ready for stores

  bool ok = true;
  // the whole of x after sweep s is in this block's copy s & 1
  auto wait_x = [&](int s) {
    if (!ok) return;
    const uint32_t bar = smem_u32(&s_bar[s & 1]), parity = (s - 1) >> 1 & 1;
    uint32_t n = 0;
    while (!test_phase(bar, parity))
      if (++n == kPollLimit) {
        ok = false;
        s_fail = 1;
        break;
      }
  };
  const uint32_t xs0 = smem_u32(xs);
#pragma unroll 1
  for (int s = 1; s <= a.sweeps; ++s) {
    const uint32_t bar = smem_u32(&s_bar[s & 1]);
    if (tid == 0) expect_bytes(bar, 4 * a.npad);
    if (s > 1) wait_x(s - 1);
    const float* x = xs + (s - 1 & 1) * nx;
    const bool first = s == 1 && a.zero_first;
    // A block that is here has the whole of sweep s - 1, so every block is
    // done with the copy of sweep s - 2 that these stores replace.
#pragma unroll 1
    for (int t = wid; t < tasks; t += kSweepWarps) {
      const int row = t * R + lane / G;
      const float2 f = bw[row];
      float y;
      if (first) {
        y = f.y * f.x;
      } else {
        const int2 q = rq[row];
        float sum = 0.0f;
        for (int k = q.x + gl; k < q.y; k += G) {
          const float4 v = val[k];
          const uint2 c = idx[k];
          sum += v.x * x[c.x & 0xffff];
          sum += v.y * x[c.x >> 16];
          sum += v.z * x[c.y & 0xffff];
          sum += v.w * x[c.y >> 16];
        }
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o, G);
        y = x[r0 + row] + f.y * (f.x - sum);
      }
      // four rows a store, a lane for each block (and half of the rows)
      const int h = R == 8 ? lane >> 4 : 0;
      const float y0 = __shfl_sync(0xffffffffu, y, (4 * h) * G),
                  y1 = __shfl_sync(0xffffffffu, y, (4 * h + 1) * G),
                  y2 = __shfl_sync(0xffffffffu, y, (4 * h + 2) * G),
                  y3 = __shfl_sync(0xffffffffu, y, (4 * h + 3) * G);
      const int to = lane & 15;
      if (to < a.blocks && (R == 8 || lane < 16))
        send_f4(map_rank(xs0 + 4 * ((s & 1) * nx + r0 + t * R + 4 * h), to), map_rank(bar, to), y0, y1,
                y2, y3);
    }
  }
  wait_x(a.sweeps);
  __syncthreads();
  const bool fail = s_fail != 0;
  const float* x = xs + (a.sweeps & 1) * nx;
  for (int row = tid; row < nr; row += kSweepThreads)
    if (r0 + row < a.n) a.x[r0 + row] = fail ? NAN : x[r0 + row];
  if (a.t.xf)
    for (int i = rank * kSweepThreads + tid; i < a.t.nf; i += a.blocks * kSweepThreads)
      a.t.xf[i] += fail ? NAN : x[a.t.agg[i]];
  if (fail) {
    if (tid == 0) atomicOr(reinterpret_cast<unsigned int*>(a.status), MGPBD_STATUS_SYNC_TIMEOUT);
    // stores to this block may still be on their way
    for (int k = 0; k < 50; ++k) __nanosleep(1000);
  }
  __syncthreads();
  cluster_meet();
}

using SweepFn = void (*)(SArgs);
SweepFn sweep_fn(int lanes) { return lanes == 8 ? k_sweeps<8> : k_sweeps<4>; }

void sweep_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute& at, int blocks, int smem,
                  cudaStream_t s) {
  cfg = {};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(kSweepThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = blocks;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
}

}  // namespace

void build_sweep_plan(const std::vector<int32_t>& indptr, int32_t n, SweepPlan& plan,
                      cudaStream_t s) {
  plan = SweepPlan();
  const int32_t npad = (n + kCutRows - 1) / kCutRows * kCutRows;
  if (n < 1 || npad + 4 > 65536) return;  // columns are 16-bit
  auto groups = [&](int32_t r) { return r < n ? (indptr[r + 1] - indptr[r] + 3) / 4 : 0; };
  const int lanes = static_cast<double>(indptr[n]) / n >= 48.0 ? 8 : 4;
  int dev = 0, limit = 0;
  MGPBD_CUDA(cudaGetDevice(&dev));
  MGPBD_CUDA(cudaDeviceGetAttribute(&limit, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  limit -= 1024;  // the static part
  const int blocks = kSweepBlocks;
  // cuts after equal shares of the groups, a row counted as two of them
  int64_t total = 0, at = 0;
  for (int32_t r = 0; r < n; ++r) total += groups(r) + 2;
  std::vector<int32_t> host(blocks + 1 + n);
  int32_t k = 1, q = 0, rows = 0, quads = 0;
  for (int32_t r = 0; r < npad; r += kCutRows) {
    while (k < blocks && at * blocks >= total * k) {
      host[k++] = r;
      q = 0;
    }
    for (int32_t i = r; i < std::min(n, r + kCutRows); ++i) {
      host[blocks + 1 + i] = q;
      q += groups(i);
      at += groups(i) + 2;
    }
    quads = std::max(quads, q);
  }
  while (k <= blocks) host[k++] = npad;
  quads += quads & 1;  // the copies of x behind them start on 16 bytes
  for (k = 0; k < blocks; ++k) rows = std::max(rows, host[k + 1] - host[k]);
  const int64_t smem = 24LL * quads + 16LL * rows + 8LL * (npad + 4);
  if (smem > limit) return;
  const void* fn = reinterpret_cast<const void*>(sweep_fn(lanes));
  MGPBD_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, limit));
  MGPBD_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr;
  sweep_config(cfg, attr, blocks, static_cast<int>(smem), s);
  int fit = 0;
  if (cudaOccupancyMaxActiveClusters(&fit, fn, &cfg) != cudaSuccess || fit < 1) {
    (void)cudaGetLastError();
    return;
  }
  plan.dev.alloc(static_cast<int64_t>(host.size()));
  MGPBD_CUDA(cudaMemcpyAsync(plan.dev.p, host.data(), sizeof(int32_t) * host.size(),
                             cudaMemcpyHostToDevice, s));
  MGPBD_CUDA(cudaStreamSynchronize(s));
  plan.blocks = blocks;
  plan.lanes = lanes;
  plan.rows = rows;
  plan.quads = quads;
  plan.smem = static_cast<int32_t>(smem);
}

void launch_sweeps(const CgState* st, const CsrView& a, const SweepPlan& plan, const float* b, float w,
                   const float* w_dev, int32_t sweeps, bool zero_first, float* x,
                   const SweepTransfer& t, int32_t* status, cudaStream_t s) {
  require(plan.blocks > 0 && sweeps >= 1, MGPBD_ESTATE, "no plan for the coarse sweeps");
  SArgs g = {};
  g.st = st;
  g.indptr = a.indptr;
  g.indices = a.indices;
  g.data = a.data;
  g.dinv = a.diag_inv;
  g.cuts = plan.dev.p;
  g.qoff = plan.dev.p + plan.blocks + 1;
  g.b = b;
  g.x = x;
  g.w = w;
  g.wp = w_dev;
  g.t = t;
  g.status = status;
  g.n = a.n;
  g.npad = (a.n + kCutRows - 1) / kCutRows * kCutRows;
  g.blocks = plan.blocks;
  g.rows = plan.rows;
  g.quads = plan.quads;
  g.sweeps = sweeps;
  g.zero_first = zero_first ? 1 : 0;
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr;
  sweep_config(cfg, attr, plan.blocks, plan.smem, s);
  MGPBD_CUDA(cudaLaunchKernelEx(&cfg, sweep_fn(plan.lanes), g));
  MGPBD_CHECK_LAUNCH();
}

}  // namespace mgpbd
