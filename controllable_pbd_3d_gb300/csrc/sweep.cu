// The coarsest level of the V-cycle takes some 50 Jacobi sweeps over a few
// thousand rows.  As launches of their own they were bound by launch and drain:
// the matrix is 1 to 3 MB, and each sweep depends on the one before it.  Here one
// cluster of 16 blocks makes them all: each block keeps its rows of A in
// shared memory with the x that they read, and sends its rows of the new x to
// the blocks that read them with st.async, whose bytes complete on the
// receiver's barrier.  A sweep is then one exchange over distributed shared
// memory: 0.7 us with 1,000 rows, 1.5 us with 6,000, where the reads of x from
// shared memory take as long.  (With the whole of x sent to every block the
// stores were the bound, 2.9 us with 6,000 rows.)  The restriction before it and the prolongation behind it ride along.
// 50 sweeps over 6,000 rows (144,000 nonzeros): 212 us as launches, 79 here.
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
constexpr int kCutRows = 16;  // rows are handed out in groups of 16
constexpr uint32_t kPollLimit = 1 << 24;  // polls of a barrier before a wait gives up

struct SArgs {
  const CgState* st;
  const int32_t* indptr;
  const float *data, *dinv;
  const int32_t* blk;   // SweepPlan::dev
  const int32_t* goff;  // first group of each row in its block
  const uint2* cols;
  const uint16_t* pos;
  const float* b;
  float* x;
  float w;
  const float* wp;
  SweepTransfer t;
  int32_t* status;
  int32_t n, blocks, rows, groups, nx, sweeps, zero_first;
};

extern __shared__ __align__(16) unsigned char s_mem[];

// G lanes of a warp share a row (32 / G rows a warp); a lane takes every G-th
// group of four elements.  Rows are padded to whole groups, the padding
// multiplies an x that stays 0.
//
// A block keeps the x that its rows read: its own rows, then the quads of rows
// that it receives.  Three copies: a block may send its x of sweep s to a
// block whose slower warps still read the x of sweep s - 2 (never s - 3: who
// sends to a block also receives from it, and a block has its own rows of
// sweep s - 1 only when all of them are done with s - 2).
template <int G>
__global__ void __launch_bounds__(kSweepThreads, 1) k_sweeps(SArgs a) {
  if (a.st && a.st->done) return;
  constexpr int R = 32 / G;
  __shared__ __align__(8) unsigned long long s_bar[3];
  __shared__ int s_fail;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, gl = lane % G;
  uint32_t rank;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const int r0 = a.blk[rank], nr = a.blk[rank + 1] - r0, recv = a.blk[a.blocks + 1 + rank];
  const int g0 = a.blk[2 * a.blocks + 1 + rank], ng = a.blk[2 * a.blocks + 2 + rank] - g0;
  float4* val = reinterpret_cast<float4*>(s_mem);
  float* xs = reinterpret_cast<float*>(val + a.groups);  // x, three copies
  uint2* idx = reinterpret_cast<uint2*>(xs + 3 * a.nx);
  float2* bw = reinterpret_cast<float2*>(idx + a.groups);  // b, w / diagonal
  int2* rg = reinterpret_cast<int2*>(bw + a.rows);         // groups of a row
  uint16_t* pos = reinterpret_cast<uint16_t*>(rg + a.rows);
  if (tid == 0) {
    s_fail = 0;
    for (int k = 0; k < 3; ++k)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&s_bar[k])) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (int i = tid; i < 3 * a.nx; i += kSweepThreads) xs[i] = 0.0f;
  for (int i = tid; i < ng; i += kSweepThreads) idx[i] = __ldg(a.cols + g0 + i);
  for (int i = tid; i < nr * kSweepBlocks / 4; i += kSweepThreads)
    pos[i] = __ldg(a.pos + r0 * (kSweepBlocks / 4) + i);
  const int tasks = nr / R;
  for (int t = wid; t < tasks; t += kSweepWarps) {
    const int row = t * R + lane / G, r = r0 + row;
    const bool in = r < a.n;
    const int k0 = in ? a.indptr[r] : 0, len = in ? a.indptr[r + 1] - k0 : 0;
    const int q0 = in ? a.goff[r] : 0, nq = (len + 3) >> 2;
    if (gl == 0) rg[row] = make_int2(q0, q0 + nq);
    float* v = reinterpret_cast<float*>(val + q0);
#pragma unroll 4
    for (int e = gl; e < 4 * nq; e += G) v[e] = e < len ? __ldg(a.data + k0 + e) : 0.0f;
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
  const uint32_t xs0 = smem_u32(xs);
  int to_slot = 0, slot = 0;  // of sweep s and s - 1: s % 3
  uint32_t parity = 0;        // of the barrier of sweep s - 1
#pragma unroll 1
  for (int s = 1; s <= a.sweeps; ++s) {
    slot = to_slot;
    to_slot = slot == 2 ? 0 : slot + 1;
    const bool last = s == a.sweeps;
    const uint32_t bar = smem_u32(&s_bar[to_slot]);
    if (tid == 0 && !last) expect_bytes(bar, 16 * recv);
    if (s > 1) {
      if (ok) {
        const uint32_t from = smem_u32(&s_bar[slot]);
        uint32_t n = 0;
        while (!try_phase(from, parity))
          if (++n == kPollLimit) {
            ok = false;
            s_fail = 1;
            break;
          }
      }
      if (slot == 0) parity ^= 1;  // (sweeps 1 to 3, 4 to 6, ...)
    }
    const float* x = xs + slot * a.nx;
    const bool first = s == 1 && a.zero_first;
#pragma unroll 1
    for (int t = wid; t < tasks; t += kSweepWarps) {
      const int row = t * R + lane / G;
      const float2 f = bw[row];
      float y;
      if (first) {
        y = f.y * f.x;
      } else {
        const int2 q = rg[row];
        float sum = 0.0f;
#pragma unroll 1  // (unrolled by two: 10 % slower)
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
        y = x[row] + f.y * (f.x - sum);
      }
      if (last) {
        if (gl == 0) xs[to_slot * a.nx + row] = y;
        continue;
      }
      // four rows a store, half a warp for the blocks
      const int to = lane & 15;
#pragma unroll
      for (int i = 0; i < (R + 7) / 8; ++i) {
        const int h = R == 4 ? 0 : 2 * i + (lane >> 4);
        const float y0 = __shfl_sync(0xffffffffu, y, (4 * h) * G),
                    y1 = __shfl_sync(0xffffffffu, y, (4 * h + 1) * G),
                    y2 = __shfl_sync(0xffffffffu, y, (4 * h + 2) * G),
                    y3 = __shfl_sync(0xffffffffu, y, (4 * h + 3) * G);
        const uint32_t p = pos[(t * R / 4 + h) * kSweepBlocks + to];
        if (p != kSweepNone && (R > 4 || lane < 16))
          send_f4(map_rank(xs0 + 4 * (to_slot * a.nx + 4 * p), to), map_rank(bar, to), y0, y1, y2, y3);
      }
    }
  }
  __syncthreads();
  const bool fail = s_fail != 0;
  const float* x = xs + to_slot * a.nx;
  for (int row = tid; row < nr; row += kSweepThreads)
    if (r0 + row < a.n) a.x[r0 + row] = fail ? NAN : x[row];
  if (a.t.xf) {
    constexpr int kL = 4;  // lanes of a row's members
    for (int i = tid; i < kL * nr; i += kSweepThreads) {
      const int row = i / kL;
      if (r0 + row >= a.n) continue;
      const float v = fail ? NAN : x[row];
      const int k1 = a.t.mem_ptr[r0 + row + 1];
#pragma unroll 4
      for (int k = a.t.mem_ptr[r0 + row] + i % kL; k < k1; k += kL) a.t.xf[a.t.mem_rows[k]] += v;
    }
  }
  if (fail) {
    if (tid == 0) atomicOr(reinterpret_cast<unsigned int*>(a.status), MGPBD_STATUS_SYNC_TIMEOUT);
    // stores to this block may still be on their way
    for (int k = 0; k < 50; ++k) __nanosleep(1000);
  }
  __syncthreads();
  cluster_meet();
}

using SweepFn = void (*)(SArgs);
SweepFn sweep_fn(int lanes) { return lanes == 8 ? k_sweeps<8> : lanes == 4 ? k_sweeps<4> : k_sweeps<2>; }

// Lanes of a row: a warp's rounds over its rows, each with a fixed part (the
// sums, the stores) and a part for each group of a lane.  Fitted to 50 sweeps
// with 2 / 4 / 8 lanes (us): 1,000 rows of 22: 46 / 40 / 42; 1,000 of 71: 81 /
// 69 / 65; 3,138 of 27: 97 / 92 / 100; 5,985 of 24: 80 / 92 / 129; 10,648 of
// 25: 130 / 141 / 201.
int sweep_lanes(int32_t n, int64_t nnz) {
  int best = 2;
  double least = 1e300;
  for (int g = 2; g <= 8; g *= 2) {
    const int rounds = ceil_div(static_cast<int64_t>(ceil_div(n, kSweepBlocks)) * g, 32 * kSweepWarps);
    const double cost = rounds * ((g == 8 ? 30.0 : 18.0) + 8.0 * ceil_div(ceil_div(nnz, 4LL * n), g));
    if (cost < least) {
      least = cost;
      best = g;
    }
  }
  return best;
}

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

void build_sweep_plan(const std::vector<int32_t>& indptr, const std::vector<int32_t>& indices,
                      int32_t n, SweepPlan& plan, cudaStream_t s) {
  plan = SweepPlan();
  if (n < 1 || indptr[n] > kSweepMaxNnz) return;
  constexpr int nb = kSweepBlocks;
  int dev = 0, limit = 0;
  MGPBD_CUDA(cudaGetDevice(&dev));
  MGPBD_CUDA(cudaDeviceGetAttribute(&limit, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  limit -= 1024;  // the static part
  auto n_groups = [&](int32_t r) { return (indptr[r + 1] - indptr[r] + 3) / 4; };
  const int lanes = sweep_lanes(n, indptr[n]);
  const int32_t npad = (n + kCutRows - 1) / kCutRows * kCutRows;
  // cuts after equal shares of the groups, a row counted as two of them
  int64_t total = 0, at = 0;
  for (int32_t r = 0; r < n; ++r) total += n_groups(r) + 2;
  std::vector<int32_t> host(3 * nb + 2 + n);
  int32_t *cut = host.data(), *recv = cut + nb + 1, *first = recv + nb, *goff = first + nb + 1;
  int32_t k = 1, q = 0, all = 0;
  for (int32_t r = 0; r < npad; r += kCutRows) {
    while (k < nb && at * nb >= total * k) {
      cut[k] = r;
      first[k++] = all;
      q = 0;
    }
    for (int32_t i = r; i < std::min(n, r + kCutRows); ++i) {
      goff[i] = q;
      q += n_groups(i);
      all += n_groups(i);
      at += n_groups(i) + 2;
    }
  }
  for (; k <= nb; ++k) {
    cut[k] = npad;
    first[k] = all;
  }
  // the quads of rows that each block reads, and where it keeps them: its own
  // first, then in the order of their first use
  std::vector<uint16_t> pos(static_cast<size_t>(npad) / 4 * nb, kSweepNone);
  auto keep = [&](int32_t quad, int32_t b) {
    uint16_t& p = pos[static_cast<size_t>(quad) * nb + b];
    if (p == kSweepNone) p = static_cast<uint16_t>(recv[b]++);
    return p;
  };
  for (int32_t b = 0; b < nb; ++b)
    if ((cut[b + 1] - cut[b]) / 4 + 1 >= kSweepNone / 4) return;
  for (int32_t b = 0; b < nb; ++b)
    for (int32_t i = cut[b] / 4; i < cut[b + 1] / 4; ++i) keep(i, b);
  std::vector<bool> reads(nb * nb);  // [b * nb + o]: block b receives from block o
  for (int32_t b = 0; b < nb; ++b)
    for (int32_t r = cut[b]; r < std::min(n, cut[b + 1]); ++r)
      for (int32_t e = indptr[r]; e < indptr[r + 1]; ++e) {
        if (recv[b] >= kSweepNone / 4 - 2) return;  // positions are 16-bit
        keep(indices[e] / 4, b);
      }
  for (int32_t quad = 0, o = 0; quad < npad / 4; ++quad) {
    while (4 * quad >= cut[o + 1]) ++o;
    for (int32_t b = 0; b < nb; ++b)
      if (pos[static_cast<size_t>(quad) * nb + b] != kSweepNone) reads[b * nb + o] = true;
  }
  for (int32_t b = 0; b < nb; ++b)
    for (int32_t o = 0; o < nb; ++o)
      if (reads[b * nb + o] && !reads[o * nb + b]) keep(cut[b] / 4, o);  // who sends also receives
  int32_t rows = 0, groups = 0, quads = 0;
  for (int32_t b = 0; b < nb; ++b) {
    rows = std::max(rows, cut[b + 1] - cut[b]);
    groups = std::max(groups, first[b + 1] - first[b]);
    quads = std::max(quads, recv[b]);
  }
  const int32_t nx = 4 * (quads + 1);  // (the last four stay 0)
  const int64_t smem = 24LL * groups + (16LL + 2 * nb / 4) * rows + 12LL * nx;
  if (smem > limit || nx > 65536) return;
  std::vector<uint16_t> cols(4LL * std::max(all, 1), static_cast<uint16_t>(nx - 1));
  for (int32_t b = 0; b < nb; ++b)
    for (int32_t r = cut[b]; r < std::min(n, cut[b + 1]); ++r)
      for (int32_t e = indptr[r]; e < indptr[r + 1]; ++e)
        cols[4LL * (first[b] + goff[r]) + e - indptr[r]] = static_cast<uint16_t>(
            4 * pos[static_cast<size_t>(indices[e] / 4) * nb + b] + indices[e] % 4);
  const void* fn = reinterpret_cast<const void*>(sweep_fn(lanes));
  MGPBD_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, limit));
  MGPBD_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr;
  sweep_config(cfg, attr, nb, static_cast<int>(smem), s);
  int fit = 0;
  if (cudaOccupancyMaxActiveClusters(&fit, fn, &cfg) != cudaSuccess || fit < 1) {
    (void)cudaGetLastError();
    return;
  }
  plan.dev.alloc(static_cast<int64_t>(host.size()));
  plan.cols.alloc(static_cast<int64_t>(cols.size()));
  plan.pos.alloc(static_cast<int64_t>(pos.size()));
  MGPBD_CUDA(cudaMemcpyAsync(plan.dev.p, host.data(), sizeof(int32_t) * host.size(),
                             cudaMemcpyHostToDevice, s));
  MGPBD_CUDA(cudaMemcpyAsync(plan.cols.p, cols.data(), sizeof(uint16_t) * cols.size(),
                             cudaMemcpyHostToDevice, s));
  MGPBD_CUDA(cudaMemcpyAsync(plan.pos.p, pos.data(), sizeof(uint16_t) * pos.size(),
                             cudaMemcpyHostToDevice, s));
  MGPBD_CUDA(cudaStreamSynchronize(s));
  plan.blocks = nb;
  plan.lanes = lanes;
  plan.rows = rows;
  plan.groups = groups;
  plan.nx = nx;
  plan.smem = static_cast<int32_t>(smem);
}

void launch_sweeps(const CgState* st, const CsrView& a, const SweepPlan& plan, const float* b, float w,
                   const float* w_dev, int32_t sweeps, bool zero_first, float* x,
                   const SweepTransfer& t, int32_t* status, cudaStream_t s) {
  require(plan.blocks > 0 && sweeps >= 1, MGPBD_ESTATE, "no plan for the coarse sweeps");
  SArgs g = {};
  g.st = st;
  g.indptr = a.indptr;
  g.data = a.data;
  g.dinv = a.diag_inv;
  g.blk = plan.dev.p;
  g.goff = plan.dev.p + 3 * plan.blocks + 2;
  g.cols = reinterpret_cast<const uint2*>(plan.cols.p);
  g.pos = plan.pos.p;
  g.b = b;
  g.x = x;
  g.w = w;
  g.wp = w_dev;
  g.t = t;
  g.status = status;
  g.n = a.n;
  g.blocks = plan.blocks;
  g.rows = plan.rows;
  g.groups = plan.groups;
  g.nx = plan.nx;
  g.sweeps = sweeps;
  g.zero_first = zero_first ? 1 : 0;
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr;
  sweep_config(cfg, attr, plan.blocks, plan.smem, s);
  MGPBD_CUDA(cudaLaunchKernelEx(&cfg, sweep_fn(plan.lanes), g));
  MGPBD_CHECK_LAUNCH();
}

}  // namespace mgpbd
