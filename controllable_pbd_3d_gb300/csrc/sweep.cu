// The coarsest level of the V-cycle takes some 50 Jacobi sweeps over a few
// thousand rows.  As launches of their own they were bound by launch and drain:
// the matrix is 1 to 3 MB, and each sweep depends on the one before it.  Here one
// cluster of 16 blocks makes them all: each block keeps its rows of A in
// shared memory with the x that they read, and sends its rows of the new x to
// the blocks that read them with st.async, whose bytes complete on the
// receiver's barrier.  A sweep is then one exchange over distributed shared
// memory: 0.65 us with 1,000 rows, 1.2 us with 6,000, where the reads from
// shared memory take as long.  (With the whole of x sent to every block the
// stores were the bound, 2.9 us with 6,000 rows; with the elements of a row in
// the matrix's order the banks were, 1.5 us.)  The restriction before it and the prolongation behind it ride along.
// 50 sweeps over 6,000 rows (144,000 nonzeros): 212 us as launches, 64 here.
#include "sweep.cuh"

#include <algorithm>
#include <cmath>
#include <utility>

#include "cluster_dev.cuh"
#include "persist.cuh"

namespace mgpbd {

namespace {

using namespace cdev;

constexpr int kSweepThreads = 1024;
constexpr int kSweepWarps = kSweepThreads / 32;
constexpr int kSweepBlocks = 16;
constexpr int kCutRows = 16;  // rows are handed out in groups of 16

struct SArgs {
  const CgState* st;
  const float *data, *dinv;
  const int32_t* blk;  // SweepPlan::dev
  const int32_t* step;
  const int32_t* src;
  const uint2* cols;
  const uint16_t* pos;
  const float* b;
  float* x;
  float w;
  const float* wp;
  SweepTransfer t;
  int32_t* timed_out;
  unsigned long long spin_ns;
  int32_t n, blocks, rows, steps, nx, sweeps, zero_first;
};

extern __shared__ __align__(16) unsigned char s_mem[];

// Waits for a phase of a barrier; false when the limit is reached or another
// warp of the block has given up.  A limit of 0 gives up at the first poll that
// finds the phase incomplete.
__device__ __forceinline__ bool wait_phase(uint32_t bar, uint32_t parity, unsigned long long limit,
                                           volatile int* fail) {
  if (limit == 0) return test_phase(bar, parity);
  unsigned long long t0 = 0;
  for (uint32_t n = 1; !try_phase(bar, parity); ++n) {
    if (n % 64 != 0) continue;
    const unsigned long long t = pdev::global_ns();
    if (t0 == 0) t0 = t;
    if (*fail != 0 || t - t0 > limit) return false;
  }
  return true;
}

// G lanes of a warp share a row (32 / G rows a warp, a task).  In each step a
// lane multiplies four elements, in the order that the plan found: the 32 reads
// of x that go out together shall fall on different banks.  The padding
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
  const int nthr = blockDim.x, nw = nthr >> 5;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, gl = lane % G;
  uint32_t rank;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const int r0 = a.blk[rank], nr = a.blk[rank + 1] - r0, recv = a.blk[a.blocks + 1 + rank];
  const int t0 = r0 / R, s0 = a.step[t0], ng = 32 * (a.step[t0 + nr / R] - s0);
  float4* val = reinterpret_cast<float4*>(s_mem);           // [step][lane]
  float* xs = reinterpret_cast<float*>(val + 32 * a.steps);  // x, three copies
  uint2* idx = reinterpret_cast<uint2*>(xs + 3 * a.nx);      // byte offsets in x
  float2* bw = reinterpret_cast<float2*>(idx + 32 * a.steps);  // b, w / diagonal
  int* first_step = reinterpret_cast<int*>(bw + a.rows);
  uint16_t* pos = reinterpret_cast<uint16_t*>(first_step + a.rows / R + 1);
  if (tid == 0) {
    s_fail = 0;
    for (int k = 0; k < 3; ++k)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&s_bar[k])) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (int i = tid; i < 3 * a.nx; i += nthr) xs[i] = 0.0f;
  for (int i = tid; i < ng; i += nthr) idx[i] = __ldg(a.cols + 32 * s0 + i);
  for (int i = tid; i < 4 * ng; i += nthr) {
    const int e = __ldg(a.src + 128 * s0 + i);
    reinterpret_cast<float*>(val)[i] = e >= 0 ? __ldg(a.data + e) : 0.0f;
  }
  for (int i = tid; i < nr * kSweepBlocks / 4; i += nthr)
    pos[i] = __ldg(a.pos + r0 * (kSweepBlocks / 4) + i);
  const int tasks = nr / R;
  for (int t = tid; t <= tasks; t += nthr) first_step[t] = 32 * (a.step[t0 + t] - s0);
  const float w = a.wp ? *a.wp : a.w;
  for (int row = tid; row < nr; row += nthr) {
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

  const uint32_t xs0 = smem_u32(xs);
  int to_slot = 0, slot = 0;  // of sweep s and s - 1: s % 3
  uint32_t parity = 0;        // of the barrier of sweep s - 1
  // Only warps with rows take part.  A phase of a block's barrier completes
  // with the rows of all of them, so none of them falls behind by more than one
  // sweep; a warp without rows holds nothing back, and three sweeps behind
  // it would find the parity that it waits for turned over.
#pragma unroll 1
  for (int s = 1; s <= a.sweeps && wid < tasks; ++s) {
    slot = to_slot;
    to_slot = slot == 2 ? 0 : slot + 1;
    const bool last = s == a.sweeps;
    const uint32_t bar = smem_u32(&s_bar[to_slot]);
    if (tid == 0 && !last) expect_bytes(bar, 16 * recv);
    if (s > 1) {
      const bool ok = wait_phase(smem_u32(&s_bar[slot]), parity, a.spin_ns, &s_fail);
      if (!__all_sync(0xffffffffu, ok)) {  // no more arrivals, no more stores
        s_fail = 1;
        break;
      }
      if (slot == 0) parity ^= 1;  // (sweeps 1 to 3, 4 to 6, ...)
    }
    const float* x = xs + slot * a.nx;
    const bool first = s == 1 && a.zero_first;
#pragma unroll 1
    for (int t = wid; t < tasks; t += nw) {
      const int row = t * R + lane / G;
      const float2 f = bw[row];
      float y;
      if (first) {
        y = f.y * f.x;
      } else {
        const int k1 = first_step[t + 1];
        const char* xb = reinterpret_cast<const char*>(x);
        auto at = [&](uint32_t o) { return *reinterpret_cast<const float*>(xb + o); };
        float sum = 0.0f;
#pragma unroll 1
        for (int k = first_step[t] + lane; k < k1; k += 32) {
          const float4 v = val[k];
          const uint2 c = idx[k];
          sum += v.x * at(c.x & 0xffff);
          sum += v.y * at(c.x >> 16);
          sum += v.z * at(c.y & 0xffff);
          sum += v.w * at(c.y >> 16);
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
  const float* x = xs + a.sweeps % 3 * a.nx;
  for (int row = tid; row < nr; row += nthr)
    if (r0 + row < a.n) a.x[r0 + row] = fail ? NAN : x[row];
  if (a.t.xf) {
    constexpr int kL = 4;  // lanes of a row's members
    for (int i = tid; i < kL * nr; i += nthr) {
      const int row = i / kL;
      if (r0 + row >= a.n) continue;
      const float v = fail ? NAN : x[row];
      const int k1 = a.t.mem_ptr[r0 + row + 1];
#pragma unroll 4
      for (int k = a.t.mem_ptr[r0 + row] + i % kL; k < k1; k += kL) a.t.xf[a.t.mem_rows[k]] += v;
    }
  }
  if (fail && tid == 0) {
    *const_cast<volatile int32_t*>(a.timed_out) = 1;
    __threadfence_system();
  }
  __syncthreads();
  cluster_meet();
  // stores to a block that gave up may still be on their way
  if (fail)
    for (int k = 0; k < 50; ++k) __nanosleep(1000);
}

using SweepFn = void (*)(SArgs);
SweepFn sweep_fn(int lanes) { return lanes == 8 ? k_sweeps<8> : lanes == 4 ? k_sweeps<4> : k_sweeps<2>; }

// Lanes of a row: a warp's rounds over its rows, each with a fixed part (the
// sums, the stores) and a part for each step.  50 sweeps with 2 / 4 / 8 lanes
// (us): 1,000 rows of 22: 43 / 39 / 39; 1,000 of 71: 74 / 62 / 60; 3,138 of 35:
// 67 / 66 / 78; 5,985 of 24: 64 / 76 / 108; 10,648 of 25: 99 / 125 / 174.
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

void sweep_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute& at, int blocks, int threads, int smem,
                  cudaStream_t s) {
  cfg = {};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(threads);
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
  auto len = [&](int32_t r) { return r < n ? indptr[r + 1] - indptr[r] : 0; };
  const int lanes = sweep_lanes(n, indptr[n]), per = 32 / lanes;
  const int32_t npad = (n + kCutRows - 1) / kCutRows * kCutRows;
  // cuts after equal shares of the elements, a row counted as eight of them
  int64_t total = 0, at = 0;
  for (int32_t r = 0; r < n; ++r) total += len(r) + 8;
  std::vector<int32_t> host(2 * nb + 1);
  int32_t *cut = host.data(), *recv = cut + nb + 1;
  int32_t k = 1;
  for (int32_t r = 0; r < npad; r += kCutRows) {
    while (k < nb && at * nb >= total * k) cut[k++] = r;
    for (int32_t i = r; i < std::min(n, r + kCutRows); ++i) at += len(i) + 8;
  }
  for (; k <= nb; ++k) cut[k] = npad;
  // steps of each task: its longest row over the lanes
  std::vector<int32_t> step(npad / per + 1, 0);
  for (int32_t t = 0; t < npad / per; ++t) {
    int32_t most = 0;
    for (int32_t r = t * per; r < (t + 1) * per; ++r) most = std::max(most, len(r));
    step[t + 1] = step[t] + ceil_div(most, 4 * lanes);
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
    if ((cut[b + 1] - cut[b]) / 4 + 1 >= kSweepNone / 16) return;
  for (int32_t b = 0; b < nb; ++b)
    for (int32_t i = cut[b] / 4; i < cut[b + 1] / 4; ++i) keep(i, b);
  std::vector<bool> reads(nb * nb);  // [b * nb + o]: block b receives from block o
  for (int32_t b = 0; b < nb; ++b)
    for (int32_t r = cut[b]; r < std::min(n, cut[b + 1]); ++r)
      for (int32_t e = indptr[r]; e < indptr[r + 1]; ++e) {
        if (recv[b] >= kSweepNone / 16 - 20) return;  // byte offsets are 16-bit
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
  int32_t rows = 0, steps = 0, quads = 0;
  for (int32_t b = 0; b < nb; ++b) {
    rows = std::max(rows, cut[b + 1] - cut[b]);
    steps = std::max(steps, step[cut[b + 1] / per] - step[cut[b] / per]);
    quads = std::max(quads, recv[b]);
  }
  const int32_t nx = 4 * (quads + 1);  // (the last four stay 0)
  const int64_t smem = 32 * 24LL * steps + 8LL * rows + 4LL * (rows / per + 4) + 2LL * nb / 4 * rows + 12LL * nx;
  if (smem > limit || 4 * nx > 65536) return;
  // the order of a row's elements: each lane takes, for the read of x that goes
  // out next, one of its row's on a bank that no other lane reads
  std::vector<int32_t> src(128LL * step.back(), -1);
  std::vector<uint16_t> cols(128LL * step.back(), static_cast<uint16_t>(4 * (nx - 1)));
#pragma omp parallel for schedule(dynamic, 8)
  for (int32_t t = 0; t < npad / per; ++t) {
    int32_t b = 0;
    while (t * per >= cut[b + 1]) ++b;
    std::vector<std::pair<int32_t, int32_t>> left[16];  // (element, position in x) of each row
    int32_t slots[16];
    const int32_t n_steps = step[t + 1] - step[t];
    for (int i = 0; i < per; ++i) {
      const int32_t r = t * per + i;
      for (int32_t e = r < n ? indptr[r] : 0; e < (r < n ? indptr[r + 1] : 0); ++e)
        left[i].push_back({e, 4 * pos[static_cast<size_t>(indices[e] / 4) * nb + b] + indices[e] % 4});
      slots[i] = 4 * lanes * n_steps;
    }
    for (int32_t s = 0; s < n_steps; ++s)
      for (int c = 0; c < 4; ++c) {
        int32_t taken[32];
        int load[32] = {};
        std::fill(taken, taken + 32, -1);
        for (int lane = 0; lane < 32; ++lane) {
          auto& row = left[lane / lanes];
          const int32_t room = slots[lane / lanes]-- - static_cast<int32_t>(row.size());
          if (row.empty()) continue;
          size_t best = 0;
          int least = 1 << 20;
          for (size_t m = 0; m < row.size() && least > 0; ++m) {
            const int32_t p = row[m].second;
            const int cost = taken[p & 31] == p ? 0 : load[p & 31];
            if (cost < least) {
              least = cost;
              best = m;
            }
          }
          if (least > 0 && room > 0) continue;  // padding does it
          const auto e = row[best];
          row[best] = row.back();
          row.pop_back();
          if (taken[e.second & 31] != e.second) ++load[e.second & 31];
          taken[e.second & 31] = e.second;
          const int64_t at4 = 4 * (32LL * (step[t] + s) + lane) + c;
          src[at4] = e.first;
          cols[at4] = static_cast<uint16_t>(4 * e.second);
        }
      }
  }
  const void* fn = reinterpret_cast<const void*>(sweep_fn(lanes));
  MGPBD_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, limit));
  MGPBD_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr;
  // a warp for each task, at least 16 to load the block (1,000 rows: 39 us with
  // 32 warps, 35 with 16; 5,985 rows in 24 tasks: 64 and 74)
  const int threads = 32 * std::min(kSweepWarps, std::max(16, rows / per));
  sweep_config(cfg, attr, nb, threads, static_cast<int>(smem), s);
  int fit = 0;
  if (cudaOccupancyMaxActiveClusters(&fit, fn, &cfg) != cudaSuccess || fit < 1) {
    (void)cudaGetLastError();
    return;
  }
  plan.dev.alloc(static_cast<int64_t>(host.size()));
  plan.step.alloc(static_cast<int64_t>(step.size()));
  plan.src.alloc(std::max<int64_t>(1, static_cast<int64_t>(src.size())));
  plan.cols.alloc(std::max<int64_t>(4, static_cast<int64_t>(cols.size())));
  plan.pos.alloc(static_cast<int64_t>(pos.size()));
  MGPBD_CUDA(cudaMemcpyAsync(plan.dev.p, host.data(), sizeof(int32_t) * host.size(),
                             cudaMemcpyHostToDevice, s));
  MGPBD_CUDA(cudaMemcpyAsync(plan.step.p, step.data(), sizeof(int32_t) * step.size(),
                             cudaMemcpyHostToDevice, s));
  MGPBD_CUDA(cudaMemcpyAsync(plan.src.p, src.data(), sizeof(int32_t) * src.size(),
                             cudaMemcpyHostToDevice, s));
  MGPBD_CUDA(cudaMemcpyAsync(plan.cols.p, cols.data(), sizeof(uint16_t) * cols.size(),
                             cudaMemcpyHostToDevice, s));
  MGPBD_CUDA(cudaMemcpyAsync(plan.pos.p, pos.data(), sizeof(uint16_t) * pos.size(),
                             cudaMemcpyHostToDevice, s));
  MGPBD_CUDA(cudaStreamSynchronize(s));
  plan.blocks = nb;
  plan.lanes = lanes;
  plan.threads = threads;
  plan.rows = rows;
  plan.steps = steps;
  plan.nx = nx;
  plan.smem = static_cast<int32_t>(smem);
}

void launch_sweeps(const CgState* st, const CsrView& a, const SweepPlan& plan, const float* b, float w,
                   const float* w_dev, int32_t sweeps, bool zero_first, float* x,
                   const SweepTransfer& t, double spin_limit_s, int32_t* timed_out, cudaStream_t s) {
  require(plan.blocks > 0 && sweeps >= 1, MGPBD_ESTATE, "no plan for the coarse sweeps");
  SArgs g = {};
  g.st = st;
  g.data = a.data;
  g.dinv = a.diag_inv;
  g.blk = plan.dev.p;
  g.step = plan.step.p;
  g.src = plan.src.p;
  g.cols = reinterpret_cast<const uint2*>(plan.cols.p);
  g.pos = plan.pos.p;
  g.b = b;
  g.x = x;
  g.w = w;
  g.wp = w_dev;
  g.t = t;
  g.timed_out = timed_out;
  g.spin_ns = static_cast<unsigned long long>(spin_limit_s * 1e9);
  g.n = a.n;
  g.blocks = plan.blocks;
  g.rows = plan.rows;
  g.steps = plan.steps;
  g.nx = plan.nx;
  g.sweeps = sweeps;
  g.zero_first = zero_first ? 1 : 0;
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr;
  sweep_config(cfg, attr, plan.blocks, plan.threads, plan.smem, s);
  MGPBD_CUDA(cudaLaunchKernelEx(&cfg, sweep_fn(plan.lanes), g));
  MGPBD_CHECK_LAUNCH();
}

}  // namespace mgpbd
