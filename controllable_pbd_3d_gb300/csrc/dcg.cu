// The dual Chebyshev-CG on a spatial partition (dcg.cuh), one launch per
// solve: a cooperative grid with one block per SM for a body that fills the
// GPU, or one thread-block cluster per problem for small bodies and packs
// of independent bodies (no synchronisation between clusters).
//
// One application of A by a block:
//   vertex sums   s_v = sum x_t g_{t,l} over the block's own constraints
//                 (x in shared memory); vertices shared with other blocks
//                 first, their partial sums go to those blocks
//   constraints   (A x)_t = g_t . u + alpha~_t x_t and the vector update,
//                 those on private vertices (u = w s)
//   collect       u = w (sum of all blocks' partials) of the shared vertices
//   constraints   the others
// so a block waits for its neighbours only, once per application, and has
// work while the partials travel.  (The kernel before this one, k_jcg, has
// two grid barriers per application and gathers x and u through L2.)
//
// The exchange.  Grid: a partial is one 16-byte store of the sum and the
// number of the exchange; a reader polls until that number is there, so
// neither side needs a fence or a counter.  Cluster: st.async into the other
// block's shared memory, counted in bytes on its barrier.  Either way the
// buffers alternate between two halves: a block writes half k again only
// after it has read its neighbours' partials of the exchange in between,
// which they sent after they had read half k.  Dot products go the same way,
// every block's partial to all blocks.
//
// Where the operator lives.  The vertex-major gradients ("rows" of 32
// entries) in shared memory beside x and u; the constraints' own gradients,
// vertex positions, r, d and p in tensor memory, 256 KB that a kernel without
// matrix products has free: a thread's lane and its warp's columns hold what
// it needs of its constraints, 13 values in one access.  (In registers they
// spill, and unrolled over them the loop no longer fits the instruction
// cache; with rows and constraints the other way round the constraint phase
// is 30 % slower.)  What does not fit streams from L2, coalesced.
//
// What bounds it: issue slots and the latency of the exchange (10 meetings an
// iteration of degree 8, 3.5 us each across the grid, 1.5 us in a cluster);
// DRAM is idle.  Measured, us per CG iteration, length + volume cubes of n^3
// hexes, before / after: n = 10 68 / 27 (cluster), 20 70 / 39, 28 77 / 45,
// 40 141 / 67; 80x20x80 332 / 135; ARAP 23x17x29 63 / 39.
//
// Arithmetic per element, the reductions and the scalar logic of the CG are
// those of k_jcg (jcg.cu): float32 per element, float32 within a warp and
// float64 across warps and blocks, Kahan-compensated solution.  The sums of the
// estimate, which k_lz_apply (jform.cu) makes in float64, have 48 bits.  Sums run in a fixed
// order, so results repeat bit for bit.
//
// Every wait is bounded as there; the blocks of a cluster meet once more at
// its end, so none leaves while another may still signal it.
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "cheb_dev.cuh"
#include "cluster_dev.cuh"
#include "common.h"
#include "dcg.cuh"
#include "jform_dev.cuh"
#include "persist.cuh"

namespace mgpbd {

namespace {

using namespace jdev;
using namespace pdev;
using namespace cdev;

struct DArgs {
  DcgDev d;
  const float* b;
  float* x;
  float* xc;
  float* r;
  const float* invm;
  JState* js;
  CgState* st;
  GridSync* gs;
  const JcgCtl* ctl;
  int32_t* iters;
  double tol_abs, tol_rel, lo_ratio;
  int32_t estimate;  // 1: the Chebyshev interval is estimated first, 0: from js
  int32_t maxiter, degree, warm, per_problem, unit_dinv;
  int32_t nblk, nprob, rmax, kT, kE;  // kT, kE: of every block of a grid
  DcgSmem o;  // byte offsets of the shared-memory parts (u is at 0)
  unsigned long long spin_ns;
};

// Shared memory by offset from the array's symbol, so that every access is
// a shared-memory instruction
extern __shared__ __align__(16) unsigned char s_dyn[];
__device__ __forceinline__ float4& sm_u(int p) { return reinterpret_cast<float4*>(s_dyn)[p]; }
__device__ __forceinline__ float4 sm_u_at(uint32_t off) {
  return *reinterpret_cast<float4*>(s_dyn + off);
}
__device__ __forceinline__ float4& sm_f4(int off, int k) {
  return reinterpret_cast<float4*>(s_dyn + off)[k];
}
__device__ __forceinline__ float& sm_f(int off, int k) {
  return reinterpret_cast<float*>(s_dyn + off)[k];
}
__device__ __forceinline__ float2& sm_f2(int off, int k) {
  return reinterpret_cast<float2*>(s_dyn + off)[k];
}
__device__ __forceinline__ int32_t& sm_i(int off, int k) {
  return reinterpret_cast<int32_t*>(s_dyn + off)[k];
}
__device__ __forceinline__ uint2& sm_i2(int off, int k) {
  return reinterpret_cast<uint2*>(s_dyn + off)[k];
}
__device__ __forceinline__ uint16_t& sm_h(int off, int k) {
  return reinterpret_cast<uint16_t*>(s_dyn + off)[k];
}

// Named barrier 1: the other warps arrive and the last one waits
__device__ __forceinline__ void bar_arrive1() {
  asm volatile("bar.arrive 1, %0;" ::"r"(blockDim.x) : "memory");
}
__device__ __forceinline__ void bar_sync1() {
  asm volatile("bar.sync 1, %0;" ::"r"(blockDim.x) : "memory");
}

// Tensor memory as a second register file: a thread's lane and the columns
// of its warp's window hold what it needs of its constraints.  Every access
// is by the whole warp, converged, with one column address.
__device__ __forceinline__ void tm_ld16(uint32_t t, uint32_t (&v)[16]) {
  __syncwarp();
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, "
      "%12, %13, %14, %15}, [%16];\n\ttcgen05.wait::ld.sync.aligned;"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
        "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
        "=r"(v[14]), "=r"(v[15])
      : "r"(t)
      : "memory");
}
__device__ __forceinline__ void tm_ld8(uint32_t t, uint32_t (&v)[8]) {
  __syncwarp();
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
      : "r"(t)
      : "memory");
}
__device__ __forceinline__ float2 tm_ld2(uint32_t t) {
  float2 v;
  __syncwarp();
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0, %1}, [%2];\n\ttcgen05.wait::ld.sync.aligned;"
      : "=f"(v.x), "=f"(v.y)
      : "r"(t)
      : "memory");
  return v;
}
__device__ __forceinline__ float tm_ld1(uint32_t t) {
  float v;
  __syncwarp();
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];\n\ttcgen05.wait::ld.sync.aligned;"
               : "=f"(v)
               : "r"(t)
               : "memory");
  return v;
}
__device__ __forceinline__ void tm_st16(uint32_t t, const uint32_t (&v)[16]) {
  __syncwarp();
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, "
      "%12, %13, %14, %15, %16};" ::"r"(t),
      "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
      "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
      : "memory");
}
__device__ __forceinline__ void tm_st8(uint32_t t, const uint32_t (&v)[8]) {
  __syncwarp();
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(t),
      "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
      : "memory");
}
__device__ __forceinline__ void tm_st2(uint32_t t, float x, float y) {
  __syncwarp();
  asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1, %2};" ::"r"(t), "f"(x), "f"(y)
               : "memory");
}
__device__ __forceinline__ void tm_st1(uint32_t t, float x) {
  __syncwarp();
  asm volatile("tcgen05.st.sync.aligned.32x32b.x1.b32 [%0], {%1};" ::"r"(t), "f"(x) : "memory");
}
// the warp's stores so far are done
__device__ __forceinline__ void tm_wait_st() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// Waits until there() holds; false when the limit is reached or another
// block has given up (the failure is recorded)
template <class F>
__device__ __forceinline__ bool bounded_wait(const DArgs& a, F there) {
  bool ok = true;
  unsigned long long t0 = 0;
  for (unsigned int k = 1; !there(); ++k) {
    if (a.spin_ns == 0) {
      ok = false;
      break;
    }
    // (reading the timer is slow: not before the wait has become a long one)
    if ((k & 255u) == 0) {
      const unsigned long long t = global_ns();
      if (t0 == 0) t0 = t;
      if (ld_relaxed(&a.gs->err) != 0u || t - t0 > a.spin_ns) {
        ok = false;
        break;
      }
    }
  }
  if (!ok) {
    atomicExch(&a.gs->err, 1u);
    atomicOr(reinterpret_cast<unsigned int*>(&a.st->status), MGPBD_STATUS_SYNC_TIMEOUT);
  }
  return ok;
}

// A sum in two float32 words, about 48 bits: the products and the errors of the
// additions are kept exactly (Knuth's two-sum, a fused multiply-add for the
// product).  (In float64, whose pipe is slow, the sums of a Lanczos step would
// take as long as the application of A.)
struct Sum2 {
  float hi = 0.0f, lo = 0.0f;
  __device__ __forceinline__ void add(float v) {
    const float s = __fadd_rn(hi, v), t = __fsub_rn(s, hi);
    lo = __fadd_rn(lo, __fadd_rn(__fsub_rn(hi, __fsub_rn(s, t)), __fsub_rn(v, t)));
    hi = s;
  }
  __device__ __forceinline__ void add_product(float a, float b) {
    const float p = __fmul_rn(a, b);
    lo = __fadd_rn(lo, __fmaf_rn(a, b, -p));
    add(p);
  }
  __device__ __forceinline__ void add_lane(int o) {
    const float h = __shfl_xor_sync(0xffffffffu, hi, o), l = __shfl_xor_sync(0xffffffffu, lo, o);
    lo = __fadd_rn(lo, l);
    add(h);
  }
};

__device__ __forceinline__ float dot3(float x, float y, float z, float4 u) {
  return x * u.x + y * u.y + z * u.z;
}

// g . u of a 4-slot constraint; g0 = -(g1 + g2 + g3) in the rounding order
// the gradients are made with
__device__ __forceinline__ float tet_dot(const float (&g)[9], uint2 q) {
  const float g0 = -g[0] - g[3] - g[6], g1 = -g[1] - g[4] - g[7], g2 = -g[2] - g[5] - g[8];
  const float4 u0 = sm_u_at(q.x & 0xffff), u1 = sm_u_at(q.x >> 16), u2 = sm_u_at(q.y & 0xffff),
               u3 = sm_u_at(q.y >> 16);
  return dot3(g0, g1, g2, u0) + dot3(g[0], g[1], g[2], u1) + dot3(g[3], g[4], g[5], u2) +
         dot3(g[6], g[7], g[8], u3);
}

// ... from the packed four gradients, for constraints that are not held
__device__ __forceinline__ float tet_dot12(float4 a, float4 b, float4 c, uint2 q) {
  const float4 u0 = sm_u_at(q.x & 0xffff), u1 = sm_u_at(q.x >> 16), u2 = sm_u_at(q.y & 0xffff),
               u3 = sm_u_at(q.y >> 16);
  return dot3(a.x, a.y, a.z, u0) + dot3(a.w, b.x, b.y, u1) + dot3(b.z, b.w, c.x, u2) +
         dot3(c.y, c.z, c.w, u3);
}

__device__ __forceinline__ float edge_dot(float x, float y, float z, uint32_t e) {
  const float4 ua = sm_u_at(e & 0xffff), ub = sm_u_at(e >> 16);
  return dot3(x, y, z, ua) - dot3(x, y, z, ub);
}

// Constraint c of a block belongs to thread c % blockDim.x (4-slot and length
// constraints counted apart); up to kT / kE of each a thread keeps in tensor
// memory (16 and 8 columns: gradients, vertex positions, r, d, p), the rest
// through global memory.  The last warp also sums the partials and runs the
// scalar logic.
//
// The loops are rolled and the code of an application of A appears once: the
// body of an iteration then stays in the instruction cache, which a version
// with the gradients in registers (unrolled, 3 times the code) did not.
constexpr int kLanczosSteps = 24;
constexpr int kColR = 12, kColP = 9, kColX = 14;  // 4-slot: g 0-8, p, q 10-11, r, d, x, xc
constexpr int kEdgeR = 4, kEdgeP = 6;             // length: n 0-2, e 3, r, d, p

template <bool CLUSTER>
__global__ void __launch_bounds__(kDMaxThreads, 1) k_dcg(DArgs a) {
  if (a.ctl && a.ctl->skip) return;
  // cluster: exchange barriers, sum barriers (two of each alternate)
  __shared__ __align__(8) unsigned long long s_bar[4];
  __shared__ double s_sum[CLUSTER ? 2 : 1][3][kDMaxCluster];  // cluster: the blocks' partials
  __shared__ float s_c1[kMaxCheb], s_c2[kMaxCheb], s_it;
  __shared__ double s_la[kLanczosSteps], s_lb[kLanczosSteps];
  __shared__ double s_red[3][kDMaxWarps];
  __shared__ float s_scal, s_inv, s_bprev;
  __shared__ int s_ok, s_stop;  // s_ok: 0 once a wait of this block has given up
  __shared__ uint32_t s_tmem;
  __shared__ DBlock s_B;  // (read where needed: registers are short)
  // CG scalars, the last warp's lane 0 only (shared memory keeps them out of
  // every thread's registers)
  __shared__ double bbs, tol2, rz, rr, pap, alpha, beta;
  __shared__ int32_t iters, maxiter;
  __shared__ uint32_t status;
  const int nthr = blockDim.x, nw = nthr / 32;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const bool syncw = wid == nw - 1;
  if (tid < static_cast<int>(sizeof(DBlock) / 4))
    reinterpret_cast<int32_t*>(&s_B)[tid] = reinterpret_cast<const int32_t*>(a.d.blocks + blockIdx.x)[tid];
  const DWarp W = a.d.warps[blockIdx.x * nw + wid];
  __syncthreads();
  const DBlock& B = s_B;
  const int64_t NC = a.d.nc;
  const int prob = CLUSTER ? B.prob : blockIdx.x / a.nblk, rank = CLUSTER ? B.rank : blockIdx.x % a.nblk;
  const int G = CLUSTER ? B.size : a.nblk;
  // the cluster's block that is the first of this problem
  uint32_t base = 0;
  if (CLUSTER) {
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(base));
    base -= rank;
  }

  // all of the SM's tensor memory: the block takes more than half of the
  // shared memory, so no second block of this kernel waits here for it
  if (syncw) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(
                     smem_u32(&s_tmem))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid < kMaxCheb && !a.estimate) {
    s_c1[tid] = a.js->cf.c1[tid];
    s_c2[tid] = a.js->cf.c2[tid];
  }
  if (tid == 0 && !a.estimate) s_it = a.js->cf.inv_theta;
  if (tid == nthr - 32) {
    bbs = tol2 = rz = rr = pap = alpha = beta = 0.0;
    iters = 0;
    status = 0;
    s_ok = 1;
    maxiter = a.ctl ? a.ctl->maxiter : a.maxiter;
    if (CLUSTER) {
      for (int k = 0; k < 4; ++k)
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&s_bar[k])) : "memory");
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
  }
  const int warm = a.ctl ? a.ctl->warm : a.warm;
  const int deg = a.degree;

  // stage the tables and rows (u.w of a position holds its vertex weight)
  for (int k = tid; k < B.npos; k += nthr) {
    const int32_t v = a.d.pos_v[B.p0 + k];
    sm_u(k) = make_float4(0.f, 0.f, 0.f, v >= 0 ? a.invm[v] : 0.0f);
    if (k < B.nposS) sm_i2(a.o.info, k) = a.d.pos_info[B.p0 + k];
  }
  for (int k = tid; k < B.nsl; k += nthr) sm_i2(a.o.slice, k) = a.d.slice[B.s0 + k];
  if (CLUSTER)
    for (int k = tid; k < B.ntgt; k += nthr) sm_i(a.o.tgt, k) = a.d.tgt[B.t0 + k];
  {
    const uint4* src = reinterpret_cast<const uint4*>(a.d.rows + static_cast<int64_t>(B.r0 + W.row) * kDRow);
    uint4* dst = reinterpret_cast<uint4*>(s_dyn + a.o.rows + W.srow * kDRow);
    for (int k = lane; k < W.held * (kDRow / 16); k += 32) dst[k] = __ldg(src + k);
  }
  // one compliance for the whole block is kept in a register
  float al0 = 0.0f;
  int general = !a.unit_dinv;
  if (B.nT + B.nE > 0) {
    al0 = __ldg(a.d.ad + B.c0).x;
    for (int k = tid; k < B.nT + B.nE; k += nthr) general |= __ldg(a.d.ad + (B.c0 + k)).x != al0;
  }
  general = __syncthreads_or(general);
  // (the barrier also orders the allocation's address before its use)
  const int colT = CLUSTER ? B.kT : a.kT, colE = CLUSTER ? B.kE : a.kE;
  const uint32_t tm0 = s_tmem + (static_cast<uint32_t>(wid & 3) << 21) +
                       static_cast<uint32_t>(wid >> 2) * (16 * colT + 8 * colE);
  const uint32_t tme = tm0 + 16 * colT;

  // in tensor memory: constraints below nTr / nEr (no 4-slot one when some
  // slot-0 gradient is not minus the sum of the others), in kT / kE rounds
  const int nT = B.nT, nE = B.nE, nC = nT + nE;
  const int nTr = *a.d.gflag ? 0 : min(nT, colT * nthr), nEr = min(nE, colE * nthr);
  // rounds in which this warp has some
  const int kT = max(0, (nTr - 32 * wid + nthr - 1) / nthr);
  const int kE = max(0, (nEr - 32 * wid + nthr - 1) / nthr);
  // of these, rounds whose constraints touch private vertices only
  const int kTi = min(kT, min(B.nTi, nTr) / nthr), kEi = min(kE, min(B.nEi, nEr) / nthr);
  const int c0 = B.c0;
  auto tg = [&](int plane, int c) { return __ldg(a.d.tg + plane * NC + (c0 + c)); };
  auto ti = [&](int c) { return __ldg(a.d.ti + (c0 + c)); };
  auto perm = [&](int c) { return __ldg(a.d.perm + (c0 + c)); };
  auto ad = [&](int c) { return __ldg(a.d.ad + (c0 + c)); };
  auto gx = [&](int c) -> float& { return a.d.x[c0 + c]; };
  auto gxc = [&](int c) -> float& { return a.d.xc[c0 + c]; };
  auto gr = [&](int c) -> float& { return a.d.r[c0 + c]; };
  auto gd = [&](int c) -> float& { return a.d.d[c0 + c]; };
  auto gp = [&](int c) -> float& { return a.d.p[c0 + c]; };
#pragma unroll 1
  for (int i = 0; i < kT; ++i) {
    const int c = i * nthr + tid;
    uint32_t v[16] = {};
    if (c < nTr) {
      const float4 g0 = tg(0, c), g1 = tg(1, c), g2 = tg(2, c);
      const uint2 q = ti(c);
      const float f[9] = {g0.w, g1.x, g1.y, g1.z, g1.w, g2.x, g2.y, g2.z, g2.w};
#pragma unroll
      for (int k = 0; k < 9; ++k) v[k] = __float_as_uint(f[k]);
      v[10] = q.x;
      v[11] = q.y;
    }
    tm_st16(tm0 + 16 * i, v);
  }
#pragma unroll 1
  for (int j = 0; j < kE; ++j) {
    const int e = j * nthr + tid;
    uint32_t v[8] = {};
    if (e < nEr) {
      const float4 g = tg(0, nT + e);
      v[0] = __float_as_uint(g.x);
      v[1] = __float_as_uint(g.y);
      v[2] = __float_as_uint(g.z);
      v[3] = __float_as_uint(g.w);
    }
    tm_st8(tme + 8 * j, v);
  }
  tm_wait_st();
  if (CLUSTER) cluster_meet();  // every block's barriers are ready

  // f(c, ok, t): the warp's rounds in tensor memory (t: the column of r; ok:
  // the lane has a constraint there)
  auto rounds = [&](auto f) {
#pragma unroll 1
    for (int i = 0; i < kT; ++i)
      f(i * nthr + tid, i * nthr + tid < nTr, tm0 + 16 * i + kColR, tm0 + 16 * i + kColP);
#pragma unroll 1
    for (int j = 0; j < kE; ++j)
      f(nT + j * nthr + tid, j * nthr + tid < nEr, tme + 8 * j + kEdgeR, tme + 8 * j + kEdgeP);
  };
  // f(c): the thread's constraints that are not held
  auto rest = [&](auto f) {
    for (int c = nTr + tid; c < nC; c += nthr)
      if (c < nT || c >= nT + nEr) f(c);
  };
  auto dinv_of = [&](int c) { return a.unit_dinv ? 1.0f : ad(c).y; };
  auto put = [&](int k, float v) {  // the warp's partial of a dot product
    v = warp_sum_f(v);
    if (lane == 0) s_red[k][wid] = static_cast<double>(v);
  };
  // ... in two words, which publish adds: a conversion occupies the float64 pipe
  // for the whole warp, so not one in each
  auto put2 = [&](int k, const Sum2& v) {
    if (lane == 0) *reinterpret_cast<float2*>(&s_red[k][wid]) = make_float2(v.hi, v.lo);
  };
  // x += alpha p, compensated (x and its low part of 4-slot rounds in tensor
  // memory)
  auto kahan = [&](float al, float p, float& s, float& c) {
    const float y = al * p - c;
    const float sn = s + y;
    c = (sn - s) - y;
    s = sn;
  };
  auto x_update = [&](float al) {
#pragma unroll 1
    for (int i = 0; i < kT; ++i) {
      const float p = tm_ld1(tm0 + 16 * i + kColP);
      float2 v = tm_ld2(tm0 + 16 * i + kColX);
      kahan(al, p, v.x, v.y);
      tm_st2(tm0 + 16 * i + kColX, v.x, v.y);
    }
    constexpr int kB = 4;  // loads in flight
#pragma unroll 1
    for (int j0 = 0; j0 < kE; j0 += kB) {
      float s[kB], c[kB];
#pragma unroll
      for (int j = 0; j < kB; ++j) {
        const int e = (j0 + j) * nthr + tid;
        s[j] = c[j] = 0.0f;
        if (e < nEr) {
          s[j] = gx(nT + e);
          c[j] = gxc(nT + e);
        }
      }
#pragma unroll
      for (int j = 0; j < kB; ++j) {
        if (j0 + j >= kE) break;
        const int e = (j0 + j) * nthr + tid;
        kahan(al, tm_ld1(tme + 8 * (j0 + j) + kEdgeP), s[j], c[j]);
        if (e < nEr) {
          gx(nT + e) = s[j];
          gxc(nT + e) = c[j];
        }
      }
    }
    rest([&](int k) { kahan(al, gp(k), gx(k), gxc(k)); });
    tm_wait_st();
  };
  // The sums s_v = sum x_t g over the block's own constraints, the warp's
  // slices of vertices; shared vertices first: their partials go out; then u
  // of the private ones.
  auto sums = [&](uint32_t gen) {
    int row = 0;
#pragma unroll 1
    for (int s = W.s; s < W.e; ++s) {
      const uint2 sl = sm_i2(a.o.slice, s);
      float ax = 0.f, ay = 0.f, az = 0.f;
      const int end = row + sl.x, held = min(end, W.held);  // in shared memory
      int o = a.o.rows + (W.srow + row) * kDRow + 8 * lane;
      auto rows = [&](auto count) {  // `count` rows at once
        constexpr int N = decltype(count)::value;
        float x[N];
#pragma unroll
        for (int k = 0; k < N; ++k)
          x[k] = sm_f(a.o.x + sm_h(o + k * kDRow + kDRowX - 6 * lane, 0), 0);
#pragma unroll
        for (int k = 0; k < N; ++k) {
          const float2 g = sm_f2(o + k * kDRow, 0);
          ax += x[k] * g.x;
          ay += x[k] * g.y;
          az += x[k] * sm_f(o + k * kDRow + kDRowZ - 4 * lane, 0);
        }
        row += N;
        o += N * kDRow;
      };
#pragma unroll 1
      while (row + 4 <= held) rows(std::integral_constant<int, 4>());
      if (row + 2 <= held) rows(std::integral_constant<int, 2>());
      if (row < held) rows(std::integral_constant<int, 1>());
      // what is not held, through L1
#pragma unroll 2
      for (; row < end; ++row) {
        const unsigned char* q = a.d.rows + static_cast<int64_t>(B.r0 + W.row + row) * kDRow;
        const float x = sm_f(a.o.x + __ldg(reinterpret_cast<const uint16_t*>(q + kDRowX) + lane), 0);
        const float2 g = __ldg(reinterpret_cast<const float2*>(q) + lane);
        ax += x * g.x;
        ay += x * g.y;
        az += x * __ldg(reinterpret_cast<const float*>(q + kDRowZ) + lane);
      }
      const int vshift = sl.y >> 16;
#pragma unroll 1
      for (int o = (1 << vshift) >> 1; o > 0; o >>= 1) {
        ax += __shfl_xor_sync(0xffffffffu, ax, o);
        ay += __shfl_xor_sync(0xffffffffu, ay, o);
        az += __shfl_xor_sync(0xffffffffu, az, o);
      }
      const int p = (sl.y & 0xffff) + (lane >> vshift), sub = lane & ((1 << vshift) - 1);
      if (s >= W.p) {
        if (sub == 0) {
          const float w = sm_u(p).w;
          sm_u(p) = make_float4(w * ax, w * ay, w * az, w);
        }
        continue;
      }
      // the partial goes out; the block's own copy waits in u
      const uint2 f = sm_i2(a.o.info, p);
      const int others = static_cast<int>(f.y >> 8) - 1;
      if (CLUSTER) {
        for (int k = sub; k < others; k += 1 << vshift) {
          const uint32_t t = sm_i(a.o.tgt, (f.x >> 16) + k);
          const uint32_t to = smem_u32(s_dyn) + a.o.rbuf + 16 * ((gen & 1) * a.rmax + (t & 0xffff));
          send_f4(map_rank(to, base + (t >> 16)), map_rank(smem_u32(&s_bar[gen & 1]), base + (t >> 16)),
                  ax, ay, az);
        }
      }
      if (sub == 0 && others > 0) {
        if (!CLUSTER)
          put_tagged(a.d.exch + ((gen & 1 ? a.d.n_slots : 0) + f.x + (f.y & 0xff)),
                     __float_as_uint(ax), __float_as_uint(ay), __float_as_uint(az), gen);
        const float w = sm_u(p).w;
        sm_u(p) = make_float4(ax, ay, az, w);
      }
    }
  };
  // u of the shared vertices, after the meeting: w times the sum of all
  // blocks' partials in block order
  auto collect = [&](uint32_t gen) {
    for (int p = tid; p < B.nposS; p += nthr) {
      const uint2 f = sm_i2(a.o.info, p);
      if (!f.y) continue;
      const int n = f.y >> 8, own = f.y & 0xff;
      const float4 m = sm_u(p);
      float x = 0.f, y = 0.f, z = 0.f;
      if (CLUSTER) {
        int o = (gen & 1) * a.rmax + (f.x & 0xffff);
        for (int k = 0; k < n; ++k) {
          const float4 s = k == own ? m : sm_f4(a.o.rbuf, o++);
          x += s.x;
          y += s.y;
          z += s.z;
        }
      } else {
        const float4* e = a.d.exch + ((gen & 1 ? a.d.n_slots : 0) + f.x);
        for (int k = 0; k < n; k += 4) {
          uint4 s[4];
          const bool ok = bounded_wait(a, [&]() {
            bool all = true;
#pragma unroll
            for (int l = 0; l < 4; ++l)
              if (k + l < n && k + l != own) s[l] = get_tagged(e + k + l);
#pragma unroll
            for (int l = 0; l < 4; ++l)
              if (k + l < n && k + l != own) all &= s[l].w == gen;
            return all;
          });
          if (!ok) s_ok = 0;
#pragma unroll
          for (int l = 0; l < 4; ++l)
            if (k + l < n) {
              const bool me = k + l == own;
              x += me ? m.x : __uint_as_float(s[l].x);
              y += me ? m.y : __uint_as_float(s[l].y);
              z += me ? m.z : __uint_as_float(s[l].z);
            }
        }
      }
      sm_u(p) = make_float4(m.w * x, m.w * y, m.w * z, m.w);
    }
  };
  // ---- the last warp's part ----
  uint32_t gen = 0, nsum = 0;  // exchanges, sums
  // Publishes the block's partials of the planes in mask (arrive: once the
  // other warps have arrived with theirs; words2: from put2)
  auto publish = [&](int mask, bool arrive, bool words2 = false) {
    ++nsum;
    if (arrive) bar_sync1();
    __syncwarp();
    const uint32_t sbar = smem_u32(&s_bar[2 + (nsum & 1)]);
    if (CLUSTER && lane == 0) expect_bytes(sbar, 8 * G * __popc(mask));
#pragma unroll 1
    for (int k = 0; k < 3; ++k)
      if (mask >> k & 1) {
        double v = 0.0;
        if (lane < nw) {
          const float2 w = *reinterpret_cast<const float2*>(&s_red[k][lane]);
          v = words2 ? static_cast<double>(w.x) + static_cast<double>(w.y) : s_red[k][lane];
        }
        v = warp_sum_d(v);
        if (CLUSTER) {
          if (lane < G)
            send_f64(map_rank(smem_u32(&s_sum[nsum & 1][k][rank]), base + lane), map_rank(sbar, base + lane), v);
        } else if (lane == 0) {
          const unsigned long long u = __double_as_longlong(v);
          put_tagged(a.d.partials + ((nsum & 1) * 3 + k) * G + rank, static_cast<uint32_t>(u),
                     static_cast<uint32_t>(u >> 32), 0u, nsum);
        }
      }
  };
  // the problem's total of plane k, published (all lanes); ok: false when
  // the wait for it gave up
  auto total = [&](int k, bool& ok) {
    double acc = 0.0;
    bool mine = true;
    if (CLUSTER) {
      const uint32_t bar = smem_u32(&s_bar[2 + (nsum & 1)]), parity = (nsum - 1) >> 1 & 1;
      mine = bounded_wait(a, [&]() { return test_phase(bar, parity); });
      if (lane < G) acc = *const_cast<volatile double*>(&s_sum[nsum & 1][k][lane]);
    } else {
      const uint4* p = a.d.partials + ((nsum & 1) * 3 + k) * G;
      for (int i = lane; i < G; i += 32) {
        uint4 v;
        mine = bounded_wait(a, [&]() {
          v = get_tagged(p + i);
          return v.w == nsum;
        }) && mine;
        acc += __longlong_as_double(static_cast<long long>(static_cast<unsigned long long>(v.y) << 32 | v.x));
      }
    }
    if (!__all_sync(0xffffffffu, mine)) ok = false;
    return warp_sum_d(acc);
  };
  auto rr_test = [&](double v) {  // lane 0
    int stop = 0;
    rr = v;
    if (!isfinite(rr)) {
      status |= MGPBD_STATUS_NAN;
      stop = 1;
    } else if (rr < tol2) {
      iters += 1;
      stop = 1;
    }
    return stop;
  };

  // epi(c, r, d, (J u)_c) -> d: the rounds on private vertices (half 0), the
  // others (half 1), and what is not held
  auto held = [&](int half, auto epi) {
#pragma unroll 1
    for (int k = half ? kTi : 0; k < (half ? kT : kTi); ++k) {
      const int c = k * nthr + tid;
      const uint32_t t = tm0 + 16 * k;
      uint32_t v[16];
      tm_ld16(t, v);
      float g[9];
#pragma unroll
      for (int m = 0; m < 9; ++m) g[m] = __uint_as_float(v[m]);
      float d = __uint_as_float(v[kColR + 1]);
      if (c < nTr) d = epi(c, __uint_as_float(v[kColR]), d, tet_dot(g, make_uint2(v[10], v[11])));
      tm_st1(t + kColR + 1, d);
    }
#pragma unroll 1
    for (int k = half ? kEi : 0; k < (half ? kE : kEi); ++k) {
      const int e = k * nthr + tid;
      const uint32_t t = tme + 8 * k;
      uint32_t v[8];
      tm_ld8(t, v);
      float d = __uint_as_float(v[kEdgeR + 1]);
      if (e < nEr)
        d = epi(nT + e, __uint_as_float(v[kEdgeR]), d,
                edge_dot(__uint_as_float(v[0]), __uint_as_float(v[1]), __uint_as_float(v[2]), v[3]));
      tm_st1(t + kEdgeR + 1, d);
    }
    tm_wait_st();
  };
  auto rest_ju = [&](auto epi) {
#pragma unroll 2
    for (int c = nTr + tid; c < nT; c += nthr)
      gd(c) = epi(c, gr(c), gd(c), tet_dot12(tg(0, c), tg(1, c), tg(2, c), ti(c)));
#pragma unroll 2
    for (int c = nT + nEr + tid; c < nC; c += nthr) {
      const float4 g = tg(0, c);
      gd(c) = epi(c, gr(c), gd(c), edge_dot(g.x, g.y, g.z, __float_as_uint(g.w)));
    }
  };
  // A x of the x in shared memory: the vertex sums, the other blocks' and the
  // constraints; between() runs while the partials travel, arrived() in the
  // last warp once they are there (before the others go on).  False when a
  // wait gave up or `stop` and s_stop is set.
  auto apply = [&](bool stop, auto epi, auto between, auto arrived) {
    if (CLUSTER && tid == nthr - 32) expect_bytes(smem_u32(&s_bar[(gen + 1) & 1]), 16 * B.nrecv);
    sums(++gen);
    between();
    __syncthreads();
#pragma unroll 1
    for (int half = 0; half < 2; ++half) {
      if (half) {
        if (CLUSTER) {
          if (tid == nthr - 32) {
            const uint32_t bar = smem_u32(&s_bar[gen & 1]), parity = (gen - 1) >> 1 & 1;
            if (!bounded_wait(a, [&]() { return test_phase(bar, parity); })) s_ok = 0;
          }
          __syncthreads();
        }
        collect(gen);
        if (syncw) arrived();
        __syncthreads();
        if (!s_ok || (stop && s_stop)) return false;
      }
      held(half, epi);
    }
    rest_ju(epi);
    return true;
  };

  // The Chebyshev interval of this problem: lambda_max of S = D^-1/2 A D^-1/2
  // by Lanczos steps from a fixed start vector (Golub & Van Loan, sec. 10.1).
  // One application and one sum a step: with q.w, w.w and q.q of
  // w = S q - b q_prev, a = q.w / q.q and b = |w - a q| follow together, from
  // sums of 48 bits.  (q.q has to be summed: taken as 1, or carried on from the
  // step before, its error grows by a^2 / b^2 a step.)  Where little is left of
  // the difference b is summed from the vector itself: a small b does not say
  // that the space is exhausted (a uniform spectrum with one stiff constraint has
  // one in the first step).  As
  // kernels of their own the 24 steps and the interval took 730 us a Newton
  // iteration, here 245 us (72,000 ARAP constraints on the grid; 250 with the
  // sums' second words): a step costs two meetings, not four launches.
  auto estimate = [&]() {
    auto sqd = [&](int c) { return a.unit_dinv ? 1.0f : sqrtf(ad(c).y); };
    {
      Sum2 qq;
      auto seed = [&](int c) {
        uint32_t h = static_cast<uint32_t>(perm(c)) * 2654435761u;
        h ^= h >> 15;
        const float v = 0.5f + (h & 0xffff) * (1.0f / 65536.0f);
        qq.add_product(v, v);
        return v;
      };
      rounds([&](int c, bool ok, uint32_t t, uint32_t) { tm_st2(t, 0.0f, ok ? seed(c) : 0.0f); });
      rest([&](int c) {
        gr(c) = 0.0f;
        gd(c) = seed(c);
      });
      tm_wait_st();
#pragma unroll 1
      for (int o = 16; o > 0; o >>= 1) qq.add_lane(o);
      put2(2, qq);
      if (!syncw) {
        bar_arrive1();
      } else {
        publish(4, true, true);
        bool ok = true;
        const double v = total(2, ok);
        if (lane == 0) {
          if (!ok) s_ok = 0;
          s_scal = 0.0f;
          s_inv = v > 0.0 ? static_cast<float>(1.0 / sqrt(v)) : 1.0f;
          s_bprev = 0.0f;
        }
      }
      __syncthreads();
      if (!s_ok) return false;
    }
    auto set_b = [&](int j, double b) {
      s_lb[j] = b;
      s_inv = b > 0.0 ? static_cast<float>(1.0 / b) : 0.0f;
      s_bprev = static_cast<float>(b);
    };
#pragma unroll 1
    for (int j = 0; j < kLanczosSteps; ++j) {
      const float aj = s_scal, inv = s_inv, bprev = s_bprev;
      // q_prev = q, q = (w - a q) / b
      auto next = [&](int c, float& r, float& d) {
        const float q = (d - aj * r) * inv;
        d = r;
        r = q;
        sm_f(a.o.x, c) = sqd(c) * q;
      };
      rounds([&](int c, bool ok, uint32_t t, uint32_t) {
        float2 v = tm_ld2(t);
        if (ok) next(c, v.x, v.y);
        tm_st2(t, v.x, v.y);
      });
      rest([&](int c) { next(c, gr(c), gd(c)); });
      tm_wait_st();
      __syncthreads();
      Sum2 qw, ww, qq;
      auto epi = [&](int c, float q, float d, float y) {
        const float w = sqd(c) * (y + ad(c).x * sm_f(a.o.x, c)) - bprev * d;
        qw.add_product(q, w);
        ww.add_product(w, w);
        qq.add_product(q, q);
        return w;
      };
      if (!apply(false, epi, []() {}, []() {})) return false;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        qw.add_lane(o);
        ww.add_lane(o);
        qq.add_lane(o);
      }
      put2(0, qw);
      put2(1, ww);
      put2(2, qq);
      if (!syncw) {
        bar_arrive1();
      } else {
        publish(7, true, true);
        bool ok = true;
        const double tqw = total(0, ok), tww = total(1, ok), tqq = total(2, ok);
        if (lane == 0) {
          if (!ok) s_ok = 0;
          const double av = tqq > 0.0 ? tqw / tqq : 0.0;
          const double b2 = tww - (2.0 * tqw - av * tqq) * av;
          s_la[j] = av;
          s_scal = static_cast<float>(av);
          // (in the limits, so that the squares' float32 words hold)
          s_stop = !(b2 > 1e-6 * tww && tww > 1e-20 && tww < 1e30);
          if (!s_stop) set_b(j, sqrt(b2));
        }
      }
      __syncthreads();
      if (!s_ok) return false;
      if (s_stop) {  // |w - a q| from the vector
        const float av = s_scal;
        double yy = 0.0;
        auto left = [&](float q, float w) {
          const double y = w - av * q;
          yy += y * y;
        };
        rounds([&](int c, bool ok, uint32_t t, uint32_t) {
          const float2 v = tm_ld2(t);
          if (ok) left(v.x, v.y);
        });
        rest([&](int c) { left(gr(c), gd(c)); });
        yy = warp_sum_d(yy);
        if (lane == 0) s_red[0][wid] = yy;
        if (!syncw) {
          bar_arrive1();
        } else {
          publish(1, true);
          bool ok = true;
          const double v = total(0, ok);
          if (lane == 0) {
            if (!ok) s_ok = 0;
            set_b(j, sqrt(v));
          }
        }
        __syncthreads();
        if (!s_ok) return false;
      }
    }
    if (syncw) {
      const double lmax = lanczos_lmax(s_la, s_lb, kLanczosSteps);
      if (lane == 0) {
        double theta;
        float it;
        const bool ok = cheb_interval(lmax, deg, a.lo_ratio, s_c1, s_c2, &theta, &it);
        if (!ok) status |= MGPBD_STATUS_NAN;
        s_it = it;
        if (prob == 0 && rank == 0) {
          ChebCoef& f = a.js->cf;
          for (int i = 0; i < kMaxCheb; ++i) {
            f.c1[i] = s_c1[i];
            f.c2[i] = s_c2[i];
          }
          f.theta = theta;
          f.lmax = ok ? lmax : (isfinite(lmax) ? lmax : NAN);
          f.inv_theta = it;
          f.degree = deg;
        }
      }
    }
    __syncthreads();
    return true;
  };

  auto run = [&]() {
    if (a.estimate) {
      bool need = true;
      if (a.per_problem) {  // a body whose Newton loop has ended needs none
        float bb = 0.0f;
        for (int c = tid; c < nC; c += nthr) {
          const float bt = a.b[perm(c)];
          bb += bt * bt;
        }
        put(0, bb);
        if (!syncw) {
          bar_arrive1();
        } else {
          publish(1, true);
          bool ok = true;
          const double v = total(0, ok);
          if (lane == 0) {
            if (!ok) s_ok = 0;
            s_stop = v == 0.0;
          }
        }
        __syncthreads();
        if (!s_ok) return;
        need = s_stop == 0;
      }
      if (need && !estimate()) return;
      if (!need && tid == 0) s_it = 0.0f;
      __syncthreads();
    }
    const float it = s_it;
    // x = 0 (or the warm start), r = b - A x, p = 0, z = d = D^-1 r / theta
    {
      float bb = 0.0f, bz = 0.0f, br = 0.0f;
      auto start = [&](int c, float& r, float& z) {
        const int32_t o = perm(c);
        const float bt = a.b[o];
        r = warm ? a.r[o] : bt;
        z = dinv_of(c) * r * it;
        sm_f(a.o.x, c) = z;
        bb += bt * bt;
        bz += r * z;
        br += r * r;
      };
      rounds([&](int c, bool ok, uint32_t t, uint32_t tp) {
        float r = 0.0f, z = 0.0f;
        if (ok) start(c, r, z);
        tm_st2(t, r, z);
        tm_st1(tp, 0.0f);
      });
      rest([&](int c) {
        start(c, gr(c), gd(c));
        gp(c) = 0.0f;
      });
      for (int i = 0; i < kT; ++i) {
        const int c = i * nthr + tid;
        tm_st2(tm0 + 16 * i + kColX, warm && c < nTr ? a.x[perm(c)] : 0.0f, 0.0f);
      }
      for (int c = nTr + tid; c < nC; c += nthr) {
        gx(c) = warm ? a.x[perm(c)] : 0.0f;
        gxc(c) = 0.0f;
      }
      tm_wait_st();
      put(0, bb);
      put(1, bz);
      put(2, br);
    }
    if (!syncw) {
      bar_arrive1();
    } else {
      publish(7, true);
      bool ok = true;
      const double sb = total(0, ok), sz = total(1, ok), sr = total(2, ok);
      if (lane == 0) {
        if (!ok) s_ok = 0;
        bbs = sb;
        rz = sz;
        rr = warm ? sr : sb;
        const double tol_abs = a.ctl ? a.ctl->tol_abs : a.tol_abs;
        const double t2 = tol_abs * tol_abs, r2 = a.tol_rel * a.tol_rel * bbs;
        tol2 = r2 > t2 ? r2 : t2;
        int stop = maxiter <= 0 || (warm && rr < tol2) || (a.per_problem && bbs == 0.0);
        if (!isfinite(bbs)) {
          status |= MGPBD_STATUS_NAN;
          stop = 1;
        }
        s_stop = stop;
      }
    }
    __syncthreads();
    if (!s_ok || s_stop) return;

    float al = 0.0f;    // alpha of the x update still to be made
    bool first = true;  // before the first A p
    int i = deg > 1 ? 1 : deg;
#pragma unroll 1
    for (;;) {
      // application i of an iteration: Chebyshev steps 1 .. deg - 1 of
      // z = M^-1 r, then (i = deg) A p.  The first step's meeting also
      // carries r.r of the update before it; x += alpha p is made while it
      // is awaited.
      const bool ap = i == deg, test = i == 1 && !ap && !first;
      if (ap) {
        // beta; p = z + beta p
        if (deg == 1 && !first) x_update(al);
        if (!syncw) {
          bar_arrive1();
        } else {
          publish(deg > 1 ? 4 : (first ? 1 : 6), true);
          bool ok = true;
          const double sr = deg == 1 && !first ? total(1, ok) : 0.0;
          const double sz = deg > 1 || !first ? total(2, ok) : 0.0;
          if (deg == 1 && first) total(0, ok);
          if (lane == 0) {
            if (!ok) s_ok = 0;
            int stop = deg == 1 && !first ? rr_test(sr) : 0;
            float bf = 0.0f;
            if (first) {
              if (deg > 1) rz = sz;
              if (!isfinite(rz)) {
                status |= MGPBD_STATUS_NAN;
                stop = 1;
              }
            } else if (!stop) {
              iters += 1;
              if (fabs(rz) < 1e-30) {
                stop = 1;
              } else {
                beta = sz / rz;
                rz = sz;
                bf = (float)beta;
                if (iters >= maxiter) {
                  status |= MGPBD_STATUS_CG_MAXITER;
                  stop = 1;
                }
              }
            }
            s_scal = bf;
            s_stop = stop;
          }
        }
        __syncthreads();
        if (!s_ok || s_stop) return;
        const float bf = s_scal;
        rounds([&](int c, bool ok, uint32_t, uint32_t tp) {
          float p = bf * tm_ld1(tp);
          if (ok) sm_f(a.o.x, c) = p = sm_f(a.o.x, c) + p;
          tm_st1(tp, p);
        });
        rest([&](int c) { sm_f(a.o.x, c) = gp(c) = sm_f(a.o.x, c) + bf * gp(c); });
        tm_wait_st();
        __syncthreads();
      }
      const float c1 = ap ? 0.0f : s_c1[i], c2 = ap ? 0.0f : s_c2[i];
      float acc = 0.0f;
      // constraint epilogue: Chebyshev step (ap: d = A p, acc = p.Ap)
      auto epi = [&](int c, float r, float d, float y) {
        float alv = al0, dv = 1.0f;
        if (general) {
          const float2 v = ad(c);
          alv = v.x;
          if (!a.unit_dinv) dv = v.y;
        }
        const float zt = sm_f(a.o.x, c);
        const float yt = y + alv * zt;
        if (ap) {
          acc += zt * yt;
          return yt;
        }
        const float dn = c1 * d + c2 * (dv * (r - yt));
        const float zn = zt + dn;
        sm_f(a.o.x, c) = zn;
        acc += r * zn;
        return dn;
      };
      if (test && syncw) publish(2, false);
      const bool on = apply(
          test, epi,
          [&]() {
            if (test) x_update(al);
          },
          [&]() {
            if (!test) return;
            bool ok = true;
            const double sr = total(1, ok);
            if (lane == 0) {
              if (!ok) s_ok = 0;
              s_stop = rr_test(sr);
            }
          });
      if (!on) return;
      if (!ap) {
        if (i == deg - 1) put(2, acc);
        else __syncthreads();
        ++i;
        continue;
      }
      // alpha; r -= alpha Ap; z = d = D^-1 r / theta (x += alpha p follows)
      put(0, acc);
      if (!syncw) {
        bar_arrive1();
      } else {
        publish(1, true);
        bool ok = true;
        const double sp = total(0, ok);
        if (lane == 0) {
          if (!ok) s_ok = 0;
          pap = sp;
          int stop = 0;
          if (!isfinite(pap)) status |= MGPBD_STATUS_NAN;
          if (!(fabs(pap) >= 1e-30) || !isfinite(pap)) {
            stop = 1;
          } else {
            if (pap <= 0.0) status |= MGPBD_STATUS_PAP_NONPOS;
            alpha = rz / pap;
          }
          s_scal = (float)alpha;
          s_stop = stop;
        }
      }
      __syncthreads();
      if (!s_ok || s_stop) return;
      al = s_scal;
      {
        float acc_rr = 0.0f, acc_rz = 0.0f;
        auto upd = [&](int c, float& r, float& d) {
          r = r - al * d;
          d = dinv_of(c) * r * it;
          sm_f(a.o.x, c) = d;
          acc_rr += r * r;
          acc_rz += r * d;
        };
        rounds([&](int c, bool ok, uint32_t t, uint32_t) {
          float2 v = tm_ld2(t);
          if (ok) upd(c, v.x, v.y);
          tm_st2(t, v.x, v.y);
        });
        rest([&](int c) { upd(c, gr(c), gd(c)); });
        tm_wait_st();
        put(1, acc_rr);
        if (deg == 1) put(2, acc_rz);
        __syncthreads();
      }
      first = false;
      i = deg > 1 ? 1 : deg;
    }
  };
  run();

  // the compensated sum, rounded once; xc keeps what the rounding dropped
  __syncthreads();
  auto finish = [&](int c, float s, float e) {
    const int32_t o = perm(c);
    const float hi = s - e;
    a.xc[o] = (s - hi) - e;
    a.x[o] = hi;
  };
  rounds([&](int c, bool ok, uint32_t t, uint32_t) {
    const float2 v = tm_ld2(t);
    if (ok) a.r[perm(c)] = v.x;
  });
  rest([&](int c) { a.r[perm(c)] = gr(c); });
  for (int i = 0; i < kT; ++i) {
    const int c = i * nthr + tid;
    const float2 v = tm_ld2(tm0 + 16 * i + kColX);
    if (c < nTr) finish(c, v.x, v.y);
  }
  for (int c = nTr + tid; c < nC; c += nthr) finish(c, gx(c), gxc(c));
  if (rank == 0 && tid == nthr - 32) {
    CgState* st = a.st;
    if (a.nprob == 1) {
      st->rz = rz;
      st->pap = pap;
      st->alpha = alpha;
      st->beta = beta;
      st->rr = rr;
      st->rr0 = bbs;
      st->tol2 = tol2;
    }
    st->done = 1;
    st->maxiter = maxiter;
    st->body_runs = 1;
    if (a.iters && prob >= 0) a.iters[prob] = iters;
    atomicMax(&st->iters, iters);
    if (status) atomicOr(reinterpret_cast<unsigned int*>(&st->status), status);
  }
  __syncthreads();
  if (syncw)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(s_tmem));
  if (CLUSTER) {
    __syncthreads();
    cluster_meet();
    // stores to a block that gave up may still be on their way: it stays until
    // they have landed
    if (!s_ok) {
      const unsigned long long t0 = global_ns();
      while (global_ns() - t0 < 50000) __nanosleep(1000);
    }
  }
}

// Gradients, compliances and 1/diag in plan order (dcg.cuh)
__global__ void k_dcg_pack(const float* __restrict__ gradC, const float* __restrict__ alpha,
                           const float* __restrict__ dinv, DcgDev d, int64_t n_entries) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t t0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  for (int64_t k = t0; k < n_entries; k += stride) {
    const int32_t e = __ldg(d.row_ent + k);
    const float* g = gradC + 3LL * (e < 0 ? 0 : e);
    unsigned char* row = d.rows + (k >> 5) * kDRow;
    reinterpret_cast<float2*>(row)[k & 31] =
        e < 0 ? make_float2(0.0f, 0.0f) : make_float2(g[0], g[1]);
    reinterpret_cast<float*>(row + kDRowZ)[k & 31] = e < 0 ? 0.0f : g[2];
    // (constant, and written again with the rest)
    reinterpret_cast<uint16_t*>(row + kDRowX)[k & 31] = static_cast<uint16_t>(4 * __ldg(d.row_idx + k));
  }
  for (int64_t k = t0; k < d.nc; k += stride) {
    const int32_t c = __ldg(d.perm + k);
    const float4* g = reinterpret_cast<const float4*>(gradC + 12LL * c);
    const float4 g0 = g[0], g1 = g[1], g2 = g[2];
    if (c < d.n4) {
      d.tg[k] = g0;
      d.tg[d.nc + k] = g1;
      d.tg[2LL * d.nc + k] = g2;
      const bool same = g0.x == -g0.w - g1.z - g2.y && g0.y == -g1.x - g1.w - g2.z &&
                        g0.z == -g1.y - g2.x - g2.w;
      if (!same) *d.gflag = 1;
    } else {
      d.tg[k] = make_float4(g0.x, g0.y, g0.z, __uint_as_float(__ldg(d.ti + k).x));
    }
    d.ad[k] = make_float2(alpha[c], dinv[c]);
  }
}

// Before each solve: the caller's compliances as they are now (he may have
// changed them since the fill) into the plan's order, and the state and the
// barrier's words zeroed.  In k_dcg itself the compliances cost more than this
// launch, which takes the place of two memsets (a cluster's iterations 1.4 %
// longer).
__global__ void k_dcg_begin(DcgDev d, const float* __restrict__ alpha, GridSync* gs, CgState* st) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t t0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  for (int64_t k = t0; k < d.nc; k += stride) d.ad[k].x = alpha[__ldg(d.perm + k)];
  if (t0 == 0) {
    *gs = GridSync();
    *st = CgState();
  }
}

// Warm start: u = W J^T x in float64, stored as a float pair, then
// r = b - A x in float64 (a residual of a good start is a small difference
// of large terms).  Once per solve; without a start nothing is done.
__global__ void k_warm_u(JView j, const float* __restrict__ x, float4* __restrict__ lo,
                         const JcgCtl* ctl) {
  if (ctl && (ctl->skip || !ctl->warm)) return;
  const int lane = threadIdx.x % 4;
  const int64_t n = ((int64_t)j.nv + 7) / 8 * 8;
  for (int64_t v = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / 4; v < n;
       v += (int64_t)gridDim.x * blockDim.x / 4) {
    double sx = 0.0, sy = 0.0, sz = 0.0;
    if (v < j.nv)
      for (int32_t k = j.inc_ptr[v] + lane; k < j.inc_ptr[v + 1]; k += 4) {
        const float4 g = __ldg(j.gV + k);
        const double xt = x[__float_as_int(g.w)];
        sx += xt * g.x;
        sy += xt * g.y;
        sz += xt * g.z;
      }
#pragma unroll
    for (int o = 2; o > 0; o >>= 1) {
      sx += __shfl_xor_sync(0xffffffffu, sx, o, 4);
      sy += __shfl_xor_sync(0xffffffffu, sy, o, 4);
      sz += __shfl_xor_sync(0xffffffffu, sz, o, 4);
    }
    if (lane == 0 && v < j.nv) {
      const double w = j.invm[v];
      sx *= w;
      sy *= w;
      sz *= w;
      const float hx = (float)sx, hy = (float)sy, hz = (float)sz;
      j.u[v] = make_float4(hx, hy, hz, 0.0f);
      lo[v] = make_float4((float)(sx - hx), (float)(sy - hy), (float)(sz - hz), 0.0f);
    }
  }
}

__global__ void k_warm_r(JView j, const float* __restrict__ b, const float* __restrict__ x,
                         const float4* __restrict__ lo, float* __restrict__ r, const JcgCtl* ctl) {
  if (ctl && (ctl->skip || !ctl->warm)) return;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < j.nt;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int4 q = reinterpret_cast<const int4*>(j.t_i)[t];
    const int32_t vs[4] = {q.x, q.y, q.z, q.w};
    const float* g = j.gradC + 12 * t;
    double acc = 0.0;
#pragma unroll
    for (int l = 0; l < 4; ++l) {
      const float4 h = j.u[vs[l]], e = lo[vs[l]];
      acc += (double)g[3 * l] * ((double)h.x + e.x) + (double)g[3 * l + 1] * ((double)h.y + e.y) +
             (double)g[3 * l + 2] * ((double)h.z + e.z);
    }
    r[t] = (float)((double)b[t] - (acc + (double)j.alpha[t] * x[t]));
  }
}

const void* kernel_of(bool cluster) {
  return cluster ? reinterpret_cast<const void*>(k_dcg<true>)
                 : reinterpret_cast<const void*>(k_dcg<false>);
}

}  // namespace

// The attributes are per function and shared by every handle in the process:
// always the same values.
int dcg_smem_limit() {
  int dev = 0, optin = 0;
  MGPBD_CUDA(cudaGetDevice(&dev));
  MGPBD_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  size_t most = 0;
  for (bool cluster : {false, true}) {
    cudaFuncAttributes fa;
    MGPBD_CUDA(cudaFuncGetAttributes(&fa, kernel_of(cluster)));
    most = std::max(most, fa.sharedSizeBytes);
  }
  const int limit = optin - static_cast<int>(most);
  for (bool cluster : {false, true})
    MGPBD_CUDA(cudaFuncSetAttribute(kernel_of(cluster), cudaFuncAttributeMaxDynamicSharedMemorySize, limit));
  MGPBD_CUDA(cudaFuncSetAttribute(kernel_of(true), cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  return limit;
}

int dcg_max_clusters(int size, int threads, int smem) {
  const void* fn = kernel_of(true);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(size);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = size;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, fn, &cfg) != cudaSuccess) {
    (void)cudaGetLastError();
    return 0;
  }
  return n;
}

void launch_dcg_pack(const JView& j, const DcgDev& d, int64_t n_rows, cudaStream_t s) {
  const int64_t n = std::max<int64_t>(32 * n_rows, d.nc);
  MGPBD_CUDA(cudaMemsetAsync(d.gflag, 0, sizeof(uint32_t), s));
  k_dcg_pack<<<static_cast<int>(std::min<int64_t>(ceil_div(n, 256), 152 * 8)), 256, 0, s>>>(
      j.gradC, j.alpha, j.dinv, d, 32 * n_rows);
  MGPBD_CHECK_LAUNCH();
}

void launch_dcg(const JView& j, const JcgVecs& v, const DcgPlan& plan, const DcgDev& d,
                JState* js, CgState* st, double tol_abs, double tol_rel, int maxiter, int degree,
                double lo_ratio, bool estimate, bool warm, bool per_problem, int32_t* iters,
                double spin_limit_s, cudaStream_t s, const JcgCtl* ctl) {
  require(degree >= 1 && degree <= kMaxCheb, MGPBD_EINVAL, "Chebyshev degree out of range");
  require(plan.nblk > 0 && d.nc == j.nt, MGPBD_ESTATE, "dual CG partition not built");
  require(!(warm || ctl) || v.ulo != nullptr, MGPBD_EINVAL, "warm start needs the ulo scratch");
  DArgs a;
  a.d = d;
  a.b = v.b;
  a.x = v.x;
  a.xc = v.xc;
  a.r = v.r;
  a.invm = j.invm;
  a.js = js;
  a.st = st;
  a.gs = v.gs;
  a.ctl = ctl;
  a.iters = iters;
  a.tol_abs = tol_abs;
  a.tol_rel = tol_rel;
  a.maxiter = maxiter;
  a.degree = degree;
  a.lo_ratio = lo_ratio;
  a.estimate = estimate ? 1 : 0;
  a.warm = warm ? 1 : 0;
  a.per_problem = per_problem ? 1 : 0;
  a.unit_dinv = j.unit_dinv ? 1 : 0;
  a.nblk = plan.nblk;
  a.nprob = plan.nprob;
  a.rmax = plan.rmax;
  a.kT = plan.kT;
  a.kE = plan.kE;
  a.o = dcg_smem_parts(plan);
  a.spin_ns = static_cast<unsigned long long>(spin_limit_s * 1e9);
  if (warm || ctl) {
    const int gv = std::min(ceil_div(4LL * j.nv, 256), 152 * 8);
    k_warm_u<<<gv, 256, 0, s>>>(j, v.x, v.ulo, ctl);
    MGPBD_CHECK_LAUNCH();
    k_warm_r<<<std::min(ceil_div(j.nt, 256), 152 * 8), 256, 0, s>>>(j, v.b, v.x, v.ulo, v.r, ctl);
    MGPBD_CHECK_LAUNCH();
  }
  k_dcg_begin<<<std::min(ceil_div(d.nc, 256), 152 * 4), 256, 0, s>>>(d, j.alpha, v.gs, st);
  MGPBD_CHECK_LAUNCH();
  if (!plan.cluster)  // the tags of the launch before (the partials follow the exchange)
    MGPBD_CUDA(cudaMemsetAsync(d.exch, 0, sizeof(float4) * (2 * d.n_slots + 6 * plan.nblk), s));
  const void* fn = kernel_of(plan.cluster);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(plan.nblk);
  cfg.blockDim = dim3(plan.threads);
  cfg.dynamicSmemBytes = plan.smem;
  cfg.stream = s;
  cudaLaunchAttribute at;
  if (plan.cluster) {
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = plan.csize;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
  } else {
    at.id = cudaLaunchAttributeCooperative;
    at.val.cooperative = 1;
  }
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  void* args[] = {&a};
  MGPBD_CUDA(cudaLaunchKernelExC(&cfg, fn, args));
  MGPBD_CHECK_LAUNCH();
}

}  // namespace mgpbd
