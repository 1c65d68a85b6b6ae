// Local XPBD (cons/deform3d.py:7-288) and Vertex Block Descent
// (cons/vbd.py:6-361) on the GPU.
//
// Layouts: positions and velocities (nv, 3) float32 as the caller's fields;
// t_i as int4 per tet; per-tet rest data as (nt, 3, 3) row-major inverse
// rest-shape matrices (Dm_inv / B) and (nt) volumes; VBD's vertex-tet
// adjacency as CSR with entries tet * 4 + local index, tets ascending
// (_build_vertex_tet_adjacency, cons/vbd.py:68-96).
//
// Arithmetic is float32 in the reference's operation order per element;
// the colour kernels are deterministic (no two threads of a colour touch the
// same vertex, fixed lane-reduction order), the XPBD default method is not
// (its position updates are atomic adds racing with other tets' reads, like
// the reference's parallel loop).
#include "local.cuh"

#include <algorithm>
#include <cmath>
#include <string>

#include "coloring.h"
#include "persist.cuh"

namespace mgpbd {

namespace {

constexpr int kLT = 256;  // threads per block
// most warps of a block of the colour kernels that wait for vertices
constexpr int kXpbdWarps = 8;
constexpr int kVbdWarps = 16;  // (8: 313 us over 32^3 hexes, 16: 232)
// lanes per vertex in the VBD colour kernels: at most three tets in a row of the
// 24 (with four lanes 10 iterations over 24^3 hexes take 244 us, with eight 196,
// with sixteen 207, and 302, 313, 463 over 32^3)
constexpr int kVL = 8;

// 3x3 helpers (row-major m[r][c]); determinant by the first column's
// cofactors, inverse = adjugate / det
__device__ __forceinline__ float det3(const float m[3][3]) {
  return m[0][0] * (m[1][1] * m[2][2] - m[2][1] * m[1][2]) -
         m[1][0] * (m[0][1] * m[2][2] - m[2][1] * m[0][2]) +
         m[2][0] * (m[0][1] * m[1][2] - m[1][1] * m[0][2]);
}

__device__ __forceinline__ void inv3(const float m[3][3], float r[3][3]) {
  const float id = 1.0f / det3(m);
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j)
      r[j][i] = id * (m[(i + 1) % 3][(j + 1) % 3] * m[(i + 2) % 3][(j + 2) % 3] -
                      m[(i + 2) % 3][(j + 1) % 3] * m[(i + 1) % 3][(j + 2) % 3]);
}

__device__ __forceinline__ void cross3(const float a[3], const float b[3], float r[3]) {
  r[0] = a[1] * b[2] - a[2] * b[1];
  r[1] = a[2] * b[0] - a[0] * b[2];
  r[2] = a[0] * b[1] - a[1] * b[0];
}

__device__ __forceinline__ float nsq3(const float a[3]) { return a[0] * a[0] + a[1] * a[1] + a[2] * a[2]; }
__device__ __forceinline__ float dot3(const float a[3], const float b[3]) {
  return a[0] * b[0] + a[1] * b[1] + a[2] * b[2];
}

// F = D B with D's columns x_k - x_4 (d[k][i] = (x_k - x_4)_i); column j of
// F is f[j][.]
__device__ __forceinline__ void deformation(const float p[4][3], const float B[3][3],
                                            float f[3][3]) {
  float d[3][3];
#pragma unroll
  for (int k = 0; k < 3; ++k)
#pragma unroll
    for (int i = 0; i < 3; ++i) d[k][i] = p[k][i] - p[3][i];
#pragma unroll
  for (int j = 0; j < 3; ++j)
#pragma unroll
    for (int i = 0; i < 3; ++i) f[j][i] = d[0][i] * B[0][j] + d[1][i] * B[1][j] + d[2][i] * B[2][j];
}

// det of the matrix whose columns are f[0], f[1], f[2]
__device__ __forceinline__ float det_cols(const float f[3][3]) {
  float m[3][3];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) m[i][j] = f[j][i];
  return det3(m);
}

// rest shape of tet k: Dm (columns r_k - r_4), its inverse and |det| / 6
// (_precompute_rest_shape, cons/vbd.py:111-124; the B of
// cons/deform3d.py:75)
__global__ void k_rest_shape(const float* __restrict__ x_ref, const int4* __restrict__ t_i,
                             int32_t nt, float* __restrict__ dm_inv, float* __restrict__ vol) {
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < nt;
       k += (int64_t)gridDim.x * blockDim.x) {
    const int4 q = t_i[k];
    const int32_t v[4] = {q.x, q.y, q.z, q.w};
    float r[4][3];
#pragma unroll
    for (int l = 0; l < 4; ++l)
#pragma unroll
      for (int c = 0; c < 3; ++c) r[l][c] = x_ref[3LL * v[l] + c];
    float dm[3][3], inv[3][3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) dm[i][j] = r[j][i] - r[3][i];
    inv3(dm, inv);
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) dm_inv[9 * k + 3 * i + j] = inv[i][j];
    if (vol) vol[k] = fabsf(det3(dm)) / 6.0f;
  }
}

// ---------------------------------------------------------------------------
// local XPBD: the coupled hydrostatic (det F - 1) and deviatoric
// (|F|^2 - 3) constraints of one tet (cons/deform3d.py:57-127)

struct XArgs {
  float* x;
  const float* invm;
  const int4* t_i;
  const float* t_m;
  const float* B;
  float* lh;
  float* ld;
  int32_t nt;
  float dt, ha, da;
};

// The update of the tet t: t.x(l, c) is coordinate c of its vertex l, t.B(m)
// entry m of its rest matrix.  (The values come through memory in each kernel
// that makes it: the compiler then orders, and rounds, them alike.)  ATOMIC: positions updated with atomic adds (the parallel
// default method); otherwise plain read-modify-write in the reference's order
// (all hydrostatic updates, then all deviatoric ones).
template <bool ATOMIC, class T>
__device__ __forceinline__ void xpbd_update(const XArgs& a, const T& t) {
  float p[4][3], w[4];
#pragma unroll
  for (int l = 0; l < 4; ++l) {
#pragma unroll
    for (int c = 0; c < 3; ++c) p[l][c] = ATOMIC ? __ldcg(&t.x(l, c)) : t.x(l, c);
    w[l] = t.w(l);
  }
  float Bm[3][3];
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int c = 0; c < 3; ++c) Bm[r][c] = t.B(3 * r + c);
  float f[3][3];
  deformation(p, Bm, f);

  const float CH = det_cols(f) - 1.0f;
  float cof[3][3];  // columns f2 x f3, f3 x f1, f1 x f2
  cross3(f[1], f[2], cof[0]);
  cross3(f[2], f[0], cof[1]);
  cross3(f[0], f[1], cof[2]);
  float gH[4][3], gD[4][3];  // gradients per vertex: columns of cof B^T and 2 F B^T
#pragma unroll
  for (int j = 0; j < 3; ++j)
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      gH[j][i] = cof[0][i] * Bm[j][0] + cof[1][i] * Bm[j][1] + cof[2][i] * Bm[j][2];
      gD[j][i] = (2.0f * f[0][i]) * Bm[j][0] + (2.0f * f[1][i]) * Bm[j][1] +
                 (2.0f * f[2][i]) * Bm[j][2];
    }
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    gH[3][i] = -gH[0][i] - gH[1][i] - gH[2][i];
    gD[3][i] = -gD[0][i] - gD[1][i] - gD[2][i];
  }
  const float SH = w[0] * nsq3(gH[0]) + w[1] * nsq3(gH[1]) + w[2] * nsq3(gH[2]) + w[3] * nsq3(gH[3]);
  const float tm = t.tm();
  const float aH = a.ha / (a.dt * a.dt * tm);
  float FF = 0.0f;
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) FF += f[j][i] * f[j][i];
  const float CD = FF - 3.0f;
  const float SD = w[0] * nsq3(gD[0]) + w[1] * nsq3(gD[1]) + w[2] * nsq3(gD[2]) + w[3] * nsq3(gD[3]);
  const float aD = a.da / (a.dt * a.dt * tm);
  const float SDH = w[0] * dot3(gD[0], gH[0]) + w[1] * dot3(gD[1], gH[1]) +
                    w[2] * dot3(gD[2], gH[2]) + w[3] * dot3(gD[3], gH[3]);
  const float lH = t.lh(), lD = t.ld();
  const float dH = (SDH * (CD + aD * lD) - (CH + aH * lH) * (aD + SD)) /
                   ((aH + SH) * (aD + SD) - SDH * SDH);
  const float dD = -(CD + aD * lD + SDH * dH) / (aD + SD);
#pragma unroll
  for (int l = 0; l < 4; ++l)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const float u = w[l] * gH[l][c] * dH;
      if (ATOMIC) atomicAdd(&t.x(l, c), u);
      else t.x(l, c) = t.x(l, c) + u;
    }
  t.lh() = lH + dH;
#pragma unroll
  for (int l = 0; l < 4; ++l)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const float u = w[l] * gD[l][c] * dD;
      if (ATOMIC) atomicAdd(&t.x(l, c), u);
      else t.x(l, c) = t.x(l, c) + u;
    }
  t.ld() = lD + dD;
}

// a tet in global memory
struct XTet {
  const XArgs& a;
  int64_t k, vid[4];
  __device__ XTet(const XArgs& args, int64_t tet) : a(args), k(tet) {
    const int4 q = a.t_i[k];
    vid[0] = q.x;
    vid[1] = q.y;
    vid[2] = q.z;
    vid[3] = q.w;
  }
  __device__ float& x(int l, int c) const { return a.x[3 * vid[l] + c]; }
  __device__ float w(int l) const { return a.invm[vid[l]]; }
  __device__ float B(int m) const { return a.B[9 * k + m]; }
  __device__ float tm() const { return a.t_m[k]; }
  __device__ float& lh() const { return a.lh[k]; }
  __device__ float& ld() const { return a.ld[k]; }
};

// solve_cons (cons/deform3d.py:55-127): every tet at once
__global__ void __launch_bounds__(kLT) k_xpbd_all(XArgs a) {
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < a.nt;
       k += (int64_t)gridDim.x * blockDim.x)
    xpbd_update<true>(a, XTet(a, k));
}

// solve_cons_gauss_seidel (:128-200): one tet at a time, in index order
__global__ void k_xpbd_serial(XArgs a, int32_t passes) {
  if (blockIdx.x != 0 || threadIdx.x != 0) return;
  for (int32_t s = 0; s < passes; ++s)
    for (int64_t k = 0; k < a.nt; ++k) xpbd_update<false>(a, XTet(a, k));
}

// The tets of one colour share no vertex, so a colour's order does not matter
// but each vertex's does: it is updated by its tets in the order of their
// colours.  Each vertex carries, beside its position and in the same 16 bytes,
// the number of updates it has had; a tet waits until its four vertices have
// had those before it, which it knows from the mesh, and no more.  That chain
// through L2 is the bound: 2.1 us a colour (24^3 hexes, 38 colours; 10 passes
// 814 us).  With a grid barrier between the colours, behind which four
// dependent loads began, and a colour's tets on the first few blocks, it was
// 8 us (3,230).
struct FlowArgs {
  const int4* vid;   // vertices of each tet in chunk order (x < 0: padding)
  const int4* rank;  // updates of each vertex before this tet's, in a pass
  const int4* deg;   // and in a whole pass
  const int32_t* tet;
  const float* B;    // [9][32 n_chunks]
  float4* xt;        // position and count of updates of each vertex
  int32_t n_chunks;  // 32 tets of one colour each
  int32_t passes;
  unsigned long long spin_ns;
  GridSync* gs;
  int32_t* status;
};

// Waits until each of K vertices has had the update it is wanted with (all are
// polled at once: one after the other, each would add its own round trip);
// false once a wait of the grid gave up
// (a null vertex is one that is not waited for; a limit of 0 gives up at the first
// poll that finds one missing)
template <int K>
__device__ __forceinline__ bool wait_vertices(const float4* const (&p)[K], const uint32_t (&want)[K],
                                              uint4 (&v)[K], unsigned long long spin_ns,
                                              GridSync* gs, int32_t* status) {
#pragma unroll
  for (int l = 0; l < K; ++l) {
    v[l].w = want[l];
    if (p[l]) v[l] = pdev::get_tagged(p[l]);
  }
  unsigned long long t0 = 0;
  for (uint32_t n = spin_ns == 0 ? 1024 : 1;; ++n) {
    bool ready = true;
#pragma unroll
    for (int l = 0; l < K; ++l) ready = ready && v[l].w == want[l];
    if (ready) return true;
#pragma unroll
    for (int l = 0; l < K; ++l)
      if (v[l].w != want[l]) v[l] = pdev::get_tagged(p[l]);
    if ((n & 1023u) == 0) {
      if (pdev::ld_relaxed(&gs->err) != 0u) return false;
      const unsigned long long t = pdev::global_ns();
      if (t0 == 0) t0 = t;
      if (t - t0 >= spin_ns) {
        atomicExch(&gs->err, 1u);
        atomicOr(reinterpret_cast<unsigned int*>(status), MGPBD_STATUS_SYNC_TIMEOUT);
        return false;
      }
    }
  }
}

// B in chunk order, one row of the arrays an entry
__global__ void k_flow_rest(const float* __restrict__ B, const int32_t* __restrict__ tet, int64_t n,
                            float* __restrict__ out) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    for (int m = 0; m < 9; ++m) out[m * n + i] = tet[i] >= 0 ? B[9LL * tet[i] + m] : 0.0f;
}

__global__ void k_flow_start(const float* __restrict__ x, float4* __restrict__ xt, int32_t nv) {
  for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < nv;
       v += (int64_t)gridDim.x * blockDim.x)
    xt[v] = make_float4(x[3 * v], x[3 * v + 1], x[3 * v + 2], __uint_as_float(0u));
}

// a thread's tet in shared memory: positions, B, inverse masses, volume,
// multipliers
struct XFlowTet {
  float* s;  // the lane's column of its warp's 32
  __device__ float& at(int m) const { return s[32 * m]; }
  __device__ float& x(int l, int c) const { return at(3 * l + c); }
  __device__ float B(int m) const { return at(12 + m); }
  __device__ float w(int l) const { return at(21 + l); }
  __device__ float tm() const { return at(25); }
  __device__ float& lh() const { return at(26); }
  __device__ float& ld() const { return at(27); }
};

// solve_cons_graph_coloring / solve_range (:210-288).  A warp takes its chunks
// in the order of the passes and colours, every wait is for an earlier chunk,
// and all warps are resident: the waits end.
__global__ void __launch_bounds__(32 * kXpbdWarps) k_xpbd_flow(XArgs a, FlowArgs c) {
  extern __shared__ float sm[];
  const int lane = threadIdx.x & 31;
  const int warp = blockIdx.x + gridDim.x * (threadIdx.x >> 5);  // neighbours on other SMs
  const int warps = gridDim.x * (blockDim.x >> 5);
  const int64_t n = 32LL * c.n_chunks;
  for (int32_t s = 0; s < c.passes; ++s)
    for (int32_t j = warp; j < c.n_chunks; j += warps) {
      const int64_t i = 32LL * j + lane;
      const int4 q = __ldg(c.vid + i);
      bool ok = true;
      if (q.x >= 0) {
        const int64_t vid[4] = {q.x, q.y, q.z, q.w};
        const int4 rk = __ldg(c.rank + i), dg = __ldg(c.deg + i);
        const uint32_t deg[4] = {(uint32_t)dg.x, (uint32_t)dg.y, (uint32_t)dg.z, (uint32_t)dg.w};
        uint32_t ver[4] = {(uint32_t)rk.x, (uint32_t)rk.y, (uint32_t)rk.z, (uint32_t)rk.w};
        const float4* const at[4] = {c.xt + vid[0], c.xt + vid[1], c.xt + vid[2], c.xt + vid[3]};
        const int64_t k = __ldg(c.tet + i);
        // all that does not wait
        const XFlowTet t = {sm + 28 * 32 * (threadIdx.x >> 5) + lane};
#pragma unroll
        for (int m = 0; m < 9; ++m) t.at(12 + m) = __ldg(c.B + m * n + i);
#pragma unroll
        for (int l = 0; l < 4; ++l) t.at(21 + l) = __ldg(a.invm + vid[l]);
        t.at(25) = __ldg(a.t_m + k);
        t.lh() = a.lh[k];
        t.ld() = a.ld[k];
#pragma unroll
        for (int l = 0; l < 4; ++l) ver[l] += (uint32_t)s * deg[l];
        uint4 v[4];
        ok = wait_vertices(at, ver, v, c.spin_ns, c.gs, c.status);
        if (ok) {
#pragma unroll
          for (int l = 0; l < 4; ++l) {
            t.x(l, 0) = __uint_as_float(v[l].x);
            t.x(l, 1) = __uint_as_float(v[l].y);
            t.x(l, 2) = __uint_as_float(v[l].z);
          }
          xpbd_update<false>(a, t);
          a.lh[k] = t.lh();
          a.ld[k] = t.ld();
#pragma unroll
          for (int l = 0; l < 4; ++l) {
            const float y[3] = {t.x(l, 0), t.x(l, 1), t.x(l, 2)};
            pdev::put_tagged(const_cast<float4*>(at[l]), __float_as_uint(y[0]), __float_as_uint(y[1]),
                             __float_as_uint(y[2]), ver[l] + 1);
            if (ver[l] + 1 == (uint32_t)c.passes * deg[l]) {
#pragma unroll
              for (int d = 0; d < 3; ++d) a.x[3 * vid[l] + d] = y[d];
            }
          }
        }
      }
      if (!__all_sync(0xffffffffu, ok)) return;
    }
}

// The order with a grid barrier between the colours, for meshes in which a tet
// lists a vertex twice (its update is then two)
struct ColorArgs {
  const int32_t* order;
  const int32_t* off;
  int32_t n_colors;
  int32_t passes;
  unsigned long long spin_ns;
  GridSync* gs;
  int32_t* status;
};

__global__ void __launch_bounds__(kLT) k_xpbd_color(XArgs a, ColorArgs c) {
  unsigned long long gen = 0;
  const int64_t tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int32_t s = 0; s < c.passes; ++s)
    for (int32_t col = 0; col < c.n_colors; ++col) {
      const int32_t b = c.off[col], e = c.off[col + 1];
      for (int64_t i = b + tid; i < e; i += stride) xpbd_update<false>(a, XTet(a, c.order[i]));
      const bool last = s == c.passes - 1 && col == c.n_colors - 1;
      if (!last && !pdev::grid_sync(c.gs, c.status, c.spin_ns, gen)) return;
    }
}

// ---------------------------------------------------------------------------
// VBD: one vertex's Newton step on its inertia + the Neo-Hookean-style
// energy of its incident tets (cons/vbd.py:186-266)

struct VArgs {
  float* x;
  const float* invm;
  const int4* t_i;
  const float* dm;
  const float* vol;
  const int32_t* adj_ptr;
  const int32_t* adj;
  const float* xt;
  const float* xo;
  float* xp;
  int32_t nv;
  float mu, lam, h2, dt, kd;
  int32_t keep_prev;
};

// force and Gauss-Newton Hessian (upper triangle 00 11 22 01 02 12) of one
// incident tet (its positions, rest matrix and volume; l: the vertex's place in
// it), added to fo / H
__device__ __forceinline__ void vbd_term(const VArgs& a, const float p[4][3], const float B[3][3],
                                         float V0, int l, float fo[3], float H[6]) {
  float f[3][3];
  deformation(p, B, f);
  const float J = det_cols(f);
  float cof[3][3];
  cross3(f[1], f[2], cof[0]);
  cross3(f[2], f[0], cof[1]);
  cross3(f[0], f[1], cof[2]);
  const float s = a.lam * (J - 1.0f);
  float b[3];
#pragma unroll
  for (int c = 0; c < 3; ++c)
    b[c] = l == 0 ? B[0][c] : l == 1 ? B[1][c] : l == 2 ? B[2][c] : -(B[0][c] + B[1][c] + B[2][c]);
  float qv[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    // P = mu F + lam (J - 1) cof F; f_e = -V0 (P b)
    const float pb = (a.mu * f[0][i] + s * cof[0][i]) * b[0] + (a.mu * f[1][i] + s * cof[1][i]) * b[1] +
                     (a.mu * f[2][i] + s * cof[2][i]) * b[2];
    fo[i] += -V0 * pb;
    qv[i] = cof[0][i] * b[0] + cof[1][i] * b[1] + cof[2][i] * b[2];
  }
  const float mb = a.mu * nsq3(b);
  H[0] += V0 * (mb + a.lam * (qv[0] * qv[0]));
  H[1] += V0 * (mb + a.lam * (qv[1] * qv[1]));
  H[2] += V0 * (mb + a.lam * (qv[2] * qv[2]));
  H[3] += V0 * (a.lam * (qv[0] * qv[1]));
  H[4] += V0 * (a.lam * (qv[0] * qv[2]));
  H[5] += V0 * (a.lam * (qv[1] * qv[2]));
}

__device__ __forceinline__ void vbd_entry(const VArgs& a, int32_t ent, float fo[3], float H[6]) {
  const int64_t tet = ent >> 2;
  const int l = ent & 3;
  const int4 q = a.t_i[tet];
  const int64_t vid[4] = {q.x, q.y, q.z, q.w};
  float p[4][3];
#pragma unroll
  for (int k = 0; k < 4; ++k)
#pragma unroll
    for (int c = 0; c < 3; ++c) p[k][c] = a.x[3 * vid[k] + c];
  float B[3][3];
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int c = 0; c < 3; ++c) B[r][c] = a.dm[9 * tet + 3 * r + c];
  vbd_term(a, p, B, a.vol[tet], l, fo, H);
}

// What a vertex's solve reads beside its tets: mass / h^2, the inertial and the
// old position
struct VInertia {
  float mh, xt[3], xo[3];
};
__device__ __forceinline__ VInertia vbd_inertia(const VArgs& a, int64_t vi, float w) {
  VInertia m;
  const float mi = 1.0f / w;
  m.mh = mi / a.h2;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    m.xt[c] = a.xt[3 * vi + c];
    m.xo[c] = a.kd > 0.0f ? a.xo[3 * vi + c] : 0.0f;
  }
  return m;
}

// inertia, damping and the 3x3 solve of a vertex at x from the summed tet
// terms: its new position in y (x, as the reference, when |det H| <= 1e-10)
__device__ __forceinline__ void vbd_solve(const VArgs& a, const VInertia& m, const float x[3],
                                          const float fs[3], const float Hs[6], float y[3]) {
  const float mh = m.mh;
  float f[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    f[c] = mh * (m.xt[c] - x[c]) + fs[c];
    y[c] = x[c];
  }
  float H[3][3] = {{mh + Hs[0], Hs[3], Hs[4]}, {Hs[3], mh + Hs[1], Hs[5]}, {Hs[4], Hs[5], mh + Hs[2]}};
  if (a.kd > 0.0f) {
    const float kdt = a.kd / a.dt;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      f[c] -= kdt * (x[c] - m.xo[c]);
      H[c][c] += kdt;
    }
  }
  if (fabsf(det3(H)) > 1e-10f) {
    float inv[3][3];
    inv3(H, inv);
#pragma unroll
    for (int i = 0; i < 3; ++i) y[i] = x[i] + (inv[i][0] * f[0] + inv[i][1] * f[1] + inv[i][2] * f[2]);
  }
}

__device__ __forceinline__ void vbd_finish(const VArgs& a, int64_t vi, float w, const float fs[3],
                                           const float Hs[6]) {
  float x[3], y[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) x[c] = a.x[3 * vi + c];
  if (a.keep_prev) {
#pragma unroll
    for (int c = 0; c < 3; ++c) a.xp[3 * vi + c] = x[c];
  }
  vbd_solve(a, vbd_inertia(a, vi, w), x, fs, Hs, y);
#pragma unroll
  for (int c = 0; c < 3; ++c) a.x[3 * vi + c] = y[c];
}

// sum of 9 values over groups of W lanes (fixed xor tree; all 32 lanes call)
template <int W>
__device__ __forceinline__ void group_sum(float f[3], float H[6]) {
#pragma unroll
  for (int sh = W / 2; sh > 0; sh >>= 1) {
#pragma unroll
    for (int c = 0; c < 3; ++c) f[c] += __shfl_xor_sync(0xffffffffu, f[c], sh, W);
#pragma unroll
    for (int c = 0; c < 6; ++c) H[c] += __shfl_xor_sync(0xffffffffu, H[c], sh, W);
  }
}

// _apply_chebyshev (cons/vbd.py:180-184) for vertices [t0, n) strided
__device__ __forceinline__ void vbd_chebyshev(const VArgs& a, float om, int64_t t0, int64_t step) {
  for (int64_t v = t0; v < a.nv; v += step) {
    if (a.invm[v] > 0.0f) {
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const float xv = a.x[3 * v + c];
        a.x[3 * v + c] = xv + om * (xv - a.xp[3 * v + c]);
      }
    }
  }
}

// solve with method 'serial' (cons/vbd.py:134-160, 186-266): one block;
// warp 0 walks the vertices in index order, its 32 lanes splitting each
// vertex's incident tets
__global__ void k_vbd_serial(VArgs a, const float* __restrict__ om, int32_t n_iter, float rho) {
  const int lane = threadIdx.x & 31;
  for (int32_t n = 0; n < n_iter; ++n) {
    if (threadIdx.x < 32) {
      for (int64_t vi = 0; vi < a.nv; ++vi) {
        const float w = a.invm[vi];
        if (w == 0.0f) continue;
        float f[3] = {0.f, 0.f, 0.f}, H[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        for (int32_t j = a.adj_ptr[vi] + lane; j < a.adj_ptr[vi + 1]; j += 32) vbd_entry(a, a.adj[j], f, H);
        group_sum<32>(f, H);
        if (lane == 0) vbd_finish(a, vi, w, f, H);
        __syncwarp();
      }
    }
    __syncthreads();
    if (rho > 0.0f && n >= 1) {
      vbd_chebyshev(a, om[n], threadIdx.x, blockDim.x);
      __syncthreads();
    }
  }
}

// As for the tets of XPBD, without a barrier: a vertex of iteration n waits for
// its neighbours' positions, those of earlier colours of iteration n and those
// of later colours of iteration n - 1 (with Chebyshev: accelerated).  Each
// vertex publishes both with the count of its iterations; it cannot overwrite
// one that a neighbour still needs, because it waits for that neighbour.  What a
// vertex reads of its tets is laid out in the order of the lanes at each solve,
// so a warp streams it from L1, and what does not wait is loaded before.  10
// iterations over 24^3 hexes: 461 us with a grid barrier between the colours, 9
// scattered words a tet and four dependent loads before them; 180 here, 3.6 us a
// colour: the exchange through L2, then the tets and the solve in a row.
struct VFlowArgs {
  const int32_t* vert;    // the vertices of a warp, of one colour, a chunk (-1: padding)
  const int32_t* nb_off;  // first round of neighbours of each chunk
  const uint32_t* nb;     // [round][32]: neighbour * 2 + (1: of an earlier colour)
  const int32_t* rec_off; // first step of each chunk
  float4* rec;            // [step][3][32]: B, V0, the tet's vertices as places in
                          // the neighbours (bytes), the vertex's place in the tet
  const int32_t* ent;     // [step][32]: tet * 4 + place, -1: none
  const uint32_t* loc;    // [step][32]: those bytes
  float4* xa;             // positions after an iteration, before Chebyshev
  float4* xb;             // and after it (the same array without)
  int32_t n_chunks, n_steps;
  int32_t max_rounds;
  int32_t n_iter;
  float rho;
  const float* om;
  unsigned long long spin_ns;
  GridSync* gs;
  int32_t* status;
};
constexpr uint32_t kNoVertex = 0xffffffffu;
constexpr int kVblk = 32 / kVL;   // vertices of a warp
constexpr int kVblkMost = 48;     // most neighbours (and itself) of one: 48 kB with 16 warps

// rest matrices and volumes as they are now, in the order of VFlowArgs::rec
__global__ void k_vbd_rest(const float* __restrict__ dm, const float* __restrict__ vol, VFlowArgs c) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < 32LL * c.n_steps;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int32_t ent = c.ent[i];
    if (ent < 0) continue;
    const float* B = dm + 9LL * (ent >> 2);
    float4* r = c.rec + 3 * (i & ~31LL) + (i & 31);
    r[0] = make_float4(B[0], B[1], B[2], B[3]);
    r[32] = make_float4(B[4], B[5], B[6], B[7]);
    r[64] = make_float4(B[8], vol[ent >> 2], __uint_as_float(c.loc[i]), __int_as_float(ent & 3));
  }
}

__global__ void __launch_bounds__(32 * kVbdWarps) k_vbd_flow(VArgs a, VFlowArgs c) {
  extern __shared__ float4 sv[];  // positions of the neighbours of a warp's vertices
  const int lane = threadIdx.x & 31, gl = lane % kVL;
  const int warp = blockIdx.x + gridDim.x * (threadIdx.x >> 5);
  const int warps = gridDim.x * (blockDim.x >> 5);
  float4* mine = sv + (threadIdx.x >> 5) * (32 * c.max_rounds) + (lane / kVL) * (kVL * c.max_rounds);
  for (int32_t n = 0; n < c.n_iter; ++n) {
    const bool cheb = c.rho > 0.0f && n >= 1;
    const float om = cheb ? __ldg(c.om + n) : 0.0f;
    for (int32_t j = warp; j < c.n_chunks; j += warps) {
      const int32_t vi = __ldg(c.vert + kVblk * j + lane / kVL);
      const float w = vi >= 0 ? __ldg(a.invm + vi) : 0.0f;
      // this lane's tets (none of a fixed vertex)
      const int32_t tets = w != 0.0f ? (__ldg(a.adj_ptr + vi + 1) - __ldg(a.adj_ptr + vi) + kVL - 1 - gl) / kVL : 0;
      const int32_t r0 = __ldg(c.nb_off + j), r1 = __ldg(c.nb_off + j + 1);
      const int32_t s0 = __ldg(c.rec_off + j), s1 = __ldg(c.rec_off + j + 1);
      VInertia inertia;
      if (gl == 0 && w != 0.0f) inertia = vbd_inertia(a, vi, w);
      bool ok = true;
      constexpr int K = 8;  // neighbours polled at once
      for (int32_t r = r0; r < r1 && ok; r += K) {
        const float4* at[K];
        uint32_t want[K];
        uint4 v[K];
#pragma unroll
        for (int k = 0; k < K; ++k) {
          const uint32_t u = r + k < r1 ? __ldg(c.nb + 32LL * (r + k) + lane) : kNoVertex;
          const bool some = u != kNoVertex;
          at[k] = some ? (u & 1 ? c.xa : c.xb) + (u >> 1) : nullptr;
          want[k] = n + (some ? u & 1 : 0);
        }
        ok = wait_vertices(at, want, v, c.spin_ns, c.gs, c.status);
#pragma unroll
        for (int k = 0; k < K; ++k)
          if (at[k])
            mine[kVL * (r - r0 + k) + gl] = make_float4(__uint_as_float(v[k].x), __uint_as_float(v[k].y),
                                                        __uint_as_float(v[k].z), 0.0f);
      }
      if (!__all_sync(0xffffffffu, ok)) return;
      __syncwarp();
      float f[3] = {0.f, 0.f, 0.f}, H[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
      for (int32_t s = s0; s < s1; ++s) {
        if (s - s0 >= tets) continue;
        const float4* r = c.rec + 96LL * s + lane;
        const float4 b0 = __ldg(r), b1 = __ldg(r + 32), b2 = __ldg(r + 64);
        const float B[3][3] = {{b0.x, b0.y, b0.z}, {b0.w, b1.x, b1.y}, {b1.z, b1.w, b2.x}};
        const uint32_t q = __float_as_uint(b2.z);
        float p[4][3];
#pragma unroll
        for (int l = 0; l < 4; ++l) {
          const float4 y = mine[q >> (8 * l) & 0xff];
          p[l][0] = y.x;
          p[l][1] = y.y;
          p[l][2] = y.z;
        }
        vbd_term(a, p, B, b2.y, __float_as_int(b2.w), f, H);
      }
      group_sum<kVL>(f, H);
      if (gl == 0 && vi >= 0) {
        const float x[3] = {mine[0].x, mine[0].y, mine[0].z};  // (the vertex itself comes first)
        float y[3] = {x[0], x[1], x[2]}, z[3];
        if (w != 0.0f) vbd_solve(a, inertia, x, f, H, y);
#pragma unroll
        for (int d = 0; d < 3; ++d) z[d] = cheb && w > 0.0f ? y[d] + om * (y[d] - x[d]) : y[d];
        pdev::put_tagged(c.xa + vi, __float_as_uint(y[0]), __float_as_uint(y[1]), __float_as_uint(y[2]),
                         n + 1);
        if (c.xb != c.xa)
          pdev::put_tagged(c.xb + vi, __float_as_uint(z[0]), __float_as_uint(z[1]),
                           __float_as_uint(z[2]), n + 1);
        if (n == c.n_iter - 1 && w != 0.0f) {
#pragma unroll
          for (int d = 0; d < 3; ++d) a.x[3LL * vi + d] = z[d];
        }
      }
      __syncwarp();
    }
  }
}

// With a grid barrier between the colours, for meshes with a vertex of more
// neighbours than a warp of the above keeps
struct VColorArgs {
  const int32_t* order;
  const int32_t* off;
  int32_t n_colors;
  int32_t n_iter;
  float rho;
  const float* om;
  unsigned long long spin_ns;
  GridSync* gs;
  int32_t* status;
};

// solve with method 'color' (_solve_vertex_range, cons/vbd.py:267-361): the
// vertices of one colour share no tet; kVL lanes per vertex; grid barriers
// between colours and around the Chebyshev step
__global__ void __launch_bounds__(kLT) k_vbd_color(VArgs a, VColorArgs c) {
  unsigned long long gen = 0;
  constexpr int kPerWarp = 32 / kVL;
  const int lane = threadIdx.x & 31;
  const int sub = lane / kVL, gl = lane % kVL;
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const int64_t tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int32_t n = 0; n < c.n_iter; ++n) {
    const bool cheb = c.rho > 0.0f && n >= 1;
    for (int32_t col = 0; col < c.n_colors; ++col) {
      const int32_t b = c.off[col], e = c.off[col + 1];
      for (int64_t base = b + warp * kPerWarp; base < e; base += nwarps * kPerWarp) {
        const int64_t idx = base + sub;
        int64_t vi = 0;
        float w = 0.0f;
        if (idx < e) {
          vi = c.order[idx];
          w = a.invm[vi];
        }
        float f[3] = {0.f, 0.f, 0.f}, H[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        if (w != 0.0f)
          for (int32_t j = a.adj_ptr[vi] + gl; j < a.adj_ptr[vi + 1]; j += kVL) vbd_entry(a, a.adj[j], f, H);
        group_sum<kVL>(f, H);
        if (gl == 0 && w != 0.0f) vbd_finish(a, vi, w, f, H);
      }
      const bool last = n == c.n_iter - 1 && col == c.n_colors - 1 && !cheb;
      if (!last && !pdev::grid_sync(c.gs, c.status, c.spin_ns, gen)) return;
    }
    if (cheb) {
      vbd_chebyshev(a, c.om[n], tid, stride);
      if (n != c.n_iter - 1 && !pdev::grid_sync(c.gs, c.status, c.spin_ns, gen)) return;
    }
  }
}

// make_prediction (cons/vbd.py:125-132)
__global__ void k_vbd_predict(float* __restrict__ x, const float* __restrict__ v,
                              float* __restrict__ xo, float* __restrict__ xt, int64_t n3, float dt,
                              float gx, float gy, float gz) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n3;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int c = static_cast<int>(i % 3);
    const float g = c == 0 ? gx : (c == 1 ? gy : gz);
    const float p = x[i];
    xo[i] = p;
    const float t = p + v[i] * dt + g * dt * dt;
    xt[i] = t;
    x[i] = t;
  }
}

// update_vel (cons/vbd.py:161-166)
__global__ void k_vbd_vel(const float* __restrict__ x, const float* __restrict__ xo,
                          float* __restrict__ v, int64_t n3, float damp, float dt) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n3;
       i += (int64_t)gridDim.x * blockDim.x)
    v[i] = damp * (x[i] - xo[i]) / dt;
}

int blocks_for(int64_t n) {
  const int64_t g = (n + kLT - 1) / kLT;
  return static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(g, 4096)));
}

// one block per SM (cooperative launches; fewer blocks keep the barrier
// cheap, and a colour rarely has more elements than 152 x 256 threads)
int coop_grid(const void* fn, int threads) {
  int dev = 0, sms = 0, occ = 0;
  MGPBD_CUDA(cudaGetDevice(&dev));
  MGPBD_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  MGPBD_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, threads, 0));
  require(occ >= 1, MGPBD_ECUDA, "local solver kernel cannot be resident");
  return sms;
}

constexpr int kFlowSmem = 28 * sizeof(float);  // bytes a thread (XFlowTet)

// Warps of a colour kernel that waits for vertices: `ahead` times the chunks of
// a colour, which have loaded what does not wait when their turn comes; others
// only poll, in the way of those that can go on.
void flow_shape(const void* fn, int smem, int most, double ahead, int64_t chunks, int32_t colors,
                int* grid, int* threads) {
  int dev = 0, sms = 0, occ = 0;
  MGPBD_CUDA(cudaGetDevice(&dev));
  MGPBD_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const int64_t warps = std::max<int64_t>(16, std::llround(ahead * chunks / std::max(colors, 1)));
  const int per = static_cast<int>(std::min<int64_t>(most, ceil_div(warps, sms)));
  *grid = static_cast<int>(std::min<int64_t>(sms, ceil_div(warps, per)));
  *threads = 32 * per;
  MGPBD_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, *threads, smem * *threads));
  require(occ >= 1, MGPBD_ECUDA, "local solver kernel cannot be resident");
}

// host copy of t_i with ids validated
std::vector<int32_t> host_tets(const int32_t* t_i, int32_t nt, int32_t nv) {
  std::vector<int32_t> h(static_cast<size_t>(nt) * 4);
  MGPBD_CUDA(cudaMemcpy(h.data(), t_i, sizeof(int32_t) * h.size(), cudaMemcpyDeviceToHost));
  for (int32_t v : h) require(v >= 0 && v < nv, MGPBD_EINVAL, "tet vertex id out of range");
  return h;
}

// whether no tet lists a vertex twice
bool distinct_vertices(const std::vector<int32_t>& ht) {
  for (size_t k = 0; k < ht.size(); k += 4) {
    const int32_t *q = &ht[k];
    if (q[0] == q[1] || q[0] == q[2] || q[0] == q[3] || q[1] == q[2] || q[1] == q[3] || q[2] == q[3])
      return false;
  }
  return true;
}

void upload(DevBuf<int32_t>& d, const std::vector<int32_t>& h, cudaStream_t s) {
  d.alloc(std::max<int64_t>(1, static_cast<int64_t>(h.size())));
  if (!h.empty())
    MGPBD_CUDA(cudaMemcpyAsync(d.p, h.data(), sizeof(int32_t) * h.size(), cudaMemcpyHostToDevice, s));
  MGPBD_CUDA(cudaStreamSynchronize(s));
}

}  // namespace

// ---------------------------------------------------------------------------

LazyStatus::~LazyStatus() {
  if (ev_) cudaEventDestroy(ev_);
  if (host_) cudaFreeHost(host_);
}

void LazyStatus::record(int32_t* dev, cudaStream_t s) {
  if (!host_) {
    MGPBD_CUDA(cudaMallocHost(&host_, sizeof(int32_t)));
    *host_ = 0;
    MGPBD_CUDA(cudaEventCreateWithFlags(&ev_, cudaEventDisableTiming));
  }
  MGPBD_CUDA(cudaMemcpyAsync(host_, dev, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
  MGPBD_CUDA(cudaEventRecord(ev_, s));
  dev_ = dev;
  stream_ = s;
  pending_ = true;
}

void LazyStatus::check(const char* what) {
  if (!pending_) return;
  const cudaError_t e = cudaEventQuery(ev_);
  if (e == cudaErrorNotReady) return;
  MGPBD_CUDA(e);
  pending_ = false;
  if (static_cast<uint32_t>(*host_) & MGPBD_STATUS_SYNC_TIMEOUT) {
    // reported once: the next launch starts afresh
    MGPBD_CUDA(cudaMemsetAsync(dev_, 0, sizeof(int32_t), stream_));
    throw Error(MGPBD_ECUDA, std::string(what) + ": a grid barrier wait timed out");
  }
}

void LazyStatus::wait(const char* what) {
  if (!pending_) return;
  MGPBD_CUDA(cudaEventSynchronize(ev_));
  check(what);
}

Xpbd::Xpbd(const mgpbd_xpbd_params& p) : p_(p) {
  require(p.dt > 0.0f, MGPBD_EINVAL, "xpbd: dt must be positive");
  require(p.method >= MGPBD_XPBD_DEFAULT && p.method <= MGPBD_XPBD_GRAPH_COLORING, MGPBD_EINVAL,
          "xpbd: unknown method");
}

void Xpbd::set_mesh(float* x, const float* x_ref, const float* invm, const int32_t* t_i,
                    const float* t_m, int32_t nv, int32_t nt) {
  require(x && x_ref && invm && t_i && t_m, MGPBD_EINVAL, "xpbd: null mesh pointer");
  require(nv > 0 && nt > 0, MGPBD_EINVAL, "xpbd: empty mesh");
  require(static_cast<int64_t>(nt) * 4 < INT32_MAX, MGPBD_ERANGE, "xpbd: too many tets");
  require(reinterpret_cast<uintptr_t>(t_i) % 16 == 0, MGPBD_EINVAL, "xpbd: t_i must be 16-byte aligned");
  const std::vector<int32_t> ht = host_tets(t_i, nt, nv);
  x_ = x;
  invm_ = invm;
  t_i_ = t_i;
  t_m_ = t_m;
  nv_ = nv;
  nt_ = nt;
  cudaStream_t s = stream_;
  B_.alloc(9LL * nt);
  lam_h_.alloc(nt);
  lam_d_.alloc(nt);
  MGPBD_CUDA(cudaMemsetAsync(lam_h_.p, 0, sizeof(float) * nt, s));
  MGPBD_CUDA(cudaMemsetAsync(lam_d_.p, 0, sizeof(float) * nt, s));
  k_rest_shape<<<blocks_for(nt), kLT, 0, s>>>(x_ref, reinterpret_cast<const int4*>(t_i), nt, B_.p,
                                              nullptr);
  MGPBD_CHECK_LAUNCH();
  status_.alloc(1);
  MGPBD_CUDA(cudaMemsetAsync(status_.p, 0, sizeof(int32_t), s));
  n_colors_ = 0;
  if (p_.method == MGPBD_XPBD_GRAPH_COLORING) {
    const Coloring col = color_elements(ht.data(), nt, 4, nv);
    n_colors_ = col.n_colors;
    gs_.alloc(1);
    n_chunks_ = 0;
    if (distinct_vertices(ht)) {
      build_flow(col, ht);
      // (57 chunks a colour, 10 passes: 76 warps 814 us, 304 warps 916; 137
      // chunks: 76 warps 1232 us, 152 886, 304 942)
      flow_shape(reinterpret_cast<const void*>(k_xpbd_flow), kFlowSmem, kXpbdWarps, 1.25, n_chunks_,
                 n_colors_, &grid_, &threads_);
    } else {
      upload(order_, col.ordered, s);
      upload(offsets_, col.offsets, s);
      grid_ = coop_grid(reinterpret_cast<const void*>(k_xpbd_color), kLT);
    }
  }
  MGPBD_CUDA(cudaStreamSynchronize(s));
}

// The tets in chunks of 32 of one colour, and each vertex's order of updates
void Xpbd::build_flow(const Coloring& col, const std::vector<int32_t>& ht) {
  std::vector<int32_t> deg(nv_, 0), tet;
  for (int32_t c = 0; c < col.n_colors; ++c) {
    for (int32_t i = col.offsets[c]; i < col.offsets[c + 1]; ++i) tet.push_back(col.ordered[i]);
    while (tet.size() % 32) tet.push_back(-1);
  }
  const size_t n = tet.size();
  std::vector<int32_t> vid(4 * n, -1), rank(4 * n, 0), total(4 * n, 0);
  for (size_t i = 0; i < n; ++i)
    for (int l = 0; l < 4 && tet[i] >= 0; ++l) {
      const int32_t v = ht[4 * static_cast<size_t>(tet[i]) + l];
      vid[4 * i + l] = v;
      rank[4 * i + l] = deg[v]++;
    }
  for (size_t i = 0; i < 4 * n; ++i)
    if (vid[i] >= 0) total[i] = deg[vid[i]];
  cudaStream_t s = stream_;
  upload(f_vid_, vid, s);
  upload(f_rank_, rank, s);
  upload(f_deg_, total, s);
  upload(order_, tet, s);
  f_B_.alloc(9 * static_cast<int64_t>(n));
  xt_.alloc(nv_);
  k_flow_rest<<<blocks_for(static_cast<int64_t>(n)), kLT, 0, s>>>(B_.p, order_.p, static_cast<int64_t>(n),
                                                                  f_B_.p);
  MGPBD_CHECK_LAUNCH();
  n_chunks_ = static_cast<int32_t>(n / 32);
}

void Xpbd::preupdate() {
  require(x_ != nullptr, MGPBD_ESTATE, "xpbd: set_mesh has not been called");
  MGPBD_CUDA(cudaMemsetAsync(lam_h_.p, 0, sizeof(float) * nt_, stream_));
  MGPBD_CUDA(cudaMemsetAsync(lam_d_.p, 0, sizeof(float) * nt_, stream_));
}

void Xpbd::update(int32_t passes) {
  require(x_ != nullptr, MGPBD_ESTATE, "xpbd: set_mesh has not been called");
  require(passes >= 0, MGPBD_EINVAL, "xpbd: negative pass count");
  lazy_.check("xpbd colour kernel");
  if (passes == 0) return;
  XArgs a;
  a.x = x_;
  a.invm = invm_;
  a.t_i = reinterpret_cast<const int4*>(t_i_);
  a.t_m = t_m_;
  a.B = B_.p;
  a.lh = lam_h_.p;
  a.ld = lam_d_.p;
  a.nt = nt_;
  a.dt = p_.dt;
  a.ha = p_.hydro_alpha;
  a.da = p_.devia_alpha;
  cudaStream_t s = stream_;
  if (p_.method == MGPBD_XPBD_DEFAULT) {
    for (int32_t i = 0; i < passes; ++i) {
      k_xpbd_all<<<blocks_for(nt_), kLT, 0, s>>>(a);
      MGPBD_CHECK_LAUNCH();
    }
    return;
  }
  if (p_.method == MGPBD_XPBD_GAUSS_SEIDEL) {
    k_xpbd_serial<<<1, 32, 0, s>>>(a, passes);
    MGPBD_CHECK_LAUNCH();
    return;
  }
  MGPBD_CUDA(cudaMemsetAsync(gs_.p, 0, sizeof(GridSync), s));
  if (n_chunks_ > 0) {
    FlowArgs f;
    f.vid = reinterpret_cast<const int4*>(f_vid_.p);
    f.rank = reinterpret_cast<const int4*>(f_rank_.p);
    f.deg = reinterpret_cast<const int4*>(f_deg_.p);
    f.tet = order_.p;
    f.B = f_B_.p;
    f.xt = xt_.p;
    f.n_chunks = n_chunks_;
    f.passes = passes;
    f.spin_ns = spin_ns_;
    f.gs = gs_.p;
    f.status = status_.p;
    k_flow_start<<<blocks_for(nv_), kLT, 0, s>>>(x_, xt_.p, nv_);
    MGPBD_CHECK_LAUNCH();
    void* args[] = {&a, &f};
    MGPBD_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(k_xpbd_flow), dim3(grid_),
                                           dim3(threads_), args, kFlowSmem * threads_, s));
  } else {
    ColorArgs c;
    c.order = order_.p;
    c.off = offsets_.p;
    c.n_colors = n_colors_;
    c.passes = passes;
    c.spin_ns = spin_ns_;
    c.gs = gs_.p;
    c.status = status_.p;
    void* args[] = {&a, &c};
    MGPBD_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(k_xpbd_color), dim3(grid_),
                                           dim3(kLT), args, 0, s));
  }
  MGPBD_CHECK_LAUNCH();
  lazy_.record(status_.p, s);
}

// ---------------------------------------------------------------------------

Vbd::Vbd(const mgpbd_vbd_params& p) : p_(p) {
  require(p.dt > 0.0f, MGPBD_EINVAL, "vbd: dt must be positive");
  require(p.method == MGPBD_VBD_SERIAL || p.method == MGPBD_VBD_COLOR, MGPBD_EINVAL,
          "vbd: unknown method");
  require(p.n_iterations >= 0, MGPBD_EINVAL, "vbd: negative iteration count");
  // Lame parameters in double, then float32 (cons/vbd.py:41-46)
  const double E = p.youngs_modulus, nu = p.poissons_ratio;
  mu_ = static_cast<float>(E / (2.0 * (1.0 + nu)));
  lam_ = static_cast<float>(E * nu / ((1.0 + nu) * (1.0 - 2.0 * nu)));
  // the omega sequence of solve (cons/vbd.py:141-151), in double like the
  // Python loop, passed to the kernel as float32
  omegas_.assign(static_cast<size_t>(p.n_iterations), 1.0f);
  double om = 1.0;
  const double r = p.rho;
  for (int32_t n = 0; n < p.n_iterations; ++n) {
    if (r > 0.0 && n >= 1) {
      om = n == 1 ? 2.0 / (2.0 - r * r) : 4.0 / (4.0 - r * r * om);
    }
    omegas_[n] = static_cast<float>(om);
  }
}

void Vbd::set_mesh(float* x, const float* x_ref, const float* invm, const int32_t* t_i, int32_t nv,
                   int32_t nt) {
  require(x && x_ref && invm && t_i, MGPBD_EINVAL, "vbd: null mesh pointer");
  require(nv > 0 && nt > 0, MGPBD_EINVAL, "vbd: empty mesh");
  require(static_cast<int64_t>(nt) * 4 < INT32_MAX, MGPBD_ERANGE, "vbd: too many tets");
  require(reinterpret_cast<uintptr_t>(t_i) % 16 == 0, MGPBD_EINVAL, "vbd: t_i must be 16-byte aligned");
  const std::vector<int32_t> ht = host_tets(t_i, nt, nv);
  x_ = x;
  x_ref_ = x_ref;
  invm_ = invm;
  t_i_ = t_i;
  nv_ = nv;
  nt_ = nt;
  inited_ = false;
  cudaStream_t s = stream_;
  // vertex -> (tet, local) entries, tets ascending (cons/vbd.py:68-96)
  std::vector<int32_t> ptr(static_cast<size_t>(nv) + 1, 0), ent(ht.size());
  for (int32_t v : ht) ptr[v + 1] += 1;
  for (int32_t v = 0; v < nv; ++v) ptr[v + 1] += ptr[v];
  std::vector<int32_t> fill(ptr.begin(), ptr.end() - 1);
  for (int32_t t = 0; t < nt; ++t)
    for (int l = 0; l < 4; ++l) ent[fill[ht[4 * static_cast<size_t>(t) + l]]++] = 4 * t + l;
  upload(adj_ptr_, ptr, s);
  upload(adj_, ent, s);
  v_.alloc(3LL * nv);
  x_old_.alloc(3LL * nv);
  x_tilde_.alloc(3LL * nv);
  x_prev_.alloc(3LL * nv);
  dm_inv_.alloc(9LL * nt);
  vol_.alloc(nt);
  MGPBD_CUDA(cudaMemsetAsync(v_.p, 0, sizeof(float) * 3 * nv, s));
  MGPBD_CUDA(cudaMemsetAsync(x_old_.p, 0, sizeof(float) * 3 * nv, s));
  MGPBD_CUDA(cudaMemsetAsync(x_tilde_.p, 0, sizeof(float) * 3 * nv, s));
  MGPBD_CUDA(cudaMemsetAsync(x_prev_.p, 0, sizeof(float) * 3 * nv, s));
  om_.alloc(std::max<int64_t>(1, static_cast<int64_t>(omegas_.size())));
  if (!omegas_.empty())
    MGPBD_CUDA(cudaMemcpyAsync(om_.p, omegas_.data(), sizeof(float) * omegas_.size(),
                               cudaMemcpyHostToDevice, s));
  status_.alloc(1);
  MGPBD_CUDA(cudaMemsetAsync(status_.p, 0, sizeof(int32_t), s));
  n_colors_ = 0;
  if (p_.method == MGPBD_VBD_COLOR) {
    const Coloring col = color_vertices(ht.data(), nt, 4, nv);
    n_colors_ = col.n_colors;
    gs_.alloc(1);
    if (!build_flow(col, ht, ptr, ent)) {
      upload(order_, col.ordered, s);
      upload(offsets_, col.offsets, s);
      grid_ = coop_grid(reinterpret_cast<const void*>(k_vbd_color), kLT);
    }
  }
  MGPBD_CUDA(cudaStreamSynchronize(s));
}

// The vertices in chunks of a warp's, of one colour, their neighbours and tets in the
// order of a warp's lanes.  False: a vertex has too many neighbours.
bool Vbd::build_flow(const Coloring& col, const std::vector<int32_t>& ht,
                     const std::vector<int32_t>& ptr, const std::vector<int32_t>& ent) {
  n_chunks_ = 0;
  std::vector<int32_t> color(nv_), vert;
  for (int32_t c = 0; c < col.n_colors; ++c) {
    for (int32_t i = col.offsets[c]; i < col.offsets[c + 1]; ++i) {
      color[col.ordered[i]] = c;
      vert.push_back(col.ordered[i]);
    }
    while (vert.size() % kVblk) vert.push_back(-1);
  }
  const size_t chunks = vert.size() / kVblk;
  std::vector<int32_t> nb_off(chunks + 1, 0), rec_off(chunks + 1, 0), entries;
  std::vector<uint32_t> nb, loc;
  std::vector<int32_t> place(nv_, -1);
  int32_t most = 0;
  std::vector<int32_t> list[kVblk];
  nb.reserve(8 * vert.size());
  loc.reserve(2 * ent.size());
  entries.reserve(2 * ent.size());
  for (size_t j = 0; j < chunks; ++j) {
    size_t rounds = 0, steps = 0;
    for (int b = 0; b < kVblk; ++b) {
      const int32_t v = vert[kVblk * j + b];
      list[b].clear();
      if (v < 0) continue;
      list[b].push_back(v);
      for (int32_t e = ptr[v]; e < ptr[v + 1]; ++e)
        for (int l = 0; l < 4; ++l) {
          const int32_t u = ht[4 * static_cast<size_t>(ent[e] >> 2) + l];
          if (u != v && place[u] < 0) {
            place[u] = 1;
            list[b].push_back(u);
          }
        }
      for (int32_t u : list[b]) place[u] = -1;
      if (list[b].size() > static_cast<size_t>(kVblkMost)) return false;
      rounds = std::max(rounds, (list[b].size() + kVL - 1) / kVL);
      steps = std::max<size_t>(steps, (ptr[v + 1] - ptr[v] + kVL - 1) / kVL);
    }
    most = std::max(most, static_cast<int32_t>(rounds));
    const size_t n0 = nb.size(), e0 = entries.size();
    nb.resize(n0 + 32 * rounds, kNoVertex);
    entries.resize(e0 + 32 * steps, -1);
    loc.resize(e0 + 32 * steps, 0);
    for (int b = 0; b < kVblk; ++b) {
      const int32_t v = vert[kVblk * j + b];
      if (v < 0) continue;
      for (size_t m = 0; m < list[b].size(); ++m) {
        const int32_t u = list[b][m];
        place[u] = static_cast<int32_t>(m);
        nb[n0 + 32 * (m / kVL) + kVL * b + m % kVL] = 2u * u + (color[u] < color[v] ? 1u : 0u);
      }
      for (int32_t e = ptr[v]; e < ptr[v + 1]; ++e) {
        const size_t k = e - ptr[v], at = e0 + 32 * (k / kVL) + kVL * b + k % kVL;
        entries[at] = ent[e];
        for (int l = 0; l < 4; ++l)
          loc[at] |= static_cast<uint32_t>(place[ht[4 * static_cast<size_t>(ent[e] >> 2) + l]]) << (8 * l);
      }
      for (int32_t u : list[b]) place[u] = -1;
    }
    nb_off[j + 1] = static_cast<int32_t>(nb.size() / 32);
    rec_off[j + 1] = static_cast<int32_t>(entries.size() / 32);
  }
  cudaStream_t s = stream_;
  upload(order_, vert, s);
  upload(f_nb_off_, nb_off, s);
  upload(f_rec_off_, rec_off, s);
  upload(f_ent_, entries, s);
  upload(f_nb_, std::vector<int32_t>(nb.begin(), nb.end()), s);
  upload(f_loc_, std::vector<int32_t>(loc.begin(), loc.end()), s);
  f_rec_.alloc(std::max<int64_t>(1, 3 * static_cast<int64_t>(entries.size())));
  xa_.alloc(nv_);
  if (p_.rho > 0.0f) xb_.alloc(nv_);
  max_rounds_ = most;
  n_steps_ = rec_off[chunks];
  n_chunks_ = static_cast<int32_t>(chunks);
  // (five colours, half of the vertices in the first; 781 chunks a colour, 10
  // iterations: 1172 warps 197 us, 1953 180)
  flow_shape(reinterpret_cast<const void*>(k_vbd_flow), flow_smem(), kVbdWarps, 2.5, n_chunks_,
             n_colors_, &grid_, &threads_);
  return true;
}

void Vbd::init() {
  require(x_ != nullptr, MGPBD_ESTATE, "vbd: set_mesh has not been called");
  k_rest_shape<<<blocks_for(nt_), kLT, 0, stream_>>>(x_ref_, reinterpret_cast<const int4*>(t_i_),
                                                     nt_, dm_inv_.p, vol_.p);
  MGPBD_CHECK_LAUNCH();
  inited_ = true;
}

void Vbd::make_prediction() {
  require(inited_, MGPBD_ESTATE, "vbd: init has not been called");
  const int64_t n3 = 3LL * nv_;
  k_vbd_predict<<<blocks_for(n3), kLT, 0, stream_>>>(x_, v_.p, x_old_.p, x_tilde_.p, n3, p_.dt,
                                                     p_.gravity[0], p_.gravity[1], p_.gravity[2]);
  MGPBD_CHECK_LAUNCH();
}

void Vbd::update_vel() {
  require(inited_, MGPBD_ESTATE, "vbd: init has not been called");
  const int64_t n3 = 3LL * nv_;
  k_vbd_vel<<<blocks_for(n3), kLT, 0, stream_>>>(x_, x_old_.p, v_.p, n3, p_.damp, p_.dt);
  MGPBD_CHECK_LAUNCH();
}

void Vbd::solve() {
  require(inited_, MGPBD_ESTATE, "vbd: init has not been called");
  lazy_.check("vbd colour kernel");
  if (p_.n_iterations == 0) return;
  VArgs a;
  a.x = x_;
  a.invm = invm_;
  a.t_i = reinterpret_cast<const int4*>(t_i_);
  a.dm = dm_inv_.p;
  a.vol = vol_.p;
  a.adj_ptr = adj_ptr_.p;
  a.adj = adj_.p;
  a.xt = x_tilde_.p;
  a.xo = x_old_.p;
  a.xp = x_prev_.p;
  a.nv = nv_;
  a.mu = mu_;
  a.lam = lam_;
  a.dt = p_.dt;
  a.h2 = p_.dt * p_.dt;
  a.kd = p_.damping;
  a.keep_prev = p_.rho > 0.0f ? 1 : 0;
  cudaStream_t s = stream_;
  if (p_.method == MGPBD_VBD_SERIAL) {
    k_vbd_serial<<<1, kLT, 0, s>>>(a, om_.p, p_.n_iterations, p_.rho);
    MGPBD_CHECK_LAUNCH();
    return;
  }
  MGPBD_CUDA(cudaMemsetAsync(gs_.p, 0, sizeof(GridSync), s));
  if (n_chunks_ > 0) {
    VFlowArgs f;
    f.vert = order_.p;
    f.nb_off = f_nb_off_.p;
    f.nb = reinterpret_cast<const uint32_t*>(f_nb_.p);
    f.rec_off = f_rec_off_.p;
    f.rec = f_rec_.p;
    f.ent = f_ent_.p;
    f.loc = reinterpret_cast<const uint32_t*>(f_loc_.p);
    f.xa = xa_.p;
    f.xb = p_.rho > 0.0f ? xb_.p : xa_.p;
    f.n_chunks = n_chunks_;
    f.n_steps = n_steps_;
    f.max_rounds = max_rounds_;
    f.n_iter = p_.n_iterations;
    f.rho = p_.rho;
    f.om = om_.p;
    f.spin_ns = spin_ns_;
    f.gs = gs_.p;
    f.status = status_.p;
    if (n_steps_ > 0) {
      k_vbd_rest<<<blocks_for(32LL * n_steps_), kLT, 0, s>>>(dm_inv_.p, vol_.p, f);
      MGPBD_CHECK_LAUNCH();
    }
    k_flow_start<<<blocks_for(nv_), kLT, 0, s>>>(x_, xa_.p, nv_);
    MGPBD_CHECK_LAUNCH();
    if (f.xb != f.xa) {
      k_flow_start<<<blocks_for(nv_), kLT, 0, s>>>(x_, xb_.p, nv_);
      MGPBD_CHECK_LAUNCH();
    }
    void* args[] = {&a, &f};
    MGPBD_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(k_vbd_flow), dim3(grid_),
                                           dim3(threads_), args, flow_smem() * threads_, s));
  } else {
    VColorArgs c;
    c.order = order_.p;
    c.off = offsets_.p;
    c.n_colors = n_colors_;
    c.n_iter = p_.n_iterations;
    c.rho = p_.rho;
    c.om = om_.p;
    c.spin_ns = spin_ns_;
    c.gs = gs_.p;
    c.status = status_.p;
    void* args[] = {&a, &c};
    MGPBD_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(k_vbd_color), dim3(grid_),
                                           dim3(kLT), args, 0, s));
  }
  MGPBD_CHECK_LAUNCH();
  lazy_.record(status_.p, s);
}

void* Vbd::field(int32_t f, int64_t* count) {
  switch (f) {
    case MGPBD_VBD_FIELD_V: *count = 3LL * nv_; return v_.p;
    case MGPBD_VBD_FIELD_X_OLD: *count = 3LL * nv_; return x_old_.p;
    case MGPBD_VBD_FIELD_X_TILDE: *count = 3LL * nv_; return x_tilde_.p;
    case MGPBD_VBD_FIELD_DM_INV: *count = 9LL * nt_; return dm_inv_.p;
    case MGPBD_VBD_FIELD_REST_VOL: *count = nt_; return vol_.p;
    default: throw Error(MGPBD_EINVAL, "vbd: unknown field");
  }
}

}  // namespace mgpbd
