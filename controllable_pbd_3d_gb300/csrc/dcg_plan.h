// The partition of the dual CG (dcg.cuh), built on the host.
#pragma once

#include <cstdint>
#include <vector>

namespace mgpbd {

constexpr int kDMaxThreads = 768;
constexpr int kDMaxWarps = kDMaxThreads / 32;
constexpr int kDColumns = 512;    // tensor memory columns
// bytes of one row of 32 entries: gradient x and y, z (from kDRowZ), 16-bit
// byte offsets of x (from kDRowX)
constexpr int kDRow = 448, kDRowZ = 256, kDRowX = 384;
constexpr int kDMaxCluster = 16;
// more than half of an SM's shared memory: one block per SM (dcg.cu)
constexpr int kDMinSmem = 120 * 1024;

// What one block owns (all offsets into the plan's arrays)
struct DBlock {
  int32_t c0, nT, nE;        // constraints: c0 .. c0 + nT + nE, 4-slot ones first,
                             // in each group those on private vertices first
  int32_t nTi, nEi;          // how many of them those are
  int32_t p0, nposS, npos;   // vertex positions from p0; shared ones (first), all
  int32_t s0, nsl;           // slices from s0
  int32_t r0, nrows;         // rows from r0
  int32_t t0, ntgt, nrecv;   // cluster: its sends from t0, partials it receives per exchange
  int32_t prob, rank, size;  // its problem (-1: none), its place among that problem's blocks, how many
  int32_t kT, kE;            // 4-slot / length constraints a thread keeps in tensor memory
};

// Where the blocks of each problem are: size[k] of them from block first[k], of
// `blocks` in clusters of `cluster`.  The blocks that no problem has only meet
// the rest of their cluster.
struct DcgPlaces {
  int32_t cluster = 0, blocks = 0;
  std::vector<int32_t> first, size;
};

// Arrangements of independent bodies, by the number of vertex entries of each
// (and how soft it is, or nothing), on clusters of 16, 8 and 4 blocks, of which
// n16, n8 and n4 are resident at once (0: none): the one whose schedule should
// be shortest first.
std::vector<DcgPlaces> dcg_place_bodies(const std::vector<double>& entries,
                                        const std::vector<double>& softness, int n16, int n8, int n4);

// The vertex sums of one warp: slices s .. p - 1 of shared vertices, p .. e - 1
// of private ones (from the block's s0); its rows from row (from r0), the
// first `held` of them in shared memory from row srow there
struct DWarp {
  int32_t s, p, e, row, rows, srow, held;
};

// Host-built partition of one or several independent problems (bodies).
struct DcgPlan {
  int32_t nprob = 0, nblk = 0;  // blocks in all
  int32_t csize = 0;            // blocks of a cluster
  bool cluster = false;  // blocks of a problem form one thread-block cluster
  bool onchip = false;   // every block's operator fits in tensor and shared memory
  int32_t threads = kDMaxThreads;  // per block, a multiple of 128
  int32_t kT = 0, kE = 0;  // the most of DBlock::kT, kE
  int32_t srows = 0;     // rows a block keeps in shared memory
  int32_t smem = 0;      // dynamic shared memory per block
  int32_t cmax = 0, posmax = 0, possmax = 0, slmax = 0, tmax = 0, rmax = 0;  // largest counts of a block
  int64_t n_rows = 0;
  int64_t n_slots = 0;   // grid: exchange slots
  std::vector<DBlock> blocks;     // nblk
  std::vector<DWarp> warps;       // threads / 32 per block
  std::vector<int32_t> perm;      // (nc) constraint of each plan position
  std::vector<uint16_t> ti;       // (nc, 4) byte offsets of its vertices' u in its block
  std::vector<int32_t> pos_v;     // (positions) vertex id, -1: empty
  // (positions, 2) shared vertices: where its partials are -- grid: the
  // first exchange slot; cluster: receive slot | first send << 16 -- and
  // blocks that touch it << 8 | this block's place among them; 0 otherwise
  std::vector<uint32_t> pos_info;
  std::vector<uint32_t> tgt;      // cluster: per send, rank << 16 | receive slot there
  // (slices, 2): rows; first position | log2 of the lanes per vertex << 16
  std::vector<uint32_t> slice;
  std::vector<int32_t> row_ent;   // (rows, 32) constraint * 4 + slot, -1: padding
  std::vector<uint16_t> row_idx;  // (rows, 32) the constraint's position in its block
};

// Shared memory of a block: u (16 B per position, at 0), x (4 B per
// constraint), the shared positions' exchange entries, slices; cluster:
// targets of the sends, receive slots (twice); rows
struct DcgSmem {
  int32_t x, info, slice, tgt, rbuf, rows;
};
inline DcgSmem dcg_smem_parts(const DcgPlan& p) {
  auto up = [](int32_t v) { return (v + 15) / 16 * 16; };
  DcgSmem m;
  m.x = 16 * p.posmax;
  m.info = m.x + up(4 * p.cmax);
  m.slice = m.info + up(8 * p.possmax);
  m.tgt = m.slice + up(8 * p.slmax);
  m.rbuf = m.tgt + up(4 * p.tmax);
  m.rows = m.rbuf + 2 * 16 * p.rmax;
  return m;
}

// smem_limit: dynamic shared memory a block may use.  prob[c]: problem of
// constraint c (null: one problem).  Returns false when some block's vectors
// do not fit (the plan is then unusable).
bool build_dcg_plan(const int32_t* t_i, int32_t nt, int32_t n4, int32_t nv, const float* x_ref,
                    const int32_t* prob, const DcgPlaces& places, bool cluster, int threads,
                    int32_t smem_limit, DcgPlan& plan);
// the places of one problem on nblk blocks, of nprob problems on nblk each
DcgPlaces dcg_places(int32_t nprob, int32_t nblk);

// y = (J W J^T + alpha~) x in float64 by way of the plan's arrays, as the
// kernel goes (tests)
void dcg_plan_apply(const DcgPlan& plan, const float* gradC, const float* invm, const float* alpha,
                    const float* x, double* y);

}  // namespace mgpbd
