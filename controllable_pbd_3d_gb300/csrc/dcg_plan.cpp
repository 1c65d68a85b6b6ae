// Host side of the partitioned dual CG (dcg.cuh): the bisection of the
// constraints and each block's local numbering.
#include "dcg_plan.h"

#include <algorithm>
#include <array>
#include <cmath>
#include <numeric>

namespace mgpbd {

namespace {

struct Item {
  float c[3];
  int32_t id;
};

// Splits items[lo, hi) so that the left part holds about `share` of the
// weight, by the coordinate `dim` (ties by constraint id, so the split is a
// function of the mesh alone).  Weighted quickselect.
int64_t split(Item* it, int64_t lo, int64_t hi, int dim, double share, int32_t n4) {
  auto weight = [n4](const Item& a) { return a.id < n4 ? 4.0 : 2.0; };
  auto less = [dim](const Item& a, const Item& b) {
    return a.c[dim] < b.c[dim] || (a.c[dim] == b.c[dim] && a.id < b.id);
  };
  double total = 0.0;
  for (int64_t i = lo; i < hi; ++i) total += weight(it[i]);
  double want = total * share;
  while (hi - lo > 32) {
    const Item a = it[lo], b = it[lo + (hi - lo) / 2], c = it[hi - 1];
    const Item p = less(a, b) ? (less(b, c) ? b : (less(a, c) ? c : a))
                              : (less(a, c) ? a : (less(b, c) ? c : b));
    Item* m = std::partition(it + lo, it + hi, [&](const Item& v) { return less(v, p); });
    const int64_t mid = m - it;
    if (mid == lo) {  // the pivot is the smallest: it alone goes left
      Item* q = std::min_element(it + lo, it + hi, less);
      std::swap(*q, it[lo]);
      if (weight(it[lo]) > want) return lo;
      want -= weight(it[lo]);
      ++lo;
      continue;
    }
    double w = 0.0;
    for (int64_t i = lo; i < mid; ++i) w += weight(it[i]);
    if (w > want) {
      hi = mid;
    } else {
      want -= w;
      lo = mid;
    }
  }
  std::sort(it + lo, it + hi, less);
  while (lo < hi && want >= weight(it[lo])) want -= weight(it[lo++]);
  return lo;
}

// Cuts items[lo, hi) into n parts of equal weight; out[k] = first item of
// part k (out[n] is the caller's).
void bisect(Item* it, int64_t lo, int64_t hi, int n, int64_t* out, int32_t n4) {
  out[0] = lo;
  if (n <= 1) return;
  float mn[3] = {1e30f, 1e30f, 1e30f}, mx[3] = {-1e30f, -1e30f, -1e30f};
  for (int64_t i = lo; i < hi; ++i)
    for (int k = 0; k < 3; ++k) {
      mn[k] = std::min(mn[k], it[i].c[k]);
      mx[k] = std::max(mx[k], it[i].c[k]);
    }
  int dim = 0;
  for (int k = 1; k < 3; ++k)
    if (mx[k] - mn[k] > mx[dim] - mn[dim]) dim = k;
  const int nl = n / 2;
  const int64_t mid = hi > lo ? split(it, lo, hi, dim, static_cast<double>(nl) / n, n4) : lo;
#pragma omp task if (mid - lo > 20000)
  bisect(it, lo, mid, nl, out, n4);
#pragma omp task if (hi - mid > 20000)
  bisect(it, mid, hi, n - nl, out + nl, n4);
#pragma omp taskwait
}

}  // namespace

DcgPlaces dcg_places(int32_t nprob, int32_t nblk) {
  DcgPlaces p;
  p.cluster = nblk;
  p.blocks = nprob * nblk;
  p.size.assign(nprob, nblk);
  for (int32_t k = 0; k < nprob; ++k) p.first.push_back(k * nblk);
  return p;
}

// A body's CG takes its iterations x (23 us + 1.9 us per 1000 entries a block,
// twice that beyond the 12k entries that stay on the chip) (measured: cubes of
// 10 to 20 hexes on 8 and 16 blocks).  The iterations follow from the softness
// (alpha~ by a unit's J W J^T) and, of stiff bodies, from the side: cubes of 6 /
// 12 / 17 hexes need 1682 / 2812 / 3309 in two solves at 0.009, 915 / 1177 / 1152
// at 0.09, 364 / 390 / 391 at 0.9.  Where the softness is not known the sides
// have to do.  An arrangement is judged by its mean over kHardness draws of a
// factor for each body: up to 1.2 for what the formula misses, 2 for an unknown
// softness.  The clusters that are resident at once take the bodies longest
// first.  A cluster of 16 holds one body, two of 8 blocks or four of 4, so that
// the bodies that everything else waits for can have more SMs than the others:
// 16 bodies of 6..18 hexes a side, compliances 1e-7..1e-5, three draws: 93 / 83
// / 109 ms a substep, on clusters of 8 each 132 / 111 / 169; 24 bodies of 8..17:
// 105 / 114 / 99 and 149 / 167 / 161.  The model is of length + volume bodies in
// that range; ARAP packs and softer ones follow the same rule (ms a substep, the
// pack in lockstep over the grid / by this rule): ARAP, 16 bodies of 6..18,
// 1e-7..1e-5 257 / 72, 1e-5..1e-3 39 / 12; 40 of 4..12 249 / 61 and 40 / 11;
// length + volume, 16 of 6..18, 1e-5..1e-3 34 / 10.
std::vector<DcgPlaces> dcg_place_bodies(const std::vector<double>& entries,
                                        const std::vector<double>& softness, int n16, int n8, int n4) {
  constexpr int kHardness = 16;
  const int32_t nb = static_cast<int32_t>(entries.size());
  const bool known = !softness.empty();
  std::vector<double> its(nb);
  for (int32_t k = 0; k < nb; ++k) {
    const double side = std::cbrt(entries[k] / 36.0);  // hexes, length + volume
    its[k] = known ? 1.0 / (std::pow(std::max(softness[k], 1e-12), 0.46) / 372.0 + 1.0 / (97.0 * side * side))
                   : 100.0 * side;
  }
  // body k on 16, 8 and 4 blocks.  All blocks have the memory layout that the
  // fullest one needs, so none is to be fuller than the largest body on 8.
  const double fullest = std::max(12.0, *std::max_element(entries.begin(), entries.end()) / 8000.0);
  auto time_of = [&](int32_t k, int q) {
    const double per = entries[k] / (16 >> q) / 1000.0;
    if (q > 0 && per > fullest) return 1e6 * its[k];
    return its[k] * (23.0 + 1.9 * per + 1.9 * std::max(0.0, per - 12.0));
  };
  std::vector<int32_t> order(nb);  // longest first
  std::iota(order.begin(), order.end(), 0);
  std::stable_sort(order.begin(), order.end(), [&](int32_t a, int32_t b) { return time_of(a, 1) > time_of(b, 1); });
  std::vector<std::array<double, kHardness>> hard(nb);
  uint32_t seed = 1;
  for (auto& h : hard)
    for (double& v : h) {
      seed = seed * 1664525u + 1013904223u;
      v = std::exp2(((seed >> 8) * (2.0 / (1 << 24)) - 1.0) * (known ? 0.25 : 1.0));
    }
  std::vector<std::array<double, 3>> time(nb);
  for (int32_t i = 0; i < nb; ++i)
    for (int q = 0; q < 3; ++q) time[i][q] = time_of(order[i], q);
  struct Job {  // a cluster's bodies: `n` from the at-th longest, on 16 >> q blocks each
    double t;
    int32_t at, n, q;
  };
  // clusters of 16 >> q0: the first `one` bodies have one each, the next `two`
  // half a one, the rest a quarter
  auto jobs_of = [&](int q0, int32_t one, int32_t two) {
    std::vector<Job> jobs;
    for (int32_t i = 0; i < nb;) {
      const int half = i < one ? 0 : i < one + two ? 1 : 2;
      const int32_t end = i < one ? one : i < one + two ? one + two : nb;
      const Job j{time[i][q0 + half], i, std::min<int32_t>(1 << half, end - i), q0 + half};
      jobs.push_back(j);
      i += j.n;
    }
    std::stable_sort(jobs.begin(), jobs.end(), [](const Job& a, const Job& b) { return a.t > b.t; });
    return jobs;
  };
  // the longest queue when `resident` clusters take the jobs in their order
  auto cost = [&](const std::vector<Job>& jobs, int resident) {
    double sum = 0.0;
    std::vector<double> busy;
    for (int h = 0; h < kHardness; ++h) {
      busy.assign(resident, 0.0);
      for (const Job& j : jobs) {
        double t = 0.0;
        for (int32_t k = 0; k < j.n; ++k) t = std::max(t, time[j.at + k][j.q] * hard[j.at + k][h]);
        *std::min_element(busy.begin(), busy.end()) += t;
      }
      sum += *std::max_element(busy.begin(), busy.end());
    }
    return sum / kHardness;
  };
  auto place = [&](int q0, const std::vector<Job>& jobs) {
    const int c = 16 >> q0;
    DcgPlaces p;
    p.cluster = c;
    p.blocks = c * static_cast<int32_t>(jobs.size());
    p.first.resize(nb);
    p.size.resize(nb);
    for (size_t b = 0; b < jobs.size(); ++b)
      for (int32_t k = 0; k < jobs[b].n; ++k) {
        const int32_t body = order[jobs[b].at + k], size = 16 >> jobs[b].q;
        p.first[body] = c * static_cast<int32_t>(b) + k * size;
        p.size[body] = size;
      }
    return p;
  };
  std::vector<std::pair<double, DcgPlaces>> all;
  if (n16 > 0) {
    double least = 1e300;
    std::vector<Job> best;
    for (int32_t a = 0; a <= std::min(nb, 48); ++a)
      for (int32_t b = 0; b <= std::min(nb - a, 48); ++b) {
        const std::vector<Job> jobs = jobs_of(0, a, b);
        const double v = cost(jobs, n16);
        if (v < least) {
          least = v;
          best = jobs;
        }
      }
    all.push_back({least, place(0, best)});
  }
  for (int q = 1; q < 3; ++q)
    if (const int n = q == 1 ? n8 : n4; n > 0) {
      std::vector<Job> jobs;
      for (int32_t i = 0; i < nb; ++i) jobs.push_back({time[i][q], i, 1, q});
      all.push_back({cost(jobs, n), place(q, jobs)});
    }
  std::stable_sort(all.begin(), all.end(), [](const auto& a, const auto& b) { return a.first < b.first; });
  std::vector<DcgPlaces> r;
  for (auto& a : all) r.push_back(std::move(a.second));
  if (n16 > 0) r.push_back(place(0, jobs_of(0, nb, 0)));  // (the most memory a body)
  return r;
}

bool build_dcg_plan(const int32_t* t_i, int32_t nt, int32_t n4, int32_t nv, const float* x_ref,
                    const int32_t* prob, const DcgPlaces& places, bool cluster, int threads,
                    int32_t smem_limit, DcgPlan& plan) {
  plan = DcgPlan();
  plan.threads = threads;
  const int32_t nprob = static_cast<int32_t>(places.first.size());
  plan.nprob = nprob;
  plan.nblk = places.blocks;
  plan.csize = places.cluster;
  plan.cluster = cluster;
  const int64_t nb = places.blocks;
  const int warps = threads / 32;
  auto slots = [n4](int32_t c) { return c < n4 ? 4 : 2; };

  // centroids, grouped by problem in the order of their blocks
  std::vector<int32_t> order(nprob);
  std::iota(order.begin(), order.end(), 0);
  std::sort(order.begin(), order.end(), [&](int32_t a, int32_t b) { return places.first[a] < places.first[b]; });
  std::vector<int64_t> count(nprob, 0), pbeg(nprob), pend(nprob);
  for (int32_t c = 0; c < nt; ++c) count[prob ? prob[c] : 0]++;
  int64_t sum = 0;
  for (int32_t k : order) {
    pbeg[k] = sum;
    pend[k] = sum += count[k];
  }
  std::vector<Item> items(nt);
  {
    std::vector<int64_t> cur(pbeg);
    std::vector<int64_t> at(nt);
    for (int32_t c = 0; c < nt; ++c) at[c] = cur[prob ? prob[c] : 0]++;
#pragma omp parallel for schedule(static)
    for (int32_t c = 0; c < nt; ++c) {
      Item& a = items[at[c]];
      a.id = c;
      const int n = slots(c);
      for (int k = 0; k < 3; ++k) {
        float s = 0.0f;
        for (int l = 0; l < n; ++l) s += x_ref[3LL * t_i[4LL * c + l] + k];
        // (a coordinate that is not finite has no place; ordered by it, the
        // bisection would take one constraint a pass)
        a.c[k] = std::isfinite(s) ? s / n : 0.0f;
      }
    }
  }
  plan.blocks.assign(nb, DBlock());
  for (DBlock& B : plan.blocks) {
    B.prob = -1;
    B.size = 1;
  }
  for (int32_t k = 0; k < nprob; ++k)
    for (int32_t r = 0; r < places.size[k]; ++r) {
      DBlock& B = plan.blocks[places.first[k] + r];
      B.prob = k;
      B.rank = r;
      B.size = places.size[k];
    }
  std::vector<int64_t> part(nb + 1, nt);
#pragma omp parallel
#pragma omp single
  for (int32_t k = 0; k < nprob; ++k) {
#pragma omp task
    bisect(items.data(), pbeg[k], pend[k], places.size[k], part.data() + places.first[k], n4);
  }
  part[nb] = nt;
  for (int64_t b = nb - 1; b >= 0; --b)
    if (plan.blocks[b].prob < 0) part[b] = part[b + 1];

  // each block's constraints (4-slot ones first, ascending) and vertices
  plan.perm.resize(nt);
  std::vector<std::vector<int32_t>> verts(nb);
#pragma omp parallel for schedule(dynamic, 1)
  for (int64_t b = 0; b < nb; ++b) {
    int32_t* pm = plan.perm.data() + part[b];
    const int32_t n = static_cast<int32_t>(part[b + 1] - part[b]);
    for (int32_t i = 0; i < n; ++i) pm[i] = items[part[b] + i].id;
    std::sort(pm, pm + n);
    DBlock& B = plan.blocks[b];
    B.c0 = static_cast<int32_t>(part[b]);
    B.nT = static_cast<int32_t>(std::lower_bound(pm, pm + n, n4) - pm);
    B.nE = n - B.nT;
    std::vector<int32_t>& v = verts[b];
    v.reserve(4LL * n);
    for (int32_t i = 0; i < n; ++i)
      for (int l = 0; l < slots(pm[i]); ++l) v.push_back(t_i[4LL * pm[i] + l]);
    std::sort(v.begin(), v.end());
    v.erase(std::unique(v.begin(), v.end()), v.end());
  }

  // vertices of several blocks: consecutive exchange slots, one per block
  // in ascending block order
  std::vector<int32_t> touch(nv, 0), first(nv, -1);
  for (int64_t b = 0; b < nb; ++b)
    for (int32_t v : verts[b]) touch[v]++;
  int64_t ns = 0;
  for (int32_t v = 0; v < nv; ++v)
    if (touch[v] > 1) {
      first[v] = static_cast<int32_t>(ns);
      ns += touch[v];
    }
  if (ns >= INT32_MAX) return false;
  plan.n_slots = ns;
  // the blocks of each shared vertex, and (cluster) where each receives the
  // others' partials: consecutive slots in block order, its own left out
  std::vector<std::vector<uint8_t>> own(nb);
  std::vector<int32_t> who(ns), recv(ns);
  std::vector<int32_t> nrecv(nb, 0);
  {
    std::vector<uint8_t> seen(nv, 0);
    for (int64_t b = 0; b < nb; ++b) {
      own[b].reserve(verts[b].size());
      for (int32_t v : verts[b]) {
        if (touch[v] > 1) {
          who[first[v] + seen[v]] = static_cast<int32_t>(b);
          recv[first[v] + seen[v]] = nrecv[b];
          nrecv[b] += touch[v] - 1;
        }
        own[b].push_back(touch[v] > 1 ? seen[v]++ : 0);
      }
    }
  }

  // local numbering: shared vertices first, each group by falling number of
  // entries
  struct Local {
    std::vector<int32_t> pos_v, row_ent;
    std::vector<uint32_t> pos_info, tgt, slice;
    std::vector<DWarp> warps;
    std::vector<uint16_t> row_idx;
  };
  std::vector<Local> loc(nb);
  plan.ti.assign(4LL * nt, 0);
#pragma omp parallel for schedule(dynamic, 1)
  for (int64_t b = 0; b < nb; ++b) {
    DBlock& B = plan.blocks[b];
    Local& L = loc[b];
    const std::vector<int32_t>& V = verts[b];
    const int32_t n = B.nT + B.nE;
    const int32_t m = static_cast<int32_t>(V.size());
    int32_t* pm = plan.perm.data() + B.c0;
    // constraints on private vertices only come first in their group
    auto inner = [&](int32_t c) {
      for (int l = 0; l < slots(c); ++l)
        if (first[t_i[4LL * c + l]] >= 0) return false;
      return true;
    };
    B.nTi = static_cast<int32_t>(std::stable_partition(pm, pm + B.nT, inner) - pm);
    B.nEi = static_cast<int32_t>(std::stable_partition(pm + B.nT, pm + n, inner) - (pm + B.nT));
    auto local = [&](int32_t v) {
      return static_cast<int32_t>(std::lower_bound(V.begin(), V.end(), v) - V.begin());
    };
    auto repeated = [&](int32_t c, int l) {
      for (int k = 0; k < l; ++k)
        if (t_i[4LL * c + k] == t_i[4LL * c + l]) return true;
      return false;
    };
    std::vector<int32_t> lv(4LL * n), ptr(m + 1, 0);
    for (int32_t i = 0; i < n; ++i)
      for (int l = 0; l < slots(pm[i]); ++l) {
        lv[4LL * i + l] = local(t_i[4LL * pm[i] + l]);
        if (!repeated(pm[i], l)) ptr[lv[4LL * i + l] + 1]++;
      }
    for (int32_t i = 0; i < m; ++i) ptr[i + 1] += ptr[i];
    std::vector<int32_t> cur(ptr.begin(), ptr.end() - 1), ent(ptr[m]), eidx(ptr[m]);
    for (int32_t i = 0; i < n; ++i)
      for (int l = 0; l < slots(pm[i]); ++l)
        if (!repeated(pm[i], l)) {
          const int32_t k = cur[lv[4LL * i + l]]++;
          ent[k] = 4 * pm[i] + l;
          eidx[k] = i;
        }
    std::vector<int32_t> order(m);
    for (int32_t i = 0; i < m; ++i) order[i] = i;
    std::sort(order.begin(), order.end(), [&](int32_t a, int32_t c) {
      const bool sa = first[V[a]] >= 0, sc = first[V[c]] >= 0;
      if (sa != sc) return sa;
      const int32_t na = ptr[a + 1] - ptr[a], nc = ptr[c + 1] - ptr[c];
      return na != nc ? na > nc : a < c;
    });
    int32_t nshared = 0;
    while (nshared < m && first[V[order[nshared]]] >= 0) ++nshared;
    // Slices: a vertex gets as many lanes as bring its run to `goal` rows
    struct Slice {
      int32_t k0, n, shift, rows, group, warp;  // order[k0 ..+ n), log2 lanes
    };
    std::vector<Slice> sl;
    const int32_t goal = std::min(13, std::max(2, ptr[m] / 32 / warps));
    for (int32_t k = 0; k < m;) {
      const int32_t end = k < nshared ? nshared : m;
      const int32_t deg = std::max(1, ptr[order[k] + 1] - ptr[order[k]]);
      int32_t shift = 0;
      while (shift < 5 && (deg + (1 << shift) - 1) >> shift > goal) ++shift;
      // the last ones of a group take the lanes that are left
      while (shift < 5 && (32 >> (shift + 1)) >= end - k) ++shift;
      const int32_t cnt = std::min(32 >> shift, end - k);
      sl.push_back({k, cnt, shift, (deg + (1 << shift) - 1) >> shift, k < nshared ? 0 : 1, 0});
      k += cnt;
    }
    // dealt to the warps, the longest first, each to the warp with the least
    // so far: the shared ones, then the private ones on top (a slice counts
    // two rows more for its overhead)
    std::stable_sort(sl.begin(), sl.end(), [](const Slice& a, const Slice& c) {
      return a.group != c.group ? a.group < c.group : a.rows > c.rows;
    });
    {
      std::vector<int32_t> load(warps, 0);
      for (Slice& s : sl) {
        s.warp = static_cast<int32_t>(std::min_element(load.begin(), load.end()) - load.begin());
        load[s.warp] += s.rows + 2;
      }
    }
    // positions by (group, kind), so that a kind's vertices may be exchanged
    B.nsl = static_cast<int32_t>(sl.size());
    std::vector<int32_t> pos0(B.nsl + 1, 0);
    for (int32_t s = 0; s < B.nsl; ++s) {
      pos0[s + 1] = pos0[s] + (32 >> sl[s].shift);
      if (sl[s].group == 0) B.nposS = pos0[s + 1];
    }
    B.npos = pos0[B.nsl];
    // the slices in warp order, shared ones first
    std::vector<int32_t> seq(B.nsl), row(B.nsl);
    for (int32_t s = 0; s < B.nsl; ++s) seq[s] = s;
    std::stable_sort(seq.begin(), seq.end(),
                     [&](int32_t a, int32_t c) { return sl[a].warp < sl[c].warp; });
    L.slice.resize(2LL * B.nsl);
    L.warps.resize(warps);
    {
      int32_t k = 0, r = 0;
      for (int32_t w = 0; w < warps; ++w) {
        DWarp& W = L.warps[w];
        W.s = k;
        W.row = r;
        while (k < B.nsl && sl[seq[k]].warp == w && sl[seq[k]].group == 0) r += sl[seq[k++]].rows;
        W.p = k;
        while (k < B.nsl && sl[seq[k]].warp == w) r += sl[seq[k++]].rows;
        W.e = k;
        W.rows = r - W.row;
      }
      B.nrows = r;
      r = 0;
      for (int32_t q = 0; q < B.nsl; ++q) {
        const int32_t s = seq[q];
        row[s] = r;
        r += sl[s].rows;
        L.slice[2LL * q] = static_cast<uint32_t>(sl[s].rows);
        L.slice[2LL * q + 1] = static_cast<uint32_t>(pos0[s]) | static_cast<uint32_t>(sl[s].shift) << 16;
      }
    }
    L.pos_v.assign(B.npos, -1);
    L.pos_info.assign(2LL * B.npos, 0);
    // Which vertex of a kind (group, lanes, rows) gets which position: its
    // bank (position mod 8) is chosen against the other vertices that the
    // same 8 threads read in one 16-byte access of u.
    std::vector<int32_t> bp(m + 1, 0), bk;
    {
      std::vector<std::vector<int32_t>> of(m);
      for (int32_t i = 0; i < n; ++i) {
        const int32_t g = i < B.nT ? i / 8 : (B.nT + 7) / 8 + (i - B.nT) / 8;
        for (int l = 0; l < slots(pm[i]); ++l) {
          std::vector<int32_t>& o = of[lv[4LL * i + l]];
          if (std::find(o.rbegin(), o.rbegin() + std::min<size_t>(o.size(), 8), 4 * g + l) ==
              o.rbegin() + std::min<size_t>(o.size(), 8))
            o.push_back(4 * g + l);
        }
      }
      for (int32_t v = 0; v < m; ++v) {
        bk.insert(bk.end(), of[v].begin(), of[v].end());
        bp[v + 1] = static_cast<int32_t>(bk.size());
      }
    }
    std::vector<uint8_t> used(8LL * 4 * ((B.nT + 7) / 8 + (B.nE + 7) / 8 + 1), 0);
    std::vector<int32_t> where(m), at(B.npos, -1);
    for (int32_t s = 0; s < B.nsl;) {
      int32_t e = s;
      std::vector<int32_t> pool;
      while (e < B.nsl && sl[e].group == sl[s].group && sl[e].shift == sl[s].shift &&
             sl[e].rows == sl[s].rows) {
        pool.insert(pool.end(), order.begin() + sl[e].k0, order.begin() + sl[e].k0 + sl[e].n);
        ++e;
      }
      size_t next = 0;
      for (; s < e; ++s)
        for (int32_t k = 0; k < sl[s].n; ++k) {
          const int32_t p = pos0[s] + k;
          size_t best = next;
          int32_t cost = INT32_MAX;
          for (size_t q = next; q < std::min(pool.size(), next + 24) && cost > 0; ++q) {
            int32_t c = 0;
            for (int32_t t = bp[pool[q]]; t < bp[pool[q] + 1]; ++t) c += used[8LL * bk[t] + p % 8];
            if (c < cost) {
              cost = c;
              best = q;
            }
          }
          const int32_t v = pool[best];
          pool[best] = pool[next++];
          for (int32_t t = bp[v]; t < bp[v + 1]; ++t) used[8LL * bk[t] + p % 8]++;
          where[v] = p;
          at[p] = v;
          L.pos_v[p] = V[v];
          if (sl[s].group != 0) continue;
          const int32_t f = first[V[v]], nt_ = touch[V[v]];
          uint32_t at0 = static_cast<uint32_t>(f);
          if (cluster) {
            at0 = static_cast<uint32_t>(recv[f + own[b][v]]) | static_cast<uint32_t>(L.tgt.size()) << 16;
            for (int32_t j = 0; j < nt_; ++j) {
              if (j == own[b][v]) continue;
              // the slots of block who[f + j] leave out its own place j
              const int32_t slot = recv[f + j] + (own[b][v] < j ? own[b][v] : own[b][v] - 1);
              L.tgt.push_back(static_cast<uint32_t>(plan.blocks[who[f + j]].rank) << 16 | static_cast<uint32_t>(slot));
            }
          }
          L.pos_info[2LL * p] = at0;
          L.pos_info[2LL * p + 1] = static_cast<uint32_t>(nt_ << 8 | own[b][v]);
        }
    }
    for (int32_t i = 0; i < n; ++i)
      for (int l = 0; l < slots(pm[i]); ++l)
        plan.ti[4LL * (B.c0 + i) + l] = static_cast<uint16_t>(16 * where[lv[4LL * i + l]]);
    // rows: each vertex's entries dealt to its lanes, row by row the ones
    // whose x lies in a bank that the row has used least (position mod 32)
    L.row_ent.assign(32LL * B.nrows, -1);
    L.row_idx.assign(32LL * B.nrows, 0);
    for (int32_t s = 0; s < B.nsl; ++s) {
      const int32_t lanes = 1 << sl[s].shift;
      for (int32_t r = 0; r < sl[s].rows; ++r) {
        uint8_t bank[32] = {};
        const int64_t o = 32LL * (row[s] + r);
        uint16_t any = 0;
        for (int32_t k = 0; k < sl[s].n; ++k) {
          const int32_t v = at[pos0[s] + k];
          int32_t& e0 = ptr[v];  // entries before it are placed
          const int32_t e1 = cur[v];
          for (int32_t q = 0; q < lanes && e0 < e1; ++q, ++e0) {
            int32_t best = e0;
            for (int32_t e = e0; e < e1 && bank[eidx[best] % 32] > 0; ++e)
              if (bank[eidx[e] % 32] < bank[eidx[best] % 32]) best = e;
            std::swap(ent[best], ent[e0]);
            std::swap(eidx[best], eidx[e0]);
            bank[eidx[e0] % 32]++;
            L.row_ent[o + lanes * k + q] = ent[e0];
            L.row_idx[o + lanes * k + q] = any = static_cast<uint16_t>(eidx[e0]);
          }
        }
        for (int q = 0; q < 32; ++q)
          if (L.row_ent[o + q] < 0) L.row_idx[o + q] = any;
      }
    }
  }

  // offsets, sizes
  int64_t np = 0, nr = 0, nsl = 0, ntg = 0;
  for (int64_t b = 0; b < nb; ++b) {
    DBlock& B = plan.blocks[b];
    const Local& L = loc[b];
    B.nrecv = cluster ? nrecv[b] : 0;
    B.ntgt = static_cast<int32_t>(L.tgt.size());
    if (B.nT + B.nE > 16383 || B.npos > 4095 || B.nrecv > 65535 || B.ntgt > 65535) return false;
    B.t0 = static_cast<int32_t>(ntg);
    B.p0 = static_cast<int32_t>(np);
    B.s0 = static_cast<int32_t>(nsl);
    B.r0 = static_cast<int32_t>(nr);
    ntg += B.ntgt;
    np += B.npos;
    nsl += B.nsl;
    nr += B.nrows;
    plan.tmax = std::max(plan.tmax, B.ntgt);
    plan.rmax = std::max(plan.rmax, B.nrecv);
    plan.cmax = std::max(plan.cmax, B.nT + B.nE);
    plan.posmax = std::max(plan.posmax, B.npos);
    plan.possmax = std::max(plan.possmax, B.nposS);
    plan.slmax = std::max(plan.slmax, B.nsl);
  }
  if (np >= INT32_MAX / 2 || nr >= INT32_MAX / 32 || ntg >= INT32_MAX) return false;
  plan.n_rows = nr;
  plan.pos_v.resize(np);
  plan.pos_info.resize(2 * np);
  plan.tgt.resize(ntg);
  plan.slice.resize(2 * nsl);
  plan.warps.resize(nb * warps);
  plan.row_ent.resize(32 * nr);
  plan.row_idx.resize(32 * nr);
  // rounds of constraints in tensor memory: as many as the block needs of both
  // kinds, cut to the columns a warp gets (4-slot ones, which save more, first)
  const int cols = kDColumns / (threads / 128);
  // A grid's blocks are alike and have the fullest one's rounds, which the
  // kernel then reads from its arguments (from the block, 40^3 takes 67.7 ms
  // instead of 64.0); packed bodies are not (16 of them 102 -> 93 ms, 24 123 ->
  // 105).
  int32_t rmax = 0, mostT = 0, mostE = 0;
  for (const DBlock& B : plan.blocks) {
    rmax = std::max(rmax, B.nrows);
    mostT = std::max(mostT, (B.nT + threads - 1) / threads);
    mostE = std::max(mostE, (B.nE + threads - 1) / threads);
  }
  bool held = true;
  for (DBlock& B : plan.blocks) {
    const int32_t needT = cluster ? (B.nT + threads - 1) / threads : mostT;
    const int32_t needE = cluster ? (B.nE + threads - 1) / threads : mostE;
    B.kT = std::min(needT, cols / 16);
    B.kE = std::min(needE, (cols - 16 * B.kT) / 8);
    held = held && B.kT == needT && B.kE == needE;
    plan.kT = std::max(plan.kT, B.kT);
    plan.kE = std::max(plan.kE, B.kE);
  }
  // shared memory: the vectors and tables, the rest holds rows
  const DcgSmem o = dcg_smem_parts(plan);
  if (o.rows > smem_limit) return false;
  plan.srows = std::min(rmax, (smem_limit - o.rows) / kDRow);
  plan.onchip = held && plan.srows == rmax;
  plan.smem = std::max(o.rows + plan.srows * kDRow, kDMinSmem);
  // the same share of every warp's rows
  for (int64_t b = 0; b < nb; ++b) {
    const DBlock& B = plan.blocks[b];
    const int32_t most = std::min(plan.srows, B.nrows);
    int32_t at = 0, seen = 0;
    for (DWarp& W : loc[b].warps) {
      seen += W.rows;
      W.srow = at;
      W.held = B.nrows > 0 ? static_cast<int32_t>(static_cast<int64_t>(most) * seen / B.nrows) - at : 0;
      W.held = std::min(W.held, W.rows);
      at += W.held;
    }
  }
#pragma omp parallel for schedule(dynamic, 1)
  for (int64_t b = 0; b < nb; ++b) {
    const DBlock& B = plan.blocks[b];
    const Local& L = loc[b];
    std::copy(L.pos_v.begin(), L.pos_v.end(), plan.pos_v.begin() + B.p0);
    std::copy(L.pos_info.begin(), L.pos_info.end(), plan.pos_info.begin() + 2LL * B.p0);
    std::copy(L.tgt.begin(), L.tgt.end(), plan.tgt.begin() + B.t0);
    std::copy(L.slice.begin(), L.slice.end(), plan.slice.begin() + 2LL * B.s0);
    std::copy(L.warps.begin(), L.warps.end(), plan.warps.begin() + b * warps);
    std::copy(L.row_ent.begin(), L.row_ent.end(), plan.row_ent.begin() + 32LL * B.r0);
    std::copy(L.row_idx.begin(), L.row_idx.end(), plan.row_idx.begin() + 32LL * B.r0);
  }
  return true;
}

void dcg_plan_apply(const DcgPlan& P, const float* gradC, const float* invm, const float* alpha,
                    const float* x, double* y) {
  struct V3 {
    double c[3];
  };
  const int nw = P.threads / 32;
  const size_t nb = P.blocks.size();
  std::vector<V3> exch(P.n_slots);
  std::vector<std::vector<V3>> u(nb), rbuf(nb);
  for (size_t b = 0; b < nb; ++b) {
    u[b].assign(P.blocks[b].npos, V3{});
    rbuf[b].assign(P.blocks[b].nrecv, V3{});
  }
  for (size_t b = 0; b < nb; ++b) {
    const DBlock& B = P.blocks[b];
    for (int w = 0; w < nw; ++w) {
      const DWarp& W = P.warps[b * nw + w];
      int64_t row = B.r0 + W.row;
      for (int32_t s = W.s; s < W.e; ++s) {
        const uint32_t rows = P.slice[2LL * (B.s0 + s)], at = P.slice[2LL * (B.s0 + s) + 1];
        const int lanes = 1 << (at >> 16);
        for (int k = 0; k < 32 / lanes; ++k) {
          V3 a{};
          for (uint32_t r = 0; r < rows; ++r)
            for (int q = 0; q < lanes; ++q) {
              const int64_t o = 32 * (row + r) + lanes * k + q;
              const int32_t e = P.row_ent[o];
              if (e < 0) continue;
              const double xt = x[P.perm[B.c0 + P.row_idx[o]]];
              for (int c = 0; c < 3; ++c) a.c[c] += xt * gradC[3LL * e + c];
            }
          const int64_t p = (at & 0xffff) + k;
          const uint32_t to = P.pos_info[2 * (B.p0 + p)], n = P.pos_info[2 * (B.p0 + p) + 1];
          u[b][p] = a;
          if (n == 0) continue;
          if (!P.cluster) {
            exch[to + (n & 0xff)] = a;
          } else {
            for (uint32_t j = 0; j + 1 < n >> 8; ++j) {
              const uint32_t t = P.tgt[B.t0 + (to >> 16) + j];
              rbuf[b - B.rank + (t >> 16)][t & 0xffff] = a;
            }
          }
        }
        row += rows;
      }
    }
  }
  for (size_t b = 0; b < nb; ++b) {
    const DBlock& B = P.blocks[b];
    for (int32_t p = 0; p < B.npos; ++p) {
      const uint32_t from = P.pos_info[2LL * (B.p0 + p)], n = P.pos_info[2LL * (B.p0 + p) + 1];
      V3 a = u[b][p];
      if (n != 0) {
        const V3 own = a;
        a = V3{};
        uint32_t o = from & 0xffff;
        for (uint32_t k = 0; k < n >> 8; ++k) {
          const V3& v = k == (n & 0xff) ? own : (P.cluster ? rbuf[b][o++] : exch[from + k]);
          for (int c = 0; c < 3; ++c) a.c[c] += v.c[c];
        }
      }
      const double w = P.pos_v[B.p0 + p] >= 0 ? invm[P.pos_v[B.p0 + p]] : 0.0;
      for (int c = 0; c < 3; ++c) u[b][p].c[c] = w * a.c[c];
    }
    for (int32_t i = 0; i < B.nT + B.nE; ++i) {
      const int32_t t = P.perm[B.c0 + i];
      double s = static_cast<double>(alpha[t]) * x[t];
      for (int l = 0; l < (i < B.nT ? 4 : 2); ++l)
        for (int c = 0; c < 3; ++c)
          s += gradC[12LL * t + 3 * l + c] * u[b][P.ti[4LL * (B.c0 + i) + l] / 16].c[c];
      y[t] = s;
    }
  }
}

}  // namespace mgpbd
