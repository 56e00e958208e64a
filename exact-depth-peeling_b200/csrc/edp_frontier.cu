// Contour-guided convex subdivision: per-source candidate lists, then rounds
// of the device-controlled loop (warp_peel/frontier.py:15-245,
// event_kernels.py:12-25).
#include "edp_filtered.cuh"
#include "edp_internal.h"
#include "edp_warp.cuh"

namespace edp {
namespace {

constexpr int kBlock = 128;
constexpr int kWarps = kBlock / 32;

// The contour segments: hierarchy leaf ids, end points and depth at the ends.
struct Segments {
  const int *ids;
  const V2 *a, *b, *near;
  const int2 *near_src;  // the sources whose planes give `near`
  const V2 *near_mag;    // their |a x| + |b y| + |c| at the ends
  const Plane *scores;
  const int2 *vid;       // the welded mesh vertex at each end, or -1
  const int *faces, *canonical, *clipped, *src_n;
  const float4 *lo, *hi;
};

__device__ inline Segments segments_of(const Dev &d) {
  return Segments{d.seg_tree.ids, d.seg_a, d.seg_b, d.seg_near, d.seg_near_src,
                  d.seg_near_mag, d.scores, d.seg_vid, d.faces, d.canonical, d.clipped,
                  d.src_n, d.seg_lo, d.seg_hi};
}

// Source `s` is an unclipped triangle with welded vertex `v`.
__device__ inline bool has_vertex(const Segments &g, int s, int v) {
  if (v < 0 || g.clipped[s] || g.src_n[s] != 3) return false;
  const int *f = g.faces + 3 * int64_t(s);
  return g.canonical[f[0]] == v || g.canonical[f[1]] == v || g.canonical[f[2]] == v;
}

// Depth order of a source and a segment at the segment's two ends, each +1
// where the segment is nearer: 3 (sa + 1) + (sb + 1), or kDepthOpen when the
// filter-only form (F = 4) leaves a sign undecided.
constexpr int kDepthOpen = 9;

// Neither end of the segment is nearer.
__device__ inline bool behind(int code) { return code / 3 <= 1 && code % 3 <= 1; }

// The plane `sc` of `source` against the plane of the source that gives
// segment c its near depth, at the segment's ends a and b.  The plain form
// compares the rounded depths.  The filtered forms: each binary64 evaluation
// is within 3.01 u of its terms' magnitudes (two products, two sums), so a
// difference above 4 u of both magnitudes has its sign.  Otherwise: zero when
// the end is a mesh vertex of both triangles (both planes pass through it: the
// projected mesh's exact depths tie there, which the rounded plane
// coefficients can only approximate), else the two planes compared exactly
// (zero when the source is the patch's own).
template <int F>
__device__ inline int depth_code(const Segments &g, int c, V2 a, V2 b, V2 near, const Plane &sc,
                                 int source, Tally &tally) {
  const double za = value(sc, a) - near.x, zb = value(sc, b) - near.y;
  if constexpr (F == 0) {
    return 3 * (sign_of(za) + 1) + sign_of(zb) + 1;
  } else {
    const V2 mag = g.near_mag[c];
    const double z[2] = {za, zb};
    const double bound[2] = {
        4.0 * pred::kU64 * (fabs(sc.a * a.x) + fabs(sc.b * a.y) + fabs(sc.c) + mag.x),
        4.0 * pred::kU64 * (fabs(sc.a * b.x) + fabs(sc.b * b.y) + fabs(sc.c) + mag.y)};
    int sign[2];
    for (int e = 0; e < 2; ++e) {
      int stage = pred::kBinary64;
      if (fabs(z[e]) > bound[e]) {
        sign[e] = sign_of(z[e]);
      } else {
        const int2 srcs = g.near_src[c], vids = g.vid[c];
        const int s = e ? srcs.y : srcs.x, v = e ? vids.y : vids.x;
        const V2 x = e ? b : a;
        if (has_vertex(g, source, v) && has_vertex(g, s, v))
          sign[e] = 0;
        else
          sign[e] = order_sign<F>(sc, value(sc, x), g.scores[s], e ? near.y : near.x, x, stage);
      }
      if constexpr (F == 2) tally.add(stage);
    }
    if (F == 4 && (sign[0] == pred::kUndecided || sign[1] == pred::kUndecided)) return kDepthOpen;
    return 3 * (sign[0] + 1) + sign[1] + 1;
  }
}

// Predicate tallies of one thread (counted form only).
struct CutTally {
  Tally side, segment, depth;
};

// ------------------------------------------------------------ candidate lists
// Only some of the contour segments over a source can ever cut a patch of it.
// The list of a source holds the ones left after three tests, each with a
// margin far above what rounding can move a patch vertex (a cut point lies on
// its patch edge within 1e-16, so every patch lies in its source within 1e-13):
//   * the segment's line has source vertices more than kSideMargin away on
//     both sides.  Any other line splits a part off a patch that is at most
//     kSideMargin wide, whose doubled area is at most kSideMargin times its
//     perimeter: clean() drops it (below kEps = 1e-10 times the perimeter) and
//     the cut is cancelled;
//   * the segment is nowhere more than kOutsideMargin outside a source edge
//     with both ends: it lies apart from every patch, and the patch edge its
//     line enters by has both ends on its outside;
//   * it is nearer than the source at an end, which depends on the source and
//     the segment alone (depth_code, stored with the entry).
// The entries are in leaf order, so a patch meets the cutting candidates in
// the order of the hierarchy walk, and takes the same cuts.
constexpr double kSideMargin = 1.0e-12;
constexpr double kOutsideMargin = 1.0e-7;
// Entries of a list, held in shared memory until it is written.  One sheet
// behind 100 tiles has 304: 0.89 ms with its list, 1.00 with the search; behind
// 400 tiles, with 1,204, 2.9 ms with the list and 2.5 with the search.
constexpr int kListMost = 384;
constexpr int kScreenMost = 2048; // candidates screened for one list
constexpr int kUnlisted = -1;     // Dev::cand_count of a source without a list

// Can segment c cut a patch of the source v[0..n)?  `code` receives its depth
// code.
template <int F>
__device__ inline bool may_cut(const Segments &g, int c, const V2 *v, int n, const Plane &sc,
                               int source, int &code, CutTally &tally) {
  const V2 a = g.a[c], b = g.b[c];
  const double margin = kSideMargin * (fabs(b.x - a.x) + fabs(b.y - a.y));
  double most = 0.0, least = 0.0;
  for (int j = 0; j < n; ++j) {
    const double side = cross(a, b, v[j]);
    most = fmax(most, side);
    least = fmin(least, side);
  }
  if constexpr (F == 2) {  // the exact sides of the same vertices, for the tally
    for (int j = 0; j < n; ++j) {
      int stage = 0;
      side_sign<F>(a, b, v[j], stage);
      tally.side.add(stage);
    }
  }
  if (!(most > margin && least < -margin)) return false;
  for (int j = 0; j < n; ++j) {
    const V2 p = v[j], q = v[j + 1 < n ? j + 1 : 0];
    const double outside = -kOutsideMargin * (fabs(q.x - p.x) + fabs(q.y - p.y));
    if (cross(p, q, a) < outside && cross(p, q, b) < outside) return false;
  }
  code = depth_code<F>(g, c, a, b, g.near[c], sc, source, tally.depth);
  return !behind(code);
}

// One warp per source: its candidate list, and its first patch.  The warp
// walks the contour hierarchy once with the source's box, and screens the
// candidates 32 at a time, one per lane.  A source with an empty list is a
// final polygon as it is; any other joins the frontier.  A source with more
// than kListMost entries or kScreenMost candidates, or whose list does not fit
// the pool, is left without a list, and its patches search the hierarchy
// themselves, in the second pass of each iteration.  A large triangle behind a
// fine mesh is such a source: one warp would list its thousands of segments
// while the rest of the GPU waits (1.5 ms for a floor behind the 65,536-face
// knot), and each of its patches would look through all of them.
// Bound by the latency of the walk's 4 to 5 dependent steps: 8 blocks per SM
// with the candidates screened together, against 6 with each leaf group's few
// by themselves, took the preparation of the 720K primitives from 2.92 to 2.55
// ms and the knot's from 0.35 to 0.32 (10 and 12 blocks spill).
// Listing once per source replaced a hierarchy walk per patch whose candidates
// were tested by a whole warp each: on the 65,536-face knot 783K patch walks
// and 3.7M candidate tests against 65K walks, 0.19 ms here.
template <int F>
__global__ void __launch_bounds__(kBlock, 8) k_candidates(Dev d) {
  __shared__ int2 s_list[kWarps][kListMost];
  __shared__ int s_queue[kWarps][64];
  __shared__ V2 s_source[kWarps][kSourceVertices];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned below = (1u << lane) - 1u;
  const bool fits = int64_t(d.n) <= d.cap.frontier;
  if (blockIdx.x == 0 && threadIdx.x == 0 && !fits) set_error(d.status, kErrResidual);
  if (!fits || d.status[kError] != 0) return;
  const Segments segs = segments_of(d);
  const int leaves = *d.seg_tree.size;
  int2 *list = s_list[warp];
  int *queue = s_queue[warp];  // candidates of the walk, in leaf order, not screened yet
  V2 *v = s_source[warp];
  CutTally tally;
  const int warps = int(gridDim.x) * kWarps;
  for (int s = int(blockIdx.x) * kWarps + warp; s < d.n; s += warps) {
    const int n = d.src_n[s];
    if (n == 0) continue;
    const Plane sc = d.scores[s];
    __syncwarp();
    V2 p = v2(0.0, 0.0);
    if (lane < n) {
      p = d.src_v[int64_t(kSourceVertices) * s + lane];
      v[lane] = p;
    }
    __syncwarp();
    float4 lo = d.src_lo[s];
    const float4 hi = d.src_hi[s];
    lo.z = -1.0e30f;
    int total = 0, start = 0;
    {
      WarpWalk w;
      walk_begin(w, d.seg_tree, leaves, lo, hi, 0);
      int budget = 0x7fffffff, first, resume, queued = 0, screened = 0;
      unsigned batch;
      // Screens the first 32 queued candidates, one per lane.
      auto screen = [&]() {
        __syncwarp();
        const int c = queue[lane], rest = queue[32 + lane];
        int code = 0;
        const bool keep = lane < queued && may_cut<F>(segs, c, v, n, sc, s, code, tally);
        const unsigned kept = __ballot_sync(kFull, keep);
        const int slot = total + __popc(kept & below);
        if (keep && slot < kListMost) list[slot] = make_int2(c, code);
        total += __popc(kept);
        screened += 32;
        __syncwarp();
        queue[lane] = rest;
        queued = max(0, queued - 32);
        __syncwarp();  // the next batch is written over the places past the rest
      };
      while (total <= kListMost && screened <= kScreenMost &&
             walk_next(w, d.seg_tree, leaves, lo, hi, 0, budget, batch, first, resume)) {
        if ((batch >> lane) & 1u)
          queue[queued + __popc(batch & below)] = __ldg(&segs.ids[first + lane]);
        queued += __popc(batch);
        if (queued >= 32) screen();
      }
      if (queued > 0 && total <= kListMost && screened <= kScreenMost) screen();
      if (total > kListMost || screened > kScreenMost) total = kUnlisted;
    }
    if (total > 0) {
      if (lane == 0)
        start = int(claim_entries(reinterpret_cast<unsigned long long *>(&d.sc[kCandidates]),
                                  total, d.cand_cap));
      start = __shfl_sync(kFull, start, 0);
      if (start < 0) {
        total = kUnlisted;
      } else {
        __syncwarp();
        for (int k = lane; k < total; k += 32) d.cand[int64_t(start) + k] = list[k];
        __syncwarp();
      }
    }
    int slot = 0;
    if (lane == 0)
      slot = atomicAdd(total == 0           ? &d.status[kPolygons]
                       : total == kUnlisted ? &d.sc[kTopLive]
                                            : &d.status[kResidual],
                       1);
    slot = __shfl_sync(kFull, slot, 0);
    if (total == 0) {
      if (slot >= d.cap.regions) {
        if (lane == 0) set_error(d.status, kErrOutput);
        continue;
      }
      if (lane < n) d.out_v[int64_t(kMaxVertices) * slot + lane] = p;
      if (lane == 0) {
        d.out_n[slot] = n;
        d.out_src[slot] = s;
        d.out_layer[slot] = 0;
      }
      continue;
    }
    // The slots of both ends: at most n <= frontier capacity of them.
    if (total == kUnlisted) slot = d.frontier_room - 1 - slot;
    if (lane < n) d.fv[0][int64_t(kMaxVertices) * slot + lane] = p;
    if (lane == 0) {
      d.fn[0][slot] = n;
      d.fsrc[0][slot] = s;
      d.fcur[0][slot] = 0;
      d.cand_start[s] = start;
      d.cand_count[s] = total;
    }
  }
  if constexpr (F == 2) {
    tally.side.flush(d, kPredSide);
    tally.depth.flush(d, kPredDepth);
  }
}

__global__ void k_loop_condition(Dev d) {
  // The frontier must have room for every source, listed or not.
  const bool fits = int64_t(d.n) <= d.cap.frontier;
  d.status[kPeakResidual] = fits ? d.n : 0;
  d.metrics[kRounds] = fits && d.n > 0 && d.status[kError] == 0 ? 1 : 0;
  int c = (d.status[kResidual] > 0 || d.sc[kTopLive] > 0) && d.status[kError] == 0;
  *d.condition = c;
  if (d.use_handle) cudaGraphSetConditional(d.cond_handle, unsigned(c));
}

// ------------------------------------------------------------ rounds
// Does segment a->b cut the patch?  Its line has patch vertices strictly on
// both sides, and the part of the segment inside the patch lies strictly in
// front of it somewhere: the segment's parameter range clipped by each patch
// edge and by the depth half-plane stays open (frontier.py:81-103).
//
// Two tests decide it.  `certainly_missed` takes a candidate per lane against
// the whole patch and rejects most of a list chunk at once; `cuts` takes one
// candidate of the few left with a lane per patch edge (p -> q).
//
// certainly_missed: no patch vertex on one of the line's sides, or a patch
// edge with both segment ends on its outside.  F = 0 takes the signs of
// `cuts`.  The filtered forms take signs that a filter decides: with one
// difference rounded per factor, the two products and their difference are
// within 5 u of S = |product| + |product|, so a determinant above 8 u S has its
// sign; it is zero when S is, and when the point is an end of the edge.
struct QuickSign {
  bool positive, negative, zero;  // none: undecided
};

template <int F>
__device__ inline QuickSign quick_side(V2 a, V2 dir, V2 b, V2 c) {
  const V2 w = c - a;
  const double s = dir.x * w.y, t = dir.y * w.x, det = s - t;
  if constexpr (F == 0) return QuickSign{det > 0.0, det < 0.0, det == 0.0};
  const double sum = fabs(s) + fabs(t), bound = 8.0 * pred::kU64 * sum;
  const bool zero = sum == 0.0 || c == b;
  return QuickSign{!zero && det > bound, !zero && det < -bound, zero};
}

template <int F>
__device__ inline bool certainly_missed(const V2 *v, int n, int most, V2 a, V2 b, bool meets) {
  const V2 dir = b - a;
  bool left = false, right = false;  // some vertex is or may be there
  for (int j = 0; j < most; ++j) {   // most: the largest n in the warp
    const QuickSign s = quick_side<F>(a, dir, b, v[j]);
    left = left || (j < n && !s.negative && !s.zero);
    right = right || (j < n && !s.positive && !s.zero);
  }
  bool missed = !left || !right;
  if (!__any_sync(kFull, meets && !missed)) return true;
  V2 p = v[0];
  for (int j = 0; j < most; ++j) {
    const V2 q = v[j + 1 < n ? j + 1 : 0], edge = q - p;
    const QuickSign sa = quick_side<F>(p, edge, q, a), sb = quick_side<F>(p, edge, q, b);
    missed = missed || (j < n && (sa.negative || sa.zero) && (sb.negative || sb.zero));
    p = q;
  }
  return missed;
}

// cuts: ballots decide the sides and the closed edges, and butterflies give
// the clip range, which is a max / min of the same quotients as the
// sequential clip and so is order-free.  F is the predicate form
// (edp_filtered.cuh): the plain form evaluates the reference's binary64
// expressions; the filtered forms take exact signs of the sides and of the
// segment ends against the patch edges, and keep binary64 for the clip
// parameters.  The filter-only form gives kOpen when its filters cannot
// decide.  `side` is left with this lane's vertex against the line (the split
// reuses it).
enum CutTest : int { kMiss = 0, kHit = 1, kOpen = 2 };

template <int F, int W>
__device__ inline int cuts(const Group<W> &g, V2 p, V2 q, int n, const Plane &sc, V2 a, V2 b,
                           V2 near, int code, int &side, CutTally &tally) {
  const bool mine = g.lane < n;
  int stage = 0, stage_a = 0, stage_b = 0, sda, sdb;
  const double da = cross(p, q, a), db = cross(p, q, b);
  if constexpr (F == 0) {
    side = sign_of(cross(a, b, p));
    sda = sign_of(da);
    sdb = sign_of(db);
  } else {
    side = mine ? side_sign<F>(a, b, p, stage) : 0;
    sda = mine ? side_sign<F>(p, q, a, stage_a) : 0;
    sdb = mine ? side_sign<F>(p, q, b, stage_b) : 0;
    if constexpr (F == 2) {
      if (mine) {
        tally.side.add(stage);
        tally.segment.add(stage_a);
        tally.segment.add(stage_b);
      }
    }
  }
  // Every ballot is taken by the whole warp, whatever the groups' answers.
  const unsigned undecided = F == 4 ? g.ballot(side == pred::kUndecided ||
                                               sda == pred::kUndecided ||
                                               sdb == pred::kUndecided)
                                    : 0u;
  const unsigned lefts = g.ballot(mine && side > 0), rights = g.ballot(mine && side < 0);
  const unsigned closed = g.ballot(mine && sda <= 0 && sdb <= 0);
  const bool open = code == kDepthOpen || undecided != 0;
  const bool miss = lefts == 0 || rights == 0 || closed != 0 || behind(code);
  const int sza = code / 3 - 1, szb = code % 3 - 1;
  double low, high, rz;
  const double za = value(sc, a) - near.x, zb = value(sc, b) - near.y;
  if constexpr (F == 0) {
    const double r = da / (da - db);
    low = mine && da < 0.0 ? fmax(0.0, r) : 0.0;
    high = mine && db < 0.0 ? fmin(1.0, r) : 1.0;
    rz = za / (za - zb);
  } else {
    const double r = crossing(da, db);
    low = mine && sda < 0 ? r : 0.0;
    high = mine && sdb < 0 ? r : 1.0;
    rz = crossing(za, zb);
  }
  const int width = W == 8 ? 8 : lane_width(n);
  for (int off = width >> 1; off > 0; off >>= 1) {  // lanes [0, width) hold the edges
    low = larger(low, g.shfl_xor(low, off));
    high = smaller(high, g.shfl_xor(high, off));
  }
  if (W > 8) {
    low = g.shfl(low, 0);
    high = g.shfl(high, 0);
  }
  if (sza < 0) low = larger(low, rz);
  if (szb < 0) high = smaller(high, rz);
  if (open) return kOpen;
  return !miss && high > low ? kHit : kMiss;
}

// A frontier's patch pool.  `n` holds the vertex count and, above it, the
// patch's generation: how many right-hand parts lie on its way from the
// source.  Generations are the reference's rounds (frontier.py:106-223, each
// round's right-hand parts make up the next one's frontier): the counter is one
// above the last generation, and a generation at Dev::cap.rounds is the
// round-capacity error.  How many iterations of the loop they take here depends
// on how the work is handed on, and is bounded by nothing but the candidates.
constexpr int kSizeBits = 6;
constexpr int kSizeMask = (1 << kSizeBits) - 1;

struct Frontier {
  V2 *v;
  int *n, *src, *cur;
  int *count, *status;
  int64_t capacity;
};

// Append the patches of the groups that `want` it (one vertex per lane) to the
// frontier, upwards from slot 0, or downwards from its last slot (`top`) for
// patches left to this round's second pass, counted in `count`.  Returns the
// slot, or -1 on overflow.
template <int W>
__device__ __noinline__ int64_t push_patch(Frontier f, int *count, bool top, bool want, V2 p,
                                           int size, int source, int cursor) {
  const Group<W> g;
  const int k = g.reserve_slot(count, want);
  if (!want) return -1;
  const int64_t slot = top ? f.capacity - 1 - k : int64_t(k);
  if (slot < 0 || slot >= f.capacity) {
    if (g.lane == 0) set_error(f.status, kErrResidual);
    return -1;
  }
  if (g.lane < (size & kSizeMask)) f.v[int64_t(kMaxVertices) * slot + g.lane] = p;
  if (g.lane == 0) {
    f.n[slot] = size;
    f.src[slot] = source;
    f.cur[slot] = cursor;
  }
  return slot;
}

// The first leaves of the contour hierarchy from leaf `cursor` on, up to 32
// together, of which some meet the box: true for the lanes whose leaf does
// (segment `id`), `base` the first one's number.  Moves the cursor past them;
// no lane's answer is true at the end.  The hierarchy's descendants five levels
// below a node are 32 consecutive nodes: a step tests them, a node per lane,
// goes down to the first that meets the box, or on and up when none does.
__device__ inline bool next_leaves(const Tree &t, int leaves, const Box &box, int &cursor,
                                   int &base, int &id) {
  const int lane = threadIdx.x & 31;
  for (int level = 0; cursor < leaves;) {
    const int nodes = leaves >> level, first = (cursor >> level) & ~31, node = first + lane;
    const bool in = node >= cursor >> level && node < nodes;
    int leaf_id = 0;
    if (in && level == 0) leaf_id = __ldg(&t.ids[node]);  // in one latency with its box
    const bool meets = in && overlaps(__ldg(&t.nodes[2 * (nodes + node)]),
                                      __ldg(&t.nodes[2 * (nodes + node) + 1]), box.lo, box.hi);
    const unsigned met = __ballot_sync(kFull, meets);
    if (met && level > 0) {
      cursor = max(cursor, (first + __ffs(int(met)) - 1) << level);
      level -= 5;
      continue;
    }
    cursor = first + 32 < nodes ? (first + 32) << level : leaves;
    if (met) {
      base = first;
      id = leaf_id;
      return meets;
    }
    if (leaves >> (level + 5) > 0) level += 5;
  }
  return false;
}

// Swap frontiers and decide whether another iteration runs
// (event_kernels.py:12-25).  The patches at the next frontier's top (parked for
// the second pass, then those without a list) share its slots with the others:
// together they must have fit.
__device__ inline void advance_round(const Dev &d) {
  // Loads past L1, of one latency together.
  const int next = __ldcg(&d.status[kNextResidual]), deferred = __ldcg(&d.sc[kDeferred]);
  const int pushed = __ldcg(&d.sc[kTopPushed]);
  const int loops = __ldcg(&d.status[kLoops]) + 1, segments = __ldcg(&d.sc[kSegmentCount]);
  const int peak = __ldcg(&d.status[kPeakResidual]), parity = __ldcg(d.parity);
  const long long parked = __ldcg(&d.metrics[kParkedPatches]);
  bool failed = __ldcg(&d.status[kError]) != 0;
  if (int64_t(next) + deferred + pushed > d.frontier_room) {
    set_error(d.status, kErrResidual);
    failed = true;
  }
  // Each iteration takes every patch past a candidate of its own at least.
  if (loops > segments + 2 && next + pushed > 0) {
    set_error(d.status, kErrWait);
    failed = true;
  }
  d.metrics[kParkedPatches] = parked + deferred;
  d.sc[kDeferred] = 0;
  d.sc[kDeferredNext] = 0;
  d.sc[kTopPushed] = 0;
  d.sc[kFrontierNext] = 0;
  d.sc[kTopFirst] = deferred;
  d.sc[kTopLive] = pushed;
  d.status[kResidual] = next;
  d.status[kNextResidual] = 0;
  d.status[kLoops] = loops;
  d.status[kPeakResidual] = max(peak, next + deferred + pushed);
  *d.parity = parity ^ 1;
  const int c = next + pushed > 0 && !failed;
  *d.condition = c;
  if (d.use_handle) cudaGraphSetConditional(d.cond_handle, unsigned(c));
}

constexpr int kStack = 8;     // patches a group keeps for itself
constexpr int kLocalCuts = 6; // cuts of one taken patch whose right parts stay local
constexpr int kMostCuts = 8;  // cuts of one taken patch before its parts go to the next round
constexpr int kFewCuts = 3;   // both, when there are fewer patches than groups

// One frontier round (frontier.py:106-223), a patch per group of W lanes.  A
// patch meets its source's listed segments whose boxes overlap its own, from
// its cursor on, in leaf order.  The first segment that cuts it splits it
// along the segment's line; a collapsed part cancels the cut.  The left part
// continues in the group, and the right part waits on the group's stack, or,
// past kStack waiting parts or kLocalCuts cuts, in the next round's frontier,
// where other groups take it; both have the cursor just past the cutting
// segment.  After kMostCuts cuts the left part goes to the next round too.  A
// patch that has met every candidate is final and goes to the output pool.
// Groups take patches from a shared counter.
//
// The groups of a warp run one loop in step: take a patch, find its next
// candidate, test it, split.  Every step is run by the whole warp when any
// group needs it.
//
// W = 8 is the first pass of a round, with the filter-only form (F = 4) under
// filtered binary64 predicates (no exact stage, so fewer registers and less
// code).  It parks a patch at the top of the next frontier, with its cursor
// at the candidate it stopped at, when its filters cannot decide, or when a
// part would have more than 8 vertices.  W = 32 is the second pass, with the
// exact stages.  It takes each parked patch past the candidate that stopped it
// and hands it, or its two parts, to the next round (a patch that no group of
// eight lanes can take goes on).  Then it takes the patches whose source has no
// list, which lie at the frontier's top: they search the contour hierarchy for
// the leaves from their cursor on that meet their box (next_leaves), the same
// segments in the same order.  Each patch meets the same tests in the same
// order as in one exact pass, so the output is the same.
//
// Reading a list of any length from end to end for every patch took 109 ms for
// 2,000 strips in front of one triangle, 53 for 10,000 tiles and 43 for a floor
// behind 200,000 faces of primitives; the search takes 27, 15 and 20.  In the
// first pass's loop, even only called from there, it costs the listed patches
// 10 to 15%.
//
// The time is instruction issue on patches of three to six vertices, and at
// small sizes the chain of one group's steps: a warp per patch left 26 of 32
// lanes idle, and a round per right-hand part made 14 rounds of the knot.
// Rounds in all (a warp per patch, then this): knot-65536 3.04 -> 0.97 ms,
// 720K primitives 11.5 -> 3.2 ms, 2,560-face icospheres 0.60 -> 0.36 ms.  The
// cut bounds trade a round's longest chain against the number of rounds:
// unbounded chains took 1.2, 3.5 and 0.43 ms, and 8 cuts even for few patches
// 1.04, 3.4 and 0.40.  4 blocks of 128 registers per SM: 5 blocks spill (1.3 ms on the knot), 3 hide less latency (1.13).
template <int F, int W>
__global__ void __launch_bounds__(kBlock, 4) k_subdivide(Dev d) {
  constexpr int kGroups = kBlock / W;
  constexpr bool kWide = W == 32;
  constexpr int kWaiting = kWide ? 1 : kStack;
  __shared__ V2 s_parts[kGroups][2][W];
  __shared__ V2 s_patch[kGroups][W];
  __shared__ V2 s_stack[kGroups][kWaiting][W];
  __shared__ int2 s_waiting[kGroups][kWaiting];  // size and generation, cursor
  const Group<W> g;
  const int slot = threadIdx.x / W, lane = threadIdx.x & 31;
  V2 *left_part = s_parts[slot][0], *right_part = s_parts[slot][1];
  const int par = *d.parity;
  // Parked in this iteration: at the next frontier's top.
  const int parked = kWide ? int(min(int64_t(d.sc[kDeferred]), int64_t(d.frontier_room))) : 0;
  const int live = kWide ? parked + d.sc[kTopLive]
                         : int(min(int64_t(d.status[kResidual]), int64_t(d.frontier_room)));
  int *taken = kWide ? &d.sc[kDeferredNext] : &d.sc[kFrontierNext];
  const V2 *fv = d.fv[par];
  const int *fn = d.fn[par], *fsrc = d.fsrc[par], *fcur = d.fcur[par];
  const Segments segs = segments_of(d);
  const Frontier next{d.fv[par ^ 1], d.fn[par ^ 1], d.fsrc[par ^ 1], d.fcur[par ^ 1],
                      &d.status[kNextResidual], d.status, int64_t(d.frontier_room) - parked};
  int visits = 0, tests = 0, splits = 0;  // each group's lane 0
  CutTally tally;
  // With fewer patches than groups the round lasts as long as one group's chain.
  const bool few = live <= int(gridDim.x) * kGroups / 2;
  const int local_cuts = few ? kFewCuts : kLocalCuts, most_cuts = few ? kFewCuts : kMostCuts;
  // The group's patch.
  bool idle = true, drained = false, changed = false;
  int waiting = 0, cut_count = 0, budget = 0;
  int n = 0, generation = 0, source = 0, cursor = 0, start = 0, count = 0;
  V2 p = v2(0.0, 0.0), q = p;
  Plane sc{0.0, 0.0, 0.0, 0.0};
  Box box{empty_lo(), empty_hi()};
  // The candidates of the current list chunk, one per lane.
  unsigned batch = 0;
  int base = 0, id = 0, code = 0;
  V2 ca = p, cb = p, cn = p;
  // To the next frontier: to its top when the source has no list.
  auto push_part = [&](bool want, V2 x, int size, int from) {
    const bool up = kWide && want && count == kUnlisted;
    if (!kWide || __any_sync(kFull, want && !up))
      push_patch<W>(next, next.count, false, want && !up, x, size, source, from);
    if (kWide && __any_sync(kFull, up))
      push_patch<W>(next, &d.sc[kTopPushed], true, up, x, size, source, from);
  };
  for (;;) {
    // Take a patch: from the group's stack, else from the frontier.
    bool fresh = false, park = false, final = false, push = false;
    if (idle && waiting > 0) {
      const int2 w = s_waiting[slot][--waiting];
      n = w.x & kSizeMask;
      generation = w.x >> kSizeBits;
      cursor = w.y;
      p = s_stack[slot][waiting][g.lane];
      fresh = true;
    }
    const bool want = idle && !fresh && !drained;
    if (__any_sync(kFull, want)) {
      const int at = g.reserve_slot(taken, want);
      const int failed = __shfl_sync(kFull, *(volatile int *)&d.status[kError], 0);
      if (want && (at >= live || failed != 0)) drained = true;
      const bool take = want && !drained;
      int i = at, size = 0;
      if (kWide) {  // from the top downwards: the parked ones, then those without a list
        const int from = at < parked ? par ^ 1 : par;
        if (at >= parked) i += d.sc[kTopFirst] - parked;
        i = d.frontier_room - 1 - i;
        fv = d.fv[from];
        fn = d.fn[from];
        fsrc = d.fsrc[from];
        fcur = d.fcur[from];
      }
      if (take) {
        size = fn[i];
        n = size & kSizeMask;
        generation = size >> kSizeBits;
        source = fsrc[i];
        cursor = fcur[i];
        p = g.lane < n ? fv[int64_t(kMaxVertices) * i + g.lane] : v2(0.0, 0.0);
        sc = d.scores[source];
        start = d.cand_start[source];
        count = d.cand_count[source];
        cut_count = 0;
        fresh = true;
      }
      if (!kWide) {
        // A patch too large for a group (left by the second pass of an earlier
        // round): to this round's second pass.
        const bool wide = take && n > W;
        if (__any_sync(kFull, wide)) {
          const int64_t to =
              push_patch<W>(next, &d.sc[kDeferred], true, wide, p, size, source, cursor);
          if (to >= 0)
            for (int j = W + g.lane; j < n; j += W)
              next.v[int64_t(kMaxVertices) * to + j] = fv[int64_t(kMaxVertices) * i + j];
          fresh = fresh && !wide;
        }
      }
    }
    if (fresh) {
      idle = false;
      ++visits;
      batch = 0;
      budget = d.step_budget;
    }
    if (__all_sync(kFull, idle && drained)) break;
    if (idle) n = 0;
    if (__any_sync(kFull, fresh || changed)) {
      q = g.shfl(p, g.lane + 1 < n ? g.lane + 1 : 0);
      box = group_bounds<W>(p, n, sc);
      box.lo.z = -1.0e30f;
      s_patch[slot][g.lane] = p;
      changed = false;
      __syncwarp();
    }
    // Find the next chunk with a candidate: of the source's list, or (second
    // pass, no list) of the contour hierarchy's leaves.
    const int most = W == 8 ? __reduce_max_sync(kFull, n) : n;
    for (;;) {
      bool look = !idle && !push && !final && batch == 0;
      if (!__any_sync(kFull, look)) break;
      const bool search = kWide && count == kUnlisted;
      const int entries = search ? *d.seg_tree.size : count;
      bool meets = false;
      if (look) {
        if (cursor >= entries) {
          final = true;
        } else if (--budget < 0) {
          push = true;  // a long walk carries over, so that one patch does not hold a round
        } else if (!search) {
          base = cursor;
          cursor += W;
          if (base + g.lane < count) {
            const int2 e = d.cand[int64_t(start) + base + g.lane];
            id = e.x;
            code = e.y;
            // The segment with its box, not after it: one latency, not two.
            const float4 lo = segs.lo[id], hi = segs.hi[id];
            ca = segs.a[id];
            cb = segs.b[id];
            cn = segs.near[id];
            meets = overlaps(lo, hi, box.lo, box.hi);
          }
        }
      }
      if (search && !final && !push) {  // the patch of the whole warp
        meets = next_leaves(d.seg_tree, entries, box, cursor, base, id);
        if (meets) {
          code = kDepthOpen;
          ca = segs.a[id];
          cb = segs.b[id];
          cn = segs.near[id];
        }
      }
      tests += __popc(g.ballot(meets));
      if ((!kWide || search) && __any_sync(kFull, meets)) {
        const bool missed = certainly_missed<F>(s_patch[slot], n, most, ca, cb, meets);
        meets = meets && !missed;
      }
      const unsigned found = g.ballot(meets);
      if (look) batch = found;
    }
    // Final patches.
    if (__any_sync(kFull, final)) {
      const int out = g.reserve_slot(&d.status[kPolygons], final);
      if (final) {
        if (out >= d.cap.regions) {
          if (g.lane == 0) set_error(d.status, kErrOutput);
        } else {
          if (g.lane < n) d.out_v[int64_t(kMaxVertices) * out + g.lane] = p;
          if (g.lane == 0) {
            d.out_n[out] = n;
            d.out_src[out] = source;
            d.out_layer[out] = generation;  // until the ranks are there (k_order_count)
          }
        }
      }
    }
    // Test the next candidate.
    const bool test = batch != 0;
    bool cut = false, moved = false;
    int side = 0, k = 0;
    V2 a = v2(0.0, 0.0), b = a;
    if (__any_sync(kFull, test)) {
      k = test ? __ffs(int(batch)) - 1 : 0;
      batch &= batch - 1;
      a = g.shfl(ca, k);
      b = g.shfl(cb, k);
      const V2 near = g.shfl(cn, k);
      int order = g.shfl(code, k);
      if constexpr (kWide) {
        const int c = g.shfl(id, k);
        if (order == kDepthOpen) {
          Tally rest;  // the same test on every lane: lane 0 counts it
          order = depth_code<F>(segs, c, a, b, near, sc, source, rest);
          if (F == 2 && lane == 0) tally.depth.add(rest);
        }
      }
      const int result = cuts<F, W>(g, p, q, test ? n : 0, sc, a, b, near, order, side, tally);
      cut = test && result == kHit;
      park = test && result == kOpen;
    }
    // Split along the segment's line.
    bool keep_right = false;
    V2 pr = p;
    int nr = 0;
    if (__any_sync(kFull, cut)) {
      const V2 dir = b - a;
      const double du = value(Plane{-dir.y, dir.x, 0.0, 0.0}, p - a);
      if constexpr (F == 0) side = sign_of(du);
      V2 pl;
      int nl;
      const bool fits = group_split<F>(g, p, q, cut ? n : 0, du, side, left_part, right_part, pl,
                                       nl, pr, nr);
      if (cut && !fits) {
        if (kWide && g.lane == 0) set_error(d.status, kErrPolygon);
        park = true;  // in the second pass, lost to the error
      }
      if (cut && nl > 0 && nr > 0) {
        ++splits;
        ++cut_count;
        keep_right = moved = true;
        p = pl;
        n = nl;
        if (generation + 1 >= d.cap.rounds && g.lane == 0) set_error(d.status, kErrRounds);
      }
    }
    // The right part: to the stack, or to the next round.
    const int right_size = nr | (generation + 1) << kSizeBits;
    if (!kWide && keep_right && waiting < kStack && cut_count < local_cuts) {
      s_stack[slot][waiting][g.lane] = pr;
      if (g.lane == 0) s_waiting[slot][waiting] = make_int2(right_size, base + k + 1);
      ++waiting;
      keep_right = false;
    }
    if (__any_sync(kFull, keep_right))
      push_part(keep_right, pr, right_size, base + k + 1);
    // The rest of the chunk is met again by the left part: a segment that ends
    // on an edge of the patch may cut a part by a rounding of that edge.
    if (moved) {
      changed = true;
      batch = 0;
      cursor = base + k + 1;
      push = !kWide && cut_count >= most_cuts;
    }
    if (kWide && test && !park && n <= 8 && count != kUnlisted) {
      cursor = base + k + 1;  // past its candidate, a group of eight lanes can go on
      push = true;
    }
    // Patches that leave the group: back to the frontier, or from the undecided
    // candidate on to the second pass.
    if (__any_sync(kFull, push)) push_part(push, p, n | generation << kSizeBits, cursor);
    if (!kWide && __any_sync(kFull, park))
      push_patch<W>(next, &d.sc[kDeferred], true, park, p, n | generation << kSizeBits, source,
                    base + k);
    if (push || park || final) {
      idle = true;
      batch = 0;
    }
    __syncwarp();  // the stack and the part buffers
  }
  if (g.lane == 0) {
    count_add(&d.metrics[kTargetVisits], visits);
    count_add(&d.metrics[kContourTests], tests);
    count_add(&d.metrics[kSplits], splits);
  }
  if constexpr (F == 2) {
    tally.side.flush(d, kPredSide);
    tally.segment.flush(d, kPredSegment);
    tally.depth.flush(d, kPredDepth);
  }
  if constexpr (kWide) {  // the second pass's last block ends the iteration
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      if (atomicAdd(&d.sc[kRoundBlocks], 1) == int(gridDim.x) - 1) {
        __threadfence();
        d.sc[kRoundBlocks] = 0;
        advance_round(d);
      }
    }
  }
}

}  // namespace

// The candidate lists, the uncut sources' final polygons and the first
// frontier.
cudaError_t stage_lists(const Dev &d, cudaStream_t st) {
  int64_t g = ceil_div(d.n > 0 ? d.n : 1, kWarps);
  if (g > 148 * 16) g = 148 * 16;
  switch (d.predicates) {
    case 0: k_candidates<0><<<unsigned(g), kBlock, 0, st>>>(d); break;
    case 1: k_candidates<1><<<unsigned(g), kBlock, 0, st>>>(d); break;
    case 2: k_candidates<2><<<unsigned(g), kBlock, 0, st>>>(d); break;
    default: k_candidates<4><<<unsigned(g), kBlock, 0, st>>>(d); break;
  }
  note_launch();
  k_loop_condition<<<1, 1, 0, st>>>(d);
  note_launch();
  return cudaGetLastError();
}

namespace {
// The first pass of a round in form N, then the second, over the few parked
// patches, in form E.
template <int N, int E>
void launch_round(const Dev &d, unsigned grid, unsigned second, cudaStream_t st) {
  k_subdivide<N, 8><<<grid, kBlock, 0, st>>>(d);
  note_launch();
  k_subdivide<E, 32><<<second, kBlock, 0, st>>>(d);
  note_launch();
}
}  // namespace

cudaError_t stage_step(const Dev &d, cudaStream_t st) {
  const int64_t most = 148 * int64_t(d.subdivide_blocks);
  const unsigned g = unsigned(std::min(ceil_div(d.cap.frontier, kBlock / 8), most));
  const unsigned second = unsigned(std::min<int64_t>(ceil_div(d.cap.frontier, kWarps), 296));
  switch (d.predicates) {
    case 0: launch_round<0, 0>(d, g, second, st); break;
    case 1: launch_round<1, 1>(d, g, second, st); break;
    case 2: launch_round<2, 2>(d, g, second, st); break;
    default: launch_round<4, 3>(d, g, second, st); break;
  }
  return cudaGetLastError();
}

}  // namespace edp
