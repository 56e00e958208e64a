// DevicePeeler: whole-source ranks, then iterative per-layer clipping
// (warp_peel/solver.py:217-379, kernels.py:539-938).
//
// Each layer pass: sources whose whole-face rank is below the current layer
// retire from the source hierarchy (a refit, no re-sort), the residual
// hierarchy is rebuilt over the patches still unresolved, and a queue of
// pieces is clipped against every candidate that can be in front of its target
// (below).  Pieces that stay visible are output for this layer; hidden pieces
// form the next pass's residual.  The layer loop is the graph's conditional
// WHILE node, the clipping launches a WHILE node nested in its body.
#include "../../include/edp.h"
#include "edp_filtered.cuh"
#include "edp_internal.h"
#include "edp_warp.cuh"

namespace edp {
namespace {

constexpr int kBlock = 128;

__device__ inline int64_t tid() { return blockIdx.x * int64_t(blockDim.x) + threadIdx.x; }
__device__ inline int64_t stride() { return int64_t(gridDim.x) * blockDim.x; }

unsigned blocks(int64_t n) {
  int64_t g = ceil_div(n > 0 ? n : 1, kBlock);
  return unsigned(g < 148 * 16 ? g : 148 * 16);
}

// Bounds of a source's contour edges, xy only (kernels.py:539-559).
__global__ void k_contour_bounds(Dev d) {
  for (int64_t i = tid(); i < d.n; i += stride()) {
    const V2 *p = d.src_v + int64_t(kSourceVertices) * i;
    const int n = d.status[kError] == 0 ? d.src_n[i] : 0;
    double lx = 1.0e30, ly = 1.0e30, hx = -1.0e30, hy = -1.0e30;
    for (int j = 0; j < n; ++j) {
      if (!contour_edge(d, i, j)) continue;
      V2 a = p[j], b = p[(j + 1) % n];
      lx = fmin(lx, fmin(a.x, b.x)); ly = fmin(ly, fmin(a.y, b.y));
      hx = fmax(hx, fmax(a.x, b.x)); hy = fmax(hy, fmax(a.y, b.y));
    }
    if (lx <= hx) {
      d.contour_lo[i] = make_float4(__double2float_rd(lx - 2.0e-7), __double2float_rd(ly - 2.0e-7),
                                    -2.0e-7f, 0.f);
      d.contour_hi[i] = make_float4(__double2float_ru(hx + 2.0e-7), __double2float_ru(hy + 2.0e-7),
                                    2.0e-7f, 0.f);
    } else {
      d.contour_lo[i] = empty_lo();
      d.contour_hi[i] = empty_hi();
    }
  }
}

// Segment a-b touches convex polygon p, conservatively by EPS (kernels.py:562-576).
__device__ inline bool touches(const V2 *p, int n, V2 a, V2 b) {
  bool hit = true;
  for (int j = 0; j < n; ++j)
    if (cross(p[j], p[(j + 1) % n], a) < -kEps && cross(p[j], p[(j + 1) % n], b) < -kEps)
      hit = false;
  bool positive = false, negative = false;
  for (int j = 0; j < n; ++j) {
    double v = cross(a, b, p[j]);
    positive = positive || v >= -kEps;
    negative = negative || v <= kEps;
  }
  return hit && positive && negative;
}

__device__ inline void save_polygon(const Dev &d, const V2 *p, int n, int source, int layer) {
  int slot = reserve(&d.status[kPolygons], 1);
  if (slot < d.cap.regions) {
    V2 *dst = d.out_v + int64_t(kMaxVertices) * slot;
    for (int j = 0; j < n; ++j) dst[j] = p[j];
    d.out_n[slot] = n;
    d.out_src[slot] = source;
    d.out_layer[slot] = layer;
    atomicMax(&d.status[kLayers], layer + 1);
  } else {
    set_error(d.status, kErrOutput);
  }
}

// Whole-source rank where no contour touches the source: count the sources
// strictly nearer at its centroid; ambiguous samples (on an edge, or a depth
// tie within 1e-12) go to clipping instead (kernels.py:599-690).
__global__ void k_classify(Dev d) {
  const int contour_leaves = *d.contour_tree.size, source_leaves = *d.source_tree.size;
  for (int64_t i = tid(); i < d.n; i += stride()) {
    const V2 *p = d.src_v + int64_t(kSourceVertices) * i;
    const int n = d.status[kError] == 0 ? d.src_n[i] : 0;
    int rank = -1;
    if (n > 0) {
      float4 lo, hi;
      polygon_bounds(p, n, Plane{0, 0, 0, 0}, lo, hi);
      lo.z = -1.0e-6f;
      hi.z = 1.0e-6f;
      bool boundary = false;
      int node = 1;
      while (node > 0 && !boundary) {
        int j;
        node = query_next(d.contour_tree, contour_leaves, lo, hi, node, 0, j);
        if (j < 0) break;
        const V2 *q = d.src_v + int64_t(kSourceVertices) * j;
        const int qn = d.src_n[j];
        for (int e = 0; e < qn && !boundary; ++e)
          if (contour_edge(d, j, e) && touches(p, n, q[e], q[(e + 1) % qn])) boundary = true;
      }
      if (!boundary) {
        V2 sample = v2(0.0, 0.0);
        for (int e = 0; e < n; ++e) sample = sample + p[e] / double(n);
        double z = value(d.scores[i], sample);
        float4 qlo = make_float4(__double2float_rd(sample.x - 2.0e-7),
                                 __double2float_rd(sample.y - 2.0e-7), -1.0e30f, 0.f);
        float4 qhi = make_float4(__double2float_ru(sample.x + 2.0e-7),
                                 __double2float_ru(sample.y + 2.0e-7),
                                 __double2float_ru(z + 2.0e-7 * fmax(1.0, fabs(z))), 0.f);
        rank = 0;
        bool ambiguous = false;
        int node2 = 1;
        while (node2 > 0) {
          int j;
          node2 = query_next(d.source_tree, source_leaves, qlo, qhi, node2, 0, j);
          if (j < 0) break;
          if (j == int(i)) continue;
          const V2 *q = d.src_v + int64_t(kSourceVertices) * j;
          const int qn = d.src_n[j];
          bool inside = qn > 0, edge = false;
          for (int e = 0; e < qn; ++e) {
            double s = cross(q[e], q[(e + 1) % qn], sample);
            inside = inside && s >= 0.0;
            edge = edge || fabs(s) <= kEps;
          }
          if (inside) {
            double delta = z - value(d.scores[j], sample);
            if (edge || fabs(delta) <= 1.0e-12 * fmax(1.0, fabs(z)))
              ambiguous = true;
            else if (delta > 0.0)
              ++rank;
          }
        }
        if (ambiguous) rank = -1;
      }
      if (rank < 0) {
        int slot = reserve(&d.status[kResidual], 1);
        if (slot < d.cap.frontier) {
          V2 *dst = d.res_v[0] + int64_t(kMaxVertices) * slot;
          for (int e = 0; e < n; ++e) dst[e] = p[e];
          d.res_n[0][slot] = n;
          d.res_src[0][slot] = int(i);
        } else {
          set_error(d.status, kErrResidual);
        }
      } else if (rank < d.limit) {
        save_polygon(d, p, n, int(i), rank);
      } else if (d.all_layers) {
        set_error(d.status, kErrLayers);
      }
    }
    d.ranks[i] = rank;
  }
}

__global__ void k_start_loop(Dev d) {
  d.status[kPeakResidual] = d.status[kResidual];
  *d.parity = 0;
  int c = d.status[kResidual] > 0 && d.status[kError] == 0;
  *d.condition = c;
  if (d.use_handle) cudaGraphSetConditional(d.cond_handle, unsigned(c));
}

// Source boxes with ranks below the current layer retire (kernels.py:717-732).
__global__ void k_retire_bounds(Dev d) {
  const int layer = d.status[kPass];
  for (int64_t i = tid(); i < d.n; i += stride()) {
    float4 lo = empty_lo(), hi = empty_hi();
    if (d.ranks[i] >= layer)
      polygon_bounds(d.src_v + int64_t(kSourceVertices) * i, d.src_n[i], d.scores[i], lo, hi);
    d.src_lo[i] = lo;
    d.src_hi[i] = hi;
  }
}

// Boxes of the current residual patches (kernels.py:699-714).
__global__ void k_active_bounds(Dev d) {
  const int par = *d.parity;
  const int live = int(min(int64_t(d.status[kResidual]), d.cap.frontier));
  for (int64_t i = tid(); i < live; i += stride()) {
    float4 lo = empty_lo(), hi = empty_hi();
    if (d.status[kError] == 0)
      polygon_bounds(d.res_v[par] + int64_t(kMaxVertices) * i, d.res_n[par][i],
                     d.scores[d.res_src[par][i]], lo, hi);
    d.res_lo[i] = lo;
    d.res_hi[i] = hi;
  }
  if (tid() == 0) d.sc[kFrontierLive] = live;
}

// ---------------------------------------------------------------- clipping
// A layer pass subtracts, from every residual patch (a target), each
// candidate that can lie in front of it: original sources of rank >= layer
// from the source hierarchy, then the other residual patches from the
// residual hierarchy (src/peel_common.h:169-199).  The work is a queue of
// pieces: a piece is a convex part of a target with the position of its
// candidate walk (which hierarchy, and the first leaf it has not met).  A
// clipping launch runs every queued piece, a warp each, against all of its
// candidates.  A candidate that cuts a piece
// splits off the parts of the piece outside the candidate (or nearer than
// it), and the part the candidate hides goes to the layer's hidden pool; one
// of the parts goes on in the same warp, the others are queued with the walk
// position past the candidate.  A piece that meets no more candidates is
// visible in this layer.  Launches repeat (a conditional WHILE node inside the
// layer loop) until no piece is left over; then a target
// none of whose pieces stayed visible is hidden whole, as the exact route
// restores it (src/bvh_peel.cpp:141-199), and the hidden pieces form the next
// layer's residual.  The work and hidden pools are shared by all targets and
// compacted by atomic appends, so their size follows the pieces alive, not a
// per-thread reservation.

constexpr int kCursorTree = 29;   // walk position: hierarchy << 29 | leaf
constexpr int kCursorLeaf = (1 << kCursorTree) - 1;
constexpr int kClipWarps = kBlock / 32;
constexpr int kClipParts = 8;     // uncovered parts of one cut held in shared memory

__device__ inline V2 *piece_at(V2 *base, int64_t slot) { return base + kMaxVertices * slot; }

// Where pieces go, by value: a helper out of line that took the kernel's
// whole Dev by reference would make every thread copy it to its stack.
struct PiecePool {
  V2 *v;
  int *n, *target, *cursor;  // cursor: null for the hidden pool
  int *count;
  int cap;
};

// The queue of a clipping launch.  Pieces are appended while other warps take
// them: `ready` holds the launch's epoch once a slot is written, and `pending`
// counts the pieces queued or in a warp.  Pieces past the pool's end go to the
// spill pool, which the next launch takes.
struct PieceQueue {
  PiecePool pool, spill;
  int *ready, *pending, *status;
  int epoch;
};

__device__ inline void write_piece(const PiecePool &f, int slot, V2 p, int n, int target,
                                   int cursor) {
  const int lane = threadIdx.x & 31;
  if (lane < n) piece_at(f.v, slot)[lane] = p;
  if (lane == 0) {
    f.n[slot] = n;
    f.target[slot] = target;
    if (f.cursor) f.cursor[slot] = cursor;
  }
}

// Appends a piece (one vertex per lane) to the hidden pool; false when it is
// full.
__device__ __noinline__ bool hide_piece(PiecePool f, V2 p, int n, int target) {
  int slot = 0;
  if ((threadIdx.x & 31) == 0) slot = atomicAdd(f.count, 1);
  slot = __shfl_sync(kFull, slot, 0);
  if (slot >= f.cap) return false;
  write_piece(f, slot, p, n, target, 0);
  return true;
}

// Queues a piece; false (and the worker-pool error) when both pools are full.
__device__ __noinline__ bool queue_piece(PieceQueue q, V2 p, int n, int target, int cursor) {
  const int lane = threadIdx.x & 31;
  int slot = 0;
  if (lane == 0) slot = atomicAdd(q.pool.count, 1);
  slot = __shfl_sync(kFull, slot, 0);
  if (slot < q.pool.cap) {
    if (lane == 0) atomicAdd(q.pending, 1);  // before this warp's own piece ends
    write_piece(q.pool, slot, p, n, target, cursor);
    __threadfence();
    __syncwarp();
    if (lane == 0) *(volatile int *)&q.ready[slot] = q.epoch;
    return true;
  }
  if (lane == 0) slot = atomicAdd(q.spill.count, 1);
  slot = __shfl_sync(kFull, slot, 0);
  if (slot >= q.spill.cap) {
    if (lane == 0) set_error(q.status, kErrWorker);
    return false;
  }
  write_piece(q.spill, slot, p, n, target, cursor);
  return true;
}

// A candidate: a projected source, or another residual patch.
struct Occluder {
  const V2 *v;
  int n, source;
};

// Can candidate `c` hide part of the piece v[0..n) (shared memory)?  Not when
// an edge of either polygon separates them, nor when the piece lies nowhere
// behind it.  One lane decides a whole candidate, so a leaf batch is rejected
// 32 candidates at a time.  Equal depth everywhere counts the lower source
// index as nearer.
template <int F>
__device__ inline bool may_hide(const Dev &d, const V2 *v, int n, const Plane &st, int source,
                                const Occluder &c, Tally &t) {
  for (int j = 0; j < c.n; ++j) {
    const V2 a = c.v[j], b = c.v[j + 1 < c.n ? j + 1 : 0];
    bool positive = false;
    for (int k = 0; k < n && !positive; ++k) {
      int stage = 0;
      positive = side_sign<F>(a, b, v[k], stage) > 0;
      if constexpr (F == 2) t.add(stage);
    }
    if (!positive) return false;
  }
  for (int j = 0; j < n; ++j) {
    const V2 a = v[j], b = v[j + 1 < n ? j + 1 : 0];
    bool positive = false;
    for (int k = 0; k < c.n && !positive; ++k) {
      int stage = 0;
      positive = side_sign<F>(a, b, c.v[k], stage) > 0;
      if constexpr (F == 2) t.add(stage);
    }
    if (!positive) return false;
  }
  const Plane so = d.scores[c.source];
  bool negative = false;
  for (int k = 0; k < n; ++k) {
    int s;
    if constexpr (F == 0) {
      s = sign_of(value(Plane{st.a - so.a, st.b - so.b, st.c - so.c, 0.0}, v[k]));
    } else {
      int stage = 0;
      s = order_sign<F>(st, value(st, v[k]), so, value(so, v[k]), v[k], stage);
      if constexpr (F == 2) t.add(stage);
    }
    if (s > 0) return true;
    negative = negative || s < 0;
  }
  if (negative) return false;
  if (source > c.source) return true;
  atomicAdd(&d.status[kDepthTies], 1);
  return false;
}

// The separating-edge test of may_hide for a piece held one vertex per lane.
template <int F>
__device__ inline bool warp_separated(V2 p, V2 q, int n, const Occluder &c, Tally &t) {
  const int lane = threadIdx.x & 31;
  const bool mine = lane < n;
  bool left = false;  // some candidate vertex is strictly left of this lane's edge
  for (int j = 0; j < c.n; ++j) {
    const V2 a = c.v[j], b = c.v[j + 1 < c.n ? j + 1 : 0];
    int stage = 0;
    const bool positive = mine && side_sign<F>(a, b, p, stage) > 0;
    if constexpr (F == 2)
      if (mine) t.add(stage);
    if (!__ballot_sync(kFull, positive)) return true;
    if (mine && !left) {
      left = side_sign<F>(p, q, a, stage) > 0;
      if constexpr (F == 2) t.add(stage);
    }
  }
  return __ballot_sync(kFull, mine && !left) != 0;
}

enum CutResult : int { kKept = 0, kCut = 1, kFailed = 2 };

// One candidate against one piece (the semantics of src/bvh_peel.cpp:141-199):
// where the piece lies behind the candidate, the part inside the candidate is
// hidden; the parts of the rest are queued with walk position `cursor` but
// for the last one, which becomes the piece (n = 0 when there is none).  A
// piece whose covered part clips away to nothing is kept unchanged (kKept).
// `tested`: may_hide() has accepted exactly this piece.
// The covered part is found first; the uncovered parts met on the way wait in
// shared memory (more than kClipParts of them are split off a second time),
// so a cut that hides nothing leaves no parts behind.
template <int F>
__device__ inline int cut_piece(const Dev &d, const PieceQueue &queue, const PiecePool &hidden,
                                V2 &p, V2 &q, int &n, const Occluder &c, const Plane &st,
                                int source, int target, int cursor,
                                bool tested, V2 *left, V2 *right, V2 *held, int *held_n,
                                Tally &t) {
  const Group<32> g;
  const int lane = g.lane;
  if (!tested && warp_separated<F>(p, q, n, c, t)) return kKept;
  const bool mine = lane < n;
  const Plane so = d.scores[c.source];
  const double behind_by = value(Plane{st.a - so.a, st.b - so.b, st.c - so.c, 0.0}, p);
  int sign;
  if constexpr (F == 0) {
    sign = sign_of(behind_by);
  } else {
    int stage = 0;
    sign = mine ? order_sign<F>(st, value(st, p), so, value(so, p), p, stage) : 0;
    if constexpr (F == 2)
      if (mine) t.add(stage);
  }
  bool positive = __ballot_sync(kFull, mine && sign > 0) != 0;
  const bool negative = __ballot_sync(kFull, mine && sign < 0) != 0;
  if (!positive && !negative) {
    positive = source > c.source;
    if (lane == 0) atomicAdd(&d.status[kDepthTies], 1);
  }
  if (!positive) return kKept;
  V2 behind = p, nearer = p;
  int behind_n = n, nearer_n = 0;
  if (negative && !group_split<F>(g, p, q, n, behind_by, sign, left, right, behind, behind_n, nearer,
                                 nearer_n)) {
    if (lane == 0) set_error(d.status, kErrPolygon);
    return kFailed;
  }
  // The part that stays with this warp; the ones before it are queued.
  V2 keep = nearer;
  int keep_n = 0;
  auto emit = [&](V2 x, int m) {
    if (keep_n > 0 && !queue_piece(queue, keep, keep_n, target, cursor)) return false;
    keep = x;
    keep_n = m;
    return true;
  };
  int parts = 0;
  for (int pass = 0; pass < 2; ++pass) {
    V2 in = behind;
    int in_n = behind_n;
    for (int e = 0; e < c.n && in_n > 0; ++e) {
      const V2 a = c.v[e], b = c.v[e + 1 < c.n ? e + 1 : 0], dir = b - a;
      const double off = value(Plane{-dir.y, dir.x, 0.0, 0.0}, in - a);
      int s, stage = 0;
      if constexpr (F == 0)
        s = sign_of(off);
      else
        s = lane < in_n ? side_sign<F>(a, b, in, stage) : 0;
      if constexpr (F == 2)
        if (lane < in_n) t.add(stage);
      // Nothing lies outside this edge: the part is inside as it is.
      if (!__ballot_sync(kFull, lane < in_n && s < 0)) continue;
      const V2 in_next = g.shfl(in, lane + 1 < in_n ? lane + 1 : 0);
      V2 inside, out;
      int inside_n, out_n;
      if (!group_split<F>(g, in, in_next, in_n, off, s, left, right, inside, inside_n, out, out_n)) {
        if (lane == 0) set_error(d.status, kErrPolygon);
        return kFailed;
      }
      if (out_n > 0) {
        if (pass == 1) {
          if (!emit(out, out_n)) return kFailed;
        } else {
          if (parts < kClipParts) {
            held[kMaxVertices * parts + lane] = out;
            held_n[parts] = out_n;
          }
          ++parts;
        }
      }
      in = inside;
      in_n = inside_n;
    }
    if (pass == 0) {
      if (in_n == 0) return kKept;  // nothing covered after all
      if (lane == 0 && atomicAdd(&d.target_hidden[target], 1) >= d.pieces)
        set_error(d.status, kErrWorker);
      if (!hide_piece(hidden, in, in_n, target) && lane == 0) set_error(d.status, kErrResidual);
      if (nearer_n > 0) emit(nearer, nearer_n);
      if (parts <= kClipParts) {
        __syncwarp();
        for (int k = 0; k < parts; ++k)
          if (!emit(held[kMaxVertices * k + lane], held_n[k])) return kFailed;
        __syncwarp();
        break;
      }
    }
  }
  p = keep;
  n = keep_n;
  q = g.shfl(p, lane + 1 < n ? lane + 1 : 0);
  return kCut;
}

// Seed the clipping queue with this layer's targets, each a whole residual
// patch at the start of its walk.
__global__ void k_clip_begin(Dev d) {
  const int par = *d.parity;
  const int live = int(min(int64_t(d.status[kResidual]), d.cap.frontier));
  for (int64_t i = tid(); i < live; i += stride()) {
    const int n = d.status[kError] == 0 ? d.res_n[par][i] : 0;
    V2 *dst = piece_at(d.work_v[0], i);
    const V2 *src = piece_at(d.res_v[par], i);
    for (int j = 0; j < n; ++j) dst[j] = src[j];
    d.work_n[0][i] = n;
    d.work_target[0][i] = int(i);
    d.work_cursor[0][i] = 0;  // the source hierarchy's first leaf
    d.target_visible[i] = 0;
    d.target_hidden[i] = 0;
  }
  if (tid() == 0) {
    const int queued = live <= d.work_cap ? live : 0;
    if (live > d.work_cap) set_error(d.status, kErrWorker);
    d.sc[kClipLive] = queued;
    d.sc[kClipNext] = queued;
    d.sc[kClipSpill] = 0;
    d.sc[kClipPending] = queued;
    d.sc[kClipTurns] = 0;
    d.sc[kClipHidden] = 0;
    d.sc[kClipParity] = 0;
    d.sc[kFrontierNext] = 0;
    ++*d.clip_epoch;
    const int c = queued > 0 && d.status[kError] == 0;
    d.sc[kClipCondition] = c;
    if (d.use_inner) cudaGraphSetConditional(d.inner_handle, unsigned(c));
  }
}

// After a launch, by its last block: the spilled pieces become the next
// launch's queue; stop when there are none.
__device__ inline void advance_clipping(const Dev &d) {
  volatile int *sc = d.sc;
  const int spilled = min(sc[kClipSpill], d.work_cap);
  sc[kClipLive] = spilled;
  sc[kClipNext] = spilled;
  sc[kClipSpill] = 0;
  sc[kClipPending] = spilled;
  sc[kFrontierNext] = 0;
  sc[kClipParity] = sc[kClipParity] ^ 1;
  d.status[kLoops] = *(volatile int *)&d.status[kLoops] + 1;
  ++*d.clip_epoch;
  const int c = spilled > 0 && *(volatile int *)&d.status[kError] == 0;
  sc[kClipCondition] = c;
  if (d.use_inner) cudaGraphSetConditional(d.inner_handle, unsigned(c));
}

// Clips the queue, one piece per warp, until it is empty.  F is the predicate
// form.  A leaf batch of the walk holds up to 32 candidates: each lane decides
// one against the piece as the batch met it (may_hide), and the few left are
// cut one by one in leaf order with a lane per piece vertex.  A part of a
// piece that may_hide rejected needs no new test: it lies in the piece.
//
// Warps take slots of the queue by ticket and wait for the slot to be written,
// or for the last piece to end.  A waited-for slot is written by a warp that
// holds a piece and waits for nothing, so every wait ends; each is bounded all
// the same (kWaitLimit polls, about a second, without a piece queued or ended
// or a turn of Dev::clip_budget walk steps), and running out is an error.
//
// A walk is not put back into the queue between its turns: the queue's slots
// are written once per launch, so that they are as many as the pieces (a target
// or an uncovered part each, which ends as a visible or a hidden piece, or
// several), however long their walks are.
//
// The bound is the serial chain of cuts of one piece, not throughput: a layer
// has a few thousand pieces for 148 SMs.  A thread per piece, with its polygons
// in local memory and every cut ending the piece's launch, took 59.8 ms per
// extraction of two nested icospheres (2,560 faces, 12 layers) and 42.6 ms of
// a crossing scene of 994 faces; a warp per piece with a launch per round of
// cuts took 10.1 and 7.0, with the queue taken while it grows 5.4 and 3.2.
// More polls, longer or shorter turns and half the blocks are all within 2%.
constexpr int kWaitLimit = 1 << 20;
constexpr int kMostSteps = 1024;  // of a turn, far less than a wait's limit takes

template <int F>
__global__ void __launch_bounds__(kBlock, 4) k_clip_round(Dev d) {
  __shared__ V2 s_piece[kClipWarps][kMaxVertices];
  __shared__ V2 s_parts[kClipWarps][2][kMaxVertices];
  __shared__ V2 s_held[kClipWarps][kClipParts * kMaxVertices];
  __shared__ int s_held_n[kClipWarps][kClipParts];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  V2 *piece = s_piece[warp];
  const int wpar = d.sc[kClipParity], next = wpar ^ 1;
  const int live = min(d.sc[kClipLive], d.work_cap);
  const int rpar = *d.parity;
  const int layer = d.status[kPass];
  const int source_leaves = *d.source_tree.size, residual_leaves = *d.residual_tree.size;
  const PieceQueue queue{
      {d.work_v[wpar], d.work_n[wpar], d.work_target[wpar], d.work_cursor[wpar],
       &d.sc[kClipNext], d.work_cap},
      {d.work_v[next], d.work_n[next], d.work_target[next], d.work_cursor[next],
       &d.sc[kClipSpill], d.work_cap},
      d.work_ready[wpar], &d.sc[kClipPending], d.status, *d.clip_epoch};
  const PiecePool hidden{d.hid_v, d.hid_n, d.hid_target, nullptr, &d.sc[kClipHidden],
                         d.hidden_cap};
  long long tested = 0;  // lane 0's tally
  Tally clip;
  for (;;) {
    int i = 0;
    if (lane == 0) {
      i = atomicAdd(&d.sc[kFrontierNext], 1);
      if (i >= d.work_cap) i = -1;
      int seen = 0;
      for (int polls = 0; i >= 0; ++polls) {
        // Loaded together, for one latency per poll.
        const int failed = *(volatile int *)&d.status[kError];
        const int ready = *(volatile int *)&queue.ready[i];
        const int pending = *(volatile int *)queue.pending;
        if (failed != 0) {
          i = -1;
          break;
        }
        // Slots below `live` were written before this launch.
        if (i < live || ready == queue.epoch) break;
        if (pending <= 0) {  // every piece has ended, so no slot is written any more
          i = -1;
          break;
        }
        if ((polls & 63) == 63) {
          const int progress = pending + *(volatile int *)queue.pool.count +
                               *(volatile int *)&d.sc[kClipTurns];
          if (progress != seen) polls = 0;
          seen = progress;
        }
        if (polls > kWaitLimit) {
          set_error(d.status, kErrWait);
          i = -1;
          break;
        }
        __nanosleep(400);
      }
      __threadfence();
    }
    i = __shfl_sync(kFull, i, 0);
    if (i < 0) break;
    // Past L1, which may hold these lines from before they were written.
    int n = __ldcg(&d.work_n[wpar][i]);
    const int target = __ldcg(&d.work_target[wpar][i]);
    const int start = __ldcg(&d.work_cursor[wpar][i]);
    V2 p = v2(0.0, 0.0);
    if (lane < n) {
      const double2 x = __ldcg(reinterpret_cast<const double2 *>(piece_at(d.work_v[wpar], i)) + lane);
      p = v2(x.x, x.y);
    }
    if (n < 3) {
      if (lane == 0) atomicSub(queue.pending, 1);
      continue;
    }
    V2 q = Group<32>().shfl(p, lane + 1 < n ? lane + 1 : 0);
    const int source = d.res_src[rpar][target];
    const Plane st = d.scores[source];
    const int turn = min(max(d.clip_budget, 8), kMostSteps);
    int budget = turn;
    bool done = false;  // nothing of the piece is left in this warp
    for (int tree = start >> kCursorTree; tree < 2 && !done; ++tree) {
      const Tree &t = tree == 0 ? d.source_tree : d.residual_tree;
      const int leaves = tree == 0 ? source_leaves : residual_leaves;
      int cursor = tree == start >> kCursorTree ? start & kCursorLeaf : 0;
      Box box = group_bounds<32>(p, n, st);
      box.lo.z = -1.0e30f;
      WarpWalk w;
      walk_begin(w, t, leaves, box.lo, box.hi, cursor);
      unsigned batch;
      int first, resume = leaves;
      while (!done) {
        if (!walk_next(w, t, leaves, box.lo, box.hi, cursor, budget, batch, first, resume)) {
          if (resume >= leaves) break;
          if (lane == 0) atomicAdd(&d.sc[kClipTurns], 1);
          done = __shfl_sync(kFull, *(volatile int *)&d.status[kError], 0) != 0;
          budget = turn;
          cursor = resume;
          walk_begin(w, t, leaves, box.lo, box.hi, cursor);  // with the box it has by now
          continue;
        }
        // Each lane's candidate of the batch.
        Occluder mine{nullptr, 0, -1};
        if ((batch >> lane) & 1u) {
          const int c = __ldg(&t.ids[first + lane]);
          bool eligible = true;
          if (tree == 0) {
            mine = Occluder{d.src_v + int64_t(kSourceVertices) * c, d.src_n[c], c};
            eligible = d.ranks[c] >= layer;
          } else {
            mine = Occluder{piece_at(d.res_v[rpar], c), d.res_n[rpar][c], d.res_src[rpar][c]};
          }
          if (!eligible || mine.source == source) mine.source = -1;
        }
        const unsigned candidates = __ballot_sync(kFull, mine.source >= 0);
        if (!candidates) continue;
        tested += __popc(candidates);
        __syncwarp();
        piece[lane] = p;
        __syncwarp();
        const bool hides = mine.source >= 0 &&
                           may_hide<F>(d, piece, n, st, source, mine, clip);
        unsigned left = __ballot_sync(kFull, hides);
        bool whole = true;
        while (left && !done) {
          const int k = __ffs(int(left)) - 1;
          left &= left - 1;
          Occluder c;
          c.v = reinterpret_cast<const V2 *>(
              __shfl_sync(kFull, reinterpret_cast<unsigned long long>(mine.v), k));
          c.n = __shfl_sync(kFull, mine.n, k);
          c.source = __shfl_sync(kFull, mine.source, k);
          const int result =
              cut_piece<F>(d, queue, hidden, p, q, n, c, st, source, target,
                           (tree << kCursorTree) | (first + k + 1), whole, s_parts[warp][0],
                           s_parts[warp][1], s_held[warp], s_held_n[warp], clip);
          if (result == kKept) continue;
          done = result == kFailed || n == 0;
          if (done) break;
          whole = false;
          box = group_bounds<32>(p, n, st);
          box.lo.z = -1.0e30f;
        }
      }
    }
    if (done) {
      __syncwarp();
      if (lane == 0) atomicSub(queue.pending, 1);
      continue;
    }
    int slot = 0;
    if (lane == 0) {
      if (atomicAdd(&d.target_visible[target], 1) >= d.pieces) set_error(d.status, kErrWorker);
      slot = atomicAdd(&d.status[kPolygons], 1);
      if (slot >= d.cap.regions) set_error(d.status, kErrOutput);
      atomicSub(queue.pending, 1);
    }
    slot = __shfl_sync(kFull, slot, 0);
    if (slot >= d.cap.regions) continue;
    if (lane < n) d.out_v[int64_t(kMaxVertices) * slot + lane] = p;
    if (lane == 0) {
      d.out_n[slot] = n;
      d.out_src[slot] = source;
      d.out_layer[slot] = layer;
      atomicMax(&d.status[kLayers], layer + 1);
    }
  }
  if (lane == 0 && layer < d.cap.layers && tested) count_add(&d.stats[3 * int64_t(layer) + 1], tested);
  if constexpr (F == 2) clip.flush(d, kPredClip);
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(&d.sc[kRoundBlocks], 1) == int(gridDim.x) - 1) {
      __threadfence();
      d.sc[kRoundBlocks] = 0;
      advance_clipping(d);
    }
  }
}

// After the last round: a target with no visible piece is hidden whole (its
// hidden pieces are dropped); every other target's hidden pieces go to the
// next layer's residual.  Threads run over targets and hidden pieces alike.
__global__ void k_clip_finish(Dev d) {
  const int rpar = *d.parity;
  const int targets = int(min(int64_t(d.status[kResidual]), d.cap.frontier));
  const int hidden = min(d.sc[kClipHidden], d.hidden_cap);
  const int layer = d.status[kPass];
  V2 *next_v = d.res_v[rpar ^ 1];
  int *next_n = d.res_n[rpar ^ 1], *next_src = d.res_src[rpar ^ 1];
  long long restored = 0;
  int most_hidden = 0;
  for (int64_t i = tid(); i < int64_t(targets) + hidden; i += stride()) {
    if (d.status[kError] != 0) break;
    const V2 *src;
    int n, source;
    if (i < targets) {
      most_hidden = max(most_hidden, d.target_hidden[i]);
      if (d.target_visible[i] > 0) continue;
      src = piece_at(d.res_v[rpar], i);
      n = d.res_n[rpar][i];
      source = d.res_src[rpar][i];
      ++restored;
    } else {
      const int h = int(i - targets), target = d.hid_target[h];
      if (d.target_visible[target] == 0) continue;
      src = piece_at(d.hid_v, h);
      n = d.hid_n[h];
      source = d.res_src[rpar][target];
    }
    const int slot = reserve(&d.status[kNextResidual], 1);
    if (slot >= d.cap.frontier) {
      set_error(d.status, kErrResidual);
      continue;
    }
    V2 *dst = piece_at(next_v, slot);
    for (int j = 0; j < n; ++j) dst[j] = src[j];
    next_n[slot] = n;
    next_src[slot] = source;
  }
  if (layer < d.cap.layers) {
    if (tid() == 0) count_add(&d.stats[3 * int64_t(layer)], targets);
    if (restored) count_add(&d.stats[3 * int64_t(layer) + 2], restored);
  }
  if (most_hidden) atomicMax(&d.status[kMaxHidden], most_hidden);
}

// The next layer's residual becomes current; the layer loop goes on while
// patches remain and the layer limit allows.
__global__ void k_layer_next(Dev d) {
  const int remaining = d.status[kNextResidual];
  d.status[kResidual] = remaining;
  d.status[kNextResidual] = 0;
  d.status[kPeakResidual] = max(d.status[kPeakResidual], remaining);
  *d.parity ^= 1;
  const int layer = ++d.status[kPass];
  if (remaining > 0 && layer >= d.limit && d.all_layers) set_error(d.status, kErrLayers);
  const int c = remaining > 0 && layer < d.limit && d.status[kError] == 0;
  *d.condition = c;
  if (d.use_handle) cudaGraphSetConditional(d.cond_handle, unsigned(c));
}

}  // namespace

cudaError_t stage_device_prepare(const Dev &d, SortScratch &s, TreeBuffers &source_tree,
                                 TreeBuffers &contour_tree, cudaStream_t st) {
  EDP_CHECK(stage_prepare_common(d, false, st));
  EDP_CHECK(tree_build(source_tree, d.src_lo, d.src_hi, nullptr, d.n, false, s, st));
  EDP_CHECK(cudaMemsetAsync(d.stats, 0, sizeof(long long) * 3 * d.cap.layers, st));
  k_contour_bounds<<<blocks(d.n), kBlock, 0, st>>>(d);
  note_launch();
  EDP_CHECK(tree_build(contour_tree, d.contour_lo, d.contour_hi, nullptr, d.n, false, s, st));
  k_classify<<<blocks(d.n), kBlock, 0, st>>>(d);
  note_launch();
  k_start_loop<<<1, 1, 0, st>>>(d);
  note_launch();
  return cudaGetLastError();
}

cudaError_t stage_device_layer(const Dev &layer_dev, SortScratch &s, TreeBuffers &source_tree,
                               TreeBuffers &residual_tree, cudaStream_t st, cudaStream_t rounds) {
  Dev d = layer_dev;
  k_retire_bounds<<<blocks(d.n), kBlock, 0, st>>>(d);
  note_launch();
  EDP_CHECK(tree_refit(source_tree, d.src_lo, d.src_hi, st));
  k_active_bounds<<<blocks(d.cap.frontier), kBlock, 0, st>>>(d);
  note_launch();
  EDP_CHECK(tree_build(residual_tree, d.res_lo, d.res_hi, d.sc + kFrontierLive, 0, false, s, st));
  const unsigned clip_blocks = 148 * 4;  // 4 blocks of 4 warps per SM, a piece per warp
  if (d.use_handle) {
    // Inside a capture: the clipping rounds are a conditional WHILE node of
    // the graph being recorded on `st` (the layer loop's body), their body
    // recorded on `rounds`.
    cudaStreamCaptureStatus cs;
    cudaGraph_t g = nullptr;
    const cudaGraphNode_t *deps = nullptr;
    size_t ndeps = 0;
    EDP_CHECK(cudaStreamGetCaptureInfo(st, &cs, nullptr, &g, &deps, &ndeps));
    cudaGraphConditionalHandle handle;
    EDP_CHECK(cudaGraphConditionalHandleCreate(&handle, g, 0, cudaGraphCondAssignDefault));
    d.use_inner = 1;
    d.inner_handle = handle;
    k_clip_begin<<<blocks(d.cap.frontier), kBlock, 0, st>>>(d);
    note_launch();
    EDP_CHECK(cudaStreamGetCaptureInfo(st, &cs, nullptr, &g, &deps, &ndeps));
    alignas(cudaGraphNodeParams) unsigned char raw[sizeof(cudaGraphNodeParams)] = {};
    cudaGraphNodeParams &params = *reinterpret_cast<cudaGraphNodeParams *>(raw);
    params.type = cudaGraphNodeTypeConditional;
    params.conditional.handle = handle;
    params.conditional.type = cudaGraphCondTypeWhile;
    params.conditional.size = 1;
    cudaGraphNode_t loop;
    EDP_CHECK(cudaGraphAddNode(&loop, g, deps, ndeps, &params));
    cudaGraph_t body = params.conditional.phGraph_out[0];
    EDP_CHECK(cudaStreamUpdateCaptureDependencies(st, &loop, 1, cudaStreamSetCaptureDependencies));
    EDP_CHECK(cudaStreamBeginCaptureToGraph(rounds, body, nullptr, nullptr, 0,
                                            cudaStreamCaptureModeRelaxed));
    EDP_LAUNCH_FORM(d.predicates, k_clip_round, clip_blocks, kBlock, rounds, d);
    note_launch();
    cudaError_t launched = cudaGetLastError();
    cudaGraph_t captured = nullptr;
    cudaError_t end = cudaStreamEndCapture(rounds, &captured);
    EDP_CHECK(launched);
    EDP_CHECK(end);
  } else {
    // Eager (warm-up): the host drives the rounds.
    d.use_inner = 0;
    k_clip_begin<<<blocks(d.cap.frontier), kBlock, 0, st>>>(d);
    for (;;) {
      int more = 0;
      EDP_CHECK(cudaMemcpyAsync(&more, d.sc + kClipCondition, sizeof(int),
                                cudaMemcpyDeviceToHost, st));
      EDP_CHECK(cudaStreamSynchronize(st));
      if (!more) break;
      EDP_LAUNCH_FORM(d.predicates, k_clip_round, clip_blocks, kBlock, st, d);
      EDP_CHECK(cudaGetLastError());
    }
  }
  k_clip_finish<<<blocks(int64_t(d.cap.frontier) + d.hidden_cap), kBlock, 0, st>>>(d);
  note_launch();
  k_layer_next<<<1, 1, 0, st>>>(d);
  note_launch();
  return cudaGetLastError();
}

}  // namespace edp
