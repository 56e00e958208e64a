// Mesh stage: boundary vertex gathering and deduplication, the layered point
// grid (or, for very deep scenes, the layered point hierarchy), per-polygon
// noding, centroid-fan triangulation and world lifting
// (warp_peel/kernels.py:941-1204, events.py:720-780).
#include "../../include/edp.h"
#include "edp_internal.h"
#include "edp_warp.cuh"

namespace edp {
namespace {

constexpr int kBlock = 128;
constexpr int kMaxEdgeVertices = 128;  // edge noding capacity (solver.py:140-143)

__device__ inline int64_t tid() { return blockIdx.x * int64_t(blockDim.x) + threadIdx.x; }
__device__ inline int64_t stride() { return int64_t(gridDim.x) * blockDim.x; }

// Grid column (or row) of a window coordinate: floor(v G) clamped to the
// grid.  Monotone in v, so a query interval's cells hold every point inside it.
__device__ inline int grid_cell(double v, int g) {
  const double c = floor(v * double(g));
  return c < 0.0 ? 0 : c > double(g - 1) ? g - 1 : int(c);
}

// Boundary vertices with their layer, one slot per polygon vertex
// (kernels.py:953-991, event_kernels.py:504-516), in the polygons' (layer,
// Morton) order, so that the copies of one point, which neighbouring polygons
// share, meet the point table close together in time.  The point grid serves
// this extraction when it has a row for every layer; otherwise the point
// hierarchy does.
__global__ void k_scatter(Dev d) {
  const int live = d.sc[kLivePolygons];
  // No block of this launch writes the count, so all of them take it alike.
  const int total = d.sc[kLiveVertices];
  const bool fits = int64_t(total) <= d.cap.vertices;
  fill_words(d.point_table, ceil_div(int64_t(d.point_mask) + 1, 4), 0xffffffffu, tid(), stride());
  if (tid() == 0) {
    const int layers = d.status[kLayers];
    const bool on = d.status[kError] == 0 && fits && layers <= d.grid_layers;
    d.sc[kGridOn] = on ? 1 : 0;
    d.sc[kGridCells] = on ? int(int64_t(layers) * d.point_grid * d.point_grid) : 0;
    d.status[kBoundaryVertices] = total;
    if (!fits) set_error(d.status, kErrVertices);
  }
  if (!fits) return;
  for (int64_t k = tid(); k < live; k += stride()) {
    if (d.status[kError] != 0) return;
    const int i = d.order[k];
    const V2 *p = d.out_v + int64_t(kMaxVertices) * i;
    const int layer = d.out_layer[i];
    const int64_t base = d.offsets[k];
    const int n = int(min(int64_t(d.out_n[i]), d.cap.vertices - base));
    for (int j = 0; j < n; ++j) {
      d.bverts[base + j] = p[j];
      d.blayers[base + j] = layer;
    }
  }
}

// Counting sort of the distinct points by (layer, cell): the scan of the
// counts gives each cell's start, and each point takes a slot of its cell.
// Taking the slots counts every cell back down to zero, so the counts need no
// clearing between extractions.
__global__ void k_grid_scatter(Dev d, cudaGraphConditionalHandle handle, int conditional) {
  if (tid() == 0) {
    // The point hierarchy's items, and in a graph whether its node runs.
    d.sc[kTreePoints] = d.sc[kGridOn] ? 0 : d.sc[kUniqueVertices];
    if (conditional) cudaGraphSetConditional(handle, d.sc[kGridOn] ? 0u : 1u);
  }
  if (!d.sc[kGridOn]) return;
  const int total = d.sc[kUniqueVertices], g = d.point_grid;
  if (tid() == 0) d.cell_start[d.sc[kGridCells]] = total;
  for (int64_t u = tid(); u < total; u += stride()) {
    const V2 x = d.uverts[u];
    const int layer = int(d.pt_lo[u].z);
    const int64_t cell = (int64_t(layer) * g + grid_cell(x.y, g)) * g + grid_cell(x.x, g);
    const int slot = atomicSub(&d.cell_count[cell], 1) - 1;
    d.grid_pts[d.cell_start[cell] + slot] = x;
  }
}

// Each distinct (layer, point) enters the point hierarchy once: a vertex
// shared by several patches would otherwise be a candidate of every query
// several times over.  One thread per boundary vertex inserts it into an
// open-addressing table keyed by its bits and layer; the first slot to claim
// an entry adds the point.
template <int kTogether>
__device__ inline void unique_points(const Dev &d, int total) {
  const int lane = threadIdx.x & 31;
  const bool grid = d.sc[kGridOn] != 0;
  const uint32_t mask = uint32_t(d.point_mask);
  for (int64_t s0 = kTogether * (tid() - lane); s0 < total; s0 += kTogether * stride()) {
    V2 x[kTogether], y[kTogether];
    int layer[kTogether], cur[kTogether], of[kTogether];
    uint32_t probe[kTogether];
#pragma unroll
    for (int j = 0; j < kTogether; ++j) {
      const int64_t slot = s0 + 32 * j + lane;
      x[j] = slot < total ? d.bverts[slot] : v2(0.0, 0.0);
      layer[j] = slot < total ? d.blayers[slot] : 0;
    }
#pragma unroll
    for (int j = 0; j < kTogether; ++j) {
      const uint64_t h = mix64(mix64(key_bits(x[j].x)) ^ key_bits(x[j].y)) ^
                         mix64(uint64_t(layer[j]) + 7ull);
      probe[j] = uint32_t(h) & mask;
      const int64_t slot = s0 + 32 * j + lane;
      if (kTogether > 1 || slot >= total)
        cur[j] = __ldcg(&d.point_table[probe[j]]);
      else
        cur[j] = atomicCAS(&d.point_table[probe[j]], -1, int(slot));
    }
    unsigned fresh = 0;
#pragma unroll
    for (int j = 0; j < kTogether; ++j) {
      if (kTogether == 1 && s0 + lane < total && cur[j] < 0) fresh = 1;
      y[j] = cur[j] >= 0 ? d.bverts[cur[j]] : v2(0.0, 0.0);
      of[j] = cur[j] >= 0 ? d.blayers[cur[j]] : -1;
    }
#pragma unroll
    for (int j = 0; j < kTogether; ++j) {
      const int64_t slot = s0 + 32 * j + lane;
      bool found = slot >= total || (fresh >> j & 1u) || (cur[j] >= 0 && y[j] == x[j] && of[j] == layer[j]);
      for (int k = 0; !found && k <= d.point_mask; ++k) {
        int c = k == 0 ? cur[j] : __ldcg(&d.point_table[probe[j]]);
        if (c < 0) c = atomicCAS(&d.point_table[probe[j]], -1, int(slot));
        if (c < 0) {
          fresh |= 1u << j;
          found = true;
        } else {
          found = d.bverts[c] == x[j] && d.blayers[c] == layer[j];
          probe[j] = (probe[j] + 1) & mask;
        }
      }
    }
    __syncwarp();
    unsigned mine[kTogether];
    int count = 0;
#pragma unroll
    for (int j = 0; j < kTogether; ++j) {
      mine[j] = __ballot_sync(kFull, fresh >> j & 1u);
      count += __popc(mine[j]);
    }
    int base = 0;
    if (lane == 0 && count) base = atomicAdd(&d.sc[kUniqueVertices], count);
    base = __shfl_sync(kFull, base, 0);
#pragma unroll
    for (int j = 0; j < kTogether; ++j) {
      if (fresh >> j & 1u) {
        const int u = base + __popc(mine[j] & ((1u << lane) - 1u));
        if (grid) {
          const int g = d.point_grid;
          atomicAdd(&d.cell_count[(int64_t(layer[j]) * g + grid_cell(x[j].y, g)) * g +
                                  grid_cell(x[j].x, g)], 1);
        }
        d.uverts[u] = x[j];
        d.pt_lo[u] = make_float4(__double2float_rd(x[j].x - 2.0e-7),
                                 __double2float_rd(x[j].y - 2.0e-7), float(layer[j]), 0.f);
        d.pt_hi[u] = make_float4(__double2float_ru(x[j].x + 2.0e-7),
                                 __double2float_ru(x[j].y + 2.0e-7), float(layer[j]), 0.f);
      }
      base += __popc(mine[j]);
    }
  }
}

// Bound by the latency of the table's accesses and by the reservations' atomics
// on one counter.  Up to one vertex per thread of the grid a lane takes one;
// above, it looks four up together, reading an entry before it claims one
// (most vertices are there already).  This stage, one at a time, then four:
// knot-65536 0.28 -> 0.19 ms (two 0.21, eight 0.24), 720K primitives 1.87 ->
// 0.95 (two 1.00, eight 1.00); four at the smallest sizes cost 0.01 ms.
__global__ void k_unique_points(Dev d) {
  if (d.status[kError] != 0) return;
  const int total = d.sc[kLiveVertices];
  if (total <= stride())
    unique_points<1>(d, total);
  else
    unique_points<4>(d, total);
}

// Sort key of each live output polygon: the Morton code of its box centre
// (the 15-bit-per-axis code of the hierarchies, kernels.py:67-91, cut to 12
// bits per axis), below its layer when `layered`.
__device__ inline uint64_t morton_of(const Dev &d, int64_t i) {
  const V2 *p = d.out_v + int64_t(kMaxVertices) * i;
  const int n = min(max(d.out_n[i], 1), kMaxVertices);
  double lx = p[0].x, ly = p[0].y, hx = p[0].x, hy = p[0].y;
  for (int j = 1; j < n; ++j) {
    lx = fmin(lx, p[j].x); ly = fmin(ly, p[j].y);
    hx = fmax(hx, p[j].x); hy = fmax(hy, p[j].y);
  }
  const float cx = fminf(fmaxf(float(0.5 * (lx + hx)), 0.f), 1.f);
  const float cy = fminf(fmaxf(float(0.5 * (ly + hy)), 0.f), 1.f);
  const uint32_t x = uint32_t(int(cx * 32767.0f)), y = uint32_t(int(cy * 32767.0f));
  // 12 bits per axis (a 4096 x 4096 grid) are plenty for locality.
  return (part1by1(x) | (part1by1(y) << 1)) >> 6;
}

__device__ inline int live_outputs(const Dev &d) {
  return int(min(int64_t(d.status[kPolygons]), d.cap.regions));
}

// The rounds that a subdivision made: one above the generations, which the
// polygons carry in place of their layers until they are ranked.
__device__ inline void count_rounds(const Dev &d, int generation) {
  generation = __reduce_max_sync(kFull, generation);
  if ((threadIdx.x & 31) == 0 && generation >= *(volatile long long *)&d.metrics[kRounds])
    atomicMax(&d.metrics[kRounds], (long long)generation + 1);
}

__global__ void k_order_keys(Dev d) {
  const int live = live_outputs(d);
  int generation = 0;
  if (tid() == 0) d.sc[kLivePolygons] = live;
  for (int64_t i = tid(); i < live; i += stride()) {
    d.order_keys[i] = morton_of(d, i);
    d.order[i] = int(i);
    generation = max(generation, d.out_layer[i]);
  }
  count_rounds(d, generation);
}

// The same order by a counting sort: buckets of the leading Morton bits, below
// the layer when `layered`, 4 to 8 per polygon (the polygons cover a small part
// of the window) and at most 2^Dev::order_bits.  Three launches where the radix
// sort took 5 and 7; the order inside a bucket is left to chance, which no
// result depends on.  Twice the buckets cost as much in their scan as they
// gain in locality (both within 0.03 ms on the 65,536-face knot), but with 2^20
// at most the rays and the noding of 2.2M polygons of the 720K primitives took
// 2.11 and 3.69 ms instead of 1.70 and 3.60.
__device__ inline int ceil_log2(int v) { return v <= 1 ? 0 : 32 - __clz(v - 1); }

__device__ inline void order_bits(const Dev &d, int live, int layered, int &layer_shift,
                                  int &layer_bits, int &morton_bits) {
  const int most = d.order_bits, want = min(most, ceil_log2(live) + 2);
  layer_bits = layered ? ceil_log2(max(d.status[kLayers], 1)) : 0;
  layer_shift = max(0, layer_bits - most);
  layer_bits -= layer_shift;
  morton_bits = max(0, want - layer_bits);
}

__global__ void k_order_count(Dev d, int layered) {
  const int live = live_outputs(d);
  int layer_shift, layer_bits, morton_bits;
  order_bits(d, live, layered, layer_shift, layer_bits, morton_bits);
  if (tid() == 0) {
    d.sc[kLivePolygons] = live;
    d.sc[kOrderLive] = 1 << (layer_bits + morton_bits);
  }
  int generation = 0;
  for (int64_t i = tid(); i < live; i += stride()) {
    int bucket = int(morton_of(d, i) >> (24 - morton_bits));
    if (layered) {
      // A layer past the limit (an error, or a suppressed polygon) shares the last.
      const int layer = min(max(d.out_layer[i], 0) >> layer_shift, (1 << layer_bits) - 1);
      bucket |= layer << morton_bits;
    }
    if (!layered) generation = max(generation, d.out_layer[i]);
    d.order_keys[i] = uint64_t(bucket) << 32 | unsigned(atomicAdd(&d.order_count[bucket], 1));
  }
  if (!layered) count_rounds(d, generation);
}

// Places the polygons, and lays out what the stage scans next: each polygon's
// vertex count in this order.
__global__ void k_order_place(Dev d, int layered) {
  const int live = d.sc[kLivePolygons];
  if (layered && tid() == 0) {
    d.sc[kUniqueVertices] = 0;
    d.sc[kHeavyPolygons] = 0;
  }
  const bool failed = layered && d.status[kError] != 0;
  for (int64_t i = tid(); i < live; i += stride()) {
    const uint64_t key = d.order_keys[i];
    const int at = d.order_start[key >> 32] + int(unsigned(key));
    d.order[at] = int(i);
    d.counts[at] = failed ? 0 : d.out_n[i];
    if (!layered) {
      d.parents[i] = int(i);
      d.group_counts[i] = 0;
      d.group_fill[i] = 0;
    }
  }
}

// World position of a window point on a source plane (kernels.py:994-1006).
__device__ inline void lift(const Dev &d, V2 x, const Plane &s, double *w) {
  const double *st = d.settings, *m = d.inverse;
  double u = st[0] + x.x * (st[2] - st[0]);
  double v = st[1] + x.y * (st[3] - st[1]);
  double z = value(s, x);
  if (st[4] != 0.0) {
    z = -1.0 / z;
    u *= z;
    v *= z;
  }
  for (int r = 0; r < 3; ++r) w[r] = m[4 * r] * u + m[4 * r + 1] * v + m[4 * r + 2] * z + m[4 * r + 3];
}

// Node every edge of one output polygon against the same-layer boundary
// vertices lying on it (collinear within EPS, strictly inside the edge), then
// emit the polygon's centroid fan with the split points, lifted to world
// space (kernels.py:1009-1125).  One point-hierarchy query per polygon (its
// box contains every edge's box) replaces the reference's query per edge; the
// acceptance test and therefore the triangles are the same.
constexpr int kPolygonSplits = 256;  // split points buffered per polygon
// Candidate points x edges above which a polygon is noded by a whole warp
// (k_mesh_heavy) rather than by eight lanes, so that a few large polygons in
// dense cells do not hold up the other groups of a warp:
// Dev::heavy_noding_work (1024 unless tuned).

// The centroid fan of polygon p (n vertices, centroid `center`) through its
// split points sorted by (edge, parameter).  Counts the fan triangles (signed
// doubled area above EPS^2: noded points 1e-13 apart can otherwise give
// slivers of area ~1e-19 whose orientation rounding decides; the reference
// tests |area|, kernels.py:1105), reserves their slots at once, then writes
// them with their world positions.
__device__ inline void emit_fan(const Dev &d, const V2 *p, int n, V2 center, int layer,
                                int source, const double *split_t,
                                const unsigned char *split_edge, int count) {
  int emitted = 0;
  for (int e = 0, k = 0; e < n; ++e) {
    const V2 a = p[e], dir = p[(e + 1) % n] - a;
    double previous = 0.0;
    V2 cursor = a;
    for (;;) {
      const bool last = !(k < count && split_edge[k] == e);
      const double following = last ? 1.0 : split_t[k++];
      if (following > previous + kEps) {
        const V2 next = a + following * dir;
        if (cross(center, cursor, next) > kEps * kEps) ++emitted;
        cursor = next;
        previous = following;
      }
      if (last) break;
    }
  }
  int slot = reserve(&d.status[kTriangles], emitted);
  if (int64_t(slot) + emitted > d.cap.triangles) {
    set_error(d.status, kErrTriangles);
    return;
  }
  const Plane sc = d.scores[source];
  double w_center[3];
  lift(d, center, sc, w_center);
  for (int e = 0, k = 0; e < n; ++e) {
    const V2 a = p[e], dir = p[(e + 1) % n] - a;
    double previous = 0.0;
    V2 cursor = a;
    double w_cursor[3];
    lift(d, cursor, sc, w_cursor);
    for (;;) {
      const bool last = !(k < count && split_edge[k] == e);
      const double following = last ? 1.0 : split_t[k++];
      if (following > previous + kEps) {
        const V2 next = a + following * dir;
        double w_next[3];
        lift(d, next, sc, w_next);
        if (cross(center, cursor, next) > kEps * kEps) {
          V2 *uv = d.tri_uv + 3 * int64_t(slot);
          double *w = d.tri_world + 9 * int64_t(slot);
          uv[0] = center;
          uv[1] = cursor;
          uv[2] = next;
          for (int c = 0; c < 3; ++c) {
            w[c] = w_center[c];
            w[3 + c] = w_cursor[c];
            w[6 + c] = w_next[c];
          }
          d.tri_src[slot] = source;
          d.tri_layer[slot] = layer;
          ++slot;
        }
        cursor = next;
        for (int c = 0; c < 3; ++c) w_cursor[c] = w_next[c];
        previous = following;
      }
      if (last) break;
    }
  }
}

// Without the point grid (more layers than it has rows for), one thread per
// polygon and one point-hierarchy query each.
__global__ void __launch_bounds__(kBlock, 8) k_mesh_polygons(Dev d, int edge_capacity) {
  if (d.sc[kGridOn] != 0) return;
  const int live = d.sc[kLivePolygons];
  const int leaves = *d.point_tree.size;
  double split_t[kPolygonSplits];
  unsigned char split_edge[kPolygonSplits];
  for (int64_t k = tid(); k < live; k += stride()) {
    if (d.status[kError] != 0) return;
    const int64_t i = d.order[k];
    const V2 *p = d.out_v + int64_t(kMaxVertices) * i;
    const int n = d.out_n[i];
    if (n < 3) continue;
    const int layer = d.out_layer[i], source = d.out_src[i];
    double lx = 1.0e30, ly = 1.0e30, hx = -1.0e30, hy = -1.0e30;
    V2 center = v2(0.0, 0.0);
    for (int j = 0; j < n; ++j) {
      lx = fmin(lx, p[j].x); ly = fmin(ly, p[j].y);
      hx = fmax(hx, p[j].x); hy = fmax(hy, p[j].y);
      center = center + p[j] / double(n);
    }
    const float4 lo = make_float4(__double2float_rd(lx - 2.0e-7), __double2float_rd(ly - 2.0e-7),
                                  float(layer), 0.f);
    const float4 hi = make_float4(__double2float_ru(hx + 2.0e-7), __double2float_ru(hy + 2.0e-7),
                                  float(layer), 0.f);
    int count = 0, per_edge[kMaxVertices];
    for (int e = 0; e < n; ++e) per_edge[e] = 0;
    bool overflow = false;
    // Test one candidate point against every edge: a split point lies on the
    // edge's line within EPS, strictly inside the edge.
    auto node_point = [&](const V2 x) {
      for (int e = 0; e < n; ++e) {
        const V2 a = p[e], b = p[(e + 1) % n];
        // An edge's own end point has parameter 0 or 1 exactly: never a split.
        if (x == a || x == b) continue;
        const V2 dir = b - a;
        const double length2 = dot(dir, dir);
        if (!(length2 > 0.0)) continue;
        // Division-free rejection of points off the edge's line (4x slack over
        // the exact test below, which alone decides).
        const double off = cross(a, b, x);
        if (off * off > 4.0 * kEps * kEps * length2) continue;
        const double tt = dot(x - a, dir) / length2;
        if (tt > kEps && tt < 1.0 - kEps && fabs(cross(a, b, x)) <= kEps * sqrt(length2)) {
          if (++per_edge[e] > edge_capacity || count == kPolygonSplits) {
            overflow = true;
            return;
          }
          split_t[count] = tt;
          split_edge[count] = (unsigned char)e;
          ++count;
        }
      }
    };
    int node = 1;
    while (node > 0 && !overflow) {
      int j;
      node = query_next(d.point_tree, leaves, lo, hi, node, 0, j);
      if (j < 0) break;
      node_point(d.uverts[j]);
    }
    if (overflow) {
      set_error(d.status, kErrEdgeNoding);
      return;
    }
    // Order the split points by (edge, parameter).
    for (int k = 1; k < count; ++k) {
      const double t = split_t[k];
      const unsigned char e = split_edge[k];
      int m = k - 1;
      while (m >= 0 && (split_edge[m] > e || (split_edge[m] == e && split_t[m] > t))) {
        split_t[m + 1] = split_t[m];
        split_edge[m + 1] = split_edge[m];
        --m;
      }
      split_t[m + 1] = t;
      split_edge[m + 1] = e;
    }
    emit_fan(d, p, n, center, layer, source, split_t, split_edge, count);
  }
}

// Noding and emission with the point grid, eight lanes per polygon, four
// polygons per warp in step.  A lane owns a polygon edge.  The rows of grid
// cells meeting the polygon's box grown by 1e-9 hold every same-layer point
// within 1e-10 of its boundary, hence every split point; eight of their points
// are loaded at a time, the box rejects most, and the ones left wait until
// there are eight to test, a point per lane, against every edge.  A lane keeps its
// edge's split points in order, so the fan needs no sort: a lane writes its
// edge's triangles, the lanes' counts are scanned in edge order, and a warp's
// triangles are staged in shared memory and written as one run.
// Polygons of more than eight vertices, with more than Dev::heavy_noding_work
// candidate x edge tests, or with more than kEdgeSplits points on an edge go
// to k_mesh_heavy, a warp each.
//
// Bound by instruction issue (about 10 of a polygon's 55 cell points lie in
// its box).  A thread per polygon ran 4.6 of 32 lanes, which waited for the
// one with the most candidates, and wrote 48- and 72-byte pieces.  Noding and
// emission together: knot-65536 1.36 -> 0.88 ms, its 9,702-face relative 0.55
// -> 0.13, 720K primitives 4.0 -> 3.6, 640-face icospheres 0.12 -> 0.03.
// Testing each near point by all edges at once instead of eight at a time took
// 1.01 ms on the knot.  6 blocks of 80 registers per SM: 4 and 5 hide less
// latency (0.97 and 0.91 ms), 7 spill (1.22).  The line to the warp kernel at
// 1024 tests takes 0.79 ms on the knot and 3.6 on the 720K primitives: 512
// takes 0.86 and 3.9, 2048 takes 0.85 and 3.5.
constexpr int kLanes = 8;
constexpr int kMeshGroups = kBlock / kLanes;
constexpr int kEdgeSplits = 8;
constexpr int kStaged = 32;  // triangles of one warp staged in shared memory
constexpr int kNear = 16;    // points in a polygon's box that wait for their edge tests

struct Staging {
  V2 uv[3 * kStaged];
  double world[9 * kStaged];
  int src[kStaged], layer[kStaged];
};

__global__ void __launch_bounds__(kBlock, 6) k_mesh_groups(Dev d, int edge_capacity) {
  __shared__ V2 s_a[kMeshGroups][kLanes], s_dir[kMeshGroups][kLanes];
  __shared__ double s_slack[kMeshGroups][kLanes];
  __shared__ V2 s_near[kMeshGroups][kNear];
  __shared__ double s_t[kMeshGroups][kLanes][kEdgeSplits];
  __shared__ Staging s_staging[kBlock / 32];
  if (d.sc[kGridOn] == 0) return;
  const Group<kLanes> w;
  const int lane = threadIdx.x & 31, slot = threadIdx.x / kLanes;
  double *split_t = s_t[slot][w.lane];
  const V2 *edge_a = s_a[slot], *edge_dir = s_dir[slot];
  const double *edge_slack = s_slack[slot];
  V2 *waiting = s_near[slot];
  Staging &out = s_staging[threadIdx.x / 32];
  const int live = d.sc[kLivePolygons], g = d.point_grid;
  for (int64_t k0 = tid() >> 5 << 2; k0 < live; k0 += stride() >> 5 << 2) {
    if (__shfl_sync(kFull, *(volatile int *)&d.status[kError], 0) != 0) return;
    const int64_t k = k0 + (lane >> 3);
    const int i = k < live ? d.order[k] : 0;
    int n = k < live ? d.out_n[i] : 0;
    const int layer = d.out_layer[i], source = d.out_src[i];
    if (n < 3) n = 0;
    bool heavy = n > kLanes;
    if (heavy) n = 0;
    const bool mine = w.lane < n;
    const V2 a = mine ? d.out_v[int64_t(kMaxVertices) * i + w.lane] : v2(0.0, 0.0);
    const V2 b = w.shfl(a, w.lane + 1 < n ? w.lane + 1 : 0);
    // Box, and the centroid summed in vertex order.
    double lx = mine ? a.x : 1.0e30, ly = mine ? a.y : 1.0e30;
    double hx = mine ? a.x : -1.0e30, hy = mine ? a.y : -1.0e30;
    for (int off = kLanes / 2; off > 0; off >>= 1) {
      lx = smaller(lx, w.shfl_xor(lx, off));
      ly = smaller(ly, w.shfl_xor(ly, off));
      hx = larger(hx, w.shfl_xor(hx, off));
      hy = larger(hy, w.shfl_xor(hy, off));
    }
    waiting[w.lane] = a / double(n > 0 ? n : 1);
    const V2 dir = b - a;
    const double length2 = dot(dir, dir);
    s_a[slot][w.lane] = a;
    s_dir[slot][w.lane] = dir;
    s_slack[slot][w.lane] = 4.0 * kEps * kEps * length2;
    __syncwarp();
    V2 center = v2(0.0, 0.0);
    for (int j = 0; j < kLanes; ++j)
      if (j < n) center = center + waiting[j];
    __syncwarp();
    const double qlx = lx - 1.0e-9, qly = ly - 1.0e-9, qhx = hx + 1.0e-9, qhy = hy + 1.0e-9;
    const int cx0 = n ? grid_cell(qlx, g) : 0, cx1 = n ? grid_cell(qhx, g) : 0;
    const int cy0 = n ? grid_cell(qly, g) : 0, cy1 = n ? grid_cell(qhy, g) : -1;
    const int most = __reduce_max_sync(kFull, n);
    int count = 0;       // this lane's edge's split points
    bool full = false;   // more than kEdgeSplits of them
    int candidates = 0;  // of the polygon, up to the current rows
    int near_n = 0;      // points waiting
    // Up to eight waiting points of each group, a point per lane: the edges
    // whose line it lies on (4x slack over the exact test) and that it does
    // not end (an edge's own end point has parameter 0 or 1 exactly: never a
    // split).  The few found are then tested by the lanes that own the edges.
    auto node_waiting = [&](bool take) {
      const int points = take ? min(near_n, kLanes) : 0;
      const V2 x = waiting[w.lane];
      unsigned on = 0, end = 0;
      for (int e = 0; e < most; ++e) {
        const V2 u = edge_a[e], dir_e = edge_dir[e], to = x - u;
        const double off = dir_e.x * to.y - dir_e.y * to.x;  // cross(a, b, x)
        on |= unsigned(!(off * off > edge_slack[e])) << e;
        end |= unsigned(x == u) << e;
      }
      if (n > 0) on &= ~(end | end >> 1 | (end & 1u) << (n - 1)) & ((1u << n) - 1u);
      unsigned found = w.ballot(w.lane < points && on != 0);
      while (__any_sync(kFull, found != 0)) {
        const int c = found ? __ffs(int(found)) - 1 : 0;
        const V2 y = w.shfl(x, c);
        const unsigned edges = w.shfl(on, c);
        if (found && (edges >> w.lane & 1u) && length2 > 0.0) {
          const V2 to = y - a;
          const double off = dir.x * to.y - dir.y * to.x;
          const double tt = dot(to, dir) / length2;
          if (tt > kEps && tt < 1.0 - kEps && fabs(off) <= kEps * sqrt(length2)) {
            full = full || count == kEdgeSplits;
            if (!full) {
              int m = count++;
              for (; m > 0 && split_t[m - 1] > tt; --m) split_t[m] = split_t[m - 1];
              split_t[m] = tt;
            }
          }
        }
        found &= found - 1;
      }
      const V2 rest = waiting[kNear - kLanes + w.lane];
      __syncwarp();
      if (take) {
        waiting[w.lane] = rest;
        near_n -= points;
      }
      __syncwarp();
    };
    for (int row0 = cy0; __any_sync(kFull, row0 <= cy1); row0 += kLanes) {
      // Eight rows, one per lane, and the scan of their point counts.
      int begin = 0, points = 0;
      if (row0 + w.lane <= cy1) {
        const int64_t row = (int64_t(layer) * g + row0 + w.lane) * g;
        begin = d.cell_start[row + cx0];
        points = d.cell_start[row + cx1 + 1] - begin;
      }
      int before = points;
      for (int off = 1; off < kLanes; off <<= 1) {
        const int y = __shfl_up_sync(kFull, before, off, kLanes);
        if (w.lane >= off) before += y;
      }
      int total = w.shfl(before, kLanes - 1);
      before -= points;
      candidates += total;
      if (int64_t(candidates) * n > d.heavy_noding_work) heavy = true;
      if (heavy) total = 0;
      for (int t0 = 0; __any_sync(kFull, t0 < total); t0 += kLanes) {
        const int t = t0 + w.lane;
        int r = 0;  // the row that holds the t-th point: the last one that begins at or before t
        for (int off = kLanes / 2; off > 0; off >>= 1)
          if (w.shfl(before, r + off) <= t) r += off;
        const int at = w.shfl(begin, r) + t - w.shfl(before, r);
        V2 x = v2(0.0, 0.0);
        bool near = t < total;
        if (near) {
          x = d.grid_pts[at];
          near = !(x.x < qlx || x.x > qhx || x.y < qly || x.y > qhy);
        }
        const unsigned nears = w.ballot(near);
        if (near) waiting[near_n + __popc(nears & ((1u << w.lane) - 1u))] = x;
        near_n += __popc(nears);
        __syncwarp();
        if (__any_sync(kFull, near_n >= kLanes)) node_waiting(near_n >= kLanes);
      }
    }
    if (__any_sync(kFull, near_n > 0)) node_waiting(true);
    if (w.ballot(full)) heavy = true;
    if (heavy && w.lane == 0) d.heavy_polygons[atomicAdd(&d.sc[kHeavyPolygons], 1)] = i;
    const bool over = !heavy && mine && count > edge_capacity;
    if (__any_sync(kFull, over)) {
      if (over) set_error(d.status, kErrEdgeNoding);
      return;
    }
    // The fan of emit_fan() with a lane per edge.
    const bool active = mine && !heavy;
    int emitted = 0;
    if (active) {
      double previous = 0.0;
      V2 cursor = a;
      for (int m = 0; m <= count; ++m) {
        const double following = m == count ? 1.0 : split_t[m];
        if (following > previous + kEps) {
          const V2 next = a + following * dir;
          if (cross(center, cursor, next) > kEps * kEps) ++emitted;
          cursor = next;
          previous = following;
        }
      }
    }
    int offset = emitted;
    for (int off = 1; off < 32; off <<= 1) {
      const int y = __shfl_up_sync(kFull, offset, off);
      if (lane >= off) offset += y;
    }
    const int total = __shfl_sync(kFull, offset, 31);
    offset -= emitted;
    int base = 0;
    if (lane == 0 && total) base = atomicAdd(&d.status[kTriangles], total);
    base = __shfl_sync(kFull, base, 0);
    if (int64_t(base) + total > d.cap.triangles) {
      if (lane == 0) set_error(d.status, kErrTriangles);
      return;
    }
    const bool staged = total <= kStaged;
    V2 *uvs = staged ? out.uv : d.tri_uv + 3 * int64_t(base);
    double *worlds = staged ? out.world : d.tri_world + 9 * int64_t(base);
    int *srcs = staged ? out.src : d.tri_src + base, *layers = staged ? out.layer : d.tri_layer + base;
    if (active) {
      const Plane sc = d.scores[source];
      double w_center[3], w_cursor[3];
      lift(d, center, sc, w_center);
      lift(d, a, sc, w_cursor);
      double previous = 0.0;
      V2 cursor = a;
      int at = offset;
      for (int m = 0; m <= count; ++m) {
        const double following = m == count ? 1.0 : split_t[m];
        if (following > previous + kEps) {
          const V2 next = a + following * dir;
          double w_next[3];
          lift(d, next, sc, w_next);
          if (cross(center, cursor, next) > kEps * kEps) {
            V2 *uv = uvs + 3 * at;
            double *v = worlds + 9 * at;
            uv[0] = center;
            uv[1] = cursor;
            uv[2] = next;
            for (int c = 0; c < 3; ++c) {
              v[c] = w_center[c];
              v[3 + c] = w_cursor[c];
              v[6 + c] = w_next[c];
            }
            srcs[at] = source;
            layers[at] = layer;
            ++at;
          }
          cursor = next;
          for (int c = 0; c < 3; ++c) w_cursor[c] = w_next[c];
          previous = following;
        }
      }
    }
    __syncwarp();
    if (staged) {
      for (int m = lane; m < 3 * total; m += 32) d.tri_uv[3 * int64_t(base) + m] = out.uv[m];
      for (int m = lane; m < 9 * total; m += 32) d.tri_world[9 * int64_t(base) + m] = out.world[m];
      for (int m = lane; m < total; m += 32) {
        d.tri_src[base + m] = out.src[m];
        d.tri_layer[base + m] = out.layer[m];
      }
    }
    __syncwarp();
  }
}

// One polygon edge as the split-point test uses it, with
// the quantities that test derives from the edge computed once.
struct NodeEdge {
  V2 a, b, dir;
  double length2, slack, tol;
};

constexpr int kHeavyWarps = kBlock / 32;

// Noding and emission of the polygons k_mesh_groups queued as heavy, one
// polygon per warp.  The warp reads the points of 32 grid rows together, 32
// at a time; those in the polygon's box wait until there are 32 to test, a
// point per lane, against every edge with k_mesh_groups' expressions, so the
// split points are the same.  Each split point is placed by its edge and its
// rank along the edge, and the fan is written with a lane per piece of edge.
//
// Bound by instruction issue.  Row by row, with the fan a lane per edge, 11
// of 32 lanes were busy: on the 65,536-face knot (14 thousand polygons) noding
// and emission took 0.91 instead of 0.79 ms, on the 9,702-face knot 0.13
// instead of 0.11, on the 50,000-face overlapping primitives 0.29 instead of
// 0.27; on the 720K primitives it makes no difference.
__global__ void __launch_bounds__(kBlock, 5) k_mesh_heavy(Dev d, int edge_capacity) {
  __shared__ NodeEdge s_edge[kHeavyWarps][kMaxVertices];
  __shared__ double s_t[kHeavyWarps][kPolygonSplits], s_sorted_t[kHeavyWarps][kPolygonSplits];
  __shared__ unsigned char s_e[kHeavyWarps][kPolygonSplits];
  __shared__ V2 s_near[kHeavyWarps][64];
  __shared__ int s_count[kHeavyWarps], s_per_edge[kHeavyWarps][kMaxVertices];
  constexpr unsigned kFull = 0xffffffffu;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int heavy = d.sc[kHeavyPolygons];
  if (tid() == 0) d.metrics[kHeavyNodedPolygons] = heavy;
  const int g = d.point_grid;
  NodeEdge *edges = s_edge[warp];
  V2 *waiting = s_near[warp];
  int *per_edge = s_per_edge[warp];
  double *split_t = s_t[warp], *sorted_t = s_sorted_t[warp];
  unsigned char *split_edge = s_e[warp];
  for (int64_t h = tid() >> 5; h < heavy; h += stride() >> 5) {
    int failed = 0;
    if (lane == 0) failed = *(volatile int *)&d.status[kError];
    if (__shfl_sync(kFull, failed, 0) != 0) return;
    const int i = d.heavy_polygons[h];
    const V2 *p = d.out_v + int64_t(kMaxVertices) * i;
    const int n = d.out_n[i];
    const int layer = d.out_layer[i], source = d.out_src[i];
    // Box, and the centroid summed in vertex order.
    const V2 own = lane < n ? p[lane] : v2(0.0, 0.0);
    double lx = lane < n ? own.x : 1.0e30, ly = lane < n ? own.y : 1.0e30;
    double hx = lane < n ? own.x : -1.0e30, hy = lane < n ? own.y : -1.0e30;
    for (int off = 16; off > 0; off >>= 1) {
      lx = smaller(lx, __shfl_xor_sync(kFull, lx, off));
      ly = smaller(ly, __shfl_xor_sync(kFull, ly, off));
      hx = larger(hx, __shfl_xor_sync(kFull, hx, off));
      hy = larger(hy, __shfl_xor_sync(kFull, hy, off));
    }
    waiting[lane] = own / double(n);
    if (lane < n) {
      NodeEdge e;
      e.a = own;
      e.b = p[(lane + 1) % n];
      e.dir = e.b - e.a;
      e.length2 = dot(e.dir, e.dir);
      e.slack = 4.0 * kEps * kEps * e.length2;
      e.tol = kEps * sqrt(e.length2);
      edges[lane] = e;
      per_edge[lane] = 0;
    }
    if (lane == 0) s_count[warp] = 0;
    __syncwarp();
    V2 center = v2(0.0, 0.0);
    for (int j = 0; j < n; ++j) center = center + waiting[j];
    __syncwarp();
    const double qlx = lx - 1.0e-9, qly = ly - 1.0e-9, qhx = hx + 1.0e-9, qhy = hy + 1.0e-9;
    const int cx0 = grid_cell(qlx, g), cx1 = grid_cell(qhx, g);
    const int cy0 = grid_cell(qly, g), cy1 = grid_cell(qhy, g);
    int near_n = 0;
    for (int row0 = cy0; row0 <= cy1; row0 += 32) {
      const bool last_rows = row0 + 32 > cy1;
      // 32 rows, one per lane, and the scan of their point counts.
      int begin = 0, points = 0;
      if (row0 + lane <= cy1) {
        const int64_t row = (int64_t(layer) * g + row0 + lane) * g;
        begin = d.cell_start[row + cx0];
        points = d.cell_start[row + cx1 + 1] - begin;
      }
      int before = points;
      for (int off = 1; off < 32; off <<= 1) {
        const int y = __shfl_up_sync(kFull, before, off);
        if (lane >= off) before += y;
      }
      const int total = __shfl_sync(kFull, before, 31);
      before -= points;
      int t0 = 0;
      do {
        const int t = t0 + lane;
        int r = 0;  // the row that holds the t-th point: the last one that begins at or before t
        for (int off = 16; off > 0; off >>= 1)
          if (__shfl_sync(kFull, before, r + off) <= t) r += off;
        const int at = __shfl_sync(kFull, begin, r) + t - __shfl_sync(kFull, before, r);
        V2 y = v2(0.0, 0.0);
        bool near = t < total;
        if (near) {
          y = d.grid_pts[at];
          near = !(y.x < qlx || y.x > qhx || y.y < qly || y.y > qhy);
        }
        const unsigned nears = __ballot_sync(kFull, near);
        if (near) waiting[near_n + __popc(nears & ((1u << lane) - 1u))] = y;
        near_n += __popc(nears);
        t0 += 32;
        __syncwarp();
        // 32 waiting points at a time, a point per lane, against every edge.
        const int need = last_rows && t0 >= total ? 1 : 32;
        while (near_n >= need) {
          const V2 x = waiting[lane];
          if (lane < near_n) {
            for (int e = 0; e < n; ++e) {
              const NodeEdge &E = edges[e];
              const double off = cross(E.a, E.b, x);
              if (off * off > E.slack) continue;
              if (x == E.a || x == E.b) continue;
              if (!(E.length2 > 0.0)) continue;
              const double tt = dot(x - E.a, E.dir) / E.length2;
              if (tt > kEps && tt < 1.0 - kEps && fabs(off) <= E.tol) {
                const int place = atomicAdd(&s_count[warp], 1);
                atomicAdd(&per_edge[e], 1);
                if (place < kPolygonSplits) {
                  split_t[place] = tt;
                  split_edge[place] = (unsigned char)e;
                }
              }
            }
          }
          const V2 rest = waiting[32 + lane];
          __syncwarp();
          waiting[lane] = rest;
          near_n = max(near_n - 32, 0);
          __syncwarp();
        }
      } while (t0 < total);
    }
    __syncwarp();
    // The thread kernel's overflow rule on the totals: more split points
    // than the buffer, or more on one edge than edge_capacity.
    const int count = s_count[warp];
    if (__any_sync(kFull, lane < n && per_edge[lane] > edge_capacity) || count > kPolygonSplits) {
      if (lane == 0) set_error(d.status, kErrEdgeNoding);
      return;
    }
    // Edge e's split points take places [first_e, first_e + count_e) of the
    // order by (edge, parameter): an exclusive scan of the per-edge counts.
    const int mine = lane < n ? per_edge[lane] : 0;
    int first = mine;
    for (int off = 1; off < 32; off <<= 1) {
      const int y = __shfl_up_sync(kFull, first, off);
      if (lane >= off) first += y;
    }
    first -= mine;
    __syncwarp();
    if (lane < n) per_edge[lane] = first;
    __syncwarp();
    // A split point's place: its edge's first place plus its rank among the
    // edge's points by parameter, ties by arrival (equal parameters give the
    // same triangles in either order).
    for (int k = lane; k < count; k += 32) {
      const double t = split_t[k];
      const int e = split_edge[k];
      int rank = per_edge[e];
      for (int m = 0; m < count; ++m) {
        const double tm = split_t[m];
        rank += (split_edge[m] == e && (tm < t || (tm == t && m < k))) ? 1 : 0;
      }
      sorted_t[rank] = t;
    }
    __syncwarp();
    // The fan of emit_fan(): a lane per edge keeps the split points that are
    // more than kEps past the one before, then a lane per piece of edge emits
    // its triangle, in the same order.
    int kept = 0;
    bool ends = false;
    if (lane < n) {
      double previous = 0.0;
      for (int k = 0; k < mine; ++k) {
        const double t = sorted_t[first + k];
        if (t > previous + kEps) {
          sorted_t[first + kept++] = t;
          previous = t;
        }
      }
      ends = 1.0 > previous + kEps;
    }
    const int pieces = kept + int(ends);
    int before = pieces;
    for (int off = 1; off < 32; off <<= 1) {
      const int y = __shfl_up_sync(kFull, before, off);
      if (lane >= off) before += y;
    }
    const int all = __shfl_sync(kFull, before, 31);
    before -= pieces;
    __syncwarp();
    // Piece s runs from `from` to `to`; `fan` says whether it has a triangle.
    V2 from = center, to = center;
    auto piece = [&](int s) {
      int e = 0;  // its edge: the last one that begins at or before s
      for (int off = 16; off > 0; off >>= 1)
        if (__shfl_sync(kFull, before, e + off) <= s) e += off;
      const int j = s - __shfl_sync(kFull, before, e), points = __shfl_sync(kFull, kept, e);
      const double *t = sorted_t + __shfl_sync(kFull, first, e);
      if (s >= all) return false;
      const V2 start = edges[e].a, dir = edges[e].dir;
      from = j == 0 ? start : start + t[j - 1] * dir;
      to = start + (j == points ? 1.0 : t[j]) * dir;
      return cross(center, from, to) > kEps * kEps;
    };
    int total = 0;
    for (int s0 = 0; s0 < all; s0 += 32) total += __popc(__ballot_sync(kFull, piece(s0 + lane)));
    int base = 0;
    if (lane == 0 && total) base = atomicAdd(&d.status[kTriangles], total);
    base = __shfl_sync(kFull, base, 0);
    if (int64_t(base) + total > d.cap.triangles) {
      if (lane == 0) set_error(d.status, kErrTriangles);
      __syncwarp();
      continue;
    }
    const Plane sc = d.scores[source];
    double w_center[3];
    lift(d, center, sc, w_center);
    for (int s0 = 0; s0 < all; s0 += 32) {
      const bool fan = piece(s0 + lane);
      const unsigned fans = __ballot_sync(kFull, fan);
      if (fan) {
        const int64_t at = base + __popc(fans & ((1u << lane) - 1u));
        double w_from[3], w_to[3];
        lift(d, from, sc, w_from);
        lift(d, to, sc, w_to);
        V2 *uv = d.tri_uv + 3 * at;
        double *w = d.tri_world + 9 * at;
        uv[0] = center;
        uv[1] = from;
        uv[2] = to;
        for (int c = 0; c < 3; ++c) {
          w[c] = w_center[c];
          w[3 + c] = w_from[c];
          w[6 + c] = w_to[c];
        }
        d.tri_src[at] = source;
        d.tri_layer[at] = layer;
      }
      base += __popc(fans);
    }
    __syncwarp();
  }
}
unsigned blocks(int64_t n) {
  int64_t g = ceil_div(n > 0 ? n : 1, kBlock);
  return unsigned(g < 148 * 16 ? g : 148 * 16);
}

}  // namespace

cudaError_t order_polygons(const Dev &d, bool layered, SortScratch &s, cudaStream_t st) {
  const int64_t R = d.cap.regions;
  k_order_count<<<blocks(R), kBlock, 0, st>>>(d, layered ? 1 : 0);
  note_launch();
  EDP_CHECK(scan_exclusive(d.order_count, d.order_start, d.sc + kOrderLive,
                           int64_t(1) << d.order_bits, nullptr, s, st, true));
  k_order_place<<<blocks(R), kBlock, 0, st>>>(d, layered ? 1 : 0);
  note_launch();
  return cudaGetLastError();
}

cudaError_t sort_polygons(const Dev &d, SortScratch &s, cudaStream_t st) {
  const int64_t R = d.cap.regions;
  k_order_keys<<<blocks(R), kBlock, 0, st>>>(d);
  note_launch();
  return sort_pairs_u64(d.order_keys, d.order_keys_tmp, d.order, d.order_tmp,
                        d.sc + kLivePolygons, R, 24, s, st);
}

cudaError_t stage_mesh_index(const Dev &d, SortScratch &s, TreeBuffers &point_tree,
                             cudaStream_t st) {
  const int64_t R = d.cap.regions, E = d.cap.vertices;
  EDP_CHECK(order_polygons(d, true, s, st));
  EDP_CHECK(scan_exclusive(d.counts, d.offsets, d.sc + kLivePolygons, R, d.sc + kLiveVertices, s, st));
  const int64_t cells = int64_t(d.grid_layers) * d.point_grid * d.point_grid;
  k_scatter<<<blocks(R), kBlock, 0, st>>>(d);
  note_launch();
  k_unique_points<<<blocks(E), kBlock, 0, st>>>(d);
  note_launch();
  EDP_CHECK(stage_mark(EDP_STAGE_MESH_VERTICES, st));
  EDP_CHECK(scan_exclusive(d.cell_count, d.cell_start, d.sc + kGridCells, cells, nullptr, s, st));
  // The point hierarchy sits in a conditional IF node of a captured graph (run
  // eagerly, it takes its count, zero with the grid, from the device).
  cudaGraphConditionalHandle handle{};
  const bool branch = d.use_handle && d.aux_stream;
  if (branch) EDP_CHECK(conditional_handle(st, handle));
  k_grid_scatter<<<blocks(E), kBlock, 0, st>>>(d, handle, branch ? 1 : 0);
  note_launch();
  if (branch) {
    EDP_CHECK(conditional_begin(st, handle, d.aux_stream));
    const int64_t first = launch_count();
    cudaError_t built = tree_build(point_tree, d.pt_lo, d.pt_hi, d.sc + kTreePoints, 0, true, s,
                                   d.aux_stream);
    EDP_CHECK(conditional_end(d.aux_stream));
    EDP_CHECK(built);
    forget_launches(launch_count() - first);
  } else {
    EDP_CHECK(tree_build(point_tree, d.pt_lo, d.pt_hi, d.sc + kTreePoints, 0, true, s, st));
  }
  EDP_CHECK(stage_mark(EDP_STAGE_MESH_INDEX, st));
  return cudaGetLastError();
}

cudaError_t stage_mesh_emit(const Dev &d, cudaStream_t st) {
  int cap = int(d.cap.edge_vertices < kMaxEdgeVertices ? d.cap.edge_vertices : kMaxEdgeVertices);
  k_mesh_groups<<<unsigned(std::min<int64_t>(ceil_div(d.cap.regions, kMeshGroups), 148 * 6)),
                  kBlock, 0, st>>>(d, cap);
  note_launch();
  k_mesh_polygons<<<blocks(d.cap.regions), kBlock, 0, st>>>(d, cap);
  note_launch();
  k_mesh_heavy<<<148 * 5, kBlock, 0, st>>>(d, cap);
  note_launch();
  EDP_CHECK(stage_mark(EDP_STAGE_MESH_EMIT, st));
  return cudaGetLastError();
}

}  // namespace edp
