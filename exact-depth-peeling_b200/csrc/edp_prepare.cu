// Preparation stage: validation, welding, projection, mesh contours, contour
// segments and the source / segment hierarchies
// (warp_peel/solver.py:217-321, warp_peel/events.py:148-220).
#include "edp_internal.h"

namespace edp {
namespace {

constexpr int kBlock = 128;

__device__ inline int64_t tid() { return blockIdx.x * int64_t(blockDim.x) + threadIdx.x; }
__device__ inline int64_t stride() { return int64_t(gridDim.x) * blockDim.x; }

// Tables to fill with one 32-bit word each, 16 bytes at a time.
struct FillList {
  static constexpr int kMost = 12;
  uint4 *at[kMost];
  int64_t quads[kMost];
  unsigned word[kMost];
  int count = 0;
  template <class T>
  void add(T *p, int64_t elements, unsigned value) {  // alloc() pads to 16 bytes
    at[count] = reinterpret_cast<uint4 *>(p);
    quads[count] = ceil_div(elements * int64_t(sizeof(T)), 16);
    word[count++] = value;
  }
};

// Counters and the tables that the preparation fills, in one launch.
__global__ void k_reset(Dev d, FillList fills) {
  const int i = int(tid());
  if (i < kStatusSlots) d.status[i] = 0;
  if (i < kMetrics) d.metrics[i] = 0;
  if (i < kPredCounters) d.pred_counts[i] = 0;
  if (i < kScalarCount)
    d.sc[i] = i == kSourceCount    ? d.n
              : i == kSegmentSlots ? kSourceVertices * d.n
              : i == kRayGridCells ? d.grid_size * d.grid_size
                                   : 0;
  if (i == 0) {
    *d.parity = 0;
    *d.condition = 0;
  }
  for (int f = 0; f < fills.count; ++f)
    fill_words(fills.at[f], fills.quads[f], fills.word[f], tid(), stride());
}

__device__ inline double det4(const double *m) {
  // Laplace expansion along the first row of a row-major 4x4 matrix.
  double s0 = m[10] * m[15] - m[11] * m[14], s1 = m[9] * m[15] - m[11] * m[13];
  double s2 = m[9] * m[14] - m[10] * m[13], s3 = m[8] * m[15] - m[11] * m[12];
  double s4 = m[8] * m[14] - m[10] * m[12], s5 = m[8] * m[13] - m[9] * m[12];
  double c0 = m[5] * s0 - m[6] * s1 + m[7] * s2;
  double c1 = m[4] * s0 - m[6] * s3 + m[7] * s4;
  double c2 = m[4] * s1 - m[5] * s3 + m[7] * s5;
  double c3 = m[4] * s2 - m[5] * s4 + m[6] * s5;
  return m[0] * c0 - m[1] * c1 + m[2] * c2 - m[3] * c3;
}

// Exact-position welding: the canonical id of a vertex is the smallest index
// with an equal position, signed zeros equal (kernels.py:269-306).  The
// reference sorts positions; an open-addressing table gives the same ids.
__device__ inline uint64_t position_hash(const double *v) {
  uint64_t h = mix64(key_bits(v[0]));
  h = mix64(h ^ key_bits(v[1]));
  return mix64(h ^ key_bits(v[2]));
}

__device__ inline void weld_insert(const Dev &d) {
  for (int64_t i = tid(); i < d.nv; i += stride()) {
    const double *v = d.vertices + 3 * i;
    uint32_t slot = uint32_t(position_hash(v)) & uint32_t(d.weld_mask);
    for (int probe = 0; probe <= d.weld_mask; ++probe) {
      int cur = atomicCAS(&d.weld_table[slot], -1, int(i));
      if (cur == -1) break;
      const double *w = d.vertices + 3 * int64_t(cur);
      if (w[0] == v[0] && w[1] == v[1] && w[2] == v[2]) break;
      slot = (slot + 1) & uint32_t(d.weld_mask);
    }
    atomicMin(&d.weld_min[slot], int(i));
    d.weld_slot[i] = int(slot);
  }
}

// The weld table, and input validation (kernels.py:309-350): finite values, face indices in
// range, an invertible affine camera and a valid window and near plane.
__global__ void k_validate(Dev d) {
  weld_insert(d);
  for (int64_t i = tid(); i < max(max(d.nv, d.n), 1); i += stride()) {
    if (i < d.nv) {
      for (int j = 0; j < 3; ++j)
        if (!isfinite(d.vertices[3 * i + j])) set_error(d.status, kErrInput);
    }
    if (i < d.n) {
      for (int j = 0; j < 3; ++j) {
        int f = d.faces[3 * i + j];
        if (f < 0 || f >= d.nv) set_error(d.status, kErrInput);
      }
    }
    if (i == 0) {
      const double *m = d.camera;
      bool bad = false;
      for (int k = 0; k < 16; ++k) bad |= !isfinite(m[k]);
      for (int k = 0; k < 6; ++k) bad |= !isfinite(d.settings[k]);
      bad |= det4(m) == 0.0 || m[12] != 0.0 || m[13] != 0.0 || m[14] != 0.0 || m[15] != 1.0;
      const double *s = d.settings;
      bad |= s[2] <= s[0] || s[3] <= s[1] || s[5] <= 0.0 || (s[4] != 0.0 && s[4] != 1.0);
      if (bad) set_error(d.status, kErrInput);
      // Inverse camera by Gauss-Jordan elimination with partial pivoting.
      double a[4][8];
      for (int r = 0; r < 4; ++r)
        for (int c = 0; c < 8; ++c) a[r][c] = c < 4 ? m[4 * r + c] : double(c - 4 == r);
      for (int k = 0; k < 4; ++k) {
        int p = k;
        for (int r = k + 1; r < 4; ++r)
          if (fabs(a[r][k]) > fabs(a[p][k])) p = r;
        for (int c = 0; c < 8; ++c) {
          double t = a[k][c]; a[k][c] = a[p][c]; a[p][c] = t;
        }
        double piv = a[k][k];
        if (piv == 0.0) piv = 1.0;  // singular input is already flagged
        for (int c = 0; c < 8; ++c) a[k][c] /= piv;
        for (int r = 0; r < 4; ++r)
          if (r != k) {
            double f = a[r][k];
            for (int c = 0; c < 8; ++c) a[r][c] -= f * a[k][c];
          }
      }
      for (int r = 0; r < 4; ++r)
        for (int c = 0; c < 4; ++c) d.inverse[4 * r + c] = a[r][c + 4];
    }
  }
}

// Camera transform, near clip, projection, depth plane, facing and window
// clip of one triangle (kernels.py:353-468), after the vertices' canonical ids.
__global__ void k_project(Dev d) {
  for (int64_t i = tid(); i < d.nv; i += stride()) d.canonical[i] = d.weld_min[d.weld_slot[i]];
  for (int64_t i = tid(); i < d.n; i += stride()) {
    V2 *out = d.src_v + kSourceVertices * i;
    if (d.status[kError] != 0) {
      d.src_n[i] = 0;
      d.src_lo[i] = empty_lo();
      d.src_hi[i] = empty_hi();
      d.scores[i] = Plane{0, 0, 0, 0};
      d.facing[i] = 0;
      d.clipped[i] = 0;
      continue;
    }
    const double *m = d.camera, *s = d.settings;
    double r[kSourceVertices][3];
    int count = 3;
    for (int j = 0; j < 3; ++j) {
      const double *w = d.vertices + 3 * int64_t(d.faces[3 * i + j]);
      for (int k = 0; k < 3; ++k)
        r[j][k] = m[4 * k] * w[0] + m[4 * k + 1] * w[1] + m[4 * k + 2] * w[2] + m[4 * k + 3];
      if (!isfinite(r[j][0]) || !isfinite(r[j][1]) || !isfinite(r[j][2]))
        set_error(d.status, kErrInput);
    }
    int was_clipped = 0;
    const bool persp = s[4] != 0.0;
    if (persp) {
      double ring[kSourceVertices][3];
      int c = 0;
      for (int j = 0; j < 3; ++j) {
        const double *a = r[j], *b = r[(j + 1) % 3];
        double da = a[2] - s[5], db = b[2] - s[5];
        if (da >= 0.0) {
          for (int k = 0; k < 3; ++k) ring[c][k] = a[k];
          ++c;
        } else {
          was_clipped = 1;
        }
        if ((da > 0.0 && db < 0.0) || (da < 0.0 && db > 0.0)) {
          double t = da / (da - db);
          for (int k = 0; k < 3; ++k) ring[c][k] = a[k] + t * (b[k] - a[k]);
          ++c;
        }
      }
      for (int j = 0; j < c; ++j)
        for (int k = 0; k < 3; ++k) r[j][k] = ring[j][k];
      count = c;
    }
    V2 p[kMaxVertices];
    double depth[kSourceVertices];
    int n = 0;
    for (int j = 0; j < count; ++j) {
      double invz = persp ? 1.0 / r[j][2] : 1.0;
      V2 x = v2((r[j][0] * invz - s[0]) / (s[2] - s[0]), (r[j][1] * invz - s[1]) / (s[3] - s[1]));
      n = append(p, n, x);
      depth[j] = persp ? -invz : r[j][2];
      if (x.x < 0.0 || x.x > 1.0 || x.y < 0.0 || x.y > 1.0) was_clipped = 1;
    }
    Plane score{0, 0, 0, 0};
    double det = 0.0;
    int index = 2;
    if (count >= 3) {
      for (int j = 2; j < count; ++j) {
        det = cross(p[0], p[1], p[j]);
        if (det != 0.0) {
          index = j;
          break;
        }
      }
    }
    int face = 0;
    if (det != 0.0) {
      V2 pa = p[1] - p[0], pb = p[index] - p[0];
      double s0 = ((depth[1] - depth[0]) * pb.y - (depth[index] - depth[0]) * pa.y) / det;
      double s1 = (pa.x * (depth[index] - depth[0]) - pb.x * (depth[1] - depth[0])) / det;
      score = Plane{s0, s1, depth[0] - s0 * p[0].x - s1 * p[0].y, 0.0};
      face = 1;
      if (det < 0.0) {
        face = -1;
        for (int j = 0; j < n / 2; ++j) {
          V2 t = p[j]; p[j] = p[n - 1 - j]; p[n - 1 - j] = t;
        }
      }
      const Plane window[4] = {{1.0, 0.0, 0.0, 0}, {-1.0, 0.0, 1.0, 0}, {0.0, 1.0, 0.0, 0},
                               {0.0, -1.0, 1.0, 0}};
      V2 q[kMaxVertices], rest[kMaxVertices];
      for (int w = 0; w < 4; ++w) {
        int nq, nr;
        split_at(p, n, window[w], v2(0.0, 0.0), q, nq, rest, nr);
        n = nq;
        for (int j = 0; j < n && j < kMaxVertices; ++j) p[j] = q[j];
      }
    } else {
      n = 0;
    }
    if (!isfinite(score.a) || !isfinite(score.b) || !isfinite(score.c) ||
        fabs(score.a) > 1.0e28 || fabs(score.b) > 1.0e28 || fabs(score.c) > 1.0e28)
      set_error(d.status, kErrInput);
    if (n > kSourceVertices) {
      set_error(d.status, kErrPolygon);
      n = 0;
    }
    for (int j = 0; j < n; ++j) out[j] = p[j];
    d.src_n[i] = n;
    d.scores[i] = score;
    d.facing[i] = face;
    d.clipped[i] = was_clipped;
    float4 lo, hi;
    polygon_bounds(p, n, score, lo, hi);
    d.src_lo[i] = lo;
    d.src_hi[i] = hi;
  }
}

// Undirected welded edge keys, grouped in an open-addressing table; the
// reference sorts them (kernels.py:471-492).
__global__ void k_edge_insert(Dev d) {
  for (int64_t e = tid(); e < 3 * int64_t(d.n); e += stride()) {
    d.masks[e] = 0;
    if (d.status[kError] != 0) {
      d.edge_slot[e] = -1;
      continue;
    }
    int64_t f = e / 3;
    int j = int(e % 3);
    int a = d.canonical[d.faces[3 * f + j]], b = d.canonical[d.faces[3 * f + (j + 1) % 3]];
    unsigned long long key =
        (static_cast<unsigned long long>(min(a, b)) << 32) | static_cast<unsigned>(max(a, b));
    d.edge_keys[e] = key;
    uint32_t slot = uint32_t(mix64(key)) & uint32_t(d.ekey_mask);
    for (int probe = 0; probe <= d.ekey_mask; ++probe) {
      unsigned long long cur = atomicCAS(&d.ekey_table[slot], ~0ull, key);
      if (cur == ~0ull || cur == key) break;
      slot = (slot + 1) & uint32_t(d.ekey_mask);
    }
    int k = atomicAdd(&d.ekey_count[slot], 1);
    if (k < 2) d.ekey_member[2 * slot + k] = int(e);
    d.edge_slot[e] = int(slot);
  }
}

// Contour = not exactly two oppositely directed incidences with the same
// facing: boundary, silhouette, non-manifold or inconsistent (kernels.py:495-520).
__global__ void k_edge_mark(Dev d) {
  for (int64_t e = tid(); e < 3 * int64_t(d.n); e += stride()) {
    int slot = d.edge_slot[e];
    if (slot < 0) continue;
    bool contour = true;
    if (d.ekey_count[slot] == 2) {
      int e0 = d.ekey_member[2 * slot], e1 = d.ekey_member[2 * slot + 1];
      int a = d.canonical[d.faces[3 * (e0 / 3) + e0 % 3]];
      int b = d.canonical[d.faces[3 * (e1 / 3) + e1 % 3]];
      if (a != b && d.facing[e0 / 3] == d.facing[e1 / 3]) contour = false;
    }
    d.masks[e] = contour ? 1 : 0;
  }
}

// Up to eight canonical contour segments per source with endpoint depths,
// deduplicated exactly; each group keeps its per-endpoint minimum depth
// (event_kernels.py:388-480).  Grouping uses a table instead of four sorts.
__global__ void k_segments(Dev d) {
  const int64_t total = int64_t(kSourceVertices) * d.n;
  for (int64_t i = tid(); i < total; i += stride()) {
    int64_t source = i / kSourceVertices;
    int edge = int(i % kSourceVertices);
    V2 a = v2(1.0e30, 1.0e30), b = a;
    double za = 1.0e30, zb = 1.0e30;
    d.seg_slot[i] = -1;
    int n = d.src_n[source];
    if (d.status[kError] == 0 && edge < n && contour_edge(d, source, edge)) {
      const V2 *p = d.src_v + kSourceVertices * source;
      a = p[edge];
      b = p[(edge + 1) % n];
      if (less(b, a)) {
        V2 t = a; a = b; b = t;
      }
      Plane sc = d.scores[source];
      za = value(sc, a);
      zb = value(sc, b);
      // Publish the endpoints before the slot can be seen by other threads.
      d.slot_a[i] = a;
      d.slot_b[i] = b;
      __threadfence();
      uint64_t h = mix64(key_bits(a.x));
      h = mix64(h ^ key_bits(a.y));
      h = mix64(h ^ key_bits(b.x));
      h = mix64(h ^ key_bits(b.y));
      uint32_t slot = uint32_t(h) & uint32_t(d.seg_mask);
      for (int probe = 0; probe <= d.seg_mask; ++probe) {
        int cur = atomicCAS(&d.seg_table[slot], -1, int(i));
        if (cur == -1) break;
        V2 ca = v2(__ldcg(&d.slot_a[cur].x), __ldcg(&d.slot_a[cur].y));
        V2 cb = v2(__ldcg(&d.slot_b[cur].x), __ldcg(&d.slot_b[cur].y));
        if (ca == a && cb == b) break;
        slot = (slot + 1) & uint32_t(d.seg_mask);
      }
      atomicMin(&d.seg_min[slot], int(i));
      atomic_min_double(&d.seg_za[slot], za);
      atomic_min_double(&d.seg_zb[slot], zb);
      d.seg_slot[i] = int(slot);
    } else {
      d.slot_a[i] = a;
      d.slot_b[i] = b;
    }
  }
}

// The first slot of each group represents it (event_kernels.py:440-501).
// Each member whose endpoint depth is the group's minimum offers its source,
// the smallest of which the exact depth tests evaluate.
__global__ void k_segment_flags(Dev d) {
  const int64_t total = int64_t(kSourceVertices) * d.n;
  for (int64_t i = tid(); i < total; i += stride()) {
    const int slot = d.seg_slot[i];
    if (slot >= 0) {
      const int source = int(i / kSourceVertices);
      const Plane sc = d.scores[source];
      if (value(sc, d.slot_a[i]) == d.seg_za[slot]) atomicMin(&d.seg_srca[slot], source);
      if (value(sc, d.slot_b[i]) == d.seg_zb[slot]) atomicMin(&d.seg_srcb[slot], source);
    }
    const bool first = slot >= 0 && d.seg_min[slot] == int(i);
    d.seg_flag[i] = first ? 1 : 0;
    count_add(&d.metrics[kUniqueContours], first ? 1 : 0);
  }
}

// Representatives, compacted in slot order (seg_pos is the scan of seg_flag),
// with their near depths and padded boxes.
__global__ void k_segment_compact(Dev d) {
  const int64_t total = int64_t(kSourceVertices) * d.n;
  for (int64_t i = tid(); i < total; i += stride()) {
    if (!d.seg_flag[i]) continue;
    const int c = d.seg_pos[i], slot = d.seg_slot[i];
    const V2 a = d.slot_a[i], b = d.slot_b[i];
    const double za = d.seg_za[slot], zb = d.seg_zb[slot];
    const double pz = 2.0e-7 * fmax(1.0, fmax(fabs(za), fabs(zb)));
    d.seg_a[c] = a;
    d.seg_b[c] = b;
    d.seg_near[c] = v2(za, zb);
    // Every group has a member attaining each minimum (the same binary64
    // expression is evaluated again); the representative's own source
    // stands in should none have been recorded.
    const int own = int(i / kSourceVertices);
    int2 near_src = make_int2(d.seg_srca[slot], d.seg_srcb[slot]);
    if (near_src.x < 0 || near_src.x >= d.n) near_src.x = own;
    if (near_src.y < 0 || near_src.y >= d.n) near_src.y = own;
    d.seg_near_src[c] = near_src;
    const Plane pa = d.scores[near_src.x], pb = d.scores[near_src.y];
    d.seg_near_mag[c] = v2(fabs(pa.a * a.x) + fabs(pa.b * a.y) + fabs(pa.c),
                           fabs(pb.a * b.x) + fabs(pb.b * b.y) + fabs(pb.c));
    // The welded mesh vertex at each end: the representative's polygon is its
    // triangle's projection (unclipped; reversed when back-facing), so its
    // vertex j is the face's vertex j, or 2 - j.
    int2 vid = make_int2(-1, -1);
    if (!d.clipped[own] && d.src_n[own] == 3) {
      const V2 *p = d.src_v + int64_t(kSourceVertices) * own;
      for (int j = 0; j < 3; ++j) {
        const int v = d.canonical[d.faces[3 * int64_t(own) + (d.facing[own] < 0 ? 2 - j : j)]];
        if (p[j] == a) vid.x = v;
        if (p[j] == b) vid.y = v;
      }
    }
    d.seg_vid[c] = vid;
    d.seg_lo[c] = make_float4(float(fmin(a.x, b.x) - 2.0e-7), float(fmin(a.y, b.y) - 2.0e-7),
                              float(fmin(za, zb) - pz), 0.f);
    d.seg_hi[c] = make_float4(float(fmax(a.x, b.x) + 2.0e-7), float(fmax(a.y, b.y) + 2.0e-7),
                              float(fmax(za, zb) + pz), 0.f);
  }
}

unsigned blocks(int64_t n) {
  int64_t g = ceil_div(n > 0 ? n : 1, kBlock);
  return unsigned(g < 148 * 16 ? g : 148 * 16);
}

}  // namespace

cudaError_t stage_prepare_common(const Dev &d, bool event, cudaStream_t st) {
  FillList fills;
  fills.add(d.weld_table, int64_t(d.weld_mask) + 1, 0xffffffffu);
  fills.add(d.weld_min, int64_t(d.weld_mask) + 1, 0x7f7f7f7fu);
  fills.add(d.ekey_table, int64_t(d.ekey_mask) + 1, 0xffffffffu);
  fills.add(d.ekey_count, int64_t(d.ekey_mask) + 1, 0u);
  if (event) {
    const int64_t slots = int64_t(d.seg_mask) + 1;
    fills.add(d.seg_table, slots, 0xffffffffu);
    fills.add(d.seg_min, slots, 0x7f7f7f7fu);
    // 0x7f bytes are 1.38e306 as binary64: above every finite depth we store.
    fills.add(d.seg_za, slots, 0x7f7f7f7fu);
    fills.add(d.seg_zb, slots, 0x7f7f7f7fu);
    fills.add(d.seg_srca, slots, 0x7f7f7f7fu);
    fills.add(d.seg_srcb, slots, 0x7f7f7f7fu);
  }
  k_reset<<<148 * 4, 256, 0, st>>>(d, fills);
  note_launch();
  k_validate<<<blocks(std::max(d.nv, d.n)), kBlock, 0, st>>>(d);
  note_launch();
  if (d.nv > 0 || d.n > 0) {
    k_project<<<blocks(std::max(d.nv, d.n)), kBlock, 0, st>>>(d);
    note_launch();
  }
  if (d.n > 0) {
    k_edge_insert<<<blocks(3 * int64_t(d.n)), kBlock, 0, st>>>(d);
    note_launch();
    k_edge_mark<<<blocks(3 * int64_t(d.n)), kBlock, 0, st>>>(d);
    note_launch();
  }
  return cudaGetLastError();
}

// The stream of the side branch, which waits for what `st` has recorded.
static cudaError_t side_fork(const Dev &d, Side &side, cudaStream_t st, cudaStream_t &on) {
  on = st;
  if (!d.use_side) return cudaSuccess;
  EDP_CHECK(cudaEventRecord(side.forked, st));
  EDP_CHECK(cudaStreamWaitEvent(side.stream, side.forked, 0));
  on = side.stream;
  return cudaSuccess;
}

cudaError_t side_join(const Dev &d, Side &side, cudaStream_t st) {
  if (!d.use_side) return cudaSuccess;
  EDP_CHECK(cudaEventRecord(side.joined, side.stream));
  return cudaStreamWaitEvent(st, side.joined, 0);
}

cudaError_t stage_prepare(const Dev &d, SortScratch &s, TreeBuffers &source_tree,
                          TreeBuffers &seg_tree, Side &side, cudaStream_t st) {
  EDP_CHECK(stage_prepare_common(d, true, st));
  // Beside the segments and the subdivision: the source hierarchy and the
  // rays' grid, and once there are segments the connection test's.  A dozen
  // launches off the chain: 0.58 -> 0.52 ms per replay of the 640-face
  // icospheres, 0.93 -> 0.84 of a 9,702-face knot.  Only in a workspace's own
  // graph: 16 extractions in one graph, which fill the GPU as they are, went
  // from 2.72 to 3.27 ms with 16 branches more.
  cudaStream_t on;
  EDP_CHECK(side_fork(d, side, st, on));
  if (d.merge_regions)
    EDP_CHECK(cudaMemsetAsync(d.merge_choice, 0x7f, sizeof(int) * d.cap.regions, on));
  SortScratch &side_scratch = on == st ? s : side.scratch;
  EDP_CHECK(tree_build(source_tree, d.src_lo, d.src_hi, nullptr, d.n, false, side_scratch, on));
  EDP_CHECK(stage_ray_grid(d, side_scratch, on));
  if (d.n > 0) {
    k_segments<<<blocks(kSourceVertices * int64_t(d.n)), kBlock, 0, st>>>(d);
    note_launch();
    k_segment_flags<<<blocks(kSourceVertices * int64_t(d.n)), kBlock, 0, st>>>(d);
    note_launch();
    EDP_CHECK(scan_exclusive(d.seg_flag, d.seg_pos, d.sc + kSegmentSlots, kSourceVertices * d.n,
                             d.sc + kSegmentCount, s, st));
    k_segment_compact<<<blocks(kSourceVertices * int64_t(d.n)), kBlock, 0, st>>>(d);
    note_launch();
  }
  if (d.propagate_ranks) {
    EDP_CHECK(side_fork(d, side, st, on));
    EDP_CHECK(stage_segment_grid(d, side_scratch, on));
  }
  EDP_CHECK(tree_build(seg_tree, d.seg_lo, d.seg_hi, d.sc + kSegmentCount, 0, false, s, st));
  return stage_lists(d, st);
}

}  // namespace edp
