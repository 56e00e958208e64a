// Convex polygons held by a group of W lanes of a warp (W = 8 or 32), one
// vertex per lane: bounds, cleanup and splits with the rounding of the
// one-thread helpers in edp_device.cuh.  Most patches have three to six
// vertices, so four groups of eight lanes do the work of four warps; the whole
// warp serves the polygons that do not fit.
//
// The groups of a warp stay converged: every helper is called by all 32 lanes
// together (a group without work passes an empty polygon), so shuffles and
// ballots name the full warp and cost no reconvergence.
#pragma once
#include "edp_filtered.cuh"

namespace edp {

constexpr unsigned kFull = 0xffffffffu;

__device__ inline double larger(double a, double b) { return a > b ? a : b; }
__device__ inline double smaller(double a, double b) { return a < b ? a : b; }

// The calling lane's group.
template <int W>
struct Group {
  int lane, shift;
  __device__ Group() {
    const int l = threadIdx.x & 31;
    lane = l & (W - 1);
    shift = l & ~(W - 1);
  }
  __device__ unsigned ballot(bool p) const {
    const unsigned b = __ballot_sync(kFull, p);
    return W == 32 ? b : (b >> shift) & ((1u << (W & 31)) - 1u);
  }
  template <class T>
  __device__ T shfl(T x, int src) const { return __shfl_sync(kFull, x, src, W); }
  __device__ V2 shfl(V2 x, int src) const { return v2(shfl(x.x, src), shfl(x.y, src)); }
  template <class T>
  __device__ T shfl_xor(T x, int off) const { return __shfl_xor_sync(kFull, x, off, W); }
  // Consecutive slots of an append counter for the groups that want one, with
  // one atomic per warp.
  __device__ int reserve_slot(int *counter, bool want) const {
    const unsigned wanting = __ballot_sync(kFull, want && lane == 0);
    int at = 0;
    if ((threadIdx.x & 31) == 0 && wanting) at = atomicAdd(counter, __popc(wanting));
    at = __shfl_sync(kFull, at, 0);
    return at + __popc(wanting & ((1u << shift) - 1u));
  }
};

// The smallest power of two holding n lanes: a butterfly over it reduces
// lanes [0, n), the lanes that hold a patch's vertices.
__device__ inline int lane_width(int n) { return n <= 1 ? 1 : 1 << (32 - __clz(n - 1)); }

// polygon_bounds() of the polygon held one vertex per lane.  Min and max are
// exact, so the butterfly order does not matter; rounding to binary32 is
// monotone, so x and y are rounded first and reduced in binary32.  The plane
// comes and the box goes by value, which keeps this out-of-line helper's call
// frame small.
template <int W>
static __device__ __noinline__ Box group_bounds(V2 p, int n, Plane score) {
  const Group<W> g;
  const bool mine = g.lane < n;
  const double z = value(score, p);
  float lx = mine ? float(p.x - 2.0e-7) : 1.0e30f, ly = mine ? float(p.y - 2.0e-7) : 1.0e30f;
  float hx = mine ? float(p.x + 2.0e-7) : -1.0e30f, hy = mine ? float(p.y + 2.0e-7) : -1.0e30f;
  double lz = mine ? z : 1.0e30, hz = mine ? z : -1.0e30;
  const int width = W == 8 ? 8 : lane_width(n);
  for (int off = width >> 1; off > 0; off >>= 1) {
    lx = fminf(lx, g.shfl_xor(lx, off));
    ly = fminf(ly, g.shfl_xor(ly, off));
    hx = fmaxf(hx, g.shfl_xor(hx, off));
    hy = fmaxf(hy, g.shfl_xor(hy, off));
    lz = smaller(lz, g.shfl_xor(lz, off));
    hz = larger(hz, g.shfl_xor(hz, off));
  }
  if (W > 8) {  // lanes past the butterfly take lane 0's result
    lx = g.shfl(lx, 0);
    ly = g.shfl(ly, 0);
    hx = g.shfl(hx, 0);
    hy = g.shfl(hy, 0);
    lz = g.shfl(lz, 0);
    hz = g.shfl(hz, 0);
  }
  const double pz = 2.0e-7 * larger(1.0, larger(fabs(lz), fabs(hz)));
  return Box{make_float4(lx, ly, float(lz - pz), 0.f), make_float4(hx, hy, float(hz + pz), 0.f)};
}

// length(a) > bound, for bound > 0.  sqrt is correctly rounded, so away from
// bound^2 the squares decide.
__device__ inline bool longer(V2 a, double bound) {
  const double square = a.x * a.x + a.y * a.y, limit = bound * bound;
  if (square > limit * (1.0 + 1.0e-12)) return true;
  if (square < limit * (1.0 - 1.0e-12)) return false;
  return sqrt(square) > bound;
}

// clean() by lane 0 of each group with m > 0 (`buf`: W points for the group).
// Returns the new size; x holds the result.
template <int W>
static __device__ __noinline__ int serial_clean(V2 &x, int m, V2 *buf) {
  const Group<W> g;
  if (g.lane < m) buf[g.lane] = x;
  __syncwarp();
  int count = 0;
  if (g.lane == 0 && m > 0) count = clean(buf, m);
  __syncwarp();
  count = g.shfl(count, 0);
  if (g.lane < count) x = buf[g.lane];
  __syncwarp();
  return count;
}

// clean() of the polygon held one vertex per lane (x, m <= W vertices).  When
// no two consecutive points are near duplicates every point stays and only
// the closing merge and the area / perimeter test remain; their sums run in
// the sequential order, so they round exactly as clean() does.  Otherwise
// lane 0 runs clean() itself.  `buf` is scratch of W points for the group.
// Returns the new size; x holds the result.
template <int W>
__device__ inline int group_clean(const Group<W> &g, V2 &x, int m, V2 *buf) {
  const double merge = kEps * 0.01;
  const V2 prev = g.shfl(x, g.lane > 0 ? g.lane - 1 : 0);
  const bool near = g.ballot(g.lane > 0 && g.lane < m && !longer(x - prev, merge)) != 0;
  int count = m;
  const V2 origin = g.shfl(x, 0), last = g.shfl(x, count > 0 ? count - 1 : 0);
  if (count > 1 && !longer(origin - last, merge)) --count;
  const V2 next = g.shfl(x, g.lane + 1 < count ? g.lane + 1 : 0);
  // Each lane's terms of the two sums, read back in order.
  buf[g.lane] = v2(cross(origin, x, next), fabs(next.x - x.x) + fabs(next.y - x.y));
  __syncwarp();
  double area2 = 0.0, perimeter = 0.0;
  for (int j = 0; j < (W == 8 ? W : count); ++j) {
    const V2 term = buf[j];
    if (j < count) {
      area2 += term.x;
      perimeter += term.y;
    }
  }
  __syncwarp();
  if (count < 3 || area2 <= kEps * perimeter) count = 0;
  if (__any_sync(kFull, near)) {
    V2 y = x;
    const int serial = serial_clean<W>(y, near ? m : 0, buf);
    if (near) {
      x = y;
      count = serial;
    }
  }
  return count;
}

// Split the polygon (one vertex per lane, q the next vertex) by the sign
// `side` of a linear function with binary64 value `du` at this lane's vertex,
// into the part where it is positive (pl, nl) and where it is negative (pr,
// nr), both cleaned: the vertex sequence of the sequential split
// (kernels.py:184-203) placed with ballots and prefix counts.  `left` and
// `right` are scratch of W points each for the group.  Returns false when a
// part has more than W vertices (the parts are then not made).
template <int F, int W>
__device__ inline bool group_split(const Group<W> &g, V2 p, V2 q, int n, double du, int side,
                                   V2 *left, V2 *right, V2 &pl, int &nl, V2 &pr, int &nr) {
  const unsigned below = (1u << g.lane) - 1u;
  const bool mine = g.lane < n;
  const int next = g.lane + 1 < n ? g.lane + 1 : 0;
  const double dv = g.shfl(du, next);
  const int sv = g.shfl(side, next);
  const bool in = mine && side >= 0, out = mine && side <= 0;
  const bool cut = mine && ((side > 0 && sv < 0) || (side < 0 && sv > 0));
  const unsigned bin = g.ballot(in), bout = g.ballot(out), bcut = g.ballot(cut);
  nl = __popc(bin) + __popc(bcut);
  nr = __popc(bout) + __popc(bcut);
  const bool fits = nl <= W && nr <= W;
  if (fits) {
    const int at_l = __popc(bin & below) + __popc(bcut & below);
    const int at_r = __popc(bout & below) + __popc(bcut & below);
    if (in) left[at_l] = p;
    if (out) right[at_r] = p;
    if (cut) {
      const V2 x = p + (F == 0 ? du / (du - dv) : crossing(du, dv)) * (q - p);
      left[at_l + (in ? 1 : 0)] = x;
      right[at_r + (out ? 1 : 0)] = x;
    }
  } else {
    nl = nr = 0;
  }
  __syncwarp();
  pl = left[g.lane];
  pr = right[g.lane];
  __syncwarp();
  // One loop body for both parts: the code is long, and its callers wait on
  // instruction fetch.
#pragma unroll 1
  for (int part = 0; part < 2; ++part) {
    V2 x = part == 0 ? pl : pr;
    const int count = group_clean(g, x, part == 0 ? nl : nr, part == 0 ? left : right);
    if (part == 0) {
      pl = x;
      nl = count;
    } else {
      pr = x;
      nr = count;
    }
  }
  return fits;
}

}  // namespace edp
