// Convex polygons held by a warp, one vertex per lane: bounds, cleanup and
// splits with the rounding of the one-thread helpers in edp_device.cuh.
#pragma once
#include "edp_filtered.cuh"

namespace edp {

constexpr unsigned kFull = 0xffffffffu;

// The smallest power of two holding n lanes: a butterfly over it reduces
// lanes [0, n), the lanes that hold a patch's vertices.
__device__ inline int lane_width(int n) { return n <= 1 ? 1 : 1 << (32 - __clz(n - 1)); }

__device__ inline V2 shfl(V2 x, int lane) {
  return v2(__shfl_sync(kFull, x.x, lane), __shfl_sync(kFull, x.y, lane));
}

// polygon_bounds() of the patch held one vertex per lane (min and max are
// exact, so the butterfly order does not matter).  The plane comes and the
// box goes by value, which keeps this out-of-line helper's call frame small.
static __device__ __noinline__ Box warp_bounds(V2 p, int n, Plane score) {
  const bool mine = int(threadIdx.x & 31) < n;
  const double z = value(score, p);
  double lx = mine ? p.x : 1.0e30, ly = mine ? p.y : 1.0e30, lz = mine ? z : 1.0e30;
  double hx = mine ? p.x : -1.0e30, hy = mine ? p.y : -1.0e30, hz = mine ? z : -1.0e30;
  // Lanes [0, width) hold every vertex; a butterfly over them leaves the
  // result in lane 0, which every lane then reads.
  const int width = lane_width(n);
  for (int off = width >> 1; off > 0; off >>= 1) {
    lx = fmin(lx, __shfl_xor_sync(kFull, lx, off));
    ly = fmin(ly, __shfl_xor_sync(kFull, ly, off));
    lz = fmin(lz, __shfl_xor_sync(kFull, lz, off));
    hx = fmax(hx, __shfl_xor_sync(kFull, hx, off));
    hy = fmax(hy, __shfl_xor_sync(kFull, hy, off));
    hz = fmax(hz, __shfl_xor_sync(kFull, hz, off));
  }
  lx = __shfl_sync(kFull, lx, 0);
  ly = __shfl_sync(kFull, ly, 0);
  lz = __shfl_sync(kFull, lz, 0);
  hx = __shfl_sync(kFull, hx, 0);
  hy = __shfl_sync(kFull, hy, 0);
  hz = __shfl_sync(kFull, hz, 0);
  double pz = 2.0e-7 * fmax(1.0, fmax(fabs(lz), fabs(hz)));
  return Box{make_float4(float(lx - 2.0e-7), float(ly - 2.0e-7), float(lz - pz), 0.f),
             make_float4(float(hx + 2.0e-7), float(hy + 2.0e-7), float(hz + pz), 0.f)};
}

// clean() of the polygon held one vertex per lane (x, m <= kMaxVertices
// vertices).  When no two consecutive points are near duplicates every point
// stays and only the closing merge and the area / perimeter test remain; their
// sums run in the sequential order through shuffles, so they round exactly as
// clean() does.  Otherwise lane 0 runs clean() itself on `buf` (a per-warp
// scratch of kMaxVertices points).  Returns the new size; x holds the result.
static __device__ __noinline__ int serial_clean(V2 &x, int m, V2 *buf) {
  const int lane = threadIdx.x & 31;
  if (lane < m) buf[lane] = x;
  __syncwarp();
  int count = 0;
  if (lane == 0) count = clean(buf, m);
  __syncwarp();
  count = __shfl_sync(kFull, count, 0);
  if (lane < count) x = buf[lane];
  __syncwarp();
  return count;
}

__device__ inline int warp_clean(V2 &x, int m, V2 *buf) {
  const int lane = threadIdx.x & 31;
  const double merge = kEps * 0.01;
  const V2 prev = shfl(x, lane > 0 ? lane - 1 : 0);
  const bool near = lane > 0 && lane < m && !(length(x - prev) > merge);
  if (__ballot_sync(kFull, near)) return serial_clean(x, m, buf);
  int count = m;
  if (count > 1 && length(shfl(x, 0) - shfl(x, count - 1)) <= merge) --count;
  if (count < 3) return 0;
  const V2 origin = shfl(x, 0), next = shfl(x, lane + 1 < count ? lane + 1 : 0);
  const double term = cross(origin, x, next);
  const double step = fabs(next.x - x.x) + fabs(next.y - x.y);
  double area2 = 0.0, perimeter = 0.0;
  for (int j = 0; j < count; ++j) {
    area2 += __shfl_sync(kFull, term, j);
    perimeter += __shfl_sync(kFull, step, j);
  }
  return area2 <= kEps * perimeter ? 0 : count;
}

// Split the polygon (one vertex per lane, q the next vertex) by the sign
// `side` of a linear function with binary64 value `du` at this lane's vertex,
// into the part where it is positive (pl, nl) and where it is negative (pr,
// nr), both cleaned: the vertex sequence of the sequential split
// (kernels.py:184-203) placed with ballots and prefix counts.  `left` and
// `right` are per-warp scratch of kMaxVertices points.  Returns false when a
// part exceeds kMaxVertices.
template <int F>
__device__ inline bool warp_split(V2 p, V2 q, int n, double du, int side, V2 *left, V2 *right,
                                  V2 &pl, int &nl, V2 &pr, int &nr) {
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  const bool mine = lane < n;
  const int next = lane + 1 < n ? lane + 1 : 0;
  const double dv = __shfl_sync(kFull, du, next);
  const int sv = __shfl_sync(kFull, side, next);
  const bool in = mine && side >= 0, out = mine && side <= 0;
  const bool cut = mine && ((side > 0 && sv < 0) || (side < 0 && sv > 0));
  const unsigned bin = __ballot_sync(kFull, in), bout = __ballot_sync(kFull, out);
  const unsigned bcut = __ballot_sync(kFull, cut);
  nl = __popc(bin) + __popc(bcut);
  nr = __popc(bout) + __popc(bcut);
  if (nl > kMaxVertices || nr > kMaxVertices) return false;
  const int at_l = __popc(bin & below) + __popc(bcut & below);
  const int at_r = __popc(bout & below) + __popc(bcut & below);
  if (in) left[at_l] = p;
  if (out) right[at_r] = p;
  if (cut) {
    const V2 x = p + (F == 0 ? du / (du - dv) : crossing(du, dv)) * (q - p);
    left[at_l + (in ? 1 : 0)] = x;
    right[at_r + (out ? 1 : 0)] = x;
  }
  __syncwarp();
  pl = left[lane];
  pr = right[lane];
  __syncwarp();
  nl = warp_clean(pl, nl, left);
  nr = warp_clean(pr, nr, right);
  return true;
}

}  // namespace edp
