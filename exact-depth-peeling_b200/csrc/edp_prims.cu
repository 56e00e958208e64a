// Device-count-aware primitives: exclusive scan, stable LSD radix sort and
// the implicit-tree hierarchy build.  Counts are device scalars so that one
// captured CUDA graph handles any live size up to the allocated capacity
// (the role of the reference's conditional sort buckets, events.py:637-718).
#include "../../include/edp.h"
#include "edp_internal.h"

namespace edp {
namespace {

__device__ inline int warp_inclusive(int v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    int t = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += t;
  }
  return v;
}

// Block-wide exclusive scan of one value per thread (blockDim.x <= 1024).
__device__ inline int block_exclusive(int v, int *smem, int &total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  int inc = warp_inclusive(v);
  if (lane == 31) smem[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    int s = lane < warps ? smem[lane] : 0;
    int si = warp_inclusive(s);
    if (lane < warps) smem[lane] = si - s;
    if (lane == warps - 1) smem[32] = si;
  }
  __syncthreads();
  int r = smem[warp] + inc - v;
  total = smem[32];
  __syncthreads();
  return r;
}

// ---------------------------------------------------------------- look-back
// Scans and radix passes run as one launch each, by decoupled look-back
// (Merrill and Garland 2016; Adinets and Merrill 2022 for the radix pass):
// blocks take tiles in order from a ticket, publish their tile's sums, and add
// up the published sums before it.  A tile waits only for tiles whose blocks
// hold earlier tickets and publish without waiting, so every wait ends; each
// is bounded all the same, and running out sets an error.
//
// A published word holds the sum, a state and the launch's epoch, so the words
// need no clearing between launches (but once in 2^30, when the epochs start
// over: a few hours of replays of a small scene).  The last block to finish gives the
// ticket back and starts the next epoch.
//
// Three launches per scan and per pass (counts, their scan, the scatter) cost
// small extractions mostly gaps between launches: 157 kernels outside the
// subdivision loop became 97.  Replays: icospheres-640 0.81 -> 0.72 ms,
// knot-9702 1.14 -> 1.03, a batch of 16 small scenes 3.44 -> 3.03.
enum Published : unsigned { kNothing = 0, kSum = 1, kPrefix = 2 };
constexpr unsigned kEpochMask = 0x3fffffffu;

__device__ inline unsigned long long publish_word(unsigned epoch, unsigned state, int value) {
  return (unsigned long long)(epoch << 2 | state) << 32 | unsigned(value);
}

// The word at `p` once it is of this epoch.  A wait that runs out sets the
// error and goes on as if nothing came before: every index stays in range.
__device__ inline unsigned long long await_word(const unsigned long long *p, unsigned epoch,
                                                const LookBack &s) {
  const volatile unsigned long long *v = p;
  unsigned long long w = *v;
  for (int polls = 0; unsigned(w >> 34) != epoch || (unsigned(w >> 32) & 3u) == kNothing; w = *v) {
    if (++polls > s.polls) {
      atomicOr(s.error, int(kErrWait));
      return publish_word(epoch, kPrefix, 0);
    }
  }
  return w;
}

// This block's tile (shared by all its threads) and the launch's epoch.
__device__ inline int take_tile(LookBack s, int *shared, unsigned &epoch) {
  if (threadIdx.x == 0) shared[0] = atomicAdd(&s.control[0], 1);
  epoch = *(volatile unsigned *)&s.control[2] & kEpochMask;
  __syncthreads();
  return shared[0];
}

// Counts the block as finished; true in thread 0 of the launch's last block,
// after the state is ready for the next launch.
__device__ inline bool finish_tile(LookBack s, int tiles, unsigned epoch) {
  __syncthreads();
  if (threadIdx.x != 0) return false;
  __threadfence();
  if (atomicAdd(&s.control[1], 1) != tiles - 1) return false;
  s.control[0] = 0;
  s.control[1] = 0;
  const unsigned next = (epoch + 1u) & kEpochMask;
  // The words' 30 epoch bits start over: a word that was last written 2^30
  // launches ago would look like this epoch's.
  if (next == 0)
    for (int64_t w = 0; w < s.size; ++w) s.words[w] = 0;
  s.control[2] = int(next);
  return true;
}

// ---------------------------------------------------------------- scan
// Exclusive scan in one launch and one pass over memory; `clear` zeroes the
// input behind itself (counters for the next extraction).
__global__ void __launch_bounds__(256)
k_scan(int *in, int *out, const int *count, LookBack s, int *total_out, int clear) {
  __shared__ int smem[33];
  __shared__ int s_tile[1], s_before;
  const int n = *count;
  if (n == 0) {
    if (blockIdx.x == 0 && threadIdx.x == 0 && total_out) *total_out = 0;
    return;
  }
  const int tiles = int(ceil_div(n, kScanTile));
  if (int(blockIdx.x) >= tiles) return;
  unsigned epoch;
  const int tile = take_tile(s, s_tile, epoch);
  constexpr int per = kScanTile / 256;  // blockDim.x == 256
  const int64_t first = int64_t(tile) * kScanTile + int64_t(threadIdx.x) * per;
  int v[per];
  int sum = 0;
#pragma unroll
  for (int k = 0; k < per; k += 4) {
    int4 x = make_int4(0, 0, 0, 0);
    if (first + k + 3 < n) {
      x = *reinterpret_cast<const int4 *>(in + first + k);
      if (clear) *reinterpret_cast<int4 *>(in + first + k) = make_int4(0, 0, 0, 0);
    } else {
      int *y = reinterpret_cast<int *>(&x);
      for (int c = 0; c < 4; ++c)
        if (first + k + c < n) {
          y[c] = in[first + k + c];
          if (clear) in[first + k + c] = 0;
        }
    }
    v[k] = x.x; v[k + 1] = x.y; v[k + 2] = x.z; v[k + 3] = x.w;
    sum += x.x + x.y + x.z + x.w;
  }
  int total;
  int e = block_exclusive(sum, smem, total);
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    int before = 0;
    if (tile > 0) {
      if (lane == 0) *(volatile unsigned long long *)&s.words[tile] = publish_word(epoch, kSum, total);
      for (int look = tile - 1;; look -= 32) {
        const int at = look - lane;
        const unsigned long long w = at >= 0 ? await_word(s.words + at, epoch, s)
                                             : publish_word(epoch, kPrefix, 0);
        const unsigned full = __ballot_sync(0xffffffffu, (unsigned(w >> 32) & 3u) == kPrefix);
        const int last = full ? __ffs(int(full)) - 1 : 31;
        before += __reduce_add_sync(0xffffffffu, lane <= last ? int(unsigned(w)) : 0);
        if (full) break;
      }
    }
    if (lane == 0) {
      *(volatile unsigned long long *)&s.words[tile] = publish_word(epoch, kPrefix, before + total);
      s_before = before;
    }
  }
  __syncthreads();
  e += s_before;
#pragma unroll
  for (int k = 0; k < per; k += 4) {
    int4 x;
    x.x = e; e += v[k];
    x.y = e; e += v[k + 1];
    x.z = e; e += v[k + 2];
    x.w = e; e += v[k + 3];
    if (first + k + 3 < n) {
      *reinterpret_cast<int4 *>(out + first + k) = x;
    } else {
      const int *y = reinterpret_cast<const int *>(&x);
      for (int c = 0; c < 4; ++c)
        if (first + k + c < n) out[first + k + c] = y[c];
    }
  }
  if (threadIdx.x == 0 && total_out && tile == tiles - 1) *total_out = s_before + total;
  finish_tile(s, tiles, epoch);
}

// ---------------------------------------------------------------- radix sort
// Digit counts of every pass at once: the digits of a key are those of the
// key set, whatever its order, so one read serves all passes.  `hist` is
// [passes][256], zero on entry (the last pass of a sort clears it).
template <class K>
__device__ inline void count_digits(K key, int passes, int *local) {
  for (int p = 0; p < passes; ++p) atomicAdd(&local[256 * p + int((key >> (8 * p)) & 255u)], 1);
}

__device__ inline void add_digits(const int *local, int passes, int *hist) {
  for (int k = threadIdx.x; k < 256 * passes; k += blockDim.x)
    if (local[k]) atomicAdd(&hist[k], local[k]);
}

template <class K>
__global__ void k_radix_hist(const K *__restrict__ keys, const int *count, int passes, int *hist) {
  __shared__ int local[256 * kSortPasses];
  const int n = *count;
  if (n == 0) return;
  for (int k = threadIdx.x; k < 256 * passes; k += blockDim.x) local[k] = 0;
  __syncthreads();
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x)
    count_digits(keys[i], passes, local);
  __syncthreads();
  add_digits(local, passes, hist);
}

// One stable pass.  Warp w of a tile owns a contiguous run of 256 keys, in
// eight rounds of 32; peers with equal digits are ranked with match_any.
// Thread d looks back over the tiles before for digit d, eight at a time.
template <class K>
__global__ void __launch_bounds__(kSortBlock) k_radix_pass(
    const K *__restrict__ keys, const int *__restrict__ vals, K *keys_out, int *vals_out,
    const int *count, int pass, int passes, int *hist, LookBack s) {
  __shared__ int wcount[kSortBlock / 32][256];
  __shared__ int smem[33];
  __shared__ int s_tile[1];
  const int n = *count;
  if (n == 0) return;
  const int tiles = int(ceil_div(n, kSortTile));
  if (int(blockIdx.x) >= tiles) return;
  unsigned epoch;
  const int tile = take_tile(s, s_tile, epoch);
  const int64_t tile0 = int64_t(tile) * kSortTile;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, shift = 8 * pass;
  int total;
  int running = block_exclusive(hist[256 * pass + threadIdx.x], smem, total);
  for (int w = 0; w < kSortBlock / 32; ++w) wcount[w][threadIdx.x] = 0;
  __syncthreads();
  K k[kSortItems];
  int d[kSortItems];
  const int64_t run = tile0 + int64_t(warp) * (32 * kSortItems);
#pragma unroll
  for (int r = 0; r < kSortItems; ++r) {
    int64_t i = run + r * 32 + lane;
    if (i < n) {
      k[r] = keys[i];
      d[r] = int((k[r] >> shift) & 255u);
    } else {
      d[r] = 256;
    }
  }
  const unsigned lt = (1u << lane) - 1u;
#pragma unroll
  for (int r = 0; r < kSortItems; ++r) {
    unsigned peers = __match_any_sync(0xffffffffu, d[r]);
    if (d[r] < 256 && lane == __ffs(peers) - 1) wcount[warp][d[r]] += __popc(peers);
    __syncwarp();
  }
  __syncthreads();
  {
    int mine = 0;
    for (int w = 0; w < kSortBlock / 32; ++w) mine += wcount[w][threadIdx.x];
    unsigned long long *words = s.words + threadIdx.x;
    int before = 0;
    if (tile > 0) {
      *(volatile unsigned long long *)&words[256 * int64_t(tile)] = publish_word(epoch, kSum, mine);
      constexpr int kWindow = 8;
      for (int look = tile - 1, done = 0; !done; look -= kWindow) {
        unsigned long long w[kWindow];
#pragma unroll
        for (int c = 0; c < kWindow; ++c)
          w[c] = look - c >= 0
                     ? *(const volatile unsigned long long *)&words[256 * int64_t(look - c)]
                     : publish_word(epoch, kPrefix, 0);
#pragma unroll
        for (int c = 0; c < kWindow; ++c) {
          if (done) continue;
          if (unsigned(w[c] >> 34) != epoch || (unsigned(w[c] >> 32) & 3u) == kNothing)
            w[c] = await_word(words + 256 * int64_t(look - c), epoch, s);
          before += int(unsigned(w[c]));
          done = (unsigned(w[c] >> 32) & 3u) == kPrefix;
        }
      }
    }
    *(volatile unsigned long long *)&words[256 * int64_t(tile)] =
        publish_word(epoch, kPrefix, before + mine);
    running += before;
    for (int w = 0; w < kSortBlock / 32; ++w) {
      int c = wcount[w][threadIdx.x];
      wcount[w][threadIdx.x] = running;
      running += c;
    }
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kSortItems; ++r) {
    unsigned peers = __match_any_sync(0xffffffffu, d[r]);
    if (d[r] < 256) {
      // Below n, unless a wait ran out and left older keys in an earlier pass.
      int pos = min(wcount[warp][d[r]] + __popc(peers & lt), n - 1);
      int64_t i = run + r * 32 + lane;
      keys_out[pos] = k[r];
      vals_out[pos] = vals[i];
    }
    __syncwarp();
    if (d[r] < 256 && lane == __ffs(peers) - 1) wcount[warp][d[r]] += __popc(peers);
    __syncwarp();
  }
  const bool last = finish_tile(s, tiles, epoch);
  if (pass == passes - 1) {  // every block has read the digit counts
    if (threadIdx.x == 0) s_tile[0] = last;
    __syncthreads();
    if (s_tile[0])
      for (int p = 0; p < passes; ++p) hist[256 * p + threadIdx.x] = 0;
  }
}

template <class K>
__global__ void k_copy_pairs(const K *keys, const int *vals, K *keys_out, int *vals_out,
                             const int *count) {
  const int n = *count;
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x) {
    keys_out[i] = keys[i];
    vals_out[i] = vals[i];
  }
}

// The passes of a sort whose digit counts are in s.hist.
template <class K>
cudaError_t sort_passes(K *keys, K *keys_tmp, int *vals, int *vals_tmp, const int *count,
                        int64_t capacity, int passes, SortScratch &s, cudaStream_t st) {
  const int64_t tiles = ceil_div(capacity, kSortTile);
  if (tiles > s.tiles || passes > kSortPasses) return cudaErrorInvalidValue;
  K *ka = keys, *kb = keys_tmp;
  int *va = vals, *vb = vals_tmp;
  for (int p = 0; p < passes; ++p) {
    k_radix_pass<K><<<unsigned(tiles), kSortBlock, 0, st>>>(ka, va, kb, vb, count, p, passes,
                                                             s.hist, s.look_back);
    note_launch();
    K *tk = ka; ka = kb; kb = tk;
    int *tv = va; va = vb; vb = tv;
  }
  if (ka != keys) {
    k_copy_pairs<K><<<592, 256, 0, st>>>(ka, va, keys, vals, count);
    note_launch();
  }
  return cudaGetLastError();
}

template <class K>
cudaError_t sort_pairs(K *keys, K *keys_tmp, int *vals, int *vals_tmp, const int *count,
                       int64_t capacity, int bits, SortScratch &s, cudaStream_t st) {
  const int passes = int(ceil_div(bits, 8));
  k_radix_hist<K><<<unsigned(std::min<int64_t>(ceil_div(capacity, kSortTile), 148 * 4)),
                    kSortBlock, 0, st>>>(keys, count, passes, s.hist);
  note_launch();
  return sort_passes(keys, keys_tmp, vals, vals_tmp, count, capacity, passes, s, st);
}

// ---------------------------------------------------------------- hierarchy
// The build's item and leaf counts, the leaves' keys, and the keys' digit
// counts for the sort.
__global__ void k_tree_keys(const float4 *lo, const float4 *hi, const int *count_ptr,
                            int static_count, int *count_out, int *size, uint64_t *keys, int *ids,
                            int layered, int passes, int *hist) {
  __shared__ int local[256 * kSortPasses];
  const int n = count_ptr ? *count_ptr : static_count;
  int leaves = 1;
  while (leaves < n) leaves <<= 1;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    *count_out = n;
    *size = leaves;
  }
  if (int64_t(blockIdx.x) * blockDim.x >= leaves) return;
  for (int k = threadIdx.x; k < 256 * passes; k += blockDim.x) local[k] = 0;
  __syncthreads();
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < leaves;
       i += int64_t(gridDim.x) * blockDim.x) {
    ids[i] = int(i);
    uint64_t key = ~0ull;
    if (i < n) {
      float4 a = lo[i], b = hi[i];
      if (a.x <= b.x && a.y <= b.y) {
        float cx = fminf(fmaxf((a.x + b.x) * 0.5f, 0.f), 1.f);
        float cy = fminf(fmaxf((a.y + b.y) * 0.5f, 0.f), 1.f);
        uint32_t x = uint32_t(int(cx * 32767.0f)), y = uint32_t(int(cy * 32767.0f));
        key = uint64_t(part1by1(x) | (part1by1(y) << 1));
        if (layered) key |= uint64_t(int(a.z)) << 32;
      }
      count_digits(key, passes, local);
    }
    keys[i] = key;
  }
  __syncthreads();
  add_digits(local, passes, hist);
}

// Every node of a fresh hierarchy holds the empty box, which overlaps nothing.
__global__ void k_tree_clear(float4 *nodes, int64_t count) {
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < count;
       i += int64_t(gridDim.x) * blockDim.x) {
    nodes[2 * i] = empty_lo();
    nodes[2 * i + 1] = empty_hi();
  }
}

__device__ inline void union_into(float4 *nodes, int node) {
  float4 a = __ldcg(&nodes[4 * node]), c = __ldcg(&nodes[4 * node + 1]);      // child 2 node
  float4 b = __ldcg(&nodes[4 * node + 2]), d = __ldcg(&nodes[4 * node + 3]);  // child 2 node + 1
  __stcg(&nodes[2 * node], make_float4(fminf(a.x, b.x), fminf(a.y, b.y), fminf(a.z, b.z), 0.f));
  __stcg(&nodes[2 * node + 1], make_float4(fmaxf(c.x, d.x), fmaxf(c.y, d.y), fmaxf(c.z, d.z), 0.f));
}

constexpr int kFitThreads = 256;
constexpr int kFitLeaves = 2 * kFitThreads;  // leaves of one block's subtree

// Leaves and every internal box in one launch.  Leaf i holds the box of item
// ids[i] (the empty box past the item count).  Each block reduces whole
// subtrees of up to kFitLeaves leaves level by level in shared memory; the
// last block to finish then reduces the levels above the subtree roots.
// Unions of binary32 boxes are exact, so the boxes do not depend on the order.
__global__ void __launch_bounds__(kFitThreads)
k_tree_fit(float4 *nodes, const int *ids, const float4 *lo, const float4 *hi, const int *count,
           const int *size, int *done) {
  __shared__ float4 s_lo[kFitThreads], s_hi[kFitThreads];
  __shared__ int s_last;
  const int n = *count, leaves = *size, t = threadIdx.x;
  const int span = leaves < kFitLeaves ? leaves : kFitLeaves;
  const int subtrees = leaves / span;
  auto leaf = [&](int i, float4 &a, float4 &b) {
    const int j = ids[i];
    a = empty_lo();
    b = empty_hi();
    if (j < n) {
      a = lo[j];
      b = hi[j];
    }
    nodes[2 * (leaves + i)] = a;
    nodes[2 * (leaves + i) + 1] = b;
  };
  for (int sub = blockIdx.x; sub < subtrees; sub += gridDim.x) {
    const int first = sub * span;
    if (span == 1) {
      float4 a, b;
      if (t == 0) leaf(first, a, b);
      continue;
    }
    int width = span >> 1, base = (leaves + first) >> 1;  // node id of slot 0 on this level
    if (t < width) {
      float4 a, b, c, e;
      leaf(first + 2 * t, a, b);
      leaf(first + 2 * t + 1, c, e);
      a = make_float4(fminf(a.x, c.x), fminf(a.y, c.y), fminf(a.z, c.z), 0.f);
      b = make_float4(fmaxf(b.x, e.x), fmaxf(b.y, e.y), fmaxf(b.z, e.z), 0.f);
      s_lo[t] = a;
      s_hi[t] = b;
      nodes[2 * (base + t)] = a;
      nodes[2 * (base + t) + 1] = b;
    }
    __syncthreads();
    for (width >>= 1; width >= 1; width >>= 1) {
      base >>= 1;
      float4 a, b;
      if (t < width) {
        const float4 l0 = s_lo[2 * t], l1 = s_lo[2 * t + 1], h0 = s_hi[2 * t], h1 = s_hi[2 * t + 1];
        a = make_float4(fminf(l0.x, l1.x), fminf(l0.y, l1.y), fminf(l0.z, l1.z), 0.f);
        b = make_float4(fmaxf(h0.x, h1.x), fmaxf(h0.y, h1.y), fmaxf(h0.z, h1.z), 0.f);
      }
      __syncthreads();
      if (t < width) {
        s_lo[t] = a;
        s_hi[t] = b;
        nodes[2 * (base + t)] = a;
        nodes[2 * (base + t) + 1] = b;
      }
      __syncthreads();
    }
  }
  __threadfence();
  __syncthreads();
  if (t == 0) s_last = atomicAdd(done, 1) == int(gridDim.x) - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  for (int width = subtrees >> 1; width >= 1; width >>= 1) {
    for (int k = t; k < width; k += blockDim.x) union_into(nodes, width + k);
    __syncthreads();
  }
  if (t == 0) *done = 0;
}

}  // namespace

cudaError_t scan_exclusive(int *in, int *out, const int *count, int64_t capacity, int *total,
                           SortScratch &s, cudaStream_t st, bool clear) {
  const int64_t tiles = ceil_div(capacity > 0 ? capacity : 1, kScanTile);
  if (tiles > s.scan_tiles) return cudaErrorInvalidValue;
  k_scan<<<unsigned(tiles), 256, 0, st>>>(in, out, count, s.look_back, total, clear ? 1 : 0);
  note_launch();
  return cudaGetLastError();
}

cudaError_t sort_pairs_u64(uint64_t *keys, uint64_t *keys_tmp, int *vals, int *vals_tmp,
                           const int *count, int64_t capacity, int bits, SortScratch &s,
                           cudaStream_t st) {
  return sort_pairs<uint64_t>(keys, keys_tmp, vals, vals_tmp, count, capacity, bits, s, st);
}

cudaError_t tree_refit(TreeBuffers &t, const float4 *lo, const float4 *hi, cudaStream_t st) {
  const int64_t subtrees = ceil_div(t.leaves_cap, int64_t(kFitLeaves));
  const unsigned g = unsigned(subtrees < 148 * 8 ? subtrees : 148 * 8);
  k_tree_fit<<<g, kFitThreads, 0, st>>>(t.nodes, t.ids, lo, hi, t.count, t.size, t.flags);
  note_launch();
  return cudaGetLastError();
}

cudaError_t tree_init(TreeBuffers &t) {
  t.count = t.size + 1;
  const int64_t count = 2 * t.leaves_cap;
  k_tree_clear<<<grid_for(count, 256) < 4 * 148 ? grid_for(count, 256) : 4 * 148, 256>>>(t.nodes, count);
  note_launch();
  return cudaGetLastError();
}

cudaError_t tree_build(TreeBuffers &t, const float4 *lo, const float4 *hi, const int *count_ptr,
                       int static_count, bool layered, SortScratch &s, cudaStream_t st) {
  // Layered keys hold the layer above 30 Morton bits; 48 key bits order them
  // for up to 65536 layers.  Deeper scenes leave higher layer bits unordered,
  // which only loosens the hierarchy: any leaf order gives the same queries.
  const int passes = layered ? 6 : 4;
  const unsigned g = grid_for(t.leaves_cap, 256) < 4 * 148 ? grid_for(t.leaves_cap, 256) : 4 * 148;
  k_tree_keys<<<g, 256, 0, st>>>(lo, hi, count_ptr, static_count, t.count, t.size, t.keys, t.ids,
                                 layered ? 1 : 0, passes, s.hist);
  note_launch();
  EDP_CHECK(sort_passes(t.keys, t.keys_tmp, t.ids, t.ids_tmp, t.count, t.leaves_cap, passes, s, st));
  return tree_refit(t, lo, hi, st);
}

}  // namespace edp

namespace edp {
namespace {
thread_local int64_t g_launches = 0;
thread_local cudaEvent_t *g_marks = nullptr;
thread_local int g_next_mark = 0;  // stages marked so far in this capture
}
void note_launch() { ++g_launches; }
void forget_launches(int64_t n) { g_launches -= n; }
int64_t launch_count() { return g_launches; }

void set_stage_marks(cudaEvent_t *events) {
  g_marks = events;
  g_next_mark = 0;
}

cudaError_t stage_mark(int stage, cudaStream_t st) {
  if (!g_marks) return cudaSuccess;
  if (stage < 0) {  // the start
    g_next_mark = 0;
    return cudaEventRecordWithFlags(g_marks[0], st, cudaEventRecordExternal);
  }
  for (; g_next_mark <= stage && g_next_mark < EDP_STAGE_COUNT; ++g_next_mark) {
    cudaError_t e = cudaEventRecordWithFlags(g_marks[g_next_mark + 1], st, cudaEventRecordExternal);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}
}  // namespace edp

namespace edp {
// A conditional IF node of the graph being captured on `st` (default: not
// taken): a kernel sets the handle, then the body is recorded on `body`
// between conditional_begin and conditional_end.
cudaError_t conditional_handle(cudaStream_t st, cudaGraphConditionalHandle &handle) {
  cudaStreamCaptureStatus cs;
  cudaGraph_t g = nullptr;
  const cudaGraphNode_t *deps = nullptr;
  size_t ndeps = 0;
  EDP_CHECK(cudaStreamGetCaptureInfo(st, &cs, nullptr, &g, &deps, &ndeps));
  return cudaGraphConditionalHandleCreate(&handle, g, 0, cudaGraphCondAssignDefault);
}

cudaError_t conditional_begin(cudaStream_t st, cudaGraphConditionalHandle handle,
                              cudaStream_t body) {
  cudaStreamCaptureStatus cs;
  cudaGraph_t g = nullptr;
  const cudaGraphNode_t *deps = nullptr;
  size_t ndeps = 0;
  EDP_CHECK(cudaStreamGetCaptureInfo(st, &cs, nullptr, &g, &deps, &ndeps));
  alignas(cudaGraphNodeParams) unsigned char raw[sizeof(cudaGraphNodeParams)] = {};
  cudaGraphNodeParams &params = *reinterpret_cast<cudaGraphNodeParams *>(raw);
  params.type = cudaGraphNodeTypeConditional;
  params.conditional.handle = handle;
  params.conditional.type = cudaGraphCondTypeIf;
  params.conditional.size = 1;
  cudaGraphNode_t node;
  EDP_CHECK(cudaGraphAddNode(&node, g, deps, ndeps, &params));
  EDP_CHECK(cudaStreamUpdateCaptureDependencies(st, &node, 1, cudaStreamSetCaptureDependencies));
  return cudaStreamBeginCaptureToGraph(body, params.conditional.phGraph_out[0], nullptr, nullptr, 0,
                                       cudaStreamCaptureModeRelaxed);
}

cudaError_t conditional_end(cudaStream_t body) {
  cudaGraph_t captured = nullptr;
  return cudaStreamEndCapture(body, &captured);
}
}  // namespace edp
