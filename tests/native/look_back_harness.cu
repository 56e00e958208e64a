// The scans and radix passes of exact-depth-peeling_b200/csrc/edp_prims.cu on
// their own, for the GPU tests: a look-back state of the caller's making, and
// the first `missing` tickets of the first launch never taken, so that the
// tiles behind them wait in vain.
#include <vector>

#include "../../exact-depth-peeling_b200/csrc/edp_prims.cu"

namespace {
template <class T>
T *device_copy(const T *host, int64_t count) {
  T *p = nullptr;
  if (cudaMalloc(&p, sizeof(T) * count) != cudaSuccess) return nullptr;
  if (host)
    cudaMemcpy(p, host, sizeof(T) * count, cudaMemcpyHostToDevice);
  else
    cudaMemset(p, 0, sizeof(T) * count);
  return p;
}

// Words and control for `tiles` tiles of `per` words each, with room for the
// tickets past the last tile that skipped ones push blocks to.
// At the last epoch the words hold sums of an old launch with the next one.
edp::SortScratch scratch(int64_t tiles, int per, int polls, int missing, unsigned epoch,
                         int *error) {
  edp::SortScratch s;
  s.tiles = s.scan_tiles = tiles;
  const int control[3] = {missing, 0, int(epoch)};
  s.look_back.size = (tiles + missing) * per;
  const std::vector<unsigned long long> old(s.look_back.size,
                                            epoch ? 2ull << 32 | 12345ull : 0ull);
  s.look_back.words = device_copy(old.data(), s.look_back.size);
  s.look_back.control = device_copy(control, 3);
  s.look_back.error = error;
  s.look_back.polls = polls;
  s.hist = device_copy<int>(nullptr, 256 * edp::kSortPasses);
  return s;
}
}  // namespace

// Scans `values` twice with one state; errors[k] is the error word after the
// k-th.  Returns the CUDA error.
extern "C" int look_back_scan(const int *values, int n, int polls, int missing,
                              unsigned epoch, int *out, int *errors) {
  const int64_t tiles = edp::ceil_div(n, edp::kScanTile);
  int *in = device_copy(values, n), *scanned = device_copy<int>(nullptr, n);
  int *count = device_copy(&n, 1), *total = device_copy<int>(nullptr, 1);
  int *error = device_copy<int>(nullptr, 1);
  edp::SortScratch s = scratch(tiles, 1, polls, missing, epoch, error);
  for (int k = 0; k < 2; ++k) {
    edp::scan_exclusive(in, scanned, count, n, total, s, nullptr);
    cudaMemcpy(errors + k, error, sizeof(int), cudaMemcpyDeviceToHost);
    cudaMemset(error, 0, sizeof(int));
  }
  cudaMemcpy(out, scanned, sizeof(int) * n, cudaMemcpyDeviceToHost);
  cudaMemcpy(out + n, total, sizeof(int), cudaMemcpyDeviceToHost);
  for (void *p : {(void *)in, (void *)scanned, (void *)count, (void *)total, (void *)error,
                  (void *)s.look_back.words, (void *)s.look_back.control, (void *)s.hist})
    cudaFree(p);
  return int(cudaDeviceSynchronize());
}

// Sorts 16-bit `keys` twice with one state, the positions beside them.
extern "C" int look_back_sort(const uint64_t *keys, int n, int polls, int missing,
                              unsigned epoch, uint64_t *out, int *positions, int *errors) {
  const int64_t tiles = edp::ceil_div(n, edp::kSortTile);
  std::vector<int> index(n);
  for (int i = 0; i < n; ++i) index[i] = i;
  uint64_t *k = device_copy(keys, n), *k_tmp = device_copy<uint64_t>(nullptr, n);
  int *v = device_copy(index.data(), n), *v_tmp = device_copy<int>(nullptr, n);
  int *count = device_copy(&n, 1), *error = device_copy<int>(nullptr, 1);
  edp::SortScratch s = scratch(tiles, 256, polls, missing, epoch, error);
  for (int round = 0; round < 2; ++round) {
    cudaMemcpy(k, keys, sizeof(uint64_t) * n, cudaMemcpyHostToDevice);
    cudaMemcpy(v, index.data(), sizeof(int) * n, cudaMemcpyHostToDevice);
    edp::sort_pairs_u64(k, k_tmp, v, v_tmp, count, n, 16, s, nullptr);
    cudaMemcpy(errors + round, error, sizeof(int), cudaMemcpyDeviceToHost);
    cudaMemset(error, 0, sizeof(int));
  }
  cudaMemcpy(out, k, sizeof(uint64_t) * n, cudaMemcpyDeviceToHost);
  cudaMemcpy(positions, v, sizeof(int) * n, cudaMemcpyDeviceToHost);
  for (void *p : {(void *)k, (void *)k_tmp, (void *)v, (void *)v_tmp, (void *)count,
                  (void *)error, (void *)s.look_back.words, (void *)s.look_back.control,
                  (void *)s.hist})
    cudaFree(p);
  return int(cudaDeviceSynchronize());
}
