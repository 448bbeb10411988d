// Row gathers for packed sequences of different lengths: between the packed rows (all sequences of step 0, then of step 1,
// ...) and the padded [T,B] grid, forwards in time or each sequence from its own end.  A gather with an index per row,
// -1 for a zero row; every map comes with its inverse, so gradients are gathers too (no atomics, no fills).  What they
// replace is a copy and a fill per time step.  Bound by memory.
#include "common.cuh"

namespace blstm {

template <typename V>
__global__ void __launch_bounds__(256) gather_rows_kernel(V* __restrict__ dst, const V* __restrict__ src, const int* __restrict__ idx,
                                                          long long n, int cols) {
  const long long total = n * cols, step = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += step) {
    const long long row = i / cols;
    const int from = idx[row];
    V v{};
    if (from >= 0) v = src[(long long)from * cols + (i - row * cols)];
    dst[i] = v;
  }
}

// batch_sizes is non-increasing: a sequence of sorted rank j has as many steps as there are entries above j.
__global__ void __launch_bounds__(256) packed_maps_kernel(const int* __restrict__ bs, const int* __restrict__ off, const long long* __restrict__ rank,
                                                          int T, int B, int* __restrict__ maps) {
  const int n = T * B;
  int* padded = maps;            // [T,B] -> packed row
  int* turned = maps + n;        // [T,B] -> packed row of the sequence read from its end
  int* rev = maps + 2 * n;       // [T,B] -> padded row, each sequence from its own end (its own inverse)
  int* inv_last = maps + 3 * n;  // [T,B] -> sequence whose last step this is
  int* last = maps + 4 * n;      // [B]   -> padded row of the last step
  int* packed = last + B;        // [N]   -> padded row
  int* packed_t = packed + off[T - 1] + bs[T - 1];   // [N] -> padded row in the turned grid
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int t = i / B, b = i - t * B;
    const int j = rank ? (int)rank[b] : b;
    int lo = 0, hi = T;          // length of sequence j: first t with bs[t] <= j
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (bs[mid] > j) lo = mid + 1; else hi = mid;
    }
    const int len = lo;
    const bool in = t < len;
    padded[i] = in ? off[t] + j : -1;
    turned[i] = in ? off[len - 1 - t] + j : -1;
    rev[i] = in ? (len - 1 - t) * B + b : i;
    inv_last[i] = t == len - 1 ? b : -1;
    if (in) {
      packed[off[t] + j] = i;
      packed_t[off[len - 1 - t] + j] = i;
    }
    if (t == len - 1) last[b] = i;
  }
}

}  // namespace blstm

using namespace blstm;

extern "C" {

int blstm_gather_rows(void* dst, const void* src, const int32_t* idx, int64_t n, int64_t row_bytes, void* stream) {
  if (!dst || !src || !idx || n < 0 || row_bytes <= 0) return BLSTM_E_INVALID_ARG;
  if (n == 0) return BLSTM_OK;
  const uintptr_t m = reinterpret_cast<uintptr_t>(dst) | reinterpret_cast<uintptr_t>(src) | (uintptr_t)row_bytes;
  const int piece = (m & 15u) == 0 ? 16 : (m & 3u) == 0 ? 4 : (m & 1u) == 0 ? 2 : 0;
  if (!piece || row_bytes / piece > INT32_MAX) return BLSTM_E_INVALID_ARG;
  const int cols = (int)(row_bytes / piece);
  const long long want = (n * cols + 1023) / 1024, cap = 8ll * plan_sm_count();
  const unsigned grid = (unsigned)(want < cap ? want : cap);
  cudaStream_t st = (cudaStream_t)stream;
  if (piece == 16) gather_rows_kernel<uint4><<<grid, 256, 0, st>>>((uint4*)dst, (const uint4*)src, idx, n, cols);
  else if (piece == 4) gather_rows_kernel<uint32_t><<<grid, 256, 0, st>>>((uint32_t*)dst, (const uint32_t*)src, idx, n, cols);
  else gather_rows_kernel<uint16_t><<<grid, 256, 0, st>>>((uint16_t*)dst, (const uint16_t*)src, idx, n, cols);
  BLSTM_CUDA_OK(cudaGetLastError());
  count_launch();
  return BLSTM_OK;
}

int blstm_packed_maps(const int32_t* batch_sizes, const int32_t* offsets, const int64_t* rank, int T, int B, int32_t* maps, void* stream) {
  if (!batch_sizes || !offsets || !maps || T <= 0 || B <= 0) return BLSTM_E_INVALID_ARG;
  const long long n = (long long)T * B;
  if (n > INT32_MAX / 8) return BLSTM_E_INVALID_ARG;
  packed_maps_kernel<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(batch_sizes, offsets, (const long long*)rank, T, B, maps);
  BLSTM_CUDA_OK(cudaGetLastError());
  count_launch();
  return BLSTM_OK;
}

}  // extern "C"
