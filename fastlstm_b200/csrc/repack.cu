// Layout and type changes of a layer's tensors on the way in and out, all of them in one launch: zero padding of ragged
// sizes (and its inverse for gradients) and the conversion to the compute type under autocast.  What they replace is a
// fill and a copy per tensor, seven tensors a layer.  Bound by the launch for weights and states, by memory for x.
#include "common.cuh"

namespace blstm {

constexpr int kMaxItems = 8;

struct RepackParams {
  blstm_repack_item it[kMaxItems];
};

template <typename S, typename D>
__device__ __forceinline__ void repack(const blstm_repack_item& t) {
  const S* src = reinterpret_cast<const S*>(t.src);
  D* dst = reinterpret_cast<D*>(t.dst);
  const unsigned long long rows = (unsigned long long)t.groups * t.dst_rows;
  const unsigned long long n = rows * t.dst_cols, step = (unsigned long long)gridDim.x * blockDim.x;
  const bool same_rows = t.src_rows == t.dst_rows && t.src_cols == t.dst_cols;
  if (same_rows && n % 8 == 0 && ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15u) == 0) {
    // conversion alone: eight elements a thread in 16-byte accesses
    for (unsigned long long i = ((unsigned long long)blockIdx.x * blockDim.x + threadIdx.x) * 8; i < n; i += step * 8) {
      __align__(16) S s[8];
      __align__(16) D d[8];
#pragma unroll
      for (unsigned q = 0; q < sizeof(S) / 2; ++q) reinterpret_cast<uint4*>(s)[q] = reinterpret_cast<const uint4*>(src + i)[q];
#pragma unroll
      for (int q = 0; q < 8; ++q) d[q] = Elem<D>::from_f(Elem<S>::to_f(s[q]));
#pragma unroll
      for (unsigned q = 0; q < sizeof(D) / 2; ++q) reinterpret_cast<uint4*>(dst + i)[q] = reinterpret_cast<uint4*>(d)[q];
    }
    return;
  }
  for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += step) {
    float v = 0.f;
    if (same_rows) {
      v = Elem<S>::to_f(src[i]);
    } else {
      const unsigned long long row = i / (unsigned)t.dst_cols;
      const unsigned c = (unsigned)(i - row * (unsigned)t.dst_cols);
      const unsigned long long g = row / (unsigned)t.dst_rows;
      const unsigned r = (unsigned)(row - g * (unsigned)t.dst_rows);
      if (c < (unsigned)t.src_cols && r < (unsigned)t.src_rows) v = Elem<S>::to_f(src[(g * t.src_rows + r) * t.src_cols + c]);
    }
    dst[i] = Elem<D>::from_f(v);
  }
}

__global__ void __launch_bounds__(256) repack_kernel(const __grid_constant__ RepackParams p) {
  const blstm_repack_item& t = p.it[blockIdx.y];
  const int k = t.src_dtype * 3 + t.dst_dtype;
  if (k == BLSTM_F32 * 3 + BLSTM_F32) repack<float, float>(t);
  else if (k == BLSTM_F32 * 3 + BLSTM_F16) repack<float, __half>(t);
  else if (k == BLSTM_F32 * 3 + BLSTM_BF16) repack<float, __nv_bfloat16>(t);
  else if (k == BLSTM_F16 * 3 + BLSTM_F16) repack<__half, __half>(t);
  else if (k == BLSTM_BF16 * 3 + BLSTM_BF16) repack<__nv_bfloat16, __nv_bfloat16>(t);
  else if (k == BLSTM_F16 * 3 + BLSTM_F32) repack<__half, float>(t);
  else if (k == BLSTM_BF16 * 3 + BLSTM_F32) repack<__nv_bfloat16, float>(t);
  else if (k == BLSTM_F16 * 3 + BLSTM_BF16) repack<__half, __nv_bfloat16>(t);
  else repack<__nv_bfloat16, __half>(t);
}

}  // namespace blstm

using namespace blstm;

extern "C" int blstm_repack(const blstm_repack_item* items, int n, void* stream) {
  if (!items || n < 0 || n > kMaxItems) return BLSTM_E_INVALID_ARG;
  if (n == 0) return BLSTM_OK;
  RepackParams p{};
  unsigned long long most = 1;
  for (int i = 0; i < n; ++i) {
    const blstm_repack_item& t = items[i];
    if (!t.src || !t.dst || t.groups <= 0 || t.src_rows <= 0 || t.src_cols <= 0 || t.dst_rows <= 0 || t.dst_cols <= 0 ||
        t.src_dtype < 0 || t.src_dtype > 2 || t.dst_dtype < 0 || t.dst_dtype > 2)
      return BLSTM_E_INVALID_ARG;
    p.it[i] = t;
    const unsigned long long e = (unsigned long long)t.groups * t.dst_rows * t.dst_cols;
    if (e > most) most = e;
  }
  const unsigned long long want = (most + 1023) / 1024;          // four elements a thread, eight blocks per SM at most
  const unsigned cap = 8u * (unsigned)plan_sm_count();
  repack_kernel<<<dim3((unsigned)(want < cap ? want : cap), n), 256, 0, (cudaStream_t)stream>>>(p);
  BLSTM_CUDA_OK(cudaGetLastError());
  count_launch();
  return BLSTM_OK;
}
