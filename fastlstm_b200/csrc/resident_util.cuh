// Device helpers of the recurrences with resident weights.
#pragma once

#include "sm100_rec_util.cuh"

namespace blstm {
namespace sm100 {

// A from tensor memory.
__device__ __forceinline__ void umma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// W 16-bit pairs
template <int W> __device__ __forceinline__ void ld_words(uint32_t (&r)[W], const void* p) {
  if constexpr (W == 4) { const uint4 v = ldg16(p); r[0] = v.x; r[1] = v.y; r[2] = v.z; r[3] = v.w; }
  else if constexpr (W == 2) { const uint2 v = *reinterpret_cast<const uint2*>(p); r[0] = v.x; r[1] = v.y; }
  else r[0] = *reinterpret_cast<const uint32_t*>(p);
}
template <int W> __device__ __forceinline__ void st_words(void* p, const uint32_t (&r)[W]) {
  if constexpr (W == 4) stg16(p, make_uint4(r[0], r[1], r[2], r[3]));
  else if constexpr (W == 2) *reinterpret_cast<uint2*>(p) = make_uint2(r[0], r[1]);
  else *reinterpret_cast<uint32_t*>(p) = r[0];
}
template <typename T16, int W> __device__ __forceinline__ void unpack_words(const uint32_t (&r)[W], float* f) {
#pragma unroll
  for (int w = 0; w < W; ++w) { const float2 v = cvt2<T16>(r[w]); f[2 * w] = v.x; f[2 * w + 1] = v.y; }
}
template <typename T16, int W> __device__ __forceinline__ void pack_words(uint32_t (&r)[W], const float* f) {
#pragma unroll
  for (int w = 0; w < W; ++w) r[w] = pk2<T16>(f[2 * w], f[2 * w + 1]);
}

// The weights' first nt K chunks (of 64, from chunk kc0 on) into tensor memory from column a_col on: lane = M row, a 32-bit
// column = two K elements.  Forward: M row = gate * 32 + unit of tile mt; backward: unit of tile mt.  By the eight epilogue
// warps (quarter q, half g).
template <bool BWD, typename T16>
__device__ __forceinline__ void weights_to_tmem(const T16* Wh, int H, int mt, int kc0, int nt, uint32_t a_col, int q, int g, int lane) {
  for (int lc = g; lc < nt; lc += 2) {
    const size_t k = (size_t)(kc0 + lc) * 64;
    const uint32_t col = a_col + lc * 32 + (uint32_t(q * 32) << 16);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      uint32_t v[8];
      if constexpr (!BWD) {
        const T16* src = Wh + ((size_t)q * H + mt * 32 + lane) * H + k + 16 * j;
        const uint4 a = ldg16(src), b = ldg16(src + 8);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
        v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
      } else {
        const int unit = mt * 128 + q * 32 + lane;
        const uint16_t* src = reinterpret_cast<const uint16_t*>(Wh) + (k + 16 * j) * H + unit;
#pragma unroll
        for (int i = 0; i < 8; ++i)
          v[i] = unit < H ? (uint32_t)src[(size_t)(2 * i) * H] | (uint32_t)src[(size_t)(2 * i + 1) * H] << 16 : 0u;
      }
      tmem_st_32x8(col + 8 * j, v);
    }
  }
  tmem_st_wait();
}

}  // namespace sm100
}  // namespace blstm
