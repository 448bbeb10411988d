// One timestep of a layer as ONE launch (streaming inference, decoding, T = 1): projection, recurrent product, gates and
// states.  Replaces torch.addmm + persistent_fwd_kernel of fastlstm/lstm.py:66-142 at T = 1, and here two copies, the
// projection GEMM, a memset and the recurrence.
//
// Bound by reading the weights once (4H (I + H) elements; 4 MB at I = H = 512, under a microsecond) and by the launch.
// A block owns 8 hidden units (their 32 gate rows) and all batch rows (at most 64); its 8 warps split K = I + H, so every
// weight is read by one warp of the chip and a warp's loads of a K slice are all in flight together.
#include <algorithm>

#include "sm100_common.cuh"
#include "sm100_rec_util.cuh"
#include "step.cuh"

namespace blstm {
namespace sm100 {

struct StepParams {
  int B, I, H;
  int inference;
  const void* x;            // [B,I]
  const void* h0;           // [B,H] or null
  const void* c0;
  const void* Wx;
  const void* Wh;
  const void* bx;           // [4H] or null
  const void* bh;
  void* out;                // [2,B,H]: initial and new state
  void* cell;               // [2,B,H]
  void* ifgo;               // [B,4H] (not written in inference mode)
  Control* ctl;             // zeroed for callers that read it, or null
};

// Gates of one (unit, row) from its four sums; writes the states and, for backward, the pre-activations.
template <typename T, bool FAST>
__device__ __forceinline__ void step_finish(const StepParams& p, int unit, int row, float (&a)[4]) {
  const int H = p.H;
  const T* bx = reinterpret_cast<const T*>(p.bx);
  const T* bh = reinterpret_cast<const T*>(p.bh);
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    if (bx) a[g] += ld_f(bx + g * H + unit);
    if (bh) a[g] += ld_f(bh + g * H + unit);
  }
  const size_t o = (size_t)row * H + unit, slot = (size_t)p.B * H;
  const T hp = p.h0 ? reinterpret_cast<const T*>(p.h0)[o] : Elem<T>::from_f(0.f);
  const T cp = p.c0 ? reinterpret_cast<const T*>(p.c0)[o] : Elem<T>::from_f(0.f);
  float c, h;
  if (FAST) {
    c = sigmoid_fast(a[1]) * Elem<T>::to_f(cp) + sigmoid_fast(a[0]) * tanh_fast(a[2]);
    h = sigmoid_fast(a[3]) * tanh_fast(c);
  } else {
    c = sigmoid_acc(a[1]) * Elem<T>::to_f(cp) + sigmoid_acc(a[0]) * tanh_acc(a[2]);
    h = sigmoid_acc(a[3]) * tanh_acc(c);
  }
  T* out = reinterpret_cast<T*>(p.out);
  T* cell = reinterpret_cast<T*>(p.cell);
  out[o] = hp;
  cell[o] = cp;
  out[slot + o] = Elem<T>::from_f(h);
  cell[slot + o] = Elem<T>::from_f(c);
  if (!p.inference) {
    T* ifgo = reinterpret_cast<T*>(p.ifgo) + (size_t)row * 4 * H + unit;
#pragma unroll
    for (int g = 0; g < 4; ++g) ifgo[(size_t)g * H] = Elem<T>::from_f(a[g]);
  }
}

template <typename T16>
__device__ __forceinline__ void step_mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  if constexpr (sizeof(T16) == 2 && __is_same(T16, __half))
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  else
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// 16-bit.  NT: n-tiles of 8 batch rows.  Both operands come straight from global memory in 16-byte pieces: the order of K
// inside an MMA is free, so lane 4u+c takes k = 8c .. 8c+7 of every 32 of weight row u and of batch row u.
template <int NT, typename T16>
__global__ void __launch_bounds__(256) step16_kernel(const StepParams p) {
  extern __shared__ __align__(16) float red[];                  // [8 warps][2 tiles][NT][32 lanes][4]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, u = lane >> 2, c = lane & 3;
  const int H = p.H, unit0 = blockIdx.x * 8;
  if (p.ctl && blockIdx.x == 0 && threadIdx.x < sizeof(Control) / 4) reinterpret_cast<int*>(p.ctl)[threadIdx.x] = 0;
  const int nbi = (p.I + 31) / 32, nb = nbi + (p.h0 ? (H + 31) / 32 : 0);
  float acc[2][NT][4] = {};
#pragma unroll 2
  for (int blk = warp; blk < nb; blk += 8) {
    const bool rec = blk >= nbi;
    const int K = rec ? H : p.I, k = (rec ? blk - nbi : blk) * 32 + 8 * c;
    const T16* W = reinterpret_cast<const T16*>(rec ? p.Wh : p.Wx) + (size_t)(unit0 + u) * K + k;
    const T16* X = reinterpret_cast<const T16*>(rec ? p.h0 : p.x) + (size_t)u * K + k;
    const bool ok = k < K;
    uint4 w[4], b[NT];
#pragma unroll
    for (int g = 0; g < 4; ++g) w[g] = ok ? ldg16(W + (size_t)g * H * K) : make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) b[nt] = (ok && nt * 8 + u < p.B) ? ldg16(X + (size_t)nt * 8 * K) : make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        step_mma<T16>(acc[t][nt], w[2 * t].x, w[2 * t + 1].x, w[2 * t].y, w[2 * t + 1].y, b[nt].x, b[nt].y);
        step_mma<T16>(acc[t][nt], w[2 * t].z, w[2 * t + 1].z, w[2 * t].w, w[2 * t + 1].w, b[nt].z, b[nt].w);
      }
  }
#pragma unroll
  for (int t = 0; t < 2; ++t)
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
      *reinterpret_cast<float4*>(red + (((warp * 2 + t) * NT + nt) * 32 + lane) * 4) = make_float4(acc[t][nt][0], acc[t][nt][1], acc[t][nt][2], acc[t][nt][3]);
  __syncthreads();
  // thread = (unit, row): lane 4u + row/2 of n-tile row/8 holds gates (2t, 2t+1) at positions row%2 and 2 + row%2
  for (int i = threadIdx.x; i < 8 * p.B; i += 256) {
    const int un = i & 7, row = i >> 3, nt = row >> 3, l = un * 4 + ((row & 7) >> 1), e = row & 1;
    float a[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int w8 = 0; w8 < 8; ++w8)
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        const float* q = red + (((w8 * 2 + t) * NT + nt) * 32 + l) * 4 + e;
        a[2 * t] += q[0];
        a[2 * t + 1] += q[2];
      }
    step_finish<T16, true>(p, unit0 + un, row, a);
  }
}

// fp32 (FFMA).  NR: batch rows of a block (blockIdx.y).  Warp = one unit: lanes split K (one or four elements each), every lane
// multiplies its piece of the unit's four gate rows with NR rows of x or h; shuffles add the lanes up.
template <int NR, bool VEC>
__global__ void __launch_bounds__(256) step32_kernel(const StepParams p) {
  constexpr int V = VEC ? 4 : 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int H = p.H, unit = blockIdx.x * 8 + warp;
  if (p.ctl && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x < sizeof(Control) / 4) reinterpret_cast<int*>(p.ctl)[threadIdx.x] = 0;
  if (unit >= H) return;
  const int r0 = blockIdx.y * NR;
  {
    float acc[4][NR] = {};
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      if (half && !p.h0) break;
      const int K = half ? H : p.I;
      const float* W = reinterpret_cast<const float*>(half ? p.Wh : p.Wx) + (size_t)unit * K;
      const float* X = reinterpret_cast<const float*>(half ? p.h0 : p.x) + (size_t)r0 * K;
#pragma unroll 2
      for (int k = lane * V; k < K; k += 32 * V) {
        float w[4][V], xv[NR][V];
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          if constexpr (VEC) *reinterpret_cast<float4*>(w[g]) = *reinterpret_cast<const float4*>(W + (size_t)g * H * K + k);
          else w[g][0] = W[(size_t)g * H * K + k];
        }
#pragma unroll
        for (int r = 0; r < NR; ++r) {
          const bool ok = r0 + r < p.B;
          if constexpr (VEC) *reinterpret_cast<float4*>(xv[r]) = ok ? *reinterpret_cast<const float4*>(X + (size_t)r * K + k) : make_float4(0.f, 0.f, 0.f, 0.f);
          else xv[r][0] = ok ? X[(size_t)r * K + k] : 0.f;
        }
#pragma unroll
        for (int v = 0; v < V; ++v)
#pragma unroll
          for (int r = 0; r < NR; ++r)
#pragma unroll
            for (int g = 0; g < 4; ++g) acc[g][r] = fmaf(w[g][v], xv[r][v], acc[g][r]);
      }
    }
#pragma unroll
    for (int r = 0; r < NR; ++r)
#pragma unroll
      for (int g = 0; g < 4; ++g)
#pragma unroll
        for (int m = 16; m >= 1; m >>= 1) acc[g][r] += __shfl_xor_sync(0xffffffffu, acc[g][r], m);
#pragma unroll
    for (int r = 0; r < NR; ++r)
      if (lane == r && r0 + r < p.B) {
        float a[4] = {acc[0][r], acc[1][r], acc[2][r], acc[3][r]};
        step_finish<float, false>(p, unit, r0 + r, a);
      }
  }
}

template <typename T16>
static int launch_step16(const StepParams& p, cudaStream_t st) {
  const int nt = cdiv(p.B, 8), grid = p.H / 8;
#define BLSTM_STEP(N)                                                                                                          \
  if (nt <= N) {                                                                                                               \
    const size_t smem = (size_t)8 * 2 * N * 512;                                                                               \
    if (smem > 48 * 1024) BLSTM_CUDA_OK(cudaFuncSetAttribute(step16_kernel<N, T16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)); \
    step16_kernel<N, T16><<<grid, 256, smem, st>>>(p);                                                                         \
    BLSTM_CUDA_OK(cudaGetLastError());                                                                                         \
    count_launch();                                                                                                            \
    return BLSTM_OK;                                                                                                           \
  }
  BLSTM_STEP(1)
  BLSTM_STEP(2)
  BLSTM_STEP(4)
  BLSTM_STEP(8)
#undef BLSTM_STEP
  return BLSTM_E_UNSUPPORTED;
}

}  // namespace sm100

using namespace sm100;

// Up to 64 rows: beyond, the weights are no longer what is read, and the GEMM's tiles reuse the activations.  (16-bit sizes
// in 16-byte pieces; other sizes take the general path.)
bool step_supported(const blstm_desc& d) {
  if (d.seq_len != 1 || d.batch > 64 || (d.flags & (BLSTM_FLAG_FORCE_GENERIC | BLSTM_FLAG_NO_FUSED))) return false;
  return d.dtype == BLSTM_F32 || (d.input_size % 8 == 0 && d.hidden_size % 8 == 0);
}

int step_fwd(const blstm_desc& d, const void* x, const void* h0, const void* c0, const void* Wx, const void* Wh, const void* bx,
             const void* bh, void* out, void* cell, void* ifgo, Control* ctl, cudaStream_t st) {
  StepParams p;
  p.B = d.batch; p.I = d.input_size; p.H = d.hidden_size;
  p.inference = (d.flags & BLSTM_FLAG_INFERENCE) ? 1 : 0;
  p.x = x; p.h0 = h0; p.c0 = c0; p.Wx = Wx; p.Wh = Wh; p.bx = bx; p.bh = bh;
  p.out = out; p.cell = cell; p.ifgo = ifgo; p.ctl = ctl;
  if (d.dtype == BLSTM_F16) return launch_step16<__half>(p, st);
  if (d.dtype == BLSTM_BF16) return launch_step16<__nv_bfloat16>(p, st);
  uintptr_t m = reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(h0) | reinterpret_cast<uintptr_t>(Wx) | reinterpret_cast<uintptr_t>(Wh);
  const bool vec = p.I % 4 == 0 && p.H % 4 == 0 && (m & 15u) == 0;
  const dim3 grid(cdiv(p.H, 8), cdiv(p.B, p.B <= 2 ? 2 : 8));
  if (p.B <= 2) { if (vec) step32_kernel<2, true><<<grid, 256, 0, st>>>(p); else step32_kernel<2, false><<<grid, 256, 0, st>>>(p); }
  else          { if (vec) step32_kernel<8, true><<<grid, 256, 0, st>>>(p); else step32_kernel<8, false><<<grid, 256, 0, st>>>(p); }
  BLSTM_CUDA_OK(cudaGetLastError());
  count_launch();
  return BLSTM_OK;
}

}  // namespace blstm
