// fp32 GEMM on the CUDA cores (FFMA; the tolerance of 1e-5 forbids TF32) for the layer's dense contractions: input
// projection (A and B contiguous along K), input gradient (B contiguous along N), weight gradients (both contiguous
// along M / N, split over K).
//
// The problems are small (a few thousand rows, a few hundred columns, any leading dimension), so blocks are small and
// many: 64 x 64 outputs by 64 threads of 8 x 8 (four 16-byte shared-memory reads per 64 FMAs, which are issued in pairs),
// six or more per SM; where those do not fill the GPU, K is split over blocks too.  A
// four-stage cp.async pipeline of 16 K steps feeds them; operands contiguous along K are transposed on the way in by
// 4-byte copies, the others move in 16-byte copies where their rows allow it.  Bound by the FMAs' register operands (without any
// shared-memory read in the loop 48 TFLOP/s, one FMA an issue slot 39) and, below a wave of blocks, by latency.  Measured (B200; every copy
// with checks and a 64-bit product of its own before; projection, input gradient, both weight gradients): T*B = 16384, H = I = 256:
// 214 / 211 / 435 -> 191 / 193 / 377 us (45 TFLOP/s of 74); T*B = 4400, H = I = 257: 72 / 97 / 201 -> 69 / 86 / 164 us.
#include "f32_gemm.cuh"

namespace blstm {

constexpr int FM = 64, FN = 64, FK = 16, FP = FM + 4, FST = 4;

struct F32GemmParams {
  int M, N, K, kper;        // kper: K steps per split, a multiple of FK
  const float* A;
  const float* B;
  float* C;                 // [splits][M][N]
  long long lda, ldb;
  const float* bias0;
  const float* bias1;
  int a_vec, b_vec, c_vec;  // rows allow 16-byte accesses (operands: those contiguous along M / N)
};

__device__ __forceinline__ void cp_async4(uint32_t dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const float* src, bool ok) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(ok ? 4 : 0) : "memory");
}
__device__ __forceinline__ void cp_async16z(uint32_t dst, const float* src, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0) : "memory");
}

// One operand's 64 x 16 tile into shared memory as [k][64 + 4].  A tile that lies inside the operand is fetched from
// addresses that differ between the copies by the same amount for all threads; checks and 64-bit products for each copy took as many
// issue slots as the FMAs left.
template <bool KC>
__device__ __forceinline__ void load_tile(uint32_t dst, const float* base, long long ld, int m0, int M, int k0, int k1, int vec) {
  const int t = threadIdx.x;
  if (m0 + FM <= M && k0 + FK <= k1) {
    if constexpr (KC) {
      const float* src = base + m0 * ld + k0;
      const int at = (t / FK) * (int)ld + t % FK;
      const uint32_t d = dst + ((t % FK) * FP + t / FK) * 4;
#pragma unroll
      for (int i = 0; i < FM * FK / 64; ++i) cp_async4(d + i * (64 / FK) * 4, src + (long long)(i * (64 / FK)) * ld + at);
    } else if (vec) {
      const float* src = base + k0 * ld + m0;
      const int at = (t / (FM / 4)) * (int)ld + 4 * (t % (FM / 4));
      const uint32_t d = dst + ((t / (FM / 4)) * FP + 4 * (t % (FM / 4))) * 4;
#pragma unroll
      for (int i = 0; i < FM * FK / 4 / 64; ++i) cp_async16(d + i * (256 / FM) * FP * 4, src + (long long)(i * (256 / FM)) * ld + at);
    } else {
      const float* src = base + k0 * ld + m0;
#pragma unroll
      for (int i = 0; i < FK; ++i) cp_async4(dst + (i * FP + t) * 4, src + (long long)i * ld + t);
    }
  } else if constexpr (KC) {
#pragma unroll
    for (int i = 0; i < FM * FK / 64; ++i) {
      const int idx = threadIdx.x + i * 64, k = idx % FK, m = idx / FK;
      const bool ok = m0 + m < M && k0 + k < k1;
      cp_async4(dst + (k * FP + m) * 4, ok ? base + (long long)(m0 + m) * ld + k0 + k : base, ok);
    }
  } else if (vec) {
#pragma unroll
    for (int i = 0; i < FM * FK / 4 / 64; ++i) {
      const int idx = threadIdx.x + i * 64, m = 4 * (idx % (FM / 4)), k = idx / (FM / 4);
      const bool ok = m0 + m < M && k0 + k < k1;
      cp_async16z(dst + (k * FP + m) * 4, ok ? base + (long long)(k0 + k) * ld + m0 + m : base, ok);
    }
  } else {
#pragma unroll
    for (int i = 0; i < FM * FK / 64; ++i) {
      const int m = threadIdx.x, k = i;
      const bool ok = m0 + m < M && k0 + k < k1;
      cp_async4(dst + (k * FP + m) * 4, ok ? base + (long long)(k0 + k) * ld + m0 + m : base, ok);
    }
  }
}

template <bool AKC, bool BKC>
__global__ void __launch_bounds__(64) f32_gemm_kernel(const F32GemmParams p) {
  __shared__ __align__(16) float sm[FST][2][FK * FP];
  const int m0 = blockIdx.x * FM, n0 = blockIdx.y * FN;
  const int ks = blockIdx.z * p.kper, ke = min(ks + p.kper, p.K);
  const int ty = threadIdx.x / 8, tx = threadIdx.x % 8;
  const int n_it = (ke - ks + FK - 1) / FK;
  const uint32_t sbase = static_cast<uint32_t>(__cvta_generic_to_shared(&sm[0][0][0]));
  auto fetch = [&](int it) {
    if (it < n_it) {
      const uint32_t d = sbase + (uint32_t)(it % FST) * (2 * FK * FP * 4);
      load_tile<AKC>(d, p.A, p.lda, m0, p.M, ks + it * FK, ke, p.a_vec);
      load_tile<BKC>(d + FK * FP * 4, p.B, p.ldb, n0, p.N, ks + it * FK, ke, p.b_vec);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int i = 0; i < FST - 1; ++i) fetch(i);
  float2 acc[8][4] = {};                                        // pairs of columns: two FMAs an issue slot
  for (int it = 0; it < n_it; ++it) {
    asm volatile("cp.async.wait_group %0;" ::"n"(FST - 2) : "memory");
    __syncthreads();
    fetch(it + FST - 1);
    const float* as = sm[it % FST][0];
    const float* bs = sm[it % FST][1];
#pragma unroll
    for (int k = 0; k < FK; ++k) {
      float a[8];
      float2 b[4];
      *reinterpret_cast<float4*>(&a[0]) = *reinterpret_cast<const float4*>(as + k * FP + ty * 4);
      *reinterpret_cast<float4*>(&a[4]) = *reinterpret_cast<const float4*>(as + k * FP + 32 + ty * 4);
      *reinterpret_cast<float4*>(&b[0]) = *reinterpret_cast<const float4*>(bs + k * FP + tx * 4);
      *reinterpret_cast<float4*>(&b[2]) = *reinterpret_cast<const float4*>(bs + k * FP + 32 + tx * 4);
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = __ffma2_rn(make_float2(a[i], a[i]), b[j], acc[i][j]);
    }
  }
  float* C = p.C + (size_t)blockIdx.z * p.M * p.N;
#pragma unroll
  for (int jb = 0; jb < 2; ++jb) {
    const int n = n0 + jb * 32 + tx * 4;
    float bias[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (n + j < p.N) bias[j] = (p.bias0 ? p.bias0[n + j] : 0.f) + (p.bias1 ? p.bias1[n + j] : 0.f);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int m = m0 + (i >> 2) * 32 + ty * 4 + (i & 3);
      if (m >= p.M || n >= p.N) continue;
      float* dst = C + (size_t)m * p.N + n;
      const float o[4] = {acc[i][2 * jb].x + bias[0], acc[i][2 * jb].y + bias[1], acc[i][2 * jb + 1].x + bias[2], acc[i][2 * jb + 1].y + bias[3]};
      if (p.c_vec) *reinterpret_cast<float4*>(dst) = make_float4(o[0], o[1], o[2], o[3]);
      else
        for (int j = 0; j < 4 && n + j < p.N; ++j) dst[j] = o[j];
    }
  }
}

__global__ void f32_splitk_reduce_kernel(const float* __restrict__ part, int splits, size_t n, float* __restrict__ out) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float s = 0.f;
  for (int z = 0; z < splits; ++z) s += part[(size_t)z * n + i];
  out[i] = s;
}

// Splits of a long K (time steps x rows, or gate rows for the input gradient): about eight blocks per SM, at least 128 K
// steps each.
int f32_gemm_splits(int M, int N, int K, int sm_count) {
  const long long tiles = (long long)cdiv(M, FM) * cdiv(N, FN);
  long long s = (8ll * sm_count + tiles - 1) / tiles;
  if (s > K / 128) s = K / 128;
  if (s > 64) s = 64;
  return s < 1 ? 1 : (int)s;
}

int f32_gemm(int M, int N, int K, const float* A, long long lda, bool a_kc, const float* B, long long ldb, bool b_kc, float* C,
             const float* bias0, const float* bias1, int splits, float* partials, cudaStream_t st) {
  F32GemmParams p;
  p.M = M; p.N = N; p.K = K;
  p.kper = (int)round_up((size_t)cdiv(K, splits), FK);
  splits = cdiv(K, p.kper);
  p.A = A; p.B = B; p.lda = lda; p.ldb = ldb;
  p.bias0 = bias0; p.bias1 = bias1;
  p.C = splits > 1 ? partials : C;
  auto vec = [](const float* q, long long ld, int n) { return ld % 4 == 0 && n % 4 == 0 && (reinterpret_cast<uintptr_t>(q) & 15u) == 0; };
  p.a_vec = vec(A, lda, M);
  p.b_vec = vec(B, ldb, N);
  p.c_vec = vec(p.C, N, N);
  const dim3 grid(cdiv(M, FM), cdiv(N, FN), splits);
  if (a_kc && b_kc) f32_gemm_kernel<true, true><<<grid, 64, 0, st>>>(p);
  else if (a_kc) f32_gemm_kernel<true, false><<<grid, 64, 0, st>>>(p);
  else f32_gemm_kernel<false, false><<<grid, 64, 0, st>>>(p);
  BLSTM_CUDA_OK(cudaGetLastError());
  count_launch();
  if (splits > 1) {
    const size_t n = (size_t)M * N;
    f32_splitk_reduce_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(partials, splits, n, C);
    BLSTM_CUDA_OK(cudaGetLastError());
    count_launch();
  }
  return BLSTM_OK;
}

}  // namespace blstm
