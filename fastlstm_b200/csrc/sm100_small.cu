// Recurrences for batches that leave the tensor pipe idle (16-bit): what bounds a step there is the chain
// h[t] -> product -> gates -> h[t+1], not arithmetic and not memory.  (Replaces persistent_fwd_kernel and
// lstm_persistent_seq_bwd, fastlstm/kernels.py:414-663 and :1201-1409, and their global-memory handshakes for
// these shapes.)
//
// A cluster of NC CTAs (1 to 16, by the hidden size) owns a few batch rows and ALL hidden units; nothing is
// exchanged between clusters, so there are no global counters, no polling and no co-residency to guarantee.
// Inside a cluster:
//   - the recurrent weights stay on the chip for the whole sequence, as mma.sync A fragments in registers (up
//     to 128 of a thread's) and the rest in fragment order in shared memory: gate rows (forward) or output
//     units (backward) are the MMA's M, so a tile of 8 batch rows is a full N - the tcgen05 kernels pad a batch
//     to M = 128 rows and pass every product through tensor memory, which costs them 5-10 k clocks a step
//     whatever the batch;
//   - a thread ends the product with all four gates of its unit and two rows: no shuffles before the gates;
//   - results go to the peers' shared memory with st.async, whose bytes complete the peers' mbarriers: one way
//     through the cluster takes ~0.5 k clocks (an all-to-all of 16 x 512 B, 1.3 k clocks with the waits), where
//     store -> release -> counter -> poll -> TMA through L2 takes 4-6 k.
// Rows are worked in chunks of 8 with barriers of their own, so that with several chunks per cluster one
// chunk's exchange hides behind the others' products.
// What it measured: at small_plan_pays below.
#include <stdio.h>
#include <algorithm>
#include <atomic>

#include "sm100.cuh"
#include "sm100_common.cuh"
#include "cluster_util.cuh"
#include "sm100_rec_util.cuh"
#include "generic.cuh"
#include "sm100_small.cuh"

namespace blstm {
namespace sm100 {

// ---------------------------------------------------------------- primitives
template <typename T16>
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1);
template <>
__device__ __forceinline__ void mma16816<__half>(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
template <>
__device__ __forceinline__ void mma16816<__nv_bfloat16>(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldmatrix_x4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
// Transposes an 8x8 matrix of 16-bit values held one pair per lane: lane 4u+c goes from (row u, columns 2c,
// 2c+1) to (column u, rows 2c, 2c+1).
__device__ __forceinline__ uint32_t transpose8x8(uint32_t v) {
  uint32_t r;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(v));
  return r;
}
__device__ __forceinline__ uint32_t ldg4(const void* p) { return *reinterpret_cast<const uint32_t*>(p); }
__device__ __forceinline__ void stg4(void* p, uint32_t v) { *reinterpret_cast<uint32_t*>(p) = v; }
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldmatrix_x2_trans(uint32_t addr, uint32_t& r0, uint32_t& r1) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];" : "=r"(r0), "=r"(r1) : "r"(addr) : "memory");
}
__device__ __forceinline__ void stmatrix_x4_trans(uint32_t addr, uint32_t r0, uint32_t r1, uint32_t r2, uint32_t r3) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1,%2,%3,%4};"
               ::"r"(addr), "r"(r0), "r"(r1), "r"(r2), "r"(r3) : "memory");
}
__device__ __forceinline__ void stmatrix_x2_trans(uint32_t addr, uint32_t r0, uint32_t r1) {
  asm volatile("stmatrix.sync.aligned.m8n8.x2.trans.shared.b16 [%0], {%1,%2};" ::"r"(addr), "r"(r0), "r"(r1) : "memory");
}
__device__ __forceinline__ uint4 ld_shared16(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}

// Swizzle of the item slots' rows (the tensor maps use the same): 64- and 128-byte rows would put the 8 rows of an
// ldmatrix into the same banks; the other widths (16 bytes times 1, 3, 5, 6, 7) do not need one.
__host__ __device__ constexpr int slot_swizzle(int gc) { return gc == 4 ? 64 : gc == 8 ? 128 : 0; }
__device__ __forceinline__ uint32_t swz(uint32_t off, int gc) {
  return off ^ ((off >> 3) & (gc == 8 ? 0x70u : gc == 4 ? 0x30u : 0u));
}

// =====================================================================================
// Forward.  Warp = 8 units x 4 gates: MMA tile 0 holds gate i (rows 0-7) and f (8-15), tile 1 gates g and o, so
// lane 4u+c ends with the four gates of unit u for batch rows 2c, 2c+1 of the n-tile.  `rpl` replicas of the
// CTA's gc warps (same weights) take the chunks in turn: one's gate maths overlaps the other's MMAs.
// All global traffic goes through TMA and a ring of item slots,
//     [gate i f g o | h | c][row][the CTA's units]:
// the pre-activations land in the first four parts, ldmatrix.trans turns them into the accumulator's layout, the
// final ones are written back in place (stmatrix.trans) next to h and c, and leave from there.  A warp of its own
// issues the boxes: loads and stores by the computing warps (32 lines an instruction) put 0.5 k clocks on a chain
// of 1.5 k, TMA issues by one of them 0.6 k.
//   warps 0 .. gc*rpl-1 (of 8)   computing, up to 232 registers
//   warp 8                       TMA (9 to 11 idle: register shares go by warpgroup)
// KR: K steps (of 16) whose fragments live in a warp's registers (8 registers a step); the rest are read from shared
// memory.  KSPL = 2 (256 < H <= 512): two warps per 8 units, each with half of K - all of it in registers - which take
// turns at passing their partial sums on and at finishing an item.
// =====================================================================================
template <int KR, int KSPL, bool CL, typename T16>
__global__ void __launch_bounds__(384, 1)
small_fwd_kernel(const __grid_constant__ CUtensorMap tmP, const __grid_constant__ CUtensorMap tmH,
                 const __grid_constant__ CUtensorMap tmC, const SmallFwdParams p) {
  constexpr int CR = 8;                                         // rows of a chunk
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const int H = p.H, T = p.T, B = p.B, KS = p.ks, gc = p.gc;
  const int pitch = KS * 32 + 16;                               // (odd number of 16-byte pieces: no bank conflicts)
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int u = lane >> 2, c = lane & 3;
  const int rank = CL ? (int)cluster_ctarank() : 0;
  const int cl = CL ? blockIdx.x / p.nc : blockIdx.x;
  const int gl = warp % gc, kh = KSPL == 2 ? warp / gc : 0, rep = KSPL == 2 ? 0 : warp / gc;
  const int S = p.slots;                                        // of the ring, a power of two
  const int unit0 = (rank * gc + gl) * 8;
  const bool live = unit0 < H;
  const int row0 = cl * p.rows;
  const int rows = min(p.rows, B - row0);                       // rows of this cluster
  const int nch = rows > 0 ? (rows + CR - 1) / CR : 0;

  // shared memory: ring | h tiles [chunk][parity][CR][pitch] | cell states | weights past KR steps | barriers
  const uint32_t part = (uint32_t)CR * gc * 16, slot_b = 6 * part;
  const uint32_t h_off = (uint32_t)S * slot_b;
  const uint32_t c_off = h_off + (uint32_t)p.nch * 2 * CR * pitch;
  const uint32_t w_off = c_off + (uint32_t)p.nch * gc * 256;
  const uint32_t b_off = w_off + (uint32_t)gc * (KSPL == 2 ? 2 : KS - KR) * 1024;
  uint64_t* hbar = reinterpret_cast<uint64_t*>(smem + b_off);   // [chunk][parity] h complete
  uint64_t* full = hbar + 2 * SB_MAX_CHUNKS;                    // [S] slot filled
  uint64_t* staged = full + SB_MAX_SLOTS;                       // [S] slot's results in place
  uint64_t* pbar = staged + SB_MAX_SLOTS;                       // [gl][item parity] partial sums passed on
  volatile int* dead = reinterpret_cast<volatile int*>(pbar + 8);
  float4* psum = reinterpret_cast<float4*>(smem + w_off) + gl * 64 + lane;   // [item parity][gl][tile][lane] (K split; no weights there)
  float2* cst = reinterpret_cast<float2*>(smem + c_off) + gl * 32 + lane;   // [chunk][gl][lane]
  const uint4* w_s = reinterpret_cast<const uint4*>(smem + w_off) + (size_t)gl * (KS - KR) * 64 + lane;
  const uint32_t sbase = smem_u32(smem);
  const T16* out = reinterpret_cast<const T16*>(p.out);
  const T16* cell = reinterpret_cast<const T16*>(p.cell);
  const T16* Wh = reinterpret_cast<const T16*>(p.Wh);
  const int mych = nch > rep ? (nch - rep + p.rpl - 1) / p.rpl : 0;
  const int last_ch = rep + (mych - 1) * p.rpl;

  if (threadIdx.x == 0) {
    *dead = 0;
    for (int i = 0; i < 2 * nch; ++i) mbar_init(&hbar[i], CL ? 1 : gc);
    for (int i = 0; i < S; ++i) { mbar_init(&full[i], 1); mbar_init(&staged[i], gc); }
    for (int i = 0; i < 8; ++i) mbar_init(&pbar[i], 1);
    fence_mbar_init();
    if (CL)
      for (int i = 0; i < 2 * nch; ++i) mbar_expect_tx(&hbar[i], 2 * H * min(CR, rows - (i >> 1) * CR));
  }
  // ---- initial h: the whole tile of every chunk (zeros past B and past H)
  for (int i = threadIdx.x; i < p.nch * 2 * CR * (pitch / 16); i += blockDim.x) {
    const int kp = i % (pitch / 16), r = i / (pitch / 16);      // r = (chunk*2 + parity)*CR + row
    const int row = (r / (2 * CR)) * CR + r % CR;
    uint4 v = make_uint4(0, 0, 0, 0);
    if ((r / CR) % 2 == 0 && row < rows && kp * 8 < H) v = ldg16(out + (size_t)(row0 + row) * H + kp * 8);
    *reinterpret_cast<uint4*>(smem + h_off + (size_t)i * 16) = v;
  }
  __syncthreads();
  if (CL) cluster_sync_all();                                   // every peer's barriers exist, every tile is in place

  if (warp >= 8) {
    // ---------------------------------------------------------------- TMA: items in the order (t, chunk)
    regs_dec<40>();
    if (warp == 8 && lane == 0) {
      const int n = nch * T, x = rank * gc * 8;
      int lt = 0, lch = 0, t = 0, ch = 0;
      auto load = [&](int k) {
        if (k >= n) return;
        uint64_t* bar = &full[k & (S - 1)];
        mbar_expect_tx(bar, 4 * part);
        tma_load_4d(smem + (size_t)(k & (S - 1)) * slot_b, &tmP, bar, x, row0 + lch * CR, 0, lt);
        if (++lch == nch) { lch = 0; ++lt; }
      };
      for (int k = 0; k < S; ++k) load(k);
      for (int k = 0; k < n; ++k) {
        if (!wait_inline(&staged[k & (S - 1)], (uint32_t)(k / S) & 1u, dead, p.ctl, p.limit_ns, t, cl)) break;
        fence_proxy_async_smem();                               // the computing warps' stores, before the TMA unit reads them
        const uint8_t* sl = smem + (size_t)(k & (S - 1)) * slot_b;
        const int y = row0 + ch * CR;
        tma_store_3d(&tmH, sl + 4 * part, x, y, t + 1);
        if (!p.inference || t == T - 1) tma_store_3d(&tmC, sl + 5 * part, x, y, t + 1);
        if (!p.inference) tma_store_4d(&tmP, sl, x, y, 0, t);
        tma_store_commit();
        if (++ch == nch) { ch = 0; ++t; }
        if (k > 0) {                                            // the item before this one has left its slot
          tma_store_wait_read<1>();
          load(k - 1 + S);
        }
      }
      tma_store_wait<0>();
    }
  } else {
  regs_inc<232>();
  if (warp < gc * KSPL * p.rpl) {
  // ---- weights: A fragments straight from global memory (rows past H and columns past H are zero)
  uint32_t w[KR][2][4];
  {
    auto frag = [&](int ks, int tile, uint32_t (&a)[4]) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int g = 2 * tile + (i & 1), k = (kh * KR + ks) * 16 + 2 * c + (i >> 1) * 8;
        a[i] = (live && k < H) ? ldg4(Wh + ((size_t)g * H + unit0 + u) * H + k) : 0u;
      }
    };
#pragma unroll
    for (int ks = 0; ks < KR; ++ks) { frag(ks, 0, w[ks][0]); frag(ks, 1, w[ks][1]); }
    if (KSPL == 1 && rep == 0)
      for (int ks = KR; ks < KS; ++ks)
        for (int tile = 0; tile < 2; ++tile) {
          uint32_t a[4];
          frag(ks, tile, a);
          const_cast<uint4*>(w_s)[((ks - KR) * 2 + tile) * 32] = make_uint4(a[0], a[1], a[2], a[3]);
        }
  }
  // ---- own cell states
  for (int ch = rep; ch < nch; ch += p.rpl) {
    const int r = ch * CR + u;
    const uint32_t v = (live && r < rows) ? ldg4(cell + (size_t)(row0 + r) * H + unit0 + 2 * c) : 0u;
    cst[ch * gc * 32] = cvt2<T16>(transpose8x8(v));
  }
  // the shared-memory weights are in place (all computing warps come here, before anything can give up)
  asm volatile("bar.sync 1, %0;" ::"r"(32 * gc * KSPL * p.rpl) : "memory");
  // shared::cluster addresses of this lane's destinations: CTAs c, c+4, c+8, c+12
  uint32_t peer[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) peer[i] = CL ? mapa_shared(sbase, min(c + 4 * i, p.nc - 1)) : sbase;
  // this lane's places in a slot: row (lane & 7) of gate (lane >> 3) and of h / c for the matrix accesses, row u of h
  const uint32_t so_g = swz((lane >> 3) * part + (lane & 7) * gc * 16 + gl * 16, gc);
  const uint32_t so_hc = swz((4 + ((lane >> 3) & 1)) * part + (lane & 7) * gc * 16 + gl * 16, gc);
  const uint32_t so_h = swz(4 * part + u * gc * 16 + gl * 16, gc);

  for (int t = 0, ch = rep; mych > 0 && t < T;) {
    const int par = t & 1, k = t * nch + ch;                    // item number
    const uint32_t sl = sbase + (uint32_t)(k & (S - 1)) * slot_b;
    // K split: the halves take turns at finishing an item (gates, sends)
    const bool finish = KSPL == 1 || (k & 1) == kh;
    if (finish && !wait_inline(&full[k & (S - 1)], (uint32_t)(k / S) & 1u, dead, p.ctl, p.limit_ns, t, cl)) break;
    uint32_t pw[4] = {0, 0, 0, 0};
    if (finish) ldmatrix_x4_trans(sl + so_g, pw);
    float acc[2][2][4] = {};                                    // [K parity][tile]
    float2 cs = cst[ch * gc * 32];
    if (t > 0) {
      uint64_t* bar = &hbar[2 * ch + par];
      if (!wait_inline(bar, (uint32_t)((t - 1) >> 1) & 1u, dead, p.ctl, p.limit_ns, t, cl)) break;
      if (CL && gl == 0 && lane == 0 && finish && t + 2 < T) mbar_expect_tx(bar, 2 * H * min(CR, rows - ch * CR));   // its next use
    }
    // operand fetches run ahead of the MMAs (one at a time they cost as much as the MMAs)
    const uint32_t hb = sbase + h_off + (uint32_t)((ch * 2 + par) * CR + (lane & 7)) * pitch + (lane >> 3) * 16 + kh * KR * 32;
    constexpr int AH = KR / 2 < 3 ? KR / 2 : 3;
    uint32_t b[AH + 1][4];
#pragma unroll
    for (int i = 0; i < AH; ++i)
      ldmatrix_x4(hb + i * 64, b[i]);
#pragma unroll
    for (int i = 0; i < KR / 2; ++i) {
      if (i + AH < KR / 2) {
        ldmatrix_x4(hb + (i + AH) * 64, b[(i + AH) % (AH + 1)]);
      }
      const uint32_t(&bb)[4] = b[i % (AH + 1)];
      mma16816<T16>(acc[0][0], w[2 * i][0], bb[0], bb[1]);
      mma16816<T16>(acc[0][1], w[2 * i][1], bb[0], bb[1]);
      mma16816<T16>(acc[1][0], w[2 * i + 1][0], bb[2], bb[3]);
      mma16816<T16>(acc[1][1], w[2 * i + 1][1], bb[2], bb[3]);
    }
    if constexpr (KSPL == 1) {
#pragma unroll 2
      for (int ks = KR; ks < KS; ks += 2) {                     // weights in shared memory
        uint32_t a[2][2][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint4 v = w_s[((ks - KR) * 2 + i) * 32];
          a[i >> 1][i & 1][0] = v.x; a[i >> 1][i & 1][1] = v.y; a[i >> 1][i & 1][2] = v.z; a[i >> 1][i & 1][3] = v.w;
        }
        uint32_t bb[4];
        ldmatrix_x4(hb + ks * 32, bb);
        mma16816<T16>(acc[0][0], a[0][0], bb[0], bb[1]);
        mma16816<T16>(acc[0][1], a[0][1], bb[0], bb[1]);
        mma16816<T16>(acc[1][0], a[1][0], bb[2], bb[3]);
        mma16816<T16>(acc[1][1], a[1][1], bb[2], bb[3]);
      }
    } else {
      // the other half's partial sums: passed on through shared memory, or taken
#pragma unroll
      for (int tile = 0; tile < 2; ++tile)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[0][tile][e] += acc[1][tile][e];
      float4* ps = psum + (k & 1) * gc * 64;
      if (!finish) {
        ps[0] = make_float4(acc[0][0][0], acc[0][0][1], acc[0][0][2], acc[0][0][3]);
        ps[32] = make_float4(acc[0][1][0], acc[0][1][1], acc[0][1][2], acc[0][1][3]);
        __syncwarp();
        if (lane == 0) mbar_arrive(&pbar[2 * gl + (k & 1)]);
        if (ch == last_ch) { ch = rep; ++t; } else ch += p.rpl;
        continue;
      }
      if (!wait_inline(&pbar[2 * gl + (k & 1)], (uint32_t)(k >> 1) & 1u, dead, p.ctl, p.limit_ns, t, cl)) break;
      const float4 o0 = ps[0], o1 = ps[32];
      acc[1][0][0] = o0.x; acc[1][0][1] = o0.y; acc[1][0][2] = o0.z; acc[1][0][3] = o0.w;
      acc[1][1][0] = o1.x; acc[1][1][1] = o1.y; acc[1][1][2] = o1.z; acc[1][1][3] = o1.w;
      cs = cst[ch * gc * 32];                                // (the other half may have written it)
    }
    uint32_t gw[4];
    float g4[4][2];
#pragma unroll
    for (int g = 0; g < 4; ++g)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const float2 f = cvt2<T16>(pw[g]);
        g4[g][e] = acc[0][g >> 1][(g & 1) * 2 + e] + acc[1][g >> 1][(g & 1) * 2 + e] + (e ? f.y : f.x);
      }
    float hv[2], cv[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      cv[e] = sigmoid_fast(g4[1][e]) * (e ? cs.y : cs.x) + sigmoid_fast(g4[0][e]) * tanh_fast(g4[2][e]);
      hv[e] = sigmoid_fast(g4[3][e]) * tanh_fast(cv[e]);
    }
    // h and c as rows of 8 units (16 bytes); row u's h goes to the whole cluster
    stmatrix_x2_trans(sl + so_hc, pk2<T16>(hv[0], hv[1]), pk2<T16>(cv[0], cv[1]));
    __syncwarp();
    const uint4 v = ld_shared16(sl + so_h);
    const uint32_t ho = h_off + (uint32_t)((ch * 2 + (par ^ 1)) * CR + u) * pitch + unit0 * 2;
    if (live && ch * CR + u < rows && t + 1 < T && !p.no_arrive) {
      if (CL) {
        const uint32_t bo = b_off + (uint32_t)(2 * ch + (par ^ 1)) * 8;
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (c + 4 * i < p.nc) st_async16(peer[i] + ho, v, peer[i] + bo);
      } else if (c == 0) {
        st_shared16(sbase + ho, v);
      }
    }
    cst[ch * gc * 32] = make_float2(cv[0], cv[1]);
#pragma unroll
    for (int g = 0; g < 4; ++g) gw[g] = pk2<T16>(g4[g][0], g4[g][1]);
    if (!CL) {
      __syncwarp();
      if (lane == 0) mbar_arrive(&hbar[2 * ch + (par ^ 1)]);
    }
    // off the chain: the final pre-activations in place, and the previous item's boxes on their way
    if (!p.inference) {
      stmatrix_x4_trans(sl + so_g, gw[0], gw[1], gw[2], gw[3]);
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&staged[k & (S - 1)]);
    if (ch == last_ch) { ch = rep; ++t; } else ch += p.rpl;
  }
  }
  }
  __syncthreads();
  if (CL) cluster_sync_all();                                   // nobody leaves while a peer may still write here
}

// =====================================================================================
// Backward.  dh[t-1] = d_ifgo[t] x Wh is split by K: a CTA multiplies its own units' d_ifgo (4 gates x 8 gc rows
// of Wh, never exchanged) into partial sums for ALL H units, and sends each 8-unit group to the CTA that owns it,
// where the NC partial sums are added in a fixed order.  Half the bytes of gathering d_ifgo instead, and the
// weights are the forward's slice.  MMA: M = 16 output units, K = the CTA's gate rows, N = 8 batch rows.
//   warps 0 .. gc-1     gate maths of 8 units each: sums of the partial dh, d_ifgo into the product's operand buffer
//   warps 8 .. 8+nm-1   products: MPW M tiles each, KR K steps of them in registers (4 MPW KR), the rest in shared memory
//   warp 7 (one CTA: 12) TMA
// The two meet at barriers over two operand buffers, so with several chunks both are busy.  Global traffic as in
// the forward kernel: slots [gate i f g o | c | dout][row][units], d_ifgo written back over the gates.
// =====================================================================================
template <int MPW, int KR, bool CL, typename T16>
__global__ void __launch_bounds__(512, 1)
small_bwd_kernel(const __grid_constant__ CUtensorMap tmP, const __grid_constant__ CUtensorMap tmC,
                 const __grid_constant__ CUtensorMap tmO, const __grid_constant__ CUtensorMap tmD, const SmallBwdParams p) {
  constexpr int CR = 8;                                         // rows of a chunk
  constexpr int S = 8;                                          // slots of the ring
  // A single tile per warp splits its K steps over two accumulators (a chain of 16 MMAs takes 350 clocks)
  constexpr int NA = MPW == 1 ? 2 : 1;
  // All K steps in registers but for five groups of units a CTA and, in one CTA, fewer than eight: elsewhere the number of
  // groups follows from KR, and a step with addresses known at compile time takes less (us, H = 384, B = 168: 2.30 -> 2.07; H = 256,
  // B = 64: 0.95 -> 0.89; H = 512, B = 128: 2.40 both; with five groups H = 640, B = 50: 2.25 -> 2.15, B = 100: 3.0 -> 3.2).
  constexpr bool TAIL = CL ? MPW == 5 : KR < 16;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const int H = p.H, T = p.T, B = p.B, gc = TAIL ? p.gc : KR / 2;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int u = lane >> 2, c = lane & 3;
  const int rank = CL ? (int)cluster_ctarank() : 0;
  const int cl = CL ? blockIdx.x / p.nc : blockIdx.x;
  const int row0 = cl * p.rows;
  const int rows = min(p.rows, B - row0);
  const int nch = rows > 0 ? (rows + CR - 1) / CR : 0;
  const int pitch = gc * 64 + 16;
  const int nm = p.mgroups;                                     // product warps
  const int lunits = min(gc * 8, max(0, H - rank * gc * 8));    // units this CTA owns

  // shared memory: ring | operand buffers [2][CR][pitch] | partial sums [chunk][parity][src][gc*8][8] | states | weights | barriers
  const uint32_t part = (uint32_t)CR * gc * 16, slot_b = 6 * part;
  const uint32_t src_b = (uint32_t)gc * 256;                    // bytes of one source's partial sums
  const uint32_t d_off = S * slot_b;
  const uint32_t r_off = d_off + 2u * CR * pitch;
  const uint32_t s_off = r_off + (uint32_t)p.nch * 2 * p.nc * src_b;
  const uint32_t w_off = s_off + (uint32_t)p.nch * gc * 512;
  const uint32_t b_off = w_off + (uint32_t)nm * MPW * (gc - KR / 2) * 1024;
  uint64_t* xbar = reinterpret_cast<uint64_t*>(smem + b_off);   // [chunk][parity] partial sums complete
  uint64_t* full = xbar + 2 * SB_MAX_CHUNKS;                    // [S] slot filled
  uint64_t* staged = full + S;                                  // [S] slot's d_ifgo in place
  uint64_t* dfull = staged + S;                                 // [2] operand buffer written
  uint64_t* dempty = dfull + 2;                                 // [2] ... and read
  volatile int* dead = reinterpret_cast<volatile int*>(dempty + 2);
  const uint32_t sbase = smem_u32(smem);
  const T16* Wh = reinterpret_cast<const T16*>(p.Wh);

  for (uint32_t i = threadIdx.x; i < (w_off - d_off) / 16; i += blockDim.x)
    *reinterpret_cast<uint4*>(smem + d_off + (size_t)i * 16) = make_uint4(0, 0, 0, 0);
  auto expect = [&](int ch) {                                   // bytes a chunk's partial sums bring in
    return p.nc * lunits * 16 * ((min(CR, rows - ch * CR) + 3) / 4);
  };
  if (threadIdx.x == 0) {
    *dead = 0;
    for (int i = 0; i < S; ++i) { mbar_init(&full[i], 1); mbar_init(&staged[i], gc); }
    for (int i = 0; i < 2; ++i) { mbar_init(&dfull[i], gc); mbar_init(&dempty[i], nm); }
    for (int i = 0; i < 2 * nch; ++i) mbar_init(&xbar[i], CL ? 1 : nm);
    fence_mbar_init();
    if (CL)
      for (int i = 0; i < 2 * nch; ++i) mbar_expect_tx(&xbar[i], expect(i >> 1));
    tma_prefetch_desc(&tmP);
    tma_prefetch_desc(&tmC);
    tma_prefetch_desc(&tmO);
    tma_prefetch_desc(&tmD);
  }
  __syncthreads();
  if (CL) cluster_sync_all();

  // Roles and register shares by warpgroup: gates and TMA | gates | products | products, or (one CTA) gates | gates |
  // products | TMA.
  auto tma_role = [&]() {
    // ---------------------------------------------------------------- TMA: items in the order (step, chunk)
    if (lane == 0) {
      const int n = nch * T, x = rank * gc * 8;
      int lt = T - 1, lch = 0, t = T - 1, ch = 0;
      auto load = [&](int k) {
        if (k >= n) return;
        uint64_t* bar = &full[k & (S - 1)];
        uint8_t* sl = smem + (size_t)(k & (S - 1)) * slot_b;
        const int y = row0 + lch * CR;
        mbar_expect_tx(bar, slot_b);
        tma_load_4d(sl, &tmP, bar, x, y, 0, lt);
        tma_load_3d(sl + 4 * part, &tmC, bar, x, y, lt);
        tma_load_3d(sl + 5 * part, &tmO, bar, x, y, lt);
        if (++lch == nch) { lch = 0; --lt; }
      };
      for (int k = 0; k < S; ++k) load(k);
      for (int k = 0; k < n; ++k) {
        if (!wait_inline(&staged[k & (S - 1)], (uint32_t)(k / S) & 1u, dead, p.ctl, p.limit_ns, t, cl)) break;
        fence_proxy_async_smem();                               // the gate warps' stores, before the TMA unit reads them
        tma_store_4d(&tmD, smem + (size_t)(k & (S - 1)) * slot_b, x, row0 + ch * CR, 0, t);
        tma_store_commit();
        if (++ch == nch) { ch = 0; --t; }
        if (k > 0) {                                            // the item before this one has left its slot
          tma_store_wait_read<1>();
          load(k - 1 + S);
        }
      }
      tma_store_wait<0>();
    }
  };
  if (warp < 8) {
  if (CL) regs_dec<80>(); else regs_dec<104>();
  if (CL && warp == 7) {
    tma_role();
  } else if (warp < gc) {
    // ---------------------------------------------------------------- gate maths
    const int unit0 = (rank * gc + warp) * 8;
    const bool live = unit0 < H;
    float4* st_s = reinterpret_cast<float4*>(smem + s_off) + warp * 32 + lane;   // [chunk][gl][lane]: dc, c[t+1] (2 rows each)
    for (int ch = 0; ch < nch; ++ch) {
      const int r = ch * CR + u;
      const bool rok = live && r < rows;
      const size_t o = (size_t)(row0 + r) * H + unit0 + 2 * c;
      const uint32_t v = (rok && p.dc_n) ? ldg4(reinterpret_cast<const T16*>(p.dc_n) + o) : 0u;
      const uint32_t v1 = rok ? ldg4(reinterpret_cast<const T16*>(p.cell) + (size_t)T * B * H + o) : 0u;
      const float2 d2 = cvt2<T16>(transpose8x8(v)), c2 = cvt2<T16>(transpose8x8(v1));
      st_s[ch * gc * 32] = make_float4(d2.x, d2.y, c2.x, c2.y);
    }
    const uint32_t so_g = swz((lane >> 3) * part + (lane & 7) * gc * 16 + warp * 16, gc);
    const uint32_t so_cd = swz((4 + ((lane >> 3) & 1)) * part + (lane & 7) * gc * 16 + warp * 16, gc);
    // dh of this lane's unit and rows: the sum of the sources' partial sums
    auto gather = [&](int st, int ch, float (&dh)[2]) {
      const float2* src = reinterpret_cast<const float2*>(smem + r_off + (size_t)(ch * 2 + ((st - 1) & 1)) * p.nc * src_b +
                                                          warp * 256) + lane;
      dh[0] = dh[1] = 0.f;
#pragma unroll 8
      for (int s = 0; s < p.nc; ++s, src += src_b / 8) {
        const float2 v = *src;
        dh[0] += v.x;
        dh[1] += v.y;
      }
    };
    float db[4] = {0.f, 0.f, 0.f, 0.f};
    bool ok = true;
    int k = 0;                                                  // item counter
    for (int st = 0; st < T && ok; ++st) {
      for (int ch = 0; ch < nch; ++ch, ++k) {
        const int par = k & 1;
        const uint32_t sl = sbase + (uint32_t)(k & (S - 1)) * slot_b;
        if (!wait_inline(&full[k & (S - 1)], (uint32_t)(k / S) & 1u, dead, p.ctl, p.limit_ns, T - 1 - st, cl)) { ok = false; break; }
        // all that does not depend on dh
        float fA[2], fO[2], fI[2], fF[2], fG[2], sF[2];
        uint32_t pw[4], pc, pd;
        ldmatrix_x4_trans(sl + so_g, pw);
        ldmatrix_x2_trans(sl + so_cd, pc, pd);
        const float4 sv = st_s[ch * gc * 32];
        const float2 cv = cvt2<T16>(pc), dv = cvt2<T16>(pd);
        const float2 x0 = cvt2<T16>(pw[0]), x1 = cvt2<T16>(pw[1]), x2 = cvt2<T16>(pw[2]), x3 = cvt2<T16>(pw[3]);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const float si = sigmoid_fast(e ? x0.y : x0.x), sf = sigmoid_fast(e ? x1.y : x1.x), so = sigmoid_fast(e ? x3.y : x3.x);
          const float tg = tanh_fast(e ? x2.y : x2.x), tc = tanh_fast(e ? sv.w : sv.z);
          fA[e] = so * (1.f - tc * tc);
          fI[e] = tg * si * (1.f - si);
          fF[e] = (e ? cv.y : cv.x) * sf * (1.f - sf);
          fG[e] = si * (1.f - tg * tg);
          fO[e] = tc * so * (1.f - so);
          sF[e] = sf;
        }
        if (st > 0) {
          uint64_t* bar = &xbar[2 * ch + ((st - 1) & 1)];
          if (!wait_inline(bar, (uint32_t)((st - 1) >> 1) & 1u, dead, p.ctl, p.limit_ns, T - 1 - st, cl)) { ok = false; break; }
          if (CL && warp == 0 && lane == 0 && st + 1 < T) mbar_expect_tx(bar, expect(ch));
        }
        float q[4][2];
        float dh[2] = {0.f, 0.f};
        if (st > 0) gather(st, ch, dh);
        else if (p.dh_n) {
          const int r = ch * CR + u;
          const uint32_t v = (live && r < rows) ? ldg4(reinterpret_cast<const T16*>(p.dh_n) + (size_t)(row0 + r) * H + unit0 + 2 * c) : 0u;
          const float2 f = cvt2<T16>(transpose8x8(v));
          dh[0] = f.x;
          dh[1] = f.y;
        }
        float dcn[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const float d = (e ? dv.y : dv.x) + dh[e];
          const float dcv = fmaf(d, fA[e], e ? sv.y : sv.x);
          q[0][e] = dcv * fI[e];
          q[1][e] = dcv * fF[e];
          q[2][e] = dcv * fG[e];
          q[3][e] = d * fO[e];
          dcn[e] = dcv * sF[e];
        }
        st_s[ch * gc * 32] = make_float4(dcn[0], dcn[1], cv.x, cv.y);
        // operand buffer `par` is free once the product two items ago has read it
        if (k >= 2 && !wait_inline(&dempty[par], (uint32_t)((k >> 1) - 1) & 1u, dead, p.ctl, p.limit_ns, T - 1 - st, cl)) { ok = false; break; }
        const uint32_t dgs = sbase + d_off + (uint32_t)(par * CR) * pitch + warp * 64;
        uint32_t w16[4];
#pragma unroll
        for (int g = 0; g < 4; ++g) w16[g] = pk2<T16>(q[g][0], q[g][1]);
        stmatrix_x4_trans(dgs + (uint32_t)(lane & 7) * pitch + (lane >> 3) * 16, w16[0], w16[1], w16[2], w16[3]);
        __syncwarp();
        if (lane == 0) mbar_arrive(&dfull[par]);
        // off the chain: d_ifgo for the TMA store, the bias gradient's sums (of the values as stored), the previous item's boxes
        stmatrix_x4_trans(sl + so_g, w16[0], w16[1], w16[2], w16[3]);
        const int rc = ch * CR + 2 * c;                         // this lane's two rows
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          const float2 f = cvt2<T16>(w16[g]);
          db[g] += (rc < rows ? f.x : 0.f) + (rc + 1 < rows ? f.y : 0.f);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&staged[k & (S - 1)]);
      }
    }
    // ---- gradients of the initial states
    for (int ch = 0; ch < nch && ok; ++ch) {
      if (!wait_inline(&xbar[2 * ch + ((T - 1) & 1)], (uint32_t)((T - 1) >> 1) & 1u, dead, p.ctl, p.limit_ns, -1, cl)) break;
      float dh[2];
      gather(T, ch, dh);
      const float4 sv = st_s[ch * gc * 32];
      const uint32_t hw = transpose8x8(pk2<T16>(dh[0], dh[1])), cw = transpose8x8(pk2<T16>(sv.x, sv.y));
      const int r = ch * CR + u;
      if (live && r < rows) {
        const size_t o = (size_t)(row0 + r) * H + unit0 + 2 * c;
        stg4(reinterpret_cast<T16*>(p.dh0) + o, hw);
        stg4(reinterpret_cast<T16*>(p.dc0) + o, cw);
      }
    }
    if (p.db_part) {
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        float v = db[g];
        v += __shfl_xor_sync(0xffffffffu, v, 1);
        v += __shfl_xor_sync(0xffffffffu, v, 2);
        if (live && c == 0 && nch > 0) p.db_part[(size_t)cl * 4 * H + (size_t)g * H + unit0 + u] = v;
      }
    }
  }
  } else if (!CL && warp >= 12) {
    regs_dec<40>();
    if (warp == 12) tma_role();
  } else {
  if (CL) regs_inc<176>(); else regs_inc<232>();
  if (warp < 8 + nm) {
    // ---------------------------------------------------------------- products
    const int mg = warp - 8;                                    // M tiles mg, mg+mgroups, ...
    const int kmem = gc - KR / 2;                               // pairs of K steps (one unit group each) kept in shared memory
    uint4* w_s = reinterpret_cast<uint4*>(smem + w_off) + (size_t)mg * MPW * kmem * 64 + lane;
    // weights: A[unit][k], k = 32*(local group) + 8*gate + unit of the group
    uint32_t w[MPW][KR][4];
    {
      auto frag = [&](int i, int ks, uint32_t (&a)[4]) {        // ks: K step
        const int m = (mg + i * p.mgroups) * 16 + u;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int mm = m + (j & 1) * 8, kg = ks >> 1, gate = (ks & 1) * 2 + (j >> 1);
          const int ku = (rank * gc + kg) * 8 + 2 * c;
          uint32_t v = 0;
          if (mm < H && kg < gc && ku < H) {
            const unsigned short* src = reinterpret_cast<const unsigned short*>(Wh) + ((size_t)gate * H + ku) * H + mm;
            v = (uint32_t)src[0] | ((uint32_t)src[H] << 16);
          }
          a[j] = v;
        }
      };
#pragma unroll
      for (int i = 0; i < MPW; ++i)
#pragma unroll
        for (int ks = 0; ks < KR; ++ks) frag(i, ks, w[i][ks]);
      for (int i = 0; i < MPW; ++i)
        for (int ks = 0; ks < 2 * kmem; ++ks) {
          uint32_t a[4];
          frag(i, KR + ks, a);
          w_s[(i * 2 * kmem + ks) * 32] = make_uint4(a[0], a[1], a[2], a[3]);
        }
      __syncwarp();
    }
    // where this lane's 16 bytes of every M tile go: an even lane sends the tile's first 8 units, an odd one its second
    uint32_t dst[MPW];
    uint32_t there = 0, owners = 0;
#pragma unroll
    for (int i = 0; i < MPW; ++i) {
      const int grp = 2 * (mg + i * p.mgroups) + (c & 1);
      const int owner = grp / gc, lg = grp - owner * gc;
      if (grp * 8 < H && !p.no_arrive) there |= 1u << i;
      owners |= (uint32_t)min(owner, p.nc - 1) << (4 * i);
      dst[i] = (CL ? mapa_shared(sbase, min(owner, p.nc - 1)) : sbase) + r_off + rank * src_b + (lg * 8 + u) * 32 + (c >> 1) * 16;
    }
    bool ok = true;
    int k = 0;
    for (int st = 0; st < T && ok; ++st) {
      for (int ch = 0; ch < nch; ++ch, ++k) {
        const int par = k & 1;
        if (!wait_inline(&dfull[par], (uint32_t)(k >> 1) & 1u, dead, p.ctl, p.limit_ns, T - 1 - st, cl)) { ok = false; break; }
        float acc[MPW * NA][4];
#pragma unroll
        for (int i = 0; i < MPW * NA; ++i)
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[i][e] = 0.f;
        const uint32_t da = sbase + d_off + (uint32_t)(par * CR + (lane & 7)) * pitch + (lane >> 3) * 16;
        constexpr int AH = KR / 2 <= 4 ? KR / 2 : 2;             // operand fetches run ahead of the MMAs
        uint32_t bf[AH][4];
#pragma unroll
        for (int kk = 0; kk < (AH == KR / 2 ? AH : 1); ++kk) ldmatrix_x4(da + kk * 64, bf[kk]);
#pragma unroll
        for (int kk = 0; kk < KR / 2; ++kk) {
          if (AH < KR / 2 && kk + 1 < KR / 2) ldmatrix_x4(da + (kk + 1) * 64, bf[(kk + 1) & 1]);
#pragma unroll
          for (int i = 0; i < MPW; ++i) mma16816<T16>(acc[i], w[i][2 * kk], bf[kk % AH][0], bf[kk % AH][1]);
#pragma unroll
          for (int i = 0; i < MPW; ++i) mma16816<T16>(acc[i + NA - 1], w[i][2 * kk + 1], bf[kk % AH][2], bf[kk % AH][3]);
        }
#pragma unroll 1
        for (int kk = KR / 2; TAIL && kk < gc; ++kk) {
          uint32_t b[4];
          ldmatrix_x4(da + kk * 64, b);
#pragma unroll
          for (int i = 0; i < MPW; ++i) {
            const uint4 v0 = w_s[(i * 2 * kmem + 2 * kk - KR) * 32], v1 = w_s[(i * 2 * kmem + 2 * kk - KR + 1) * 32];
            const uint32_t a0[4] = {v0.x, v0.y, v0.z, v0.w}, a1[4] = {v1.x, v1.y, v1.z, v1.w};
            mma16816<T16>(acc[i], a0, b[0], b[1]);
            mma16816<T16>(acc[i + NA - 1], a1, b[2], b[3]);
          }
        }
        if (NA == 2) {
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[0][e] += acc[MPW * NA - 1][e];
        }
        const uint32_t bufo = (uint32_t)(ch * 2 + (st & 1)) * p.nc * src_b;
        const uint32_t bo = sbase + b_off + (uint32_t)(2 * ch + (st & 1)) * 8;
        const int valid = rows - ch * CR;
#pragma unroll
        for (int i = 0; i < MPW; ++i) {
          const float s0 = (c & 1) ? acc[i][0] : acc[i][2], s1 = (c & 1) ? acc[i][1] : acc[i][3];
          const float r0 = __shfl_xor_sync(0xffffffffu, s0, 1), r1 = __shfl_xor_sync(0xffffffffu, s1, 1);
          const uint4 v = (c & 1) ? make_uint4(__float_as_uint(r0), __float_as_uint(r1), __float_as_uint(acc[i][2]), __float_as_uint(acc[i][3]))
                                  : make_uint4(__float_as_uint(acc[i][0]), __float_as_uint(acc[i][1]), __float_as_uint(r0), __float_as_uint(r1));
          if ((there >> i & 1u) && 4 * (c >> 1) < valid) {
            const uint32_t a = dst[i] + bufo;
            if (CL) st_async16(a, v, mapa_shared(bo, owners >> (4 * i) & 15u)); else st_shared16(a, v);
          }
        }
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(&dempty[par]);                            // (every lane's fragments have been read)
          if (!CL) mbar_arrive(&xbar[2 * ch + (st & 1)]);
        }
      }
    }
  }
  }
  __syncthreads();
  if (CL) cluster_sync_all();
}

// ---------------------------------------------------------------- plans and launches
// CTAs per cluster: one while a single SM holds the weights and does a step's product in less time than an exchange
// takes, then as few as keep a step short.  By the hidden size alone, so that the order of the sums - and with it
// every bit of a row's results - does not depend on the batch.
static int small_cluster(int H) { return H <= 64 ? 1 : H <= 128 ? 4 : H <= 256 ? 8 : 16; }

__global__ void one_cta_per_sm_kernel() {}

// Asked of the occupancy calculator once per size from 5 CTAs on: clusters do not tile every GPC without a remainder.
int resident_clusters(int nc) {
  static std::atomic<int> cached[17];
  static const int b200[17] = {0, 148, 74, 45, 33, 26, 22, 15, 15, 15, 11, 7, 7, 7, 7, 7, 7};     // its answers with 148 SMs
  const int sms = plan_sm_count();
  if (nc <= 4) return sms * 132 / 148 / nc;
  int c = cached[nc].load(std::memory_order_relaxed);
  if (c > 0) return c;
  c = sms * b200[nc] / 148;
  DeviceInfo di;
  auto kern = one_cta_per_sm_kernel;
  if (get_device_info(&di) == BLSTM_OK && di.sm_count > 0 &&
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024) == cudaSuccess &&
      cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(nc);
    cfg.blockDim = dim3(384);
    cfg.dynamicSmemBytes = 200 * 1024;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = nc;
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int mc = 0;
    if (cudaOccupancyMaxActiveClusters(&mc, kern, &cfg) == cudaSuccess && mc > 0) c = mc;
  }
  (void)cudaGetLastError();
  cached[nc].store(c, std::memory_order_relaxed);
  return c;
}

// Whether the plan beats the tcgen05 kernels: those with resident weights (multiples of 64 from 256 on; smaller sizes: the
// general ones) take nearly the same time for any batch of up to several hundred rows, these about the same for
// every chunk of 8 rows after the first, so the line is a number of chunks per cluster.  us per step (B200), these against
// the others at 1, 2, 3, ... chunks, a dash where the line lies.
// Forward: H = 192: 8: 3.5 / 5.3 (nothing saved: 4.6) - 10: 4.3 / 5.4 (4.7), 12: 5.2 / 5.4 (4.7; and two layers as a wavefront beat both);
// H = 256: 3: 2.1 / 2.7, 4: 2.3 / 3.1 - 5: 3.2 / 3.1; H = 320: 3: 2.0 / 2.8, 4: 2.7 / 2.8 - 5: 3.4 / 3.2; H = 384: 2: 1.7 / 2.9, 3: 2.3 / 2.9 -
// 4: 3.1 / 3.2; H = 448: 3: 2.7 / 3.3 - 4: 3.6 / 3.3; H = 512: 1: 1.6 / 3.0, 2: 2.2 / 3.1 - 3: 3.1 to 3.2 / 3.1 to 3.4, 5: 5.3 / 3.5;
// H = 576: 1: 1.9 / 3.1 - 2: 3.8 / 3.1; H = 640: 1: 2.2 / 3.2 - 2: 4.1 / 3.2; H = 768: 1: 2.5 / 3.4.
// Backward: H = 192: 8: 4.4 / 4.9 - 9: 4.95 / 4.95; H = 256: 5: 3.0 / 3.5, 6: 3.6 / 4.8; H = 320: 4: 3.1 / 3.5 - 5: 3.6 / 3.5; H = 384: 4: 2.8 / 3.6 -
// 5: 3.5 / 3.6; H = 448: 4: 3.5 / 3.8 - 5: 3.9 / 3.8; H = 512: 3: 2.6 / 3.3, 4: 3.4 / 3.8, 5: 4.1 / 3.8 (B = 256), 4.1 / 5.3 (B = 280); H = 576: 2: 3.4
// to 3.9 / 3.4 to 3.9; H = 640: 2: 3.4 / 3.5 to 3.9 (more does not fit).  At H = 512 the fifth chunk costs 9 % up to 256 rows and is
// taken there so that a batch of 256 rows and its halves go through the same kernels and agree bit for bit, which they do not
// across a line.
// (General kernels, forward: H = 64, B = 64: 1.9 -> 0.59; H = 192: 4.4 a step at any of these batches.)
static bool small_plan_pays(int H, const SmallPlan& p, int phase) {
  if (H <= 128) return true;
  if (phase == BLSTM_PHASE_BWD && H < 256 && H % 64 != 0) return true;      // (the others would be the CUDA-core kernels)
  if (phase == BLSTM_PHASE_BWD) return p.nch <= (H < 256 ? 8 : H == 256 ? 6 : H <= 448 ? 4 : H <= 512 ? 5 : 2);
  return p.nch <= (H < 256 ? 8 : H <= 320 ? 4 : H <= 448 ? 3 : H <= 512 ? 2 : 1);
}

SmallPlan small_plan(const blstm_desc& d, int phase) {
  SmallPlan p{};
  if (d.flags & (BLSTM_FLAG_FORCE_GENERIC | BLSTM_FLAG_NO_CLUSTER)) return p;
  if (d.dtype != BLSTM_F16 && d.dtype != BLSTM_BF16) return p;
  const int H = d.hidden_size, B = d.batch;
  if (H % 8 != 0 || H > 768) return p;
  const int G = H / 8;
  p.gc = cdiv(G, small_cluster(H));
  p.nc = cdiv(G, p.gc);
  if (p.nc == 1 && (d.flags & BLSTM_FLAG_TEST_NO_ARRIVE)) return p;     // (no wait that could run out)
  // (No cluster waits for another, so half a device is only a hint: two launches side by side share it as they fit.)
  const int cap = d.flags & BLSTM_FLAG_HALF_DEVICE ? (resident_clusters(p.nc) + 1) / 2 : resident_clusters(p.nc);
  p.ks = 2 * cdiv(H, 32);
  const int tiles = cdiv(B, 8);
  p.ncl = std::min(cap, tiles);
  const size_t fixed = 1024 + 2 * SB_MAX_CHUNKS * 8 + 2048;              // alignment, barriers
  if (phase == BLSTM_PHASE_FWD) {
    p.kspl = H > 256 && p.gc <= 4 ? 2 : 1;
    p.kr = p.nc == 1 ? std::min(p.ks, 4) : p.nc <= 4 ? std::min(p.ks, 8) : p.nc <= 8 ? (p.ks >= 16 ? 16 : p.ks >= 12 ? 12 : 10)
         : p.kspl == 2 ? 2 * cdiv(p.ks, 4) : 18;
    if (p.kspl == 2) p.ks = 2 * p.kr;
    p.nch = cdiv(tiles, p.ncl);
    p.rpl = 1;
    while (2 * p.rpl <= p.nch && 2 * p.rpl * p.gc * p.kspl <= 8) p.rpl *= 2;
    p.slots = (p.nc == 1 ? 8 : 4) * std::min(p.rpl, 4);
    p.threads = 384;
    p.smem = fixed + (size_t)p.slots * 768 * p.gc + (size_t)p.nch * 2 * 8 * (p.ks * 32 + 16) +
             (size_t)p.nch * p.gc * 256 + (size_t)p.gc * (p.kspl == 2 ? 2 : p.ks - p.kr) * 1024;
  } else {
    if (H > 640) return p;
    const int mt = cdiv(H, 16);
    p.mpw = p.nc == 1 ? 1 : cdiv(mt, 8);
    p.mgroups = cdiv(mt, p.mpw);
    p.nch = cdiv(tiles, p.ncl);
    p.threads = 512;
    if (p.nc == 1) p.kr = p.gc == 8 ? 16 : p.gc >= 4 ? 8 : 2;
    else if (p.nc <= 4) p.kr = p.gc == 4 ? 8 : 6;
    else p.kr = p.gc == 5 ? 6 : 2 * p.gc;
    p.smem = fixed + (size_t)8 * 768 * p.gc + (size_t)2 * 8 * (p.gc * 64 + 16) +
             (size_t)p.nch * 2 * p.nc * p.gc * 256 + (size_t)p.nch * p.gc * 512 +
             (size_t)p.mgroups * p.mpw * (p.gc - p.kr / 2) * 1024;
  }
  p.rows = 8 * p.nch;
  p.ncl = p.nparts = cdiv(B, p.rows);
  if (phase == BLSTM_PHASE_BWD)
    while (p.ncl * p.nc % 4 != 0) ++p.ncl;                               // whole groups of four CTAs; the extra clusters have no rows
  p.grid = p.ncl * p.nc;
  if (p.smem > 232448 || p.nch > SB_MAX_CHUNKS) return p;
  p.ok = small_plan_pays(H, p, phase);
  return p;
}

template <typename T16>
static int small_fwd_t(const SmallPlan& pl, const CUtensorMap& tp, const CUtensorMap& th, const CUtensorMap& tc,
                       const SmallFwdParams& p, cudaStream_t st) {
#define BLSTM_SMALL_FWD(K, N, C) \
  if (pl.kr == K && pl.kspl == N && (pl.nc > 1) == C) return launch_clusters(small_fwd_kernel<K, N, C, T16>, pl.grid, pl.threads, pl.smem, pl.nc, st, tp, th, tc, p);
  BLSTM_SMALL_FWD(2, 1, false)
  BLSTM_SMALL_FWD(4, 1, false)
  BLSTM_SMALL_FWD(6, 1, true)
  BLSTM_SMALL_FWD(8, 1, true)
  BLSTM_SMALL_FWD(10, 1, true)
  BLSTM_SMALL_FWD(12, 1, true)
  BLSTM_SMALL_FWD(16, 1, true)
  BLSTM_SMALL_FWD(18, 1, true)
  BLSTM_SMALL_FWD(10, 2, true)
  BLSTM_SMALL_FWD(12, 2, true)
  BLSTM_SMALL_FWD(14, 2, true)
  BLSTM_SMALL_FWD(16, 2, true)
#undef BLSTM_SMALL_FWD
  return BLSTM_E_UNSUPPORTED;
}

template <typename T16>
static int small_bwd_t(const SmallPlan& pl, const CUtensorMap& tp, const CUtensorMap& tc, const CUtensorMap& to,
                       const CUtensorMap& td, const SmallBwdParams& p, cudaStream_t st) {
#define BLSTM_SMALL_BWD(M, K, C) \
  if (pl.mpw == M && pl.kr == K && (pl.nc > 1) == C && ((C ? M == 5 : K < 16) || pl.gc == K / 2)) return launch_clusters(small_bwd_kernel<M, K, C, T16>, pl.grid, pl.threads, pl.smem, pl.nc, st, tp, tc, to, td, p);
  BLSTM_SMALL_BWD(1, 2, false)
  BLSTM_SMALL_BWD(1, 8, false)
  BLSTM_SMALL_BWD(1, 16, false)
  BLSTM_SMALL_BWD(1, 6, true)
  BLSTM_SMALL_BWD(1, 8, true)
  BLSTM_SMALL_BWD(2, 6, true)
  BLSTM_SMALL_BWD(2, 8, true)
  BLSTM_SMALL_BWD(3, 6, true)
  BLSTM_SMALL_BWD(4, 8, true)
  BLSTM_SMALL_BWD(5, 6, true)
#undef BLSTM_SMALL_BWD
  return BLSTM_E_UNSUPPORTED;
}

// Item boxes: the CTA's units x a chunk's rows (x 4 gates) of one step.
static int gates_map(CUtensorMap* m, const void* base, const blstm_desc& d, const SmallPlan& pl) {
  const uint64_t H = d.hidden_size, B = d.batch;
  uint64_t dims[4] = {H, B, 4, (uint64_t)d.seq_len};
  uint64_t str[3] = {4 * H * 2, H * 2, B * 4 * H * 2};
  uint32_t box[4] = {(uint32_t)pl.gc * 8, 8u, 4, 1};
  return encode_tensor_map(m, base, 4, dims, str, box, 2, slot_swizzle(pl.gc));
}
static int states_map(CUtensorMap* m, const void* base, const blstm_desc& d, const SmallPlan& pl, int steps) {
  const uint64_t H = d.hidden_size, B = d.batch;
  uint64_t dims[3] = {H, B, (uint64_t)steps};
  uint64_t str[2] = {H * 2, B * H * 2};
  uint32_t box[3] = {(uint32_t)pl.gc * 8, 8u, 1};
  return encode_tensor_map(m, base, 3, dims, str, box, 2, slot_swizzle(pl.gc));
}

}  // namespace sm100

using namespace sm100;

size_t small_workspace(const blstm_desc& d, const SmallPlan& pl, int phase) {
  return sizeof(Control) + (phase == BLSTM_PHASE_BWD ? round_up((size_t)pl.nparts * 4 * d.hidden_size * sizeof(float), 256) : 0);
}

int small_fwd_recurrence(const blstm_desc& d, const SmallPlan& pl, void* ifgo, const void* Wh, void* out, void* cell,
                         void* ws, cudaStream_t st) {
  SmallFwdParams p;
  p.T = d.seq_len; p.B = d.batch; p.H = d.hidden_size;
  p.nc = pl.nc; p.gc = pl.gc; p.ks = pl.ks; p.rows = pl.rows; p.nch = pl.nch; p.rpl = pl.rpl; p.slots = pl.slots;
  p.no_arrive = (d.flags & BLSTM_FLAG_TEST_NO_ARRIVE) ? 1 : 0;
  p.inference = (d.flags & BLSTM_FLAG_INFERENCE) ? 1 : 0;
  p.limit_ns = d.wait_limit_us > 0 ? (unsigned long long)d.wait_limit_us * 1000ull : kDefaultWaitNs;
  p.ctl = reinterpret_cast<Control*>(ws);
  p.Wh = Wh; p.out = out; p.cell = cell;
  CUtensorMap tp, th, tc;
  int rc = gates_map(&tp, ifgo, d, pl);
  if (!rc) rc = states_map(&th, out, d, pl, d.seq_len + 1);
  if (!rc) rc = states_map(&tc, cell, d, pl, d.seq_len + 1);
  if (rc) return rc;
  return d.dtype == BLSTM_BF16 ? small_fwd_t<__nv_bfloat16>(pl, tp, th, tc, p, st) : small_fwd_t<__half>(pl, tp, th, tc, p, st);
}

int small_bwd_recurrence(const blstm_desc& d, const SmallPlan& pl, const void* dout, const void* dh_n, const void* dc_n,
                         const void* ifgo, const void* cell, const void* Wh, void* d_ifgo, void* dh0, void* dc0,
                         float* db, void* ws, cudaStream_t st) {
  SmallBwdParams p;
  p.T = d.seq_len; p.B = d.batch; p.H = d.hidden_size;
  p.nc = pl.nc; p.gc = pl.gc; p.rows = pl.rows; p.nch = pl.nch; p.mgroups = pl.mgroups;
  p.no_arrive = (d.flags & BLSTM_FLAG_TEST_NO_ARRIVE) ? 1 : 0;
  p.limit_ns = d.wait_limit_us > 0 ? (unsigned long long)d.wait_limit_us * 1000ull : kDefaultWaitNs;
  p.ctl = reinterpret_cast<Control*>(ws);
  p.dh_n = dh_n; p.dc_n = dc_n; p.cell = cell; p.Wh = Wh; p.dh0 = dh0; p.dc0 = dc0;
  p.db_part = db ? reinterpret_cast<float*>(static_cast<char*>(ws) + sizeof(Control)) : nullptr;
  CUtensorMap tp, tc, to, td;
  int rc = gates_map(&tp, ifgo, d, pl);
  if (!rc) rc = states_map(&tc, cell, d, pl, d.seq_len + 1);
  if (!rc) rc = states_map(&to, dout, d, pl, d.seq_len);
  if (!rc) rc = gates_map(&td, d_ifgo, d, pl);
  if (rc) return rc;
  rc = d.dtype == BLSTM_BF16 ? small_bwd_t<__nv_bfloat16>(pl, tp, tc, to, td, p, st) : small_bwd_t<__half>(pl, tp, tc, to, td, p, st);
  if (rc) return rc;
  return db ? reduce_db(p.db_part, pl.nparts, 4 * d.hidden_size, db, st) : BLSTM_OK;
}

int small_plan_detail(const blstm_desc& d, const SmallPlan& p, int phase, char* buf, size_t n) {
  (void)d;
  if (phase == BLSTM_PHASE_BWD)
    return snprintf(buf, n, "sm100 bwd small-batch cluster=%d units_per_cta=%d rows_per_cluster=%d chunks=%d m_tiles_per_warp=%d "
                    "register_steps=%d grid=%d threads=%d smem=%zu", p.nc, p.gc * 8, p.rows, p.nch, p.mpw, p.kr,
                    p.grid, p.threads, p.smem);
  return snprintf(buf, n, "sm100 fwd small-batch cluster=%d units_per_cta=%d rows_per_cluster=%d chunks=%d k_split=%d replicas=%d "
                  "register_steps=%d/%d grid=%d threads=%d smem=%zu", p.nc, p.gc * 8, p.rows, p.nch, p.kspl, p.rpl,
                  std::min(p.kr, p.ks), p.ks, p.grid, p.threads, p.smem);
}

}  // namespace blstm
