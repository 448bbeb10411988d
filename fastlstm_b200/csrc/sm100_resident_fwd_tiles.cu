// Forward recurrence with resident weights for batches of several tiles per group (16-bit, H = 256 to 1024): as in
// sm100_resident.cu the gate rows are the M side of the MMAs and the weights their A operand, up to 192 KB of a CTA's slice in
// tensor memory and the rest in shared memory, but a group of CTAs works through three to sixteen tiles of 32 batch rows in
// turn, so that one tile's hand-off hides behind the others'.
//
// Throughput bound: the eight epilogue warps (a tile takes them 2.4 k clocks) never wait for a round trip.  Two issuers take every
// other tile, each with its own accumulator and its own buffer for the batch rows; a warp of its own counts the tiles in; the
// pre-activations of the next tile are on their way while this one's gates are formed; cell states lie in tensor memory (fp32).
// us a step, the kernel with the batch on the M side -> this (B200): B = 1024, H = 1024 19.9 -> 14.3, B = 300 11.5 -> 6.4; B = 400,
// H = 768 8.2 -> 5.1, B = 2048 21.7 -> 15.3; B = 800, H = 640 9.5 -> 5.5; B = 1300, H = 512 9.1 -> 6.7; B = 2300, H = 256 6.0 -> 5.3.
#include <algorithm>
#include <cstdio>

#include "cluster_util.cuh"
#include "generic.cuh"
#include "resident_util.cuh"
#include "sm100_resident.cuh"

namespace blstm {
namespace sm100 {

constexpr int RF_N = 32;                   // batch rows per tile
constexpr int RF_TILES = 16;               // most tiles of a group
constexpr int RF_THREADS = 384;            // producer, two issuers, publisher, eight epilogue warps
constexpr int RF_SLOT = RF_N * 128;        // a K chunk of a tile: 4 KB
constexpr int RF_MAX_KG = 2;               // groups of chunks that are fetched, waited for and multiplied at once
constexpr int RF_STATE = 2 * RF_N;         // tensor memory columns: two accumulators, eight for each tile's states, weights

struct FwdTilesParams {
  int T, B, H;
  int mt, ng, nbt;                         // M tiles; groups; batch tiles
  int kc, nt, w_col, group;                // K chunks; of these in tensor memory, from which column on; at once
  int fmt, no_arrive, inference;
  unsigned long long limit_ns;
  Control* ctl;
  int* flags;                              // [T+1][tiles / 4], a byte for each tile
  const void* Wh;
  void* ifgo;
  void* out;
  void* cell;
};

template <typename T16>
__global__ void __launch_bounds__(RF_THREADS, 1)
fwd_tiles_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmX1,
                 const FwdTilesParams p) {
  constexpr int N = RF_N, UT = 32, UP = 4, W = 2, TPR = UT / UP, EW = 8, BLK = N * 128;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int H = p.H, T = p.T, KC = p.kc, KG = p.group, nt = p.nt, n_kg = (KC + KG - 1) / KG;
  uint8_t* w_s = smem;                                              // [KC - nt][16 KB]
  uint8_t* x_s = w_s + (size_t)(KC - nt) * 16384;                   // [2][KC][32 rows][128 B]
  uint8_t* recv = x_s + (size_t)2 * KC * RF_SLOT;                   // [2][4 gates][32 rows][32 units] fp32
  uint64_t* full = reinterpret_cast<uint64_t*>(recv + 2 * 4 * BLK); // [2][RF_MAX_KG]
  uint64_t* w_full = full + 2 * RF_MAX_KG;
  uint64_t* acc_full = w_full + 1;                                  // [2] each
  uint64_t* acc_empty = acc_full + 2;
  uint64_t* xchg = acc_empty + 2;
  uint64_t* stored = xchg + 2;                                      // [4] a tile's rows are stored / counted in
  uint64_t* counted = stored + 4;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(counted + 4);
  volatile int* dead = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int mt = blockIdx.x % p.mt, grp = blockIdx.x / p.mt;
  const int NT = (p.nbt - grp + p.ng - 1) / p.ng;                   // tiles grp, grp + ng, ... (two at least)
  const int total = T * NT, words = (p.nbt + 3) / 4;

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2 * RF_MAX_KG; ++i) mbar_init(&full[i], 1);
    mbar_init(w_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&acc_full[i], 1);
      mbar_init(&acc_empty[i], EW);
      mbar_init(&xchg[i], EW);
    }
    for (int i = 0; i < 4; ++i) {
      mbar_init(&stored[i], EW);
      mbar_init(&counted[i], 1);
    }
    *dead = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmX);
    tma_prefetch_desc(&tmX1);
  }
  if (warp == 1) tmem_alloc(tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  if (warp >= 4) {
    weights_to_tmem<false>(reinterpret_cast<const T16*>(p.Wh), H, mt, 0, nt, tmem_base + p.w_col, warp & 3, (warp - 4) >> 2, lane);
    tc_fence_before();
  }
  __syncthreads();
  tc_fence_after();
  WaitCtx wc{dead, p.ctl, p.limit_ns, -1, (int)blockIdx.x};
  auto tile_of = [&](int j) { return grp + j * p.ng; };
  // Item n = (step t = n / NT, tile j = n % NT): reads h[t].
  if (warp == 0) {
    // ---------------------------------------------------------------- TMA producer
    if (lane == 0 && KC > nt) {
      mbar_expect_tx(w_full, (uint32_t)(KC - nt) * 16384);
      for (int kc = nt; kc < KC; ++kc) tma_load_3d(w_s + (size_t)(kc - nt) * 16384, &tmW, w_full, kc * 64, mt * 32, 0);   // 4 gates x 32 units x 64 k
    }
    int early = 0, t = 0, j = 0;
    for (int n = 0; n < total; ++n) {
      const int tile = tile_of(j), b = n & 1;
      const int early_now = __shfl_sync(0xffffffffu, early, 31);
      int nj = j + 1, ns = t;
      if (nj == NT) { nj = 0; ++ns; }
      int seen = 1;
      if (lane == 0) {
        // the buffer is free once the products of the item before the last are formed
        if (n >= 2) seen = mbar_wait(&acc_full[b], ((uint32_t)(n >> 1) & 1u) ^ 1u, wc) ? 1 : 0;
        if (seen && t > 0 && early_now < p.mt)
          seen = wait_flag_ge(&p.flags[(size_t)t * words + (tile >> 2)], p.mt, p.ctl, p.limit_ns, t, tile, 8 * (tile & 3)) ? 1 : 0;
      }
      seen = __shfl_sync(0xffffffffu, seen, 0);
      __syncwarp();      // (a shuffle orders no memory: the issuing lanes come behind the acquire)
      if (!seen) { *dead = 1; break; }
      fence_proxy_async_global();
      if (lane < n_kg) {
        const int kc = lane * KG, m = min(KG, KC - kc);
        uint64_t* bar = &full[b * RF_MAX_KG + lane];
        uint8_t* dst = x_s + (size_t)(b * KC + kc) * RF_SLOT;
        mbar_expect_tx(bar, m * RF_SLOT);
        if (m == KG) {
          tma_load_4d(dst, &tmX, bar, 0, tile * N, kc, t);
        } else {
          for (int i = 0; i < m; ++i) tma_load_4d(dst + i * RF_SLOT, &tmX1, bar, 0, tile * N, kc + i, t);
        }
      } else if (lane == 31) {
        // (the other arm of the same branch: the issuing lanes do not wait for this read)
        early = 0;
        if (ns < T && ns > 0) {
          const int next = tile_of(nj);
          early = (int)((unsigned)ld_acquire_gpu(&p.flags[(size_t)ns * words + (next >> 2)]) >> 8 * (next & 3) & 0xffu);
        }
      }
      __syncwarp();
      j = nj; t = ns;
    }
  } else if (warp < 3) {
    // ---------------------------------------------------------------- MMA issuers: items x, x + 2, ...
    // (the warp waits, then one lane issues a group's MMAs without a branch that depends on data: see sm100_resident.cu)
    const int x = warp - 1;
    constexpr uint64_t descK = smem_desc_base(16, 1024);
    const uint32_t idesc = instr_desc(p.fmt, 0, 0, 128, N);
    const uint32_t d_tmem = tmem_base + x * N, a_tmem = tmem_base + p.w_col, wa = smem_u32(w_s), xa = smem_u32(x_s) + x * KC * RF_SLOT;
    bool ok = KC <= nt || warp_wait_all(w_full, 0, wc);
    for (int n = x; n < total && ok; n += 2) {
      const uint32_t k = (uint32_t)(n >> 1) & 1u;
      wc.d0 = n;
      if (!warp_wait_all(&acc_empty[x], k ^ 1u, wc)) break;
      for (int kg = 0; kg < n_kg; ++kg) {
        if (!warp_wait_all(&full[x * RF_MAX_KG + kg], k, wc)) { ok = false; break; }
        tc_fence_after();
        if (elect_one()) {
          const int l0 = kg * KG, l1 = min(KC, l0 + KG), lt = max(l0, min(nt, l1));
          for (int lc = l0; lc < lt; ++lc) {
            const uint32_t sb = xa + lc * RF_SLOT;
#pragma unroll
            for (int q = 0; q < 4; ++q)
              umma_f16_ts(d_tmem, a_tmem + lc * 32 + q * 8, smem_desc(descK, sb + q * 32), idesc, (q > 0 || lc > 0) ? 1u : 0u);
          }
          for (int lc = lt; lc < l1; ++lc) {
            const uint32_t sb = xa + lc * RF_SLOT, sa = wa + (lc - nt) * 16384;
#pragma unroll
            for (int q = 0; q < 4; ++q)
              umma_f16(d_tmem, smem_desc(descK, sa + q * 32), smem_desc(descK, sb + q * 32), idesc, (q > 0 || lc > 0) ? 1u : 0u);
          }
          if (kg + 1 == n_kg) umma_commit(&acc_full[x]);
        }
        __syncwarp();
      }
    }
  } else if (warp == 3) {
    // ---------------------------------------------------------------- publisher
    if (lane == 0) {
      int t = 0, j = 0;
      for (int n = 0; n < total; ++n) {
        const int tile = tile_of(j);
        wc.d0 = t; wc.d1 = tile;
        if (!mbar_wait_spin(&stored[n & 3], (uint32_t)(n >> 2) & 1u, wc)) break;
        if (!p.no_arrive) red_release_gpu_add(&p.flags[(size_t)(t + 1) * words + (tile >> 2)], 1 << 8 * (tile & 3));
        mbar_arrive(&counted[n & 3]);
        if (++j == NT) { j = 0; ++t; }
      }
    }
  } else {
    // ---------------------------------------------------------------- epilogue
    const int ew = warp - 4, q = ew & 3, g = ew >> 2, et = ew * 32 + lane;
    const int lr = et / TPR, u = (et % TPR) * UP, unit = mt * UT + u;      // this thread's row of a tile, first unit
    const size_t H4 = 4 * (size_t)H;
    const uint32_t d_addr = tmem_base + (uint32_t(q * 32) << 16) + g * (N / 2);
    const uint32_t s_addr = tmem_base + RF_STATE + (uint32_t(q * 32) << 16) + g * 4;
    T16* const ifgo = reinterpret_cast<T16*>(p.ifgo) + unit;
    T16* const out = reinterpret_cast<T16*>(p.out) + unit;
    T16* const cell = reinterpret_cast<T16*>(p.cell) + unit;
    // (pieces of 16 bytes at places xor'ed with row and gate: see sm100_resident.cu)
    auto piece = [](int row, int gate, int i) { return i ^ (((row ^ gate) & 7) << 2); };
    for (int j = 0; j < NT; ++j) {
      const int row = tile_of(j) * N + lr;
      float c[UP] = {0.f, 0.f, 0.f, 0.f};
      if (row < p.B) {
        uint32_t w[W];
        ld_words<W>(w, cell + (size_t)row * H);
        unpack_words<T16, W>(w, c);
      }
      uint32_t v[4];
#pragma unroll
      for (int i = 0; i < UP; ++i) v[i] = __float_as_uint(c[i]);
      tmem_st_32x4(s_addr + j * 8, v);
    }
    tmem_st_wait();
    uint32_t pre[4][W];                     // pre-activations of the next item
    auto load_pre = [&](int t, int j) {
      const int row = tile_of(j) * N + lr;
      if (t < T && row < p.B)
#pragma unroll
        for (int gg = 0; gg < 4; ++gg) ld_words<W>(pre[gg], ifgo + ((size_t)t * p.B + row) * H4 + (size_t)gg * H);
    };
    // the item behind it only into L2: a row's eight threads ask for its four runs of 64 bytes
    auto prefetch_far = [&](int t, int j) {
      const int row = tile_of(j) * N + lr;
      if (t < T && row < p.B && (lane & 1) == 0) prefetch_l2(ifgo - u + ((size_t)t * p.B + row) * H4 + (size_t)((lane & 7) >> 1) * H);
    };
    load_pre(0, 0);
    // what only backward needs of an item is stored during the next one's exchange: the release waits for every store under way
    uint32_t kept[5][W];
    int kept_t = -1, kept_row = 0;
    auto store_kept = [&] {
      if (kept_t < 0 || kept_row >= p.B) return;
      if (!p.inference)
#pragma unroll
        for (int gg = 0; gg < 4; ++gg) st_words<W>(ifgo + ((size_t)kept_t * p.B + kept_row) * H4 + (size_t)gg * H, kept[gg]);
      if (!p.inference || kept_t == T - 1) st_words<W>(cell + ((size_t)(kept_t + 1) * p.B + kept_row) * H, kept[4]);
    };
    int t = 0, j = 0, n = 0;
    for (; n < total; ++n) {
      const int b = n & 1;
      const uint32_t k = (uint32_t)(n >> 1) & 1u;
      wc.d0 = n;
      if (!mbar_wait(&acc_full[b], k, wc)) break;
      tc_fence_after();
      uint32_t a[16], st[4];
      tmem_ld_32x16(d_addr + b * N, a);
      tmem_ld_32x4(s_addr + j * 8, st);
      tmem_ld_wait();
      tc_fence_before();
      uint8_t* rv = recv + b * (4 * BLK);
#pragma unroll
      for (int c = 0; c < 16; ++c) {
        const int rr = g * 16 + c;
        reinterpret_cast<uint32_t*>(rv + q * BLK + rr * 128)[piece(rr, q, lane)] = a[c];
      }
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&acc_empty[b]);
        mbar_arrive(&xchg[b]);
      }
      store_kept();
      if (!mbar_wait(&xchg[b], k, wc)) break;
      float pa[4][UP], cs[UP], hv[UP];
#pragma unroll
      for (int gg = 0; gg < 4; ++gg) {
        const float4 v = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(rv + gg * BLK + lr * 128) + piece(lr, gg, u));
        const float2 f0 = cvt2<T16>(pre[gg][0]), f1 = cvt2<T16>(pre[gg][1]);
        pa[gg][0] = v.x + f0.x; pa[gg][1] = v.y + f0.y; pa[gg][2] = v.z + f1.x; pa[gg][3] = v.w + f1.y;
      }
      const int row = tile_of(j) * N + lr;
      int nj = j + 1, ns = t;
      if (nj == NT) { nj = 0; ++ns; }
#pragma unroll
      for (int i = 0; i < UP; ++i) {
        cs[i] = sigmoid_fast(pa[1][i]) * __uint_as_float(st[i]) + sigmoid_fast(pa[0][i]) * tanh_fast(pa[2][i]);
        hv[i] = sigmoid_fast(pa[3][i]) * tanh_fast(cs[i]);
        st[i] = __float_as_uint(cs[i]);
      }
      tmem_st_32x4(s_addr + j * 8, st);
      uint32_t hw[W];
      pack_words<T16, W>(hw, hv);
      if (row < p.B) st_words<W>(out + ((size_t)(t + 1) * p.B + row) * H, hw);
      tmem_st_wait();
      __syncwarp();
      if (lane == 0) {
        if (mbar_wait(&counted[n & 3], ((uint32_t)(n >> 2) & 1u) ^ 1u, wc)) mbar_arrive(&stored[n & 3]);
      }
      __syncwarp();
      load_pre(ns, nj);
      {
        int fj = nj + 1, fs = ns;
        if (fj == NT) { fj = 0; ++fs; }
        prefetch_far(fs, fj);
      }
      kept_t = t;
      kept_row = row;
#pragma unroll
      for (int gg = 0; gg < 4; ++gg) pack_words<T16, W>(kept[gg], pa[gg]);
      pack_words<T16, W>(kept[4], cs);
      j = nj; t = ns;
    }
    if (n == total) store_kept();
  }
  // ---------------------------------------------------------------- teardown
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

FwdTilesPlan fwd_tiles_plan(const blstm_desc& d, int phase) {
  FwdTilesPlan p{};
  const int H = d.hidden_size;
  if ((d.flags & BLSTM_FLAG_FORCE_GENERIC) || (d.dtype != BLSTM_F16 && d.dtype != BLSTM_BF16)) return p;
  if (phase != BLSTM_PHASE_FWD || H % 64 != 0 || H < RES_MIN_H || H > 1024) return p;
  p.mt = H / 32;
  p.ng = plan_sm_count() / ((d.flags & BLSTM_FLAG_HALF_DEVICE) ? 2 : 1) / p.mt;
  if (p.ng < 1) return p;
  p.nbt = cdiv(d.batch, RF_N);
  const int most = cdiv(p.nbt, p.ng);
  // us a step, the kernel with the batch on the M side / this: H = 512, 6 and 7 tiles 9.3 / 8.1 and 9.3 / 9.3; H = 448, 6 and 8 9.2 / 7.9
  // and 9.4 / 10.5; H = 256, 4 and 6 6.0 / 5.3 and 7.4 / 7.8; from H = 576 on all that fit: every count of three to sixteen takes 0.43 to 0.89 of
  // that kernel's time, H = 832, 7 tiles 24.2 / 10.4, H = 576, 8 and 16 12.3 / 10.9 and 24.3 / 21.4, H = 1024, 8 20.0 / 14.6
  if (most < 3 || most > (H > 512 ? RF_TILES : H > 320 ? 6 : 4)) return p;
  p.kc = H / 64;
  p.w_col = RF_STATE + 8 * most;
  p.nt = std::min(p.kc, (512 - p.w_col) / 32);
  p.group = cdiv(p.kc, RF_MAX_KG);
  p.grid = p.ng * p.mt;
  p.smem = 1024 + (size_t)(p.kc - p.nt) * 16384 + (size_t)2 * p.kc * RF_SLOT + 2 * 4 * RF_SLOT + 512;
  p.ws_bytes = sizeof(Control) + round_up((size_t)(d.seq_len + 1) * cdiv(p.nbt, 4) * sizeof(int), 256);
  p.ok = p.smem <= 232448;
  return p;
}

}  // namespace sm100

using namespace sm100;

int fwd_tiles_recurrence(const blstm_desc& d, const FwdTilesPlan& pl, void* ifgo, const void* Wh, void* out, void* cell, void* ws, cudaStream_t st) {
  const int H = d.hidden_size, B = d.batch, T = d.seq_len;
  FwdTilesParams p{};
  p.T = T; p.B = B; p.H = H;
  p.mt = pl.mt; p.ng = pl.ng; p.nbt = pl.nbt; p.kc = pl.kc; p.nt = pl.nt; p.w_col = pl.w_col; p.group = pl.group;
  p.fmt = d.dtype == BLSTM_BF16 ? 1 : 0;
  p.no_arrive = (d.flags & BLSTM_FLAG_TEST_NO_ARRIVE) ? 1 : 0;
  p.inference = (d.flags & BLSTM_FLAG_INFERENCE) ? 1 : 0;
  p.limit_ns = d.wait_limit_us > 0 ? (unsigned long long)d.wait_limit_us * 1000ull : kDefaultWaitNs;
  p.ctl = reinterpret_cast<Control*>(ws);
  p.flags = reinterpret_cast<int*>(static_cast<char*>(ws) + sizeof(Control));
  p.Wh = Wh; p.ifgo = ifgo; p.out = out; p.cell = cell;
  CUtensorMap tw, tx, tx1;
  {  // Wh as {k, unit row, gate}
    uint64_t dims[3] = {(uint64_t)H, (uint64_t)H, 4}, str[2] = {(uint64_t)H * 2, (uint64_t)H * H * 2};
    uint32_t box[3] = {64, 32, 4};
    const int rc = encode_tensor_map(&tw, Wh, 3, dims, str, box);
    if (rc) return rc;
  }
  {  // out as {k of a chunk, batch row, chunk, step}: a group of chunks, or one
    uint64_t dims[4] = {64, (uint64_t)B, (uint64_t)H / 64, (uint64_t)T + 1}, str[3] = {(uint64_t)H * 2, 128, (uint64_t)B * H * 2};
    uint32_t box[4] = {64, RF_N, (uint32_t)pl.group, 1};
    int rc = encode_tensor_map(&tx, out, 4, dims, str, box);
    if (rc) return rc;
    box[2] = 1;
    rc = encode_tensor_map(&tx1, out, 4, dims, str, box);
    if (rc) return rc;
  }
  return p.fmt ? launch_coresident(fwd_tiles_kernel<__nv_bfloat16>, pl.grid, RF_THREADS, pl.smem, 1, st, tw, tx, tx1, p)
               : launch_coresident(fwd_tiles_kernel<__half>, pl.grid, RF_THREADS, pl.smem, 1, st, tw, tx, tx1, p);
}

int fwd_tiles_plan_detail(const FwdTilesPlan& p, char* buf, size_t n) {
  return snprintf(buf, n, "sm100 fwd resident weights tiles=%d groups=%d n=%d m_tiles=%d chunks=%d in_tmem=%d grid=%d threads=%d smem=%zu",
                  cdiv(p.nbt, p.ng), p.ng, RF_N, p.mt, p.kc, p.nt, p.grid, RF_THREADS, p.smem);
}

}  // namespace blstm
