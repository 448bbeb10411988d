// Backward recurrence with resident weights for large batches (16-bit, H = 256 to 1024): as in sm100_resident.cu the units are the
// M side of the MMAs and a CTA's slice of the weights lives in tensor memory - past H = 512 or so the rest of it in shared memory -
// but a group of CTAs works through several tiles of 64 or 32 batch rows in turn, so that one tile's hand-off hides behind the
// others'.
//
// Throughput bound, so the eight epilogue warps are not to wait for round trips: the read-out of the next tile's accumulator
// (part A: to the exchange buffers, shipped to the cluster's owners) comes before the gate maths of this one (part B),
// whose slices have arrived by then; exchange buffers, staging and output boxes are double; a warp of its own stores the
// boxes and counts the tiles in; the cell gradients of the tiles lie in the tensor memory that weights and
// accumulators leave.  Two issuers take every other tile, each with its own accumulator and its own half of the ring, which
// is what weights and exchange leave of shared memory, in stages of up to eight K chunks.  A CTA has 128 units where the
// kernel with the batch on the M side had 64 a cluster, which halves what a step reads of d_ifgo (67 MB at B = 4096, H = 512).
// us per step, that kernel -> this, launched alone: B = 4096, H = 512: 25.5 -> 20.2 (25.6 inside a training step, under the power cap);
// B = 2048: 12.9 -> 11.0; B = 4096, H = 256: 12.5 -> 9.1; B = 3000, H = 384: 19.1 -> 11.7.  Tiles of 32 rows: B = 1024,
// H = 1024 27.8 -> 19.3, B = 600 20.5 -> 12.4; B = 1500, H = 768 25.7 -> 18.9, B = 600 12.6 -> 8.3; B = 700, H = 896 16.1 -> 11.4;
// B = 1024, H = 512 8.4 -> 7.6; B = 1400, H = 384 9.5 -> 7.6.
// The epilogue warps set the pace (a 64-row tile takes them 4.4 k clocks: read-out and shipping 1.2, gate maths 1.1, bias gradient
// 0.9, fetching 0.5); sixteen of them with half the cells each were no faster (22.4).
#include <algorithm>
#include <cstdio>

#include "cluster_util.cuh"
#include "generic.cuh"
#include "resident_util.cuh"
#include "sm100_resident.cuh"

namespace blstm {
namespace sm100 {

constexpr int RT_THREADS = 384;            // producer, two issuers, publisher, eight epilogue warps
constexpr int RT_MAX_S = 8;                // stages of an issuer's ring

struct TilesParams {
  int T, B, H;
  int mt, ng, nbt;                         // M tiles; groups; batch tiles
  int kc, nt, w_col;                       // K chunks of a CTA; of these in tensor memory, from which column on
  int s2, group;                           // ring stages per issuer; chunks of a stage
  int fmt, no_arrive, flag_target;
  unsigned long long limit_ns;
  Control* ctl;
  int* flags;                              // [T+1][tiles]
  const void* Wh;
  const void* ifgo;
  const void* cell;
  const void* dout;
  const void* dh_n;
  const void* dc_n;
  void* dh0;
  void* dc0;
  float* db_part;                          // [groups * 32][4H] or null
};

// N: batch rows per tile, 64 or 32.
template <int N, typename T16>
__global__ void __launch_bounds__(RT_THREADS, 1)
tiles_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmX1,
             const __grid_constant__ CUtensorMap tmO, const TilesParams p) {
  constexpr int KS = 4, UT = 128, RO = N / KS, UP = UT * RO / 256, W = UP / 2, TPR = UT / UP;
  constexpr int SLOT = N * 128;                                     // a K chunk of a tile
  constexpr int STATE = 2 * N;                                      // tensor memory columns: two accumulators, states, weights
  constexpr int BLK = RO * 128, XB = KS * 4 * BLK;                  // exchanged block; one set of receive slots
  constexpr int SB = 3 * 4 * BLK;                                   // one set of staging slots (own slices stay here)
  constexpr int BOX = RO * 128 * 2 * 4;                             // the CTA's rows on their way out
  constexpr int EW = 8;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int H = p.H, T = p.T, KC = p.kc, S2 = p.s2;
  const int KG = p.group, nt = p.nt, n_kg = (KC + KG - 1) / KG, SG = KG * SLOT;
  uint8_t* w_s = smem;                                              // [KC - nt][16 KB]
  uint8_t* ring = w_s + (size_t)(KC - nt) * 16384;                  // [2 issuers][S2][group of chunks]
  uint8_t* recv = ring + (size_t)2 * S2 * SG;                       // [2][KS senders][4][RO][32] fp32
  uint8_t* stage = recv + 2 * XB;                                   // [2][3 receivers][4][RO][32] fp32
  uint8_t* boxes = stage + 2 * SB;                                  // [2][BOX]
  uint64_t* full = reinterpret_cast<uint64_t*>(boxes + 2 * BOX);    // [2][RT_MAX_S]
  uint64_t* empty = full + 2 * RT_MAX_S;                            // [2][RT_MAX_S]
  uint64_t* acc_full = empty + 2 * RT_MAX_S;                                  // [2] each from here on
  uint64_t* acc_empty = acc_full + 2;
  uint64_t* xchg = acc_empty + 2;
  uint64_t* consumed = xchg + 2;                                    // receive slots read by all owners
  uint64_t* box_full = consumed + 2;
  uint64_t* box_free = box_full + 2;
  uint64_t* taken = box_free + 2;                                   // receive slots read by this CTA's warps
  uint64_t* w_full = taken + 2;                                     // [1]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(w_full + 1);
  volatile int* dead = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int r = blockIdx.x % KS, mt = (blockIdx.x / KS) % p.mt, grp = blockIdx.x / KS / p.mt;
  const int kc0 = r * KC;
  const int NT = (p.nbt - grp + p.ng - 1) / p.ng;                   // tiles grp, grp + ng, ... (two at least)
  const int total = T * NT;                                         // items with a product

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2 * RT_MAX_S; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&acc_full[i], 1);
      mbar_init(&acc_empty[i], EW);
      mbar_init(&xchg[i], EW + 1);
      mbar_init(&consumed[i], KS);
      mbar_init(&taken[i], EW);
      mbar_init(&box_full[i], EW);
      mbar_init(&box_free[i], 1);
    }
    mbar_init(w_full, 1);
    *dead = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmX);
    tma_prefetch_desc(&tmX1);
    tma_prefetch_desc(&tmO);
  }
  if (warp == 1) tmem_alloc(tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  if (warp >= 4) {
    weights_to_tmem<true>(reinterpret_cast<const T16*>(p.Wh), H, mt, kc0, nt, tmem_base + p.w_col, warp & 3, (warp - 4) >> 2, lane);
    tc_fence_before();
  }
  __syncthreads();
  tc_fence_after();
  cluster_sync_all();
  WaitCtx wc{dead, p.ctl, p.limit_ns, -1, (int)blockIdx.x};
  auto tile_of = [&](int j) { return grp + j * p.ng; };
  // Item n = (step s = n / NT, tile j = n % NT): reads d_ifgo[T-1-s].
  if (warp == 0) {
    // ---------------------------------------------------------------- TMA producer
    if (lane == 0 && KC > nt) {
      mbar_expect_tx(w_full, (uint32_t)(KC - nt) * 16384);
      for (int kc = nt; kc < KC; ++kc) {
        uint8_t* dst = w_s + (size_t)(kc - nt) * 16384;
        tma_load_2d(dst, &tmW, w_full, mt * 128, (kc0 + kc) * 64);               // 64 k x 64 units, twice
        tma_load_2d(dst + 8192, &tmW, w_full, mt * 128 + 64, (kc0 + kc) * 64);
      }
    }
    // A stage has one lane that fills it, in the order in which it is consumed: a wait for a parity cannot tell a stage's next turn from the one
    // after it, so two lanes must not meet in a stage.  Lanes 0 and 1 take the even and the odd stages of an even ring; lane 0 takes all of an
    // odd one, and of a ring of 32-row tiles with four groups an item, where that is faster (us a step, two lanes / one: H = 1024, B = 1024 21.4 / 20.3,
    // H = 960, B = 2048 41.0 / 39.3; but 64-row tiles H = 512, B = 2048 12.7 / 13.7).
    const int two = S2 % 2 == 0 && (N == 64 || n_kg < 4);
    int early = 0, s = 0, j = 0;
    int gs[2] = {0, 0};                   // ring position of each issuer's next item
    uint32_t ph[2] = {0, 0};
    for (int n = 0; n < total; ++n) {
      const int t = T - 1 - s, tile = tile_of(j), x = n & 1;
      const int early_now = __shfl_sync(0xffffffffu, early, 31);
      int nj = j + 1, ns = s;
      if (nj == NT) { nj = 0; ++ns; }
      int seen = 1;
      if (lane == 0 && early_now < p.flag_target)
        seen = wait_flag_ge(&p.flags[(size_t)t * p.nbt + tile], p.flag_target, p.ctl, p.limit_ns, t, tile) ? 1 : 0;
      seen = __shfl_sync(0xffffffffu, seen, 0);
      __syncwarp();      // (a shuffle orders no memory: the issuing lanes come behind the acquire)
      if (!seen) { *dead = 1; break; }
      fence_proxy_async_global();
      bool ok = true;
      int pos = gs[0], po = ph[0];
      if (x) { pos = gs[1]; po = ph[1]; }
      if (lane <= two) {
        for (int kg = (lane + pos) & two; kg < n_kg; kg += 1 + two) {
          int st = pos + kg;
          uint32_t pp = po;
          while (st >= S2) { st -= S2; pp ^= 1; }
          uint64_t* f = &full[x * RT_MAX_S + st];
          if (!mbar_wait(&empty[x * RT_MAX_S + st], pp ^ 1, wc)) { ok = false; break; }
          const int kc = kg * KG, m = min(KG, KC - kc);
          uint8_t* dst = ring + (size_t)(x * S2 + st) * SG;
          mbar_expect_tx(f, m * SLOT);
          tma_load_4d(dst, m == KG ? &tmX : &tmX1, f, 0, tile * N, kc0 + kc, t);
        }
      } else if (lane == 31) {
        early = 0;
        if (ns < T) early = ld_acquire_gpu(&p.flags[(size_t)(T - 1 - ns) * p.nbt + tile_of(nj)]);
      }
      if (__any_sync(0xffffffffu, !ok)) break;
      pos += n_kg;
      while (pos >= S2) { pos -= S2; po ^= 1; }
      if (x) { gs[1] = pos; ph[1] = po; } else { gs[0] = pos; ph[0] = po; }
      j = nj; s = ns;
    }
  } else if (warp < 3) {
    // ---------------------------------------------------------------- MMA issuers: items x, x + 2, ...
    // (the warp waits, then one lane issues a group's MMAs without a branch that depends on data: see sm100_resident.cu)
    const int x = warp - 1;
    constexpr uint64_t descK = smem_desc_base(16, 1024), descA = smem_desc_base(8192, 1024);
    const uint32_t idesc_t = instr_desc(p.fmt, 0, 0, 128, N), idesc_s = instr_desc(p.fmt, 1, 0, 128, N);
    const uint32_t d_tmem = tmem_base + x * N, a_tmem = tmem_base + p.w_col, wa = smem_u32(w_s), ring_a = smem_u32(ring) + x * S2 * SG;
    int st = 0;
    uint32_t ph = 0;
    bool ok = KC <= nt || warp_wait_all(w_full, 0, wc);
    for (int n = x; n < total && ok; n += 2) {
      wc.d0 = n;
      if (!warp_wait_all(&acc_empty[x], ((uint32_t)(n >> 1) & 1u) ^ 1u, wc)) break;
      for (int kg = 0; kg < n_kg; ++kg) {
        if (!warp_wait_all(&full[x * RT_MAX_S + st], ph, wc)) { ok = false; break; }
        tc_fence_after();
        if (elect_one()) {
          const uint32_t sg = ring_a + st * SG;
          const int l0 = kg * KG, l1 = min(KC, l0 + KG), lt = max(l0, min(nt, l1));
          for (int lc = l0; lc < lt; ++lc) {
            const uint32_t sb = sg + (lc - l0) * SLOT;
#pragma unroll
            for (int k = 0; k < 4; ++k)
              umma_f16_ts(d_tmem, a_tmem + lc * 32 + k * 8, smem_desc(descK, sb + k * 32), idesc_t, (k > 0 || lc > 0) ? 1u : 0u);
          }
          for (int lc = lt; lc < l1; ++lc) {
            const uint32_t sb = sg + (lc - l0) * SLOT, sa = wa + (lc - nt) * 16384;
#pragma unroll
            for (int k = 0; k < 4; ++k)
              umma_f16(d_tmem, smem_desc(descA, sa + k * 2048), smem_desc(descK, sb + k * 32), idesc_s, (k > 0 || lc > 0) ? 1u : 0u);
          }
          umma_commit(&empty[x * RT_MAX_S + st]);
          if (kg + 1 == n_kg) umma_commit(&acc_full[x]);
        }
        __syncwarp();
        if (++st == S2) { st = 0; ph ^= 1; }
      }
    }
  } else if (warp == 3) {
    // ---------------------------------------------------------------- publisher: stores a tile's rows, counts the CTA in,
    // and tells the cluster when all eight warps have read an item's receive slots (for all of them: a release at cluster
    // scope stalls its thread for 0.7 k clocks and more)
    if (lane == 0) {
      const int items = total;            // (of steps T-1 .. 0: as many as have a product)
      int s = 0, j = 0;
      for (int m = 0; m < items + NT; ++m) {
        const int n = m - NT, b = m & 1;
        if (n >= 0 && n + 2 < total) {
          const int c = n & 1;
          wc.d0 = n;
          if (!mbar_wait(&taken[c], (uint32_t)(n >> 1) & 1u, wc)) break;
          fence_acq_rel_cluster();
#pragma unroll
          for (int dst = 0; dst < KS; ++dst) mbar_arrive_remote_relaxed(mapa_shared(smem_u32(&consumed[c]), dst));
        }
        if (m >= items) continue;
        const int t = T - 1 - s, tile = tile_of(j);
        wc.d0 = t; wc.d1 = tile;
        if (!mbar_wait(&box_full[b], (uint32_t)(m >> 1) & 1u, wc)) break;
        tma_store_4d(&tmO, boxes + b * BOX, mt * 128, tile * N + r * RO, 0, t);
        tma_store_commit();
        tma_store_wait<0>();
        mbar_arrive(&box_free[b]);
        if (!p.no_arrive) red_release_gpu_add(&p.flags[(size_t)t * p.nbt + tile], 1);
        if (++j == NT) { j = 0; ++s; }
      }
    }
  } else {
    // ---------------------------------------------------------------- epilogue
    const int ew = warp - 4, q = ew & 3, g = ew >> 2, et = ew * 32 + lane;
    const int lr = et / TPR, u = (et % TPR) * UP;                 // this thread's row of the owner's, first unit
    const int unit = mt * UT + u;
    const bool unit_ok = unit < H;
    const size_t H4 = 4 * (size_t)H;
    const T16* ifgo = reinterpret_cast<const T16*>(p.ifgo);
    const T16* cell = reinterpret_cast<const T16*>(p.cell);
    // on its way out: [4 gates][RO rows][128 units]
    constexpr int GS = RO * 256;
    uint8_t* mine = boxes + lr * (UT * 2) + u * 2;
    // (pieces of 16 bytes at places xor'ed with row and M quarter: see sm100_resident.cu)
    auto piece = [](int row, int quarter, int i) { return i ^ (((row ^ quarter) & 7) << 2); };
    const float* rd = reinterpret_cast<const float*>(recv) + lr * 32 + (u >> 5) * (BLK / 4);
    const uint32_t d_addr = tmem_base + (uint32_t(q * 32) << 16) + g * (N / 2);
    const uint32_t s_addr = tmem_base + STATE + (uint32_t(q * 32) << 16) + g * UP;
    // where this warp's half of an accumulator's columns goes: RO rows each for two owners
    constexpr int NB = 2;
    uint8_t* put[NB];
    int put_step[NB];                     // distance of the second buffer
#pragma unroll
    for (int i = 0; i < NB; ++i) {
      const int dst = g * 2 + i;
      const bool own = dst == r;
      put[i] = (own ? recv + (size_t)r * 4 * BLK : stage + (size_t)(dst < r ? dst : dst - 1) * 4 * BLK) + q * BLK;
      put_step[i] = own ? XB : SB;
    }
    // part A of item n
    auto part_a = [&](int n) -> bool {
      const int b = n & 1;
      const uint32_t k = (uint32_t)(n >> 1) & 1u;
      if (ew == 0 && lane == 0) mbar_expect_tx(&xchg[b], 3 * 4 * BLK);
      if (n >= 2 && !mbar_wait_cluster(&consumed[b], k ^ 1u, wc)) return false;
      if (!mbar_wait(&acc_full[b], k, wc)) return false;
      tc_fence_after();
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        uint32_t v[RO];
        tmem_ld_cols<RO>(d_addr + b * N + RO * i, v);
        tmem_ld_wait();
        uint8_t* to = put[i] + b * put_step[i];
#pragma unroll
        for (int c = 0; c < RO; ++c) reinterpret_cast<uint32_t*>(to + c * 128)[piece(c, q, lane)] = v[c];
      }
      tc_fence_before();
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&acc_empty[b]);
#pragma unroll
        for (int i = 0; i < NB; ++i) {
          const int dst = g * 2 + i;
          if (dst != r)
            dsmem_bulk_copy(mapa_shared(smem_u32(recv) + b * XB + (r * 4 + q) * BLK, dst), put[i] + b * SB, BLK, mapa_shared(smem_u32(&xchg[b]), dst));
        }
        mbar_arrive(&xchg[b]);
      }
      __syncwarp();
      return true;
    };
    // the cluster's products of item n, summed (part B)
    auto gather = [&](int n, float (&sum)[UP]) -> bool {
      const int b = n & 1;
      if (!mbar_wait_cluster(&xchg[b], (uint32_t)(n >> 1) & 1u, wc)) return false;
#pragma unroll
      for (int i = 0; i < UP; ++i) sum[i] = 0.f;
#pragma unroll
      for (int k = 0; k < KS; ++k)
#pragma unroll
        for (int i = 0; i < UP; i += 4) {
          const float4 v = *reinterpret_cast<const float4*>(rd + (size_t)b * (XB / 4) + k * BLK + piece(lr, u >> 5, (u & 31) + i));
          sum[i] += v.x;
          sum[i + 1] += v.y;
          sum[i + 2] += v.z;
          sum[i + 3] += v.w;
        }
      __syncwarp();
      if (lane == 0) mbar_arrive(&taken[b]);
      return true;
    };
    // the box of the m-th tile handed on: free to write / written
    auto box_wait = [&](int m) -> bool { return m < 2 || mbar_wait(&box_free[m & 1], ((uint32_t)(m >> 1) & 1u) ^ 1u, wc); };
    auto box_done = [&](int m) {
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&box_full[m & 1]);
    };
    auto row_of = [&](int j) { return tile_of(j) * N + r * RO + lr; };
    auto ld_state = [&](int j, float (&c)[UP]) {
      uint32_t v[UP];
      if constexpr (UP == 8) tmem_ld_32x8(s_addr + j * 16, v); else tmem_ld_32x4(s_addr + j * 8, v);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < UP; ++i) c[i] = __uint_as_float(v[i]);
    };
    auto st_state = [&](int j, const float (&c)[UP]) {
      uint32_t v[UP];
#pragma unroll
      for (int i = 0; i < UP; ++i) v[i] = __float_as_uint(c[i]);
      if constexpr (UP == 8) tmem_st_32x8(s_addr + j * 16, v); else tmem_st_32x4(s_addr + j * 8, v);
      tmem_st_wait();
    };
    const T16* dout = reinterpret_cast<const T16*>(p.dout);
    // Bias gradient: where a warp has two rows each half of it keeps two gates of both (registers are short).
    constexpr int DBG = UP == 8 ? 2 : 4;
    const int hi = UP == 8 ? lane >> 4 : 0;
    float db[DBG][UP];
#pragma unroll
    for (int gg = 0; gg < DBG; ++gg)
#pragma unroll
      for (int i = 0; i < UP; ++i) db[gg][i] = 0.f;
    uint32_t pf[7][W];                    // gates, c[t], c[t+1], dout[t]
#pragma unroll
    for (int k = 0; k < 7; ++k)
#pragma unroll
      for (int w = 0; w < W; ++w) pf[k][w] = 0u;
    auto prefetch = [&](int t, int j) {
      const int row = row_of(j);
      if (t < 0 || row >= p.B || !unit_ok) return;
      const size_t m = (size_t)t * p.B + row;
#pragma unroll
      for (int k = 0; k < 4; ++k) ld_words<W>(pf[k], ifgo + m * H4 + (size_t)k * H + unit);
      ld_words<W>(pf[4], cell + m * H + unit);
      ld_words<W>(pf[5], cell + (m + p.B) * H + unit);
      ld_words<W>(pf[6], dout + m * H + unit);
    };
    // two items ahead only into L2: a row's threads ask for its six runs of two lines
    auto prefetch_far = [&](int t, int j) {
      const int row = row_of(j), k = (lane & (TPR - 1)) >> 1, un = mt * 128 + (lane & 1) * 64;
      if (t < 0 || row >= p.B || k > 5 || un >= H) return;
      const size_t m = (size_t)t * p.B + row;
      prefetch_l2(k < 4 ? ifgo + m * H4 + (size_t)k * H + un : (k == 4 ? cell : dout) + m * H + un);
    };
    for (int j = 0; j < NT; ++j) {
      float c[UP];
#pragma unroll
      for (int i = 0; i < UP; ++i) c[i] = 0.f;
      const int row = row_of(j);
      if (p.dc_n && row < p.B && unit_ok) {
        uint32_t w[W];
        ld_words<W>(w, reinterpret_cast<const T16*>(p.dc_n) + (size_t)row * H + unit);
        unpack_words<T16, W>(w, c);
      }
      st_state(j, c);
    }
    // gate maths of step t, tile j; m: how many tiles have been handed on before
    auto maths = [&](int m, int t, int j, const float (&dh)[UP]) -> bool {
      const bool ok_cell = row_of(j) < p.B && unit_ok;
      float dc[UP];
      ld_state(j, dc);
      uint32_t dw[4][W];
#pragma unroll
      for (int w = 0; w < W; ++w) {
        const float2 pi = cvt2<T16>(pf[0][w]), pff = cvt2<T16>(pf[1][w]), pg = cvt2<T16>(pf[2][w]), po = cvt2<T16>(pf[3][w]);
        const float2 c0 = cvt2<T16>(pf[4][w]), c1 = cvt2<T16>(pf[5][w]), dd = cvt2<T16>(pf[6][w]);
        float d[2][4];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int i = 2 * w + e;
          const float si = sigmoid_fast(e ? pi.y : pi.x), sf = sigmoid_fast(e ? pff.y : pff.x), so = sigmoid_fast(e ? po.y : po.x);
          const float tg = tanh_fast(e ? pg.y : pg.x), tc = tanh_fast(e ? c1.y : c1.x);
          const float dv = (e ? dd.y : dd.x) + dh[i];
          const float dcv = fmaf(dv * so, 1.f - tc * tc, dc[i]);
          d[e][0] = dcv * (tg * si * (1.f - si));
          d[e][1] = dcv * ((e ? c0.y : c0.x) * sf * (1.f - sf));
          d[e][2] = dcv * (si * (1.f - tg * tg));
          d[e][3] = dv * (tc * so * (1.f - so));
          dc[i] = dcv * sf;
        }
#pragma unroll
        for (int gg = 0; gg < 4; ++gg) dw[gg][w] = pk2<T16>(d[0][gg], d[1][gg]);
      }
      st_state(j, dc);
      if (!box_wait(m)) return false;
#pragma unroll
      for (int gg = 0; gg < 4; ++gg) st_words<W>(mine + (m & 1) * BOX + gg * GS, dw[gg]);
      box_done(m);
      int nj = j + 1, nt = t;
      if (nj == NT) { nj = 0; --nt; }
      prefetch(nt, nj);
      int fj = nj + 1, ft = nt;
      if (fj == NT) { fj = 0; --ft; }
      prefetch_far(ft, fj);
      if (p.db_part)
#pragma unroll
        for (int gg = 0; gg < DBG; ++gg)
#pragma unroll
          for (int w = 0; w < W; ++w) {
            uint32_t keep = dw[gg][w];
            if constexpr (UP == 8) {
              const float2 o = cvt2<T16>(__shfl_xor_sync(0xffffffffu, ok_cell ? (hi ? dw[gg][w] : dw[gg + 2][w]) : 0u, 16));
              if (hi) keep = dw[gg + 2][w];
              db[gg][2 * w] += o.x;
              db[gg][2 * w + 1] += o.y;
            }
            const float2 f = cvt2<T16>(ok_cell ? keep : 0u);
            db[gg][2 * w] += f.x;
            db[gg][2 * w + 1] += f.y;
          }
      return true;
    };
    prefetch(T - 1, 0);
    bool ok = true;
    for (int j = 0; j < NT && ok; ++j) {
      float dh[UP];
#pragma unroll
      for (int i = 0; i < UP; ++i) dh[i] = 0.f;
      const int row = row_of(j);
      if (p.dh_n && row < p.B && unit_ok) {
        uint32_t w[W];
        ld_words<W>(w, reinterpret_cast<const T16*>(p.dh_n) + (size_t)row * H + unit);
        unpack_words<T16, W>(w, dh);
      }
      ok = maths(j, T - 1, j, dh);
    }
    int s = 0, j = 0;
    ok = ok && part_a(0);
    for (int n = 0; n < total && ok; ++n) {
      wc.d0 = n;
      if (n + 1 < total && !part_a(n + 1)) break;
      float dh[UP];
      if (!gather(n, dh)) break;
      if (s < T - 1) {
        if (!maths(NT + n, T - 2 - s, j, dh)) break;
      } else {
        const int row = row_of(j);
        float dc[UP];
        ld_state(j, dc);
        if (row < p.B && unit_ok) {
          uint32_t w[W];
          pack_words<T16, W>(w, dh);
          st_words<W>(reinterpret_cast<T16*>(p.dh0) + (size_t)row * H + unit, w);
          pack_words<T16, W>(w, dc);
          st_words<W>(reinterpret_cast<T16*>(p.dc0) + (size_t)row * H + unit, w);
        }
      }
      if (++j == NT) { j = 0; ++s; }
    }
    if (p.db_part && unit_ok) {
      float* dst = p.db_part + ((size_t)(grp * 4 + r) * EW + ew) * H4 + (size_t)2 * hi * H + unit;
#pragma unroll
      for (int gg = 0; gg < DBG; ++gg)
#pragma unroll
        for (int i = 0; i < UP; i += 4)
          *reinterpret_cast<float4*>(dst + (size_t)gg * H + i) = make_float4(db[gg][i], db[gg][i + 1], db[gg][i + 2], db[gg][i + 3]);
    }
  }
  // ---------------------------------------------------------------- teardown
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
  cluster_sync_all();     // no CTA leaves while a peer may still write into its shared memory
}

// Tiles of 64 rows up to H = 512 where there are four to eight.  Tiles of 32 rows from H = 768 on, where the kernel with the batch on the
// M side works with narrow slices or a short ring, and four of them from H = 384 to 512.  us a step, that kernel / this: H = 1024, 3, 4, 5
// and 8 tiles 14.3 / 10.3, 14.6 / 10.3, 21.2 / 13.6, 28.2 / 20.4; H = 896, 6 and 16 16.6 / 12.7, 42.6 / 32.5; H = 768, 4, 10 and 16 13.4 / 9.2,
// 29.4 / 20.1, 42.8 / 31.4; H = 512, 448 and 384, 4 9.0 / 8.5, 8.9 / 8.6, 10.2 / 8.4.  Not taken, measured while a shorter last stage took a load for each
// of its chunks: H = 768, 3 9.6 / 10.2; H = 704, 7 and 10 12.9 / 14.4, 16.5 / 20.9, H = 640, 8 15.2 / 15.5, H = 576, 8 13.3 / 15.9; H = 512, 6 9.7 / 11.2;
// H = 320, 6 9.6 / 11.1.
TilesPlan tiles_plan(const blstm_desc& d, int phase) {
  TilesPlan p{};
  const int H = d.hidden_size;
  if ((d.flags & BLSTM_FLAG_FORCE_GENERIC) || (d.dtype != BLSTM_F16 && d.dtype != BLSTM_BF16)) return p;
  if (phase != BLSTM_PHASE_BWD || H % 64 != 0 || H < RES_MIN_H || H > 1024) return p;
  p.mt = cdiv(H, 128);
  p.ng = resident_clusters(4) / ((d.flags & BLSTM_FLAG_HALF_DEVICE) ? 2 : 1) / p.mt;
  if (p.ng < 1) return p;
  p.N = H <= 512 && cdiv(cdiv(d.batch, 64), p.ng) >= 4 ? 64 : 32;
  p.nbt = cdiv(d.batch, p.N);
  const int most = cdiv(p.nbt, p.ng);
  if (p.N == 64 ? most > 8 : H >= 768 ? most < (H > 768 ? 3 : 4) || most > 16 : H < 384 || H > 512 || most != 4) return p;
  // a group of two tiles is two hand-off chains long: H = 832, that kernel / this, B = 289 (groups of three and two) 10.9 / 11.2, B = 384 (three each)
  // 11.1 / 9.2; from H = 896 on this wins all the same, B = 289 12.8 / 12.0
  if (H <= 832 && p.N == 32 && p.nbt < 3 * p.ng) return p;
  p.kc = H / 64;
  p.w_col = 2 * p.N + most * p.N / 4;
  p.nt = std::min(p.kc, (512 - p.w_col) / 32);
  // what weights and exchange leave of shared memory is the ring
  const int slot = p.N * 128, blk = p.N / 4 * 128;
  const size_t rest = 1024 + (size_t)(p.kc - p.nt) * 16384 + 2 * (16 * blk + 12 * blk + p.N / 4 * 1024) + 512;
  if (rest > 232448) return p;
  if (p.N == 64) {
    // Two stages of two chunks, or one of four.  us a step, two / one, four to eight tiles a group: H = 512 12.0 / 13.4, 14.1 / 13.5, 16.6 / 15.8,
    // 19.2 / 18.3, 22.0 / 20.9; H = 448 12.2 / 13.0, 14.1 / 13.6, 16.4 / 15.5, 18.8 / 17.6, 21.3 / 20.0; H = 384 10.9 / 12.9, 12.7 / 13.7, 15.0 / 15.7,
    // 17.4 / 17.9, 19.7 / 20.6; H = 320 10.9 / 12.7, 12.7 / 14.1, 14.9 / 16.0, 17.2 / 18.0, 19.5 / 20.5; H = 256, where four chunks are all, 10.0 / 10.0,
    // 12.3 / 12.1, 14.4 / 14.4, 17.7 / 17.4, 20.2 / 19.7.
    p.group = p.kc == 4 || (p.kc >= 7 && most > 4) ? 4 : 2;
    p.s2 = 4 / p.group;
  } else {
    // two stages an issuer, in as few and as equal groups as that allows; with fewer than four chunks a stage they do not pay (H = 1024, 16
    // tiles, stages of three: 65.9 us a step, the other kernel 56.1)
    const int room = (int)((232448 - rest) / slot);
    if (room < 16) return p;
    p.group = cdiv(p.kc, cdiv(p.kc, std::min(8, room / 4)));
    p.s2 = std::min({RT_MAX_S, 2 * cdiv(p.kc, p.group), room / (2 * p.group)});
  }
  p.smem = rest + (size_t)2 * p.s2 * p.group * slot;
  p.grid = p.ng * p.mt * 4;
  p.off_db = sizeof(Control) + round_up((size_t)d.seq_len * p.nbt * sizeof(int), 256);
  p.ws_bytes = p.off_db + (size_t)p.ng * 32 * 4 * H * sizeof(float);
  p.ok = true;
  return p;
}

}  // namespace sm100

using namespace sm100;

int tiles_bwd_recurrence(const blstm_desc& d, const TilesPlan& pl, const void* dout, const void* dh_n, const void* dc_n, const void* ifgo,
                         const void* cell, const void* Wh, void* d_ifgo, void* dh0, void* dc0, float* db, void* ws, cudaStream_t st) {
  const int H = d.hidden_size, B = d.batch, T = d.seq_len;
  TilesParams p{};
  p.T = T; p.B = B; p.H = H;
  p.mt = pl.mt; p.ng = pl.ng; p.nbt = pl.nbt; p.kc = pl.kc; p.nt = pl.nt; p.w_col = pl.w_col; p.s2 = pl.s2; p.group = pl.group;
  p.fmt = d.dtype == BLSTM_BF16 ? 1 : 0;
  p.no_arrive = (d.flags & BLSTM_FLAG_TEST_NO_ARRIVE) ? 1 : 0;
  p.flag_target = pl.mt * 4;
  p.limit_ns = d.wait_limit_us > 0 ? (unsigned long long)d.wait_limit_us * 1000ull : kDefaultWaitNs;
  p.ctl = reinterpret_cast<Control*>(ws);
  p.flags = reinterpret_cast<int*>(static_cast<char*>(ws) + sizeof(Control));
  p.Wh = Wh; p.ifgo = ifgo; p.cell = cell; p.dout = dout; p.dh_n = dh_n; p.dc_n = dc_n; p.dh0 = dh0; p.dc0 = dc0;
  p.db_part = db ? reinterpret_cast<float*>(static_cast<char*>(ws) + pl.off_db) : nullptr;
  CUtensorMap tw, tx, tx1, to;
  int rc;
  {  // Wh as {unit, k}
    uint64_t dims[2] = {(uint64_t)H, (uint64_t)4 * H}, str[1] = {(uint64_t)H * 2};
    uint32_t box[2] = {64, 64};
    rc = encode_tensor_map(&tw, Wh, 2, dims, str, box);
    if (rc) return rc;
  }
  {  // d_ifgo as {k of a chunk, batch row, chunk, step}: a stage's chunks, or those of an item's last stage
    uint64_t dims[4] = {64, (uint64_t)B, (uint64_t)H / 16, (uint64_t)T}, str[3] = {(uint64_t)4 * H * 2, 128, (uint64_t)B * 4 * H * 2};
    uint32_t box[4] = {64, (uint32_t)pl.N, (uint32_t)pl.group, 1};
    rc = encode_tensor_map(&tx, d_ifgo, 4, dims, str, box);
    if (rc) return rc;
    box[2] = pl.kc - (cdiv(pl.kc, pl.group) - 1) * pl.group;
    rc = encode_tensor_map(&tx1, d_ifgo, 4, dims, str, box);
    if (rc) return rc;
  }
  {  // ... as {unit, batch row, gate, step}
    uint64_t dims[4] = {(uint64_t)H, (uint64_t)B, 4, (uint64_t)T};
    uint64_t str[3] = {(uint64_t)4 * H * 2, (uint64_t)H * 2, (uint64_t)B * 4 * H * 2};
    uint32_t box[4] = {128, (uint32_t)pl.N / 4, 4, 1};
    rc = encode_tensor_map(&to, d_ifgo, 4, dims, str, box, 2, 0);
    if (rc) return rc;
  }
  auto launch = [&](auto kern) { return launch_coresident(kern, pl.grid, RT_THREADS, pl.smem, 4, st, tw, tx, tx1, to, p); };
  if (pl.N == 64) rc = p.fmt ? launch(tiles_kernel<64, __nv_bfloat16>) : launch(tiles_kernel<64, __half>);
  else            rc = p.fmt ? launch(tiles_kernel<32, __nv_bfloat16>) : launch(tiles_kernel<32, __half>);
  return rc || !db ? rc : reduce_db(p.db_part, pl.ng * 32, 4 * H, db, st);
}

int tiles_plan_detail(const TilesPlan& p, char* buf, size_t n) {
  return snprintf(buf, n, "sm100 bwd resident weights tiles=%d cluster=4 groups=%d n=%d m_tiles=%d chunks=%d in_tmem=%d stages=%d chunks_per_stage=%d grid=%d threads=%d smem=%zu",
                  cdiv(p.nbt, p.ng), p.ng, p.N, p.mt, p.kc, p.nt, 2 * p.s2, p.group, p.grid, RT_THREADS, p.smem);
}

}  // namespace blstm
