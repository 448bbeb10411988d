// Recurrences for large hidden sizes and up to a few hundred rows (16-bit): the weights stay on the chip for the whole
// sequence.  The gate rows (forward) or the units (backward) are the M side of the MMAs, so that the weights can be the A
// operand and live in TENSOR MEMORY - 192 to 240 KB of a CTA's slice of up to 256 - with the rest in shared memory, and a
// step only has to fetch the batch rows, the N side: 16 or twice 16 or 32 of them.  The recurrences with the batch on the M
// side fetch 128 rows per CTA whatever the batch, and from H = 1088 on the weights too, every step.
//
// Forward: a CTA has 32 units (128 gate rows) and K/KS of the H columns of Wh, KS = 1 or 2 CTAs in a cluster; backward:
// 128 units and a KS-th of the 4H rows, KS = 4 to 8.  The partial products of a cluster are reduce-scattered by batch
// rows through distributed shared memory to the first OWN CTAs, which do the gate maths of their rows: a thread has one
// row and UP adjacent units, their cell state or gradient in registers.  The same shared memory turns the accumulator
// (gate rows across lanes) into rows of units, for KS = 1 too.  h or d_ifgo leaves through plain stores, one release per
// owner, tile and step on the tile's counter behind them (TMA stores that the warps wait for in front of the release: 0.06 us a
// step more forward, 0.13 backward), and the whole K slice of the next step is fetched at once (no ring).
// Batch rows are divided over groups of CTAs that know nothing of each other.
//
// A step is a chain - products, exchange, gate maths, hand-off through L2 - of which the hand-off alone is half: release 1.1 k
// clocks, counter and acquire 1.2 k, first load 1 k.  So a group of more than 16 rows is two tiles that take turns: while one's
// rows are handed on, the other's products are formed.  Both tiles at half of N cost the tensor cores no more (an MMA of
// N = 32 takes 18 clocks, of N = 64 34; N = 16 11).
//
// us per step, one tile and MMAs issued behind a wait for each chunk -> now (B200, gates saved, inputs out of HBM, launch included):
// forward B=32 H=2048 4.4 -> 3.9, B=256 H=1024 5.8 -> 4.6, B=128 H=1024 4.3 -> 3.6, B=256 H=768 4.8 -> 4.3, B=512 H=512 4.5 -> 4.3; backward
// B=32 H=2048 6.9 -> 5.3, B=256 H=1024 6.3 -> 5.4, B=256 H=768 5.7 -> 4.9, B=512 H=512 5.4 -> 4.7, B=32 H=1536 4.6 -> 4.2.
// Bound by a tile's chain (some 7 to 9 k clocks a step), with K in four parts and 64 rows by the epilogue warps.
#include <algorithm>
#include <cstdio>

#include "cluster_util.cuh"
#include "generic.cuh"
#include "resident_util.cuh"
#include "sm100_resident.cuh"

namespace blstm {
namespace sm100 {

constexpr int RK = 64;                     // K chunk: one 128-byte swizzle row
constexpr int RES_MAX_KC = 22;             // chunks of a CTA's K slice
constexpr int RES_GROUP = 8;               // chunks that are fetched, waited for and multiplied at once, at most
constexpr int RES_MAX_KG = 8;              // groups of a K slice
constexpr int RES_THREADS = 384;           // producer, two issuers, publisher, eight epilogue warps

struct ResParams {
  int T, B, H;
  int mt, ks, rows;                        // M tiles; CTAs per cluster; batch rows per tile
  int kcm, nt;                             // most chunks of a K slice; chunks in tensor memory
  int x_bytes;                             // shared memory of a tile's batch rows, or of the staging laid over them if that is more
  int kc_total, group;                     // chunks of K; of these at once
  int fmt, no_arrive, inference, flag_target, n_groups;
  unsigned long long limit_ns;
  Control* ctl;
  int* flags;                              // [T+1][groups], a byte for each tile
  const void* Wh;
  void* ifgo;                              // forward: in/out; backward: in
  void* cell;
  void* x;                                 // what the steps hand on: out or d_ifgo
  const void* dout;
  const void* dh_n;
  const void* dc_n;
  void* dh0;
  void* dc0;
  float* db_part;                          // [groups * N][4H] partial sums, or null
};

// TI: tiles of N batch rows that a group works through in turn; NI: MMA issuers, each with an accumulator of its own per tile.
template <bool BWD, int TI, int N, int OWN, int NI, typename T16>
__global__ void __launch_bounds__(RES_THREADS, 1)
resident_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmX1,
                const ResParams p) {
  constexpr int UT = BWD ? 128 : 32;             // units per CTA
  constexpr int RO = N / OWN;                    // rows per owner
  constexpr int UP = UT * RO / 256 > 2 ? UT * RO / 256 : 2, W = UP / 2;  // units per epilogue thread
  constexpr int TPR = UT / UP;                   // threads per row
  constexpr int BLK = RO * 128;                  // exchanged block: RO rows x 32 M rows, fp32
  constexpr int A_COL = TI * NI * N;             // tensor memory: the accumulators, then the weights
  constexpr int EW = 8;
  // Who counts the CTA in: the last of its eight warps whose rows are stored, or a warp of its own, which keeps the 1.1 k clocks of
  // the release off the eight but comes some 200 later.  us a step, last warp / own warp: backward, two tiles of 32 rows,
  // B=512 H=512 5.28 / 4.59, B=256 H=768 5.41 / 4.77; B=32 H=2048 5.00 / 5.91.  Forward, where the last warp does it, two tiles of 32 rows: B=512
  // H=512 4.24 / 3.80, B=256 H=768 4.32 / 3.95, B=400 H=384 4.16 / 3.52, but H=1024 B=256 4.60 / 4.64 and, without gradients, 4.34 / 4.45.
  constexpr bool PUBLISHER = BWD && TI == 2 && N == 32;
  static_assert(UP <= 4, "");
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int H = p.H, T = p.T, KS = p.ks;
  uint8_t* w_s = smem;                                              // [kcm - nt][16 KB]
  uint8_t* x_s = w_s + (size_t)(p.kcm - p.nt) * 16384;              // per tile [kcm][rows][128 B]
  // ... and in it, per tile, idle from the item's last MMA until the CTA's rows have been counted in: [OWN receivers][4][RO][32] fp32
  uint8_t* recv = x_s + TI * p.x_bytes;                             // per tile [KS senders][4][RO][32] fp32
  const uint32_t recv_bytes = KS * 4 * BLK;
  uint64_t* full = reinterpret_cast<uint64_t*>(recv + TI * recv_bytes);   // [TI][RES_MAX_KG]
  uint64_t* w_full = full + TI * RES_MAX_KG;
  uint64_t* acc_full = w_full + 1;                                  // [TI]
  uint64_t* xchg = acc_full + TI;                                   // [TI]
  uint64_t* stored = xchg + TI;                                     // [TI] the CTA's rows are
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(stored + TI);
  volatile int* dead = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int* pub_cnt = const_cast<int*>(dead) + 1;                        // [TI]

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int r = blockIdx.x % KS;                                    // rank in the cluster
  const int mt = (blockIdx.x / KS) % p.mt, grp = blockIdx.x / KS / p.mt;
  const int kc0 = r * p.kc_total / KS, n_kc = (r + 1) * p.kc_total / KS - kc0;
  const int nt = min(p.nt, n_kc);
  const int tile0 = grp * TI;
  const int KG = p.group, n_kg = (n_kc + KG - 1) / KG, slot = p.rows * 128;     // groups of chunks; bytes of a chunk's rows

  if (threadIdx.x == 0) {
    for (int i = 0; i < TI * RES_MAX_KG; ++i) mbar_init(&full[i], 1);
    mbar_init(w_full, 1);
    for (int j = 0; j < TI; ++j) {
      mbar_init(&acc_full[j], NI);
      mbar_init(&xchg[j], 1 + EW);
      mbar_init(&stored[j], EW);
    }
    *dead = 0;
    for (int j = 0; j < TI; ++j) pub_cnt[j] = 0;
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
    weights_to_tmem<BWD>(reinterpret_cast<const T16*>(p.Wh), H, mt, kc0, nt, tmem_base + A_COL, warp & 3, (warp - 4) >> 2, lane);
    tc_fence_before();
  }
  __syncthreads();
  tc_fence_after();
  if (KS > 1) cluster_sync_all();     // peers' barriers exist before anyone ships to them
  WaitCtx wc{dead, p.ctl, p.limit_ns, -1, (int)blockIdx.x};
  // Products are formed for items 0 .. T-1: forward item s reads h[s]; backward item s reads d_ifgo[T-1-s].
  if (warp == 0) {
    // ---------------------------------------------------------------- TMA producer
    if (lane == 0 && n_kc > nt) {
      mbar_expect_tx(w_full, (uint32_t)(n_kc - nt) * 16384);
      for (int lc = nt; lc < n_kc; ++lc) {
        uint8_t* dst = w_s + (size_t)(lc - nt) * 16384;
        if constexpr (!BWD) {
          tma_load_3d(dst, &tmW, w_full, (kc0 + lc) * RK, mt * 32, 0);          // 4 gates x 32 units x 64 k
        } else {
          tma_load_2d(dst, &tmW, w_full, mt * 128, (kc0 + lc) * RK);            // 64 k x 64 units, twice
          tma_load_2d(dst + 8192, &tmW, w_full, mt * 128 + 64, (kc0 + lc) * RK);
        }
      }
    }
    for (int it = 0; it < TI * T; ++it) {
      const int s = it / TI, j = it % TI, t = BWD ? T - 1 - s : s;
      if (BWD || t > 0) {
        int seen = 1;
        if (lane == 0) seen = wait_flag_ge(&p.flags[(size_t)t * p.n_groups + grp], p.flag_target, p.ctl, p.limit_ns, t, tile0 + j, 8 * j) ? 1 : 0;
        seen = __shfl_sync(0xffffffffu, seen, 0);
        __syncwarp();      // (a shuffle orders no memory: the issuing lanes come behind the acquire)
        if (!seen) { *dead = 1; break; }
        fence_proxy_async_global();
      }
      if (lane < n_kg) {
        const int lc = lane * KG, n = min(KG, n_kc - lc);
        uint64_t* bar = &full[j * RES_MAX_KG + lane];
        uint8_t* dst = x_s + (size_t)j * p.x_bytes + lc * slot;
        mbar_expect_tx(bar, n * slot);
        if (n == KG) {
          tma_load_4d(dst, &tmX, bar, 0, (tile0 + j) * p.rows, kc0 + lc, t);
        } else {
          for (int i = 0; i < n; ++i) tma_load_4d(dst + i * slot, &tmX1, bar, 0, (tile0 + j) * p.rows, kc0 + lc + i, t);
        }
      }
      __syncwarp();
    }
  } else if (warp < 1 + NI) {
    // ---------------------------------------------------------------- MMA issuers: groups x, x + NI, ... of the chunks each
    // The warp waits for a group of chunks, then one lane issues all of their MMAs without a branch that depends on
    // data (one thread issues an MMA of N = 32 every 25 clocks so, every 85 with a wait for each chunk in between; a group
    // costs some 250 clocks besides: B=32 H=2048 backward in groups of 2, 4 and 8 chunks 7.5, 6.0 and 5.0 us a step).
    // The first chunks' weights lie in tensor memory, the others' in shared memory.
    const int x = warp - 1;
    constexpr uint64_t descK = smem_desc_base(16, 1024);
    constexpr uint64_t descA = BWD ? smem_desc_base(8192, 1024) : descK;
    const uint32_t idesc_t = instr_desc(p.fmt, 0, 0, 128, N), idesc_s = instr_desc(p.fmt, BWD ? 1 : 0, 0, 128, N);
    const uint32_t a_tmem = tmem_base + A_COL, wa = smem_u32(w_s);
    bool ok = n_kc <= nt || warp_wait_all(w_full, 0, wc);
    for (int it = 0; it < TI * T && ok; ++it) {
      const int s = it / TI, i = it % TI;
      const uint32_t d_tmem = tmem_base + (i * NI + x) * N, xa = smem_u32(x_s) + i * p.x_bytes;
      wc.d0 = s;
      for (int kg = x; kg < n_kg; kg += NI) {
        if (!warp_wait_all(&full[i * RES_MAX_KG + kg], s & 1, wc)) { ok = false; break; }
        tc_fence_after();
        if (elect_one()) {
          const int l0 = kg * KG, l1 = min(n_kc, l0 + KG), lt = max(l0, min(nt, l1));
          for (int lc = l0; lc < lt; ++lc) {
            const uint32_t sb = xa + lc * slot;
#pragma unroll
            for (int k = 0; k < 4; ++k)
              umma_f16_ts(d_tmem, a_tmem + lc * 32 + k * 8, smem_desc(descK, sb + k * 32), idesc_t, (k > 0 || lc != x * KG) ? 1u : 0u);
          }
          for (int lc = lt; lc < l1; ++lc) {
            const uint32_t sb = xa + lc * slot, sa = wa + (lc - nt) * 16384;
#pragma unroll
            for (int k = 0; k < 4; ++k)
              umma_f16(d_tmem, smem_desc(descA, sa + k * (BWD ? 2048 : 32)), smem_desc(descK, sb + k * 32), idesc_s, (k > 0 || lc != x * KG) ? 1u : 0u);
          }
          if (kg + NI >= n_kg) umma_commit(&acc_full[i]);
        }
        __syncwarp();
      }
    }
  } else if (warp == 3) {
    // ---------------------------------------------------------------- publisher
    for (int it = 0; PUBLISHER && it < TI * T && r < OWN; ++it) {
      const int s = it / TI, j = it % TI, t = BWD ? T - 1 - s : s + 1;
      int ok = 1;
      if (lane == 0) {
        ok = mbar_wait_spin(&stored[j], s & 1, wc);
        if (ok && !p.no_arrive) red_release_gpu_add(&p.flags[(size_t)t * p.n_groups + grp], 1 << 8 * j);
      }
      if (!__shfl_sync(0xffffffffu, ok, 0)) break;
    }
  } else if (warp >= 4) {
    // ---------------------------------------------------------------- epilogue
    const int ew = warp - 4, q = ew & 3, g = ew >> 2, et = ew * 32 + lane;
    const bool owner = r < OWN;
    const int lr = et / TPR, u = (et % TPR) * UP;                 // this thread's row among the owner's, first unit
    const int grow = r * RO + lr, unit = mt * UT + u;
    auto row_of = [&](int j) { return (tile0 + j) * p.rows + grow; };
    bool ok_cell[TI];
#pragma unroll
    for (int j = 0; j < TI; ++j) ok_cell[j] = owner && lr < RO && grow < p.rows && row_of(j) < p.B && unit < H;
    const size_t H4 = 4 * (size_t)H;
    const T16* ifgo = reinterpret_cast<const T16*>(p.ifgo);
    T16* cell = reinterpret_cast<T16*>(p.cell);
    const uint32_t tx = owner ? (uint32_t)(KS - 1) * 4 * BLK : 0u;
    // Exchanged rows (of 32 M rows) keep their 16-byte pieces at places xor'ed with row and M quarter: a warp reads several rows, or
    // quarters of a row, at a time, which would all begin in the same bank.
    auto piece = [](int row, int quarter, int i) { return i ^ (((row ^ quarter) & 7) << 2); };

    // where this warp's half of the accumulator's columns goes: RW_ rows each for NB receivers
    constexpr int NB = OWN > 1 ? OWN / 2 : 1, RW_ = N / 2 / NB, C = RW_ < 16 ? 8 : 16;
    const uint32_t taddr0 = tmem_base + (uint32_t(q * 32) << 16) + g * (N / 2);
    // this CTA's products of tile j's item s to the owners of the rows
    auto ship = [&](int s, int j) -> bool {
      if (ew == 0 && lane == 0) mbar_expect_tx(&xchg[j], tx);
      if (!mbar_wait(&acc_full[j], s & 1, wc)) return false;
      tc_fence_after();
      uint8_t* rv = recv + j * recv_bytes;
      uint8_t* stage = x_s + (size_t)j * p.x_bytes;
      const uint32_t taddr = taddr0 + j * NI * N;
#pragma unroll
      for (int c0 = 0; c0 < N / 2; c0 += C) {
        uint32_t a0[C], a1[C];
        tmem_ld_cols<C>(taddr + c0, a0);
        if constexpr (NI > 1) tmem_ld_cols<C>(taddr + N + c0, a1);
        tmem_ld_wait();
#pragma unroll
        for (int c = 0; c < C; ++c) {
          const int dst = OWN > 1 ? g * NB + (c0 + c) / RW_ : 0, rr = (c0 + c) % RW_ + (OWN > 1 ? 0 : g * RW_);
          uint8_t* put = (dst == r ? rv + (size_t)r * 4 * BLK : stage + (size_t)dst * 4 * BLK) + q * BLK + rr * 128;
          reinterpret_cast<float*>(put)[piece(rr, q, lane)] = NI > 1 ? __uint_as_float(a0[c]) + __uint_as_float(a1[c]) : __uint_as_float(a0[c]);
        }
      }
      tc_fence_before();
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        if constexpr (OWN > 1) {
#pragma unroll
          for (int i = 0; i < NB; ++i) {
            const int dst = g * NB + i;
            if (dst != r)
              dsmem_bulk_copy(mapa_shared(smem_u32(rv) + (r * 4 + q) * BLK, dst), stage + (size_t)(dst * 4 + q) * BLK, BLK,
                              mapa_shared(smem_u32(&xchg[j]), dst));
          }
        }
        mbar_arrive(&xchg[j]);
      }
      __syncwarp();
      return true;
    };
    // the cluster's products, summed
    constexpr int G = BWD ? 1 : 4;
    auto collect = [&](int s, int j, float (&sum)[G][UP]) -> bool {
      const uint8_t* rv = recv + j * recv_bytes;
      if (!(OWN > 1 ? mbar_wait_cluster(&xchg[j], s & 1, wc) : mbar_wait(&xchg[j], s & 1, wc))) return false;
#pragma unroll
      for (int gg = 0; gg < G; ++gg)
#pragma unroll
        for (int i = 0; i < UP; ++i) sum[gg][i] = 0.f;
      if (lr < RO)
        for (int k = 0; k < KS; ++k)
#pragma unroll
          for (int gg = 0; gg < G; ++gg) {
            const int quarter = BWD ? u >> 5 : gg;
            const float* rd = reinterpret_cast<const float*>(rv + (size_t)(k * 4 + quarter) * BLK) + lr * 32 + piece(lr, quarter, u & 31);
            if constexpr (UP == 4) {
              const float4 v = *reinterpret_cast<const float4*>(rd);
              sum[gg][0] += v.x; sum[gg][1] += v.y; sum[gg][2] += v.z; sum[gg][3] += v.w;
            } else {
              const float2 v = *reinterpret_cast<const float2*>(rd);
              sum[gg][0] += v.x; sum[gg][1] += v.y;
            }
          }
      return true;
    };
    // This warp's rows of step t are stored: the CTA is counted in once all eight warps' are.
    auto publish = [&](int t, int j) {
      __syncwarp();
      if (lane == 0) {
        if constexpr (PUBLISHER) mbar_arrive(&stored[j]);
        else if ((smem_count_arrive(&pub_cnt[j]) & (EW - 1)) == EW - 1 && !p.no_arrive)
          red_release_gpu_add(&p.flags[(size_t)t * p.n_groups + grp], 1 << 8 * j);
      }
      __syncwarp();
    };
    if constexpr (!BWD) {
      float c[TI][UP];
      uint32_t pre[TI][4][W];
      auto load_pre = [&](int t, int j) {
        if (ok_cell[j] && t < T)
#pragma unroll
          for (int gg = 0; gg < 4; ++gg) ld_words<W>(pre[j][gg], ifgo + ((size_t)t * p.B + row_of(j)) * H4 + (size_t)gg * H + unit);
      };
#pragma unroll
      for (int j = 0; j < TI; ++j) {
#pragma unroll
        for (int i = 0; i < UP; ++i) c[j][i] = 0.f;
        if (ok_cell[j]) {
          uint32_t w[W];
          ld_words<W>(w, cell + (size_t)row_of(j) * H + unit);
          unpack_words<T16, W>(w, c[j]);
        }
        load_pre(0, j);
      }
      // What only backward needs of an item is stored during the next one's exchange: the release waits for every store of the SM that
      // is under way.
      uint32_t kept[5][W];
      int kept_t = -1;
      auto store_kept = [&](int j) {
        if (kept_t < 0 || !ok_cell[j]) return;
        if (!p.inference)
#pragma unroll
          for (int gg = 0; gg < 4; ++gg)
            st_words<W>(reinterpret_cast<T16*>(p.ifgo) + ((size_t)kept_t * p.B + row_of(j)) * H4 + (size_t)gg * H + unit, kept[gg]);
        if (!p.inference || kept_t == T - 1) st_words<W>(cell + ((size_t)(kept_t + 1) * p.B + row_of(j)) * H + unit, kept[4]);
      };
      bool go = true;
      for (int t = 0; t < T && go; ++t) {
        wc.d0 = t;
#pragma unroll
        for (int j = 0; j < TI; ++j) {
          float pa[4][UP];
          if (!go || !ship(t, j)) { go = false; break; }
          store_kept((j + TI - 1) % TI);
          if (!collect(t, j, pa)) { go = false; break; }
          uint32_t hw[W];
          float hv[UP];
#pragma unroll
          for (int gg = 0; gg < 4; ++gg)
#pragma unroll
            for (int w = 0; w < W; ++w) {
              const float2 f = cvt2<T16>(pre[j][gg][w]);
              pa[gg][2 * w] += f.x;
              pa[gg][2 * w + 1] += f.y;
            }
#pragma unroll
          for (int i = 0; i < UP; ++i) {
            c[j][i] = sigmoid_fast(pa[1][i]) * c[j][i] + sigmoid_fast(pa[0][i]) * tanh_fast(pa[2][i]);
            hv[i] = sigmoid_fast(pa[3][i]) * tanh_fast(c[j][i]);
          }
          pack_words<T16, W>(hw, hv);
          if (ok_cell[j]) st_words<W>(reinterpret_cast<T16*>(p.x) + ((size_t)(t + 1) * p.B + row_of(j)) * H + unit, hw);
          publish(t + 1, j);
          load_pre(t + 1, j);
          kept_t = t;
#pragma unroll
          for (int gg = 0; gg < 4; ++gg) pack_words<T16, W>(kept[gg], pa[gg]);
          pack_words<T16, W>(kept[4], c[j]);
        }
      }
      if (go) store_kept(TI - 1);
    } else {
      const T16* dout = reinterpret_cast<const T16*>(p.dout);
      float dc[TI][UP], dh[1][UP], db[4][UP];             // db: the bias gradient, of the d_ifgo values as stored, of all tiles
      float fA[UP], fBi[UP], fBg[UP], fBo[UP], fSf[UP];
      uint32_t dd[W], c0[W];                              // dout[t], c[t]
      uint32_t pf[TI][6][W], cn[TI][W];                   // gates, c[t], dout[t]; c[t+1]
      float dhn[TI][UP];                                  // gradient of the last output
      auto prefetch = [&](int t, int j) {
        if (!ok_cell[j]) return;
        const size_t m = (size_t)t * p.B + row_of(j);
#pragma unroll
        for (int k = 0; k < 4; ++k) ld_words<W>(pf[j][k], ifgo + m * H4 + (size_t)k * H + unit);
        ld_words<W>(pf[j][4], cell + m * H + unit);
        ld_words<W>(pf[j][5], dout + m * H + unit);
      };
#pragma unroll
      for (int j = 0; j < TI; ++j) {
#pragma unroll
        for (int k = 0; k < 6; ++k)
#pragma unroll
          for (int w = 0; w < W; ++w) pf[j][k][w] = 0u;
#pragma unroll
        for (int w = 0; w < W; ++w) cn[j][w] = 0u;
#pragma unroll
        for (int i = 0; i < UP; ++i) dc[j][i] = dhn[j][i] = 0.f;
        if (ok_cell[j]) {
          uint32_t w[W];
          ld_words<W>(cn[j], cell + ((size_t)T * p.B + row_of(j)) * H + unit);
          if (p.dc_n) { ld_words<W>(w, reinterpret_cast<const T16*>(p.dc_n) + (size_t)row_of(j) * H + unit); unpack_words<T16, W>(w, dc[j]); }
          if (p.dh_n) { ld_words<W>(w, reinterpret_cast<const T16*>(p.dh_n) + (size_t)row_of(j) * H + unit); unpack_words<T16, W>(w, dhn[j]); }
        }
        prefetch(T - 1, j);
      }
#pragma unroll
      for (int gg = 0; gg < 4; ++gg)
#pragma unroll
        for (int i = 0; i < UP; ++i) db[gg][i] = 0.f;
      // everything that does not depend on dh, while the products are being formed:
      //   dh = dout + carry;  dcv = dh*fA + dc;  d_i = dcv*fBi;  d_f = dcv*c*fSf*(1-fSf);  d_g = dcv*fBg;  d_o = dh*fBo;  dc' = dcv*fSf
      // (c = c[t] and dout stay packed: registers are short)
      auto factors = [&](int j) {
#pragma unroll
        for (int w = 0; w < W; ++w) {
          const float2 pi = cvt2<T16>(pf[j][0][w]), pff = cvt2<T16>(pf[j][1][w]), pg = cvt2<T16>(pf[j][2][w]), po = cvt2<T16>(pf[j][3][w]);
          const float2 c1 = cvt2<T16>(cn[j][w]);
          cn[j][w] = c0[w] = pf[j][4][w];
          dd[w] = pf[j][5][w];
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int i = 2 * w + e;
            const float si = sigmoid_fast(e ? pi.y : pi.x), sf = sigmoid_fast(e ? pff.y : pff.x), so = sigmoid_fast(e ? po.y : po.x);
            const float tg = tanh_fast(e ? pg.y : pg.x), tc = tanh_fast(e ? c1.y : c1.x);
            fA[i] = so * (1.f - tc * tc);
            fBi[i] = tg * si * (1.f - si);
            fBg[i] = si * (1.f - tg * tg);
            fBo[i] = tc * so * (1.f - so);
            fSf[i] = sf;
          }
        }
      };
      bool go = true;
      for (int st = 0; st <= T && go; ++st) {
        wc.d0 = T - st;
        const int t = T - 1 - st;
#pragma unroll
        for (int j = 0; j < TI; ++j) {
          if (owner && st < T) factors(j);
          if (st == 0) {
#pragma unroll
            for (int i = 0; i < UP; ++i) dh[0][i] = dhn[j][i];
          } else if (!go || !ship(st - 1, j) || (owner && !collect(st - 1, j, dh))) {
            go = false;
            break;
          }
          if (!owner) continue;
          if (st == T) {
            if (ok_cell[j]) {
              uint32_t w[W];
              pack_words<T16, W>(w, dh[0]);
              st_words<W>(reinterpret_cast<T16*>(p.dh0) + (size_t)row_of(j) * H + unit, w);
              pack_words<T16, W>(w, dc[j]);
              st_words<W>(reinterpret_cast<T16*>(p.dc0) + (size_t)row_of(j) * H + unit, w);
            }
            continue;
          }
          float d[4][UP];
          uint32_t dw[4][W];
#pragma unroll
          for (int i = 0; i < UP; ++i) {
            const float2 d2 = cvt2<T16>(dd[i / 2]), c2 = cvt2<T16>(c0[i / 2]);
            const float dv = (i & 1 ? d2.y : d2.x) + dh[0][i], dcv = fmaf(dv, fA[i], dc[j][i]);
            d[0][i] = dcv * fBi[i];
            d[1][i] = dcv * ((i & 1 ? c2.y : c2.x) * (fSf[i] * (1.f - fSf[i])));
            d[2][i] = dcv * fBg[i];
            d[3][i] = dv * fBo[i];
            dc[j][i] = dcv * fSf[i];
          }
#pragma unroll
          for (int gg = 0; gg < 4; ++gg) {
            pack_words<T16, W>(dw[gg], d[gg]);
            if (ok_cell[j]) st_words<W>(reinterpret_cast<T16*>(p.x) + ((size_t)t * p.B + row_of(j)) * H4 + (size_t)gg * H + unit, dw[gg]);
          }
          publish(t, j);
          if (t > 0) prefetch(t - 1, j);
          if (p.db_part)
#pragma unroll
            for (int gg = 0; gg < 4; ++gg)
#pragma unroll
              for (int w = 0; w < W; ++w) {
                const float2 f = cvt2<T16>(ok_cell[j] ? dw[gg][w] : 0u);
                db[gg][2 * w] += f.x;
                db[gg][2 * w + 1] += f.y;
              }
        }
      }
      if (p.db_part && owner && unit < H) {
        float* dst = p.db_part + ((size_t)grp * N + grow) * H4 + unit;
#pragma unroll
        for (int gg = 0; gg < 4; ++gg)
#pragma unroll
          for (int i = 0; i < UP; i += 2) *reinterpret_cast<float2*>(dst + (size_t)gg * H + i) = make_float2(db[gg][i], db[gg][i + 1]);
      }
    }
  }
  // ---------------------------------------------------------------- teardown
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
  if (KS > 1) cluster_sync_all();     // no CTA leaves while a peer may still write into its shared memory
}

// The smallest split of K whose slice fits the chip, and as many groups of rows as fit beside each other.  Backward, a slice
// of 22 chunks and 32 rows fits with one issuer only (one accumulator instead of two leaves tensor memory for the chunk
// that would not fit); one more CTA a cluster makes room for two, which is worth it while a group keeps to 32 rows.  us a
// step: H = 1728, B = 32: 5.1 -> 4.1, H = 1408, B = 64: 5.0 -> 4.1; B = 96, then 48 rows a group, stays at 5.1.
// H = 2048 with 17 to 32 rows is left with one issuer over six CTAs (5.0; two take 4.4 at H = 1984): a B200 holds
// 15 clusters of seven or eight CTAs and 16 M tiles need 16; the kernel with the batch on the M side takes 8.6.
ResPlan resident_plan(const blstm_desc& d, int phase) {
  const int H = d.hidden_size, B = d.batch;
  const bool bwd = phase == BLSTM_PHASE_BWD;
  if ((d.flags & BLSTM_FLAG_FORCE_GENERIC) || (d.dtype != BLSTM_F16 && d.dtype != BLSTM_BF16)) return ResPlan{};
  if (phase != BLSTM_PHASE_FWD && !bwd) return ResPlan{};
  if (H % 64 != 0 || H < RES_MIN_H || H > 2048) return ResPlan{};
  ResPlan one{};                         // what fits with one issuer
  for (int ks = bwd ? 4 : 1; ks <= (bwd ? 8 : 2); ++ks) {
    ResPlan p{};
    p.ks = ks;
    p.mt = bwd ? cdiv(H, 128) : H / 32;
    p.kc_total = bwd ? H / 16 : H / 64;
    int cap = p.ks == 1 ? plan_sm_count() : resident_clusters(p.ks);
    if (d.flags & BLSTM_FLAG_HALF_DEVICE) cap /= 2;
    p.ng = cap / p.mt;
    if (p.ng < 1) continue;
    // (tiles of eight rows do not pay: B = 64, H = 1024 backward 3.64 us a step as one tile, 3.89 as two, B = 16, H = 2048 4.21 / 4.89)
    // Backward up to H = 448 one tile of 32 rows beats two of 16: H = 320, 308 and 352 rows 4.37 / 4.40 and 4.36 / 4.55, H = 384, 264, 308 and 352 rows
    // 4.31 / 4.41, 4.42 / 4.60 and 4.44 / 4.64, H = 448, 256 rows 4.54 / 4.72; from H = 576 on two win (120 rows 4.36 / 4.09, 168 4.65 / 4.66).
    const int group_rows = cdiv(B, p.ng);
    p.ti = group_rows <= 16 || (bwd && H <= 448 && group_rows <= 32) ? 1 : 2;
    p.rows = (int)round_up((size_t)cdiv(B, p.ng * p.ti), 8);
    p.ng = cdiv(B, p.rows * p.ti);
    p.own = bwd ? 4 : p.ks;
    p.N = p.rows <= 16 ? 16 : 32;
    if (p.rows > 32) continue;
    p.kcm = cdiv(p.kc_total, p.ks);
    const size_t x = std::max((size_t)p.kcm * p.N * 128, (size_t)p.N * 512);
    p.x_bytes = (int)x;
    for (p.ni = 2; p.ni >= 1; --p.ni) {
      p.nt = std::min(p.kcm, (512 - p.ti * p.ni * p.N) / 32);
      p.smem = 1024 + (size_t)(p.kcm - p.nt) * 16384 + p.ti * (x + (size_t)p.ks * 4 * (p.N / p.own) * 128) + 512;
      if (p.smem <= 232448 || !(bwd && p.ti * p.N == 32)) break;
    }
    if (p.smem > 232448 || p.ni < 1 || p.kcm > RES_MAX_KC) continue;
    p.group = cdiv(p.kcm, p.ni * cdiv(p.kcm, p.ni * RES_GROUP));      // as many groups for each issuer
    if (cdiv(p.kc_total / p.ks, p.group) < p.ni) continue;            // (an issuer without a group would never commit)
    if (one.ok && (p.ni < 2 || p.ti * p.N > 32)) continue;
    p.grid = p.ng * p.mt * p.ks;
    p.off_db = sizeof(Control) + round_up((size_t)(d.seq_len + 1) * p.ng * sizeof(int), 256);
    p.ws_bytes = p.off_db + (bwd ? (size_t)p.ng * p.N * 4 * H * sizeof(float) : 0);
    p.ok = true;
    if (p.ni == 2) return p;
    one = p;
  }
  return one;
}

template <bool BWD, int TI, int N, int OWN, int NI, typename T16>
static int launch_t(const ResPlan& pl, const CUtensorMap& tw, const CUtensorMap& tx, const CUtensorMap& tx1, const ResParams& p, cudaStream_t st) {
  return launch_coresident(resident_kernel<BWD, TI, N, OWN, NI, T16>, pl.grid, RES_THREADS, pl.smem, pl.ks, st, tw, tx, tx1, p);
}

static int launch(const blstm_desc& d, const ResPlan& pl, bool bwd, void* x, ResParams& p, void* ws, cudaStream_t st) {
  const int H = d.hidden_size, B = d.batch, T = d.seq_len;
  p.T = T; p.B = B; p.H = H; p.x = x;
  p.mt = pl.mt; p.ks = pl.ks; p.rows = pl.rows; p.kcm = pl.kcm; p.nt = pl.nt; p.x_bytes = pl.x_bytes; p.kc_total = pl.kc_total; p.group = pl.group;
  p.fmt = d.dtype == BLSTM_BF16 ? 1 : 0;
  p.no_arrive = (d.flags & BLSTM_FLAG_TEST_NO_ARRIVE) ? 1 : 0;
  p.inference = (d.flags & BLSTM_FLAG_INFERENCE) ? 1 : 0;
  p.flag_target = pl.mt * pl.own;
  p.n_groups = pl.ng;
  p.limit_ns = d.wait_limit_us > 0 ? (unsigned long long)d.wait_limit_us * 1000ull : kDefaultWaitNs;
  p.ctl = reinterpret_cast<Control*>(ws);
  p.flags = reinterpret_cast<int*>(static_cast<char*>(ws) + sizeof(Control));
  CUtensorMap tw, tx, tx1;
  const uint64_t K = bwd ? 4 * H : H, steps = bwd ? T : T + 1;
  int rc;
  if (bwd) {  // Wh as {unit, k}
    uint64_t dims[2] = {(uint64_t)H, (uint64_t)4 * H}, str[1] = {(uint64_t)H * 2};
    uint32_t box[2] = {64, 64};
    rc = encode_tensor_map(&tw, p.Wh, 2, dims, str, box);
  } else {    // Wh as {k, unit row, gate}
    uint64_t dims[3] = {(uint64_t)H, (uint64_t)H, 4}, str[2] = {(uint64_t)H * 2, (uint64_t)H * H * 2};
    uint32_t box[3] = {RK, 32, 4};
    rc = encode_tensor_map(&tw, p.Wh, 3, dims, str, box);
  }
  if (rc) return rc;
  {  // the product's other operand as {k of a chunk, batch row, chunk, step}: a group of chunks, or one
    uint64_t dims[4] = {RK, (uint64_t)B, K / RK, steps}, str[3] = {K * 2, RK * 2, (uint64_t)B * K * 2};
    uint32_t box[4] = {RK, (uint32_t)pl.rows, (uint32_t)pl.group, 1};
    rc = encode_tensor_map(&tx, x, 4, dims, str, box);
    if (rc) return rc;
    box[2] = 1;
    rc = encode_tensor_map(&tx1, x, 4, dims, str, box);
    if (rc) return rc;
  }
#define BLSTM_RES(BW, TT, NN, OO, II)                                                                 \
  if (bwd == BW && pl.ti == TT && pl.N == NN && pl.own == OO && pl.ni == II)                          \
    return p.fmt ? launch_t<BW, TT, NN, OO, II, __nv_bfloat16>(pl, tw, tx, tx1, p, st) : launch_t<BW, TT, NN, OO, II, __half>(pl, tw, tx, tx1, p, st);
  BLSTM_RES(false, 1, 16, 1, 2) BLSTM_RES(false, 1, 16, 2, 2) BLSTM_RES(false, 2, 16, 1, 2) BLSTM_RES(false, 2, 16, 2, 2)
  BLSTM_RES(false, 2, 32, 1, 2) BLSTM_RES(false, 2, 32, 2, 2)
  BLSTM_RES(true, 1, 16, 4, 2) BLSTM_RES(true, 1, 32, 4, 2) BLSTM_RES(true, 2, 16, 4, 2) BLSTM_RES(true, 2, 16, 4, 1) BLSTM_RES(true, 2, 32, 4, 2)
#undef BLSTM_RES
  return BLSTM_E_UNSUPPORTED;
}

}  // namespace sm100

using namespace sm100;

int resident_fwd_recurrence(const blstm_desc& d, const ResPlan& pl, void* ifgo, const void* Wh, void* out, void* cell, void* ws, cudaStream_t st) {
  ResParams p{};
  p.Wh = Wh; p.ifgo = ifgo; p.cell = cell;
  return launch(d, pl, false, out, p, ws, st);
}

int resident_bwd_recurrence(const blstm_desc& d, const ResPlan& pl, const void* dout, const void* dh_n, const void* dc_n, const void* ifgo,
                            const void* cell, const void* Wh, void* d_ifgo, void* dh0, void* dc0, float* db, void* ws, cudaStream_t st) {
  ResParams p{};
  p.Wh = Wh; p.ifgo = const_cast<void*>(ifgo); p.cell = const_cast<void*>(cell);
  p.dout = dout; p.dh_n = dh_n; p.dc_n = dc_n; p.dh0 = dh0; p.dc0 = dc0;
  p.db_part = db ? reinterpret_cast<float*>(static_cast<char*>(ws) + pl.off_db) : nullptr;
  const int rc = launch(d, pl, true, d_ifgo, p, ws, st);
  return rc || !db ? rc : reduce_db(p.db_part, pl.ng * pl.N, 4 * d.hidden_size, db, st);
}

int resident_plan_detail(const ResPlan& p, int phase, char* buf, size_t n) {
  return snprintf(buf, n, "sm100 %s resident weights cluster=%d groups=%d tiles=%d rows_per_tile=%d n=%d m_tiles=%d chunks=%d in_tmem=%d issuers=%d grid=%d threads=%d smem=%zu",
                  phase == BLSTM_PHASE_BWD ? "bwd" : "fwd", p.ks, p.ng, p.ti, p.rows, p.N, p.mt, p.kcm, p.nt, p.ni, p.grid, RES_THREADS, p.smem);
}

}  // namespace blstm
