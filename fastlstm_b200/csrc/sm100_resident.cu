// Recurrences for large hidden sizes and up to a few hundred rows (16-bit): the weights stay on the chip for the whole
// sequence.  The gate rows (forward) or the units (backward) are the M side of the MMAs, so that the weights can be the A
// operand and live in TENSOR MEMORY - 192 to 240 KB of a CTA's slice of up to 256 - with the rest in shared memory, and a
// step only has to fetch the batch rows, the N side: 16 to 64 of them.  The recurrences with the batch on the M side
// fetch 128 rows per CTA whatever the batch, and from H = 1088 on the weights too, every step.
//
// Forward: a CTA has 32 units (128 gate rows) and K/KS of the H columns of Wh, KS = 1 or 2 CTAs in a cluster; backward:
// 128 units and a KS-th of the 4H rows, KS = 4 to 8.  The partial products of a cluster are reduce-scattered by batch
// rows through distributed shared memory to the first OWN CTAs, which do the gate maths of their rows: a thread has one
// row and UP adjacent units, their cell state or gradient in registers.  The same shared memory turns the accumulator
// (gate rows across lanes) into rows of units, for KS = 1 too.  h or d_ifgo leaves through plain stores, one release per
// owner and step on the group's counter behind them (TMA stores that the warps wait for in front of the release: 0.06 us a
// step more forward, 0.13 backward), and the whole K slice of the next step is fetched at once (no ring).
// Batch rows are divided over groups of CTAs that know nothing of each other.
//
// us per step, the recurrences with the batch on the M side -> these (B200): forward B=32 H=2048 7.9 -> 4.4, B=256 H=1024
// 7.2 -> 5.7, B=128 H=1024 4.2, B=256 H=768 6.7 -> 4.7; backward B=32 H=2048 10.0 -> 6.8, B=256 H=1024 7.6 -> 6.1, B=256 H=768
// 6.8 -> 5.6, B=32 H=1536 4.5.
// Bound by the chain of a step: hand-off through L2 (its release alone 0.5 us), fetch of N rows, 64 MMAs of some 50 clocks,
// exchange, gate maths.
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
constexpr int RES_THREADS = 384;           // producer, two issuers, one idle warp, eight epilogue warps

struct ResParams {
  int T, B, H;
  int mt, ks, rows;                        // M tiles; CTAs per cluster; batch rows per group
  int kcm, nt;                             // most chunks of a K slice; chunks in tensor memory
  int x_bytes;                             // shared memory of the batch rows, or of the staging laid over them if that is more
  int kc_total;
  int fmt, no_arrive, inference, flag_target, n_groups;
  unsigned long long limit_ns;
  Control* ctl;
  int* flags;                              // [T+1][groups]
  const void* Wh;
  void* ifgo;                              // forward: in/out; backward: in
  void* cell;
  void* x;                                 // what the steps hand on: out or d_ifgo
  const void* dout;
  const void* dh_n;
  const void* dc_n;
  void* dh0;
  void* dc0;
  float* db_part;                          // [groups * N][4H] partial sums (N = 64: half as many), or null
};

// NI: MMA issuers, each with an accumulator of its own.
template <bool BWD, int N, int OWN, int NI, typename T16>
__global__ void __launch_bounds__(RES_THREADS, 1)
resident_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const ResParams p) {
  constexpr int UT = BWD ? 128 : 32;             // units per CTA
  constexpr int RO = N / OWN;                    // rows per owner
  constexpr int UP = UT * RO / 256, W = UP / 2;  // units per epilogue thread
  constexpr int TPR = UT / UP;                   // threads per row
  constexpr int BLK = RO * 128;                  // exchanged block: RO rows x 32 M rows, fp32
  constexpr int A_COL = NI * N;                  // tensor memory: the accumulators, then the weights
  constexpr int EW = 8;
  static_assert(W >= 1 && UP <= 8, "");
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int H = p.H, T = p.T, KS = p.ks;
  uint8_t* w_s = smem;                                              // [kcm - nt][16 KB]
  uint8_t* x_s = w_s + (size_t)(p.kcm - p.nt) * 16384;              // [kcm][N rows][128 B]
  uint8_t* recv = x_s + p.x_bytes;                                  // [KS senders][4][RO][32] fp32
  // in the x slots, which are idle from the item's last MMA until the CTA's rows have been counted in:
  uint8_t* stage = x_s;                                             // [OWN receivers][4][RO][32] fp32
  uint64_t* full = reinterpret_cast<uint64_t*>(recv + (size_t)KS * 4 * BLK);   // [RES_MAX_KC]
  uint64_t* w_full = full + RES_MAX_KC;
  uint64_t* acc_full = w_full + 1;
  uint64_t* xchg = acc_full + 1;
  uint64_t* counted = xchg + 1;                                     // forward: the CTA is counted in
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(counted + 1);
  volatile int* dead = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int* pub_cnt = const_cast<int*>(dead) + 1;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int r = blockIdx.x % KS;                                    // rank in the cluster
  const int mt = (blockIdx.x / KS) % p.mt, grp = blockIdx.x / KS / p.mt;
  const int kc0 = r * p.kc_total / KS, n_kc = (r + 1) * p.kc_total / KS - kc0;
  const int nt = min(p.nt, n_kc);
  const int row0 = grp * p.rows;

  if (threadIdx.x == 0) {
    for (int i = 0; i < RES_MAX_KC; ++i) mbar_init(&full[i], 1);
    mbar_init(w_full, 1);
    mbar_init(acc_full, NI);
    mbar_init(xchg, 1 + EW);
    mbar_init(counted, 1);
    *dead = 0;
    *pub_cnt = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmX);
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
    for (int s = 0; s < T; ++s) {
      const int t = BWD ? T - 1 - s : s;
      if (BWD || t > 0) {
        int seen = 1;
        if (lane == 0) seen = wait_flag_ge(&p.flags[(size_t)t * p.n_groups + grp], p.flag_target, p.ctl, p.limit_ns, t, grp) ? 1 : 0;
        seen = __shfl_sync(0xffffffffu, seen, 0);
        __syncwarp();      // (a shuffle orders no memory: the issuing lanes come behind the acquire)
        if (!seen) { *dead = 1; break; }
        fence_proxy_async_global();
      }
      if (lane < 4)
        for (int lc = lane; lc < n_kc; lc += 4) {
          mbar_expect_tx(&full[lc], p.rows * 128);
          tma_load_3d(x_s + (size_t)lc * N * 128, &tmX, &full[lc], (kc0 + lc) * RK, row0, t);
        }
      __syncwarp();
    }
  } else if (warp < 1 + NI) {
    // ---------------------------------------------------------------- MMA issuers: chunks x, x + NI, ... each
    const int x = warp - 1;
    if (elect_one()) {
      constexpr uint64_t descK = smem_desc_base(16, 1024);
      constexpr uint64_t descA = BWD ? smem_desc_base(8192, 1024) : descK;
      const uint32_t idesc_t = instr_desc(p.fmt, 0, 0, 128, N), idesc_s = instr_desc(p.fmt, BWD ? 1 : 0, 0, 128, N);
      const uint32_t d_tmem = tmem_base + x * N, a_tmem = tmem_base + A_COL;
      const uint32_t xa = smem_u32(x_s), wa = smem_u32(w_s);
      bool ok = n_kc <= nt || mbar_wait(w_full, 0, wc);
      for (int s = 0; s < T && ok; ++s) {
        wc.d0 = s;
        for (int lc = x; lc < n_kc; lc += NI) {
          if (!mbar_wait_spin(&full[lc], s & 1, wc)) { ok = false; break; }
          tc_fence_after();
          const uint32_t sb = xa + lc * (N * 128);
          if (lc < nt) {
#pragma unroll
            for (int k = 0; k < 4; ++k)
              umma_f16_ts(d_tmem, a_tmem + lc * 32 + k * 8, smem_desc(descK, sb + k * 32), idesc_t, (k > 0 || lc != x) ? 1u : 0u);
          } else {
            const uint32_t sa = wa + (lc - nt) * 16384;
#pragma unroll
            for (int k = 0; k < 4; ++k)
              umma_f16(d_tmem, smem_desc(descA, sa + k * (BWD ? 2048 : 32)), smem_desc(descK, sb + k * 32), idesc_s, (k > 0 || lc != x) ? 1u : 0u);
          }
        }
        if (ok) umma_commit(acc_full);
      }
    }
  } else if (warp >= 4) {
    // ---------------------------------------------------------------- epilogue
    const int ew = warp - 4, q = ew & 3, g = ew >> 2, et = ew * 32 + lane;
    const bool owner = r < OWN;
    const int lr = et / TPR, u = (et % TPR) * UP;                 // this thread's row among the owner's, first unit
    const int grow = r * RO + lr, row = row0 + grow, unit = mt * UT + u;
    const bool ok_cell = owner && grow < p.rows && row < p.B && unit < H;
    const size_t H4 = 4 * (size_t)H;
    const T16* ifgo = reinterpret_cast<const T16*>(p.ifgo);
    T16* cell = reinterpret_cast<T16*>(p.cell);
    const float* rd = reinterpret_cast<const float*>(recv) + lr * 32 + (BWD ? (u >> 5) * (BLK / 4) + (u & 31) : u);
    const uint32_t tx = owner ? (uint32_t)(KS - 1) * 4 * BLK : 0u;

    // where this warp's half of the accumulator's columns goes: RW_ rows each for NB receivers
    constexpr int NB = OWN > 1 ? OWN / 2 : 1, RW_ = N / 2 / NB, C = RW_ < 16 ? 8 : 16;
    const uint32_t taddr = tmem_base + (uint32_t(q * 32) << 16) + g * (N / 2);
    uint8_t* put[NB];
#pragma unroll
    for (int i = 0; i < NB; ++i) {
      const int dst = OWN > 1 ? g * NB + i : 0;
      put[i] = (dst == r ? recv + (size_t)r * 4 * BLK : stage + (size_t)dst * 4 * BLK) + q * BLK + (OWN > 1 ? 0 : g * RW_ * 128) + lane * 4;
    }
    // the cluster's products of item s, summed: acc[G][UP]
    constexpr int G = BWD ? 1 : 4;
    auto exchange = [&](int s, float (&sum)[G][UP]) -> bool {
      if (ew == 0 && lane == 0) mbar_expect_tx(xchg, tx);
      if (!mbar_wait(acc_full, s & 1, wc)) return false;
      tc_fence_after();
#pragma unroll
      for (int c0 = 0; c0 < N / 2; c0 += C) {
        uint32_t a0[C], a1[C];
        tmem_ld_cols<C>(taddr + c0, a0);
        if constexpr (NI > 1) tmem_ld_cols<C>(taddr + N + c0, a1);
        tmem_ld_wait();
#pragma unroll
        for (int c = 0; c < C; ++c)
          *reinterpret_cast<float*>(put[(c0 + c) / RW_] + ((c0 + c) % RW_) * 128) =
              NI > 1 ? __uint_as_float(a0[c]) + __uint_as_float(a1[c]) : __uint_as_float(a0[c]);
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
              dsmem_bulk_copy(mapa_shared(smem_u32(recv) + (r * 4 + q) * BLK, dst), stage + (size_t)(dst * 4 + q) * BLK, BLK,
                              mapa_shared(smem_u32(xchg), dst));
          }
        }
        mbar_arrive(xchg);
      }
      __syncwarp();
      if (!owner) return true;
      if (!mbar_wait_cluster(xchg, s & 1, wc)) return false;
#pragma unroll
      for (int gg = 0; gg < G; ++gg)
#pragma unroll
        for (int i = 0; i < UP; ++i) sum[gg][i] = 0.f;
      for (int k = 0; k < KS; ++k)
#pragma unroll
        for (int gg = 0; gg < G; ++gg)
#pragma unroll
          for (int i = 0; i < UP; i += 2) {
            const float2 v = *reinterpret_cast<const float2*>(rd + (size_t)(k * 4 + gg) * (BLK / 4) + i);
            sum[gg][i] += v.x;
            sum[gg][i + 1] += v.y;
          }
      return true;
    };
    // this warp's rows are stored: count the CTA in on flag t once all eight warps' are
    auto publish = [&](int t) {
      __syncwarp();
      if (lane == 0 && (smem_count_arrive(pub_cnt) & (EW - 1)) == EW - 1) {
        if (!p.no_arrive) red_release_gpu_add(&p.flags[(size_t)t * p.n_groups + grp], 1);
        if constexpr (!BWD) mbar_arrive(counted);
      }
      __syncwarp();
    };
    if constexpr (!BWD) {
      float c[UP];
      uint32_t pre[4][W];
#pragma unroll
      for (int i = 0; i < UP; ++i) c[i] = 0.f;
      auto load_pre = [&](int t) {
        if (ok_cell && t < T)
#pragma unroll
          for (int gg = 0; gg < 4; ++gg) ld_words<W>(pre[gg], ifgo + ((size_t)t * p.B + row) * H4 + (size_t)gg * H + unit);
      };
      if (ok_cell) {
        uint32_t w[W];
        ld_words<W>(w, cell + (size_t)row * H + unit);
        unpack_words<T16, W>(w, c);
      }
      load_pre(0);
      for (int t = 0; t < T; ++t) {
        wc.d0 = t;
        float pa[4][UP];
        if (!exchange(t, pa)) break;
        uint32_t hw[W];
        float hv[UP];
#pragma unroll
        for (int gg = 0; gg < 4; ++gg)
#pragma unroll
          for (int w = 0; w < W; ++w) {
            const float2 f = cvt2<T16>(pre[gg][w]);
            pa[gg][2 * w] += f.x;
            pa[gg][2 * w + 1] += f.y;
          }
#pragma unroll
        for (int i = 0; i < UP; ++i) {
          c[i] = sigmoid_fast(pa[1][i]) * c[i] + sigmoid_fast(pa[0][i]) * tanh_fast(pa[2][i]);
          hv[i] = sigmoid_fast(pa[3][i]) * tanh_fast(c[i]);
        }
        pack_words<T16, W>(hw, hv);
        if (ok_cell) st_words<W>(reinterpret_cast<T16*>(p.x) + ((size_t)(t + 1) * p.B + row) * H + unit, hw);
        publish(t + 1);
        load_pre(t + 1);
        // what only backward needs, behind the release, which waits for every store of the SM that is under way (B=512, H=512
        // 4.51 -> 4.43 us a step, B=200, H=1024 5.45 -> 5.22)
        if (!mbar_wait(counted, t & 1, wc)) break;
        if (ok_cell && !p.inference) {
#pragma unroll
          for (int gg = 0; gg < 4; ++gg) {
            uint32_t w[W];
            pack_words<T16, W>(w, pa[gg]);
            st_words<W>(reinterpret_cast<T16*>(p.ifgo) + ((size_t)t * p.B + row) * H4 + (size_t)gg * H + unit, w);
          }
        }
        if (ok_cell && (!p.inference || t == T - 1)) {
          uint32_t w[W];
          pack_words<T16, W>(w, c);
          st_words<W>(cell + ((size_t)(t + 1) * p.B + row) * H + unit, w);
        }
      }
    } else {
      const T16* dout = reinterpret_cast<const T16*>(p.dout);
      // Bias gradient: the d_ifgo values as stored.  Where a warp has two rows each half of it keeps two gates of both rows'
      // sums (registers are short).
      constexpr int DBG = UP == 8 ? 2 : 4;
      const int hi = UP == 8 ? lane >> 4 : 0;
      float dc[UP], dh[1][UP], db[DBG][UP];
      float fA[UP], fBi[UP], fBg[UP], fBo[UP], fSf[UP];
      uint32_t dd[W];                       // dout[t]
      uint32_t pf[6][W], cn[W];             // gates, c[t], dout[t]; c[t+1]
#pragma unroll
      for (int k = 0; k < 6; ++k)
#pragma unroll
        for (int w = 0; w < W; ++w) pf[k][w] = 0u;
#pragma unroll
      for (int w = 0; w < W; ++w) cn[w] = 0u;
#pragma unroll
      for (int i = 0; i < UP; ++i) {
        dc[i] = dh[0][i] = 0.f;
#pragma unroll
        for (int gg = 0; gg < DBG; ++gg) db[gg][i] = 0.f;
      }
      if (ok_cell) {
        uint32_t w[W];
        ld_words<W>(cn, cell + ((size_t)T * p.B + row) * H + unit);
        if (p.dc_n) { ld_words<W>(w, reinterpret_cast<const T16*>(p.dc_n) + (size_t)row * H + unit); unpack_words<T16, W>(w, dc); }
        if (p.dh_n) { ld_words<W>(w, reinterpret_cast<const T16*>(p.dh_n) + (size_t)row * H + unit); unpack_words<T16, W>(w, dh[0]); }
      }
      auto prefetch = [&](int t) {
        if (!ok_cell) return;
        const size_t m = (size_t)t * p.B + row;
#pragma unroll
        for (int k = 0; k < 4; ++k) ld_words<W>(pf[k], ifgo + m * H4 + (size_t)k * H + unit);
        ld_words<W>(pf[4], cell + m * H + unit);
        ld_words<W>(pf[5], dout + m * H + unit);
      };
      // everything that does not depend on dh, while the products are being formed:
      //   dh = dout + carry;  dcv = dh*fA + dc;  d_i = dcv*fBi;  d_f = dcv*c*fSf*(1-fSf);  d_g = dcv*fBg;  d_o = dh*fBo;  dc' = dcv*fSf
      // (c = c[t] and dout stay packed: registers are short)
      auto factors = [&]() {
#pragma unroll
        for (int w = 0; w < W; ++w) {
          const float2 pi = cvt2<T16>(pf[0][w]), pff = cvt2<T16>(pf[1][w]), pg = cvt2<T16>(pf[2][w]), po = cvt2<T16>(pf[3][w]);
          const float2 c1 = cvt2<T16>(cn[w]);
          cn[w] = pf[4][w];
          dd[w] = pf[5][w];
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
      prefetch(T - 1);
      factors();
      for (int st = 0; st <= T; ++st) {
        wc.d0 = T - st;
        if (st > 0 && !exchange(st - 1, dh)) break;
        if (!owner) { if (st == T) break; continue; }
        if (st == T) {
          if (ok_cell) {
            uint32_t w[W];
            pack_words<T16, W>(w, dh[0]);
            st_words<W>(reinterpret_cast<T16*>(p.dh0) + (size_t)row * H + unit, w);
            pack_words<T16, W>(w, dc);
            st_words<W>(reinterpret_cast<T16*>(p.dc0) + (size_t)row * H + unit, w);
          }
          break;
        }
        const int t = T - 1 - st;
        float d[4][UP];
        uint32_t dw[4][W];
#pragma unroll
        for (int i = 0; i < UP; ++i) {
          const float2 d2 = cvt2<T16>(dd[i / 2]), c2 = cvt2<T16>(cn[i / 2]);
          const float dv = (i & 1 ? d2.y : d2.x) + dh[0][i], dcv = fmaf(dv, fA[i], dc[i]);
          d[0][i] = dcv * fBi[i];
          d[1][i] = dcv * ((i & 1 ? c2.y : c2.x) * (fSf[i] * (1.f - fSf[i])));
          d[2][i] = dcv * fBg[i];
          d[3][i] = dv * fBo[i];
          dc[i] = dcv * fSf[i];
        }
#pragma unroll
        for (int gg = 0; gg < 4; ++gg) {
          pack_words<T16, W>(dw[gg], d[gg]);
          if (ok_cell) st_words<W>(reinterpret_cast<T16*>(p.x) + ((size_t)t * p.B + row) * H4 + (size_t)gg * H + unit, dw[gg]);
        }
        publish(t);
        if (t > 0) prefetch(t - 1);
        if (p.db_part)
#pragma unroll
          for (int gg = 0; gg < DBG; ++gg)
#pragma unroll
            for (int w = 0; w < W; ++w) {
              uint32_t keep = dw[gg][w];
              if constexpr (UP == 8) {
                const uint32_t other = __shfl_xor_sync(0xffffffffu, ok_cell ? (hi ? dw[gg][w] : dw[gg + 2][w]) : 0u, 16);
                if (hi) keep = dw[gg + 2][w];
                const float2 f = cvt2<T16>(other);
                db[gg][2 * w] += f.x;
                db[gg][2 * w + 1] += f.y;
              }
              const float2 f = cvt2<T16>(ok_cell ? keep : 0u);
              db[gg][2 * w] += f.x;
              db[gg][2 * w + 1] += f.y;
            }
        if (t > 0) factors();
      }
      if (p.db_part && owner && unit < H) {
        constexpr int RP = UP == 8 ? 2 : 1;      // rows per partial sum
        float* dst = p.db_part + ((size_t)grp * N + grow) / RP * H4 + (size_t)2 * hi * H + unit;
#pragma unroll
        for (int gg = 0; gg < DBG; ++gg)
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
// step: H = 1728, B = 32: 6.8 -> 4.9, H = 1408, B = 64: 6.8 -> 4.8, but B = 96, then 48 rows a group, 6.7 -> 7.1.
// H = 2048 with 17 to 32 rows is left with one issuer over six CTAs (6.8; two take 5.2 at H = 1984): a B200 holds
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
    p.rows = (int)round_up((size_t)cdiv(B, p.ng), 8);
    p.ng = cdiv(B, p.rows);
    p.own = bwd ? 4 : p.ks;
    p.N = p.rows <= 16 && p.own != 2 ? 16 : p.rows <= 32 ? 32 : 64;
    if (p.rows > 64) continue;
    p.kcm = cdiv(p.kc_total, p.ks);
    const size_t x = std::max((size_t)p.kcm * p.N * 128, (size_t)p.N * 512);
    p.x_bytes = (int)x;
    for (p.ni = 2; p.ni >= 1; --p.ni) {
      p.nt = std::min(p.kcm, (512 - p.ni * p.N) / 32);
      p.smem = 1024 + (size_t)(p.kcm - p.nt) * 16384 + x + (size_t)p.ks * 4 * (p.N / p.own) * 128 + 512;
      if (p.smem <= 232448 || !(bwd && p.N == 32)) break;
    }
    if (p.smem > 232448 || p.ni < 1 || p.kcm > RES_MAX_KC) continue;
    if (one.ok && (p.ni < 2 || p.N > 32)) continue;
    p.grid = p.ng * p.mt * p.ks;
    p.off_db = sizeof(Control) + round_up((size_t)(d.seq_len + 1) * p.ng * sizeof(int), 256);
    p.ws_bytes = p.off_db + (bwd ? (size_t)p.ng * p.N * 4 * H * sizeof(float) : 0);
    p.ok = true;
    if (p.ni == 2) return p;
    one = p;
  }
  return one;
}

template <bool BWD, int N, int OWN, int NI, typename T16>
static int launch_t(const ResPlan& pl, const CUtensorMap& tw, const CUtensorMap& tx, const ResParams& p, cudaStream_t st) {
  return launch_coresident(resident_kernel<BWD, N, OWN, NI, T16>, pl.grid, RES_THREADS, pl.smem, pl.ks, st, tw, tx, p);
}

static int launch(const blstm_desc& d, const ResPlan& pl, bool bwd, void* x, ResParams& p, void* ws, cudaStream_t st) {
  const int H = d.hidden_size, B = d.batch, T = d.seq_len;
  p.T = T; p.B = B; p.H = H; p.x = x;
  p.mt = pl.mt; p.ks = pl.ks; p.rows = pl.rows; p.kcm = pl.kcm; p.nt = pl.nt; p.x_bytes = pl.x_bytes; p.kc_total = pl.kc_total;
  p.fmt = d.dtype == BLSTM_BF16 ? 1 : 0;
  p.no_arrive = (d.flags & BLSTM_FLAG_TEST_NO_ARRIVE) ? 1 : 0;
  p.inference = (d.flags & BLSTM_FLAG_INFERENCE) ? 1 : 0;
  p.flag_target = pl.mt * pl.own;
  p.n_groups = pl.ng;
  p.limit_ns = d.wait_limit_us > 0 ? (unsigned long long)d.wait_limit_us * 1000ull : kDefaultWaitNs;
  p.ctl = reinterpret_cast<Control*>(ws);
  p.flags = reinterpret_cast<int*>(static_cast<char*>(ws) + sizeof(Control));
  CUtensorMap tw, tx;
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
  {  // the product's other operand as {k, batch row, step}
    uint64_t dims[3] = {K, (uint64_t)B, steps}, str[2] = {K * 2, (uint64_t)B * K * 2};
    uint32_t box[3] = {RK, (uint32_t)pl.rows, 1};
    rc = encode_tensor_map(&tx, x, 3, dims, str, box);
    if (rc) return rc;
  }
#define BLSTM_RES(BW, NN, OO, II)                                                                     \
  if (bwd == BW && pl.N == NN && pl.own == OO && pl.ni == II)                                         \
    return p.fmt ? launch_t<BW, NN, OO, II, __nv_bfloat16>(pl, tw, tx, p, st) : launch_t<BW, NN, OO, II, __half>(pl, tw, tx, p, st);
  BLSTM_RES(false, 16, 1, 2) BLSTM_RES(false, 32, 1, 2) BLSTM_RES(false, 64, 1, 2) BLSTM_RES(false, 32, 2, 2) BLSTM_RES(false, 64, 2, 2)
  BLSTM_RES(true, 16, 4, 2) BLSTM_RES(true, 32, 4, 2) BLSTM_RES(true, 32, 4, 1) BLSTM_RES(true, 64, 4, 2)
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
  return rc || !db ? rc : reduce_db(p.db_part, pl.ng * pl.N / (pl.N == 64 ? 2 : 1), 4 * d.hidden_size, db, st);
}

int resident_plan_detail(const ResPlan& p, int phase, char* buf, size_t n) {
  return snprintf(buf, n, "sm100 %s resident weights cluster=%d groups=%d rows_per_group=%d n=%d m_tiles=%d chunks=%d in_tmem=%d issuers=%d grid=%d threads=%d smem=%zu",
                  phase == BLSTM_PHASE_BWD ? "bwd" : "fwd", p.ks, p.ng, p.rows, p.N, p.mt, p.kcm, p.nt, p.ni, p.grid, RES_THREADS, p.smem);
}

}  // namespace blstm
