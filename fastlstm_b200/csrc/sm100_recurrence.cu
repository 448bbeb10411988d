// Persistent tcgen05 recurrence kernels for 16-bit LSTM layers.
//
// Forward (replaces persistent_fwd_kernel, fastlstm/kernels.py:414-663):
//   CTA (pb, ht) owns UH hidden units (their 4 gate rows of Wh: N = 4*UH rows, all
//   K = H columns) and keeps that slice RESIDENT in shared memory for the whole
//   sequence.  Per (timestep, batch tile of 128 rows) it computes
//       D[128, N] = h[t][tile rows, :] (TMA-streamed, K-major)  x  Wh_slice^T
//   with tcgen05.mma into a TMEM accumulator, then the epilogue warps add the
//   projected pre-activations, write the final pre-activations back (saved for
//   backward), apply the gates with c carried in fp32 registers, and publish
//   h[t+1] / c[t+1].  h is exchanged between the CTAs of a batch tile through
//   global memory (L2): one arrival counter per (timestep, batch tile), released
//   by the epilogue warps (or, with interleaved tiles, by a publisher warp on their
//   behalf) and acquired (bounded spin) by the TMA producer of each CTA before it
//   streams h[t+1].  Each CTA interleaves up to four independent batch tiles so the
//   hand-off latency of one hides behind the work of the others.
//
//   warp 0        TMA producer (flag wait, h tiles, Wh slice once)
//   warps 1..NACC tcgen05.mma issuers (each owns whole K chunks and its own TMEM
//                 accumulator; warp 1 owns the TMEM allocation)
//   next warp     publisher (interleaved tiles only): proxy fence + release per item
//   last 8        epilogue: thread = batch row x 8 or 16 hidden units x 4 gates
#include <stdio.h>
#include <algorithm>
#include <atomic>
#include <stdlib.h>

#include "generic.cuh"
#include "sm100.cuh"
#include "sm100_common.cuh"
#include "sm100_rec_util.cuh"
#include "sm100_small.cuh"
#include "sm100_resident.cuh"
#include "cluster_util.cuh"

namespace blstm {
namespace sm100 {

constexpr int RB = 128;                 // batch rows per tile (MMA M)
constexpr int RK = 64;                  // K chunk (one 128-byte swizzle row)
constexpr int R_MAX_STAGES = 16;
constexpr int R_STAGE_BYTES = RB * RK * 2;   // 16 KB: what an M = 128 MMA reads of a stage's activation rows

// Ring depth: the most stages that fit; and MMA issuers: both (max_ni allows up to two) where they can share the stages.
// Every stage barrier must always be waited on by the SAME thread of each role (a parity wait cannot tell phase n from
// phase n+2, so two threads sharing a barrier could lap each other): stage s belongs to issuer s % ni, which needs
// ni | stages; and an issuer without a chunk of the item (kc) would leave a stale accumulator.
static bool pick_ring(size_t fixed_bytes, size_t stage_bytes, int max_ni, int kc, int* stages, int* ni) {
  for (const int r : {16, 12, 8, 6, 4, 3, 2}) {
    if (fixed_bytes + (size_t)r * stage_bytes > 232448) continue;
    *stages = r;
    *ni = r % 2 ? 1 : std::min(max_ni, kc);
    return true;
  }
  return false;
}

struct RecPlan {
  bool ok;
  int UH, N, nh, nbt, nb_par, ntl, TI, grid, epi_warps, threads, stages, ni, nl, ws;
  int npb;                  // interleaved tiles: TMA landing buffers per epilogue warp (1 or 2), else 0
  int hb;                   // bytes of the h rows in a ring stage: 128 rows, or a single smaller tile's own rows
  size_t w_bytes, stage_bytes, smem, ep_bytes;
  size_t off_flags, n_flags, ws_bytes;
};

// Geometry follows the SM count of the current device (a B200 with all 148 SMs when no device can
// be queried, e.g. when only a workspace size is asked for on a host without a GPU); the
// cooperative launch refuses if the device cannot hold the grid.
static RecPlan make_plan(const blstm_desc& d, int phase) {
  RecPlan p{};
  p.ok = false;
  if (d.flags & BLSTM_FLAG_FORCE_GENERIC) return p;
  if (phase != BLSTM_PHASE_FWD) return p;
  if (d.dtype != BLSTM_F16 && d.dtype != BLSTM_BF16) return p;
  const int H = d.hidden_size, B = d.batch;
  if (H % 64 != 0 || H < 64 || H > 2048) return p;
  p.nbt = cdiv(B, RB);
  int UH = 16;
  // Wider slices when they fill the GPU AND leave every CTA two or more tiles to interleave (a single
  // tile of 32 units per CTA is latency bound and measured slower than two interleaved tiles of 16:
  // 2.12 against 1.87 ms at B=1024, H=512, T=256).
  const int sm_share = (d.flags & BLSTM_FLAG_HALF_DEVICE) ? 2 : 1;   // half the device: two kernels side by side
  if (H <= 512 && p.nbt * (H / 32) >= 74) {
    const int sms32 = plan_sm_count() / sm_share;
    int par32 = sms32 / (H / 32);
    if (par32 > p.nbt) par32 = p.nbt;
    if (par32 > 0 && cdiv(p.nbt, par32) >= 2) UH = 32;
  }
  p.UH = UH;
  p.N = 4 * UH;
  p.nh = H / UH;
  const int sms = plan_sm_count() / sm_share;
  if (p.nh > sms) return p;
  p.nb_par = sms / p.nh;
  if (p.nb_par > p.nbt) p.nb_par = p.nbt;
  p.ntl = cdiv(p.nbt, p.nb_par);
  p.TI = p.ntl >= 3 ? 4 : p.ntl >= 2 ? 2 : 1;     // batch tiles interleaved per CTA (state: cell rows in registers)
  p.grid = p.nh * p.nb_par;
  p.epi_warps = 8;
  // two issuers, eight epilogue warps and, for interleaved tiles, the publisher (32-unit slices: N = 128 runs the
  // tensor pipe at full rate from ONE issuing thread, and a single accumulator per item leaves tensor-memory columns
  // for the cell rows of four tiles)
  const int n_issuers = UH == 32 ? 1 : 2;
  const int n_publisher = p.TI >= 2 ? 1 : 0;
  p.threads = 32 * (1 + n_issuers + n_publisher + p.epi_warps);   // producer + MMA issuers [+ publisher] + epilogue
  // Wh slice resident in shared memory when it fits next to a useful ring; otherwise (H > 1024) it is
  // streamed through the ring with h, chunk by chunk, every step (it stays in L2).  A single batch tile
  // of fewer than 128 rows only stages its own rows (the MMA's rows past them read whatever follows:
  // accumulator rows nobody uses), which makes room for up to 16 stages.
  p.w_bytes = (size_t)p.N * H * 2;
  p.ws = p.w_bytes > 128 * 1024 ? 1 : 0;
  p.hb = (p.nbt == 1 ? (int)round_up((size_t)B, 8) : RB) * 128;
  const size_t w_chunk = (size_t)p.N * 128;
  p.stage_bytes = p.hb + (p.ws ? w_chunk : 0);
  // (a stage that holds fewer than 128 rows is still READ as 128 rows by the MMA: the ring is followed by
  //  enough shared memory for the last stage's read to stay inside the allocation)
  const size_t tail_pad = p.stage_bytes < (size_t)R_STAGE_BYTES ? R_STAGE_BYTES - p.stage_bytes : 0;
  // Streamed means ALL of it: keeping 18 of H=2048's 32 chunks resident (6-stage ring) measured 10.2 ms
  // against 8.1 ms with none resident and a 16-stage ring - the depth of the ring is worth more than
  // the bytes saved.
  // Interleaved tiles: the epilogue's gate traffic goes through TMA.  Every epilogue warp owns
  // landing buffers for its 32 rows' projected pre-activations (4 gates x NU units; the final
  // pre-activations are written back in place and leave from there).
  // Two landing buffers per warp (the next item's box is fetched a whole item ahead) when the ring
  // still gets four stages, else one.
  p.npb = 0;
  p.ep_bytes = 0;
  size_t fixed = 1024 + (p.ws ? 0 : p.w_bytes) + 512 + tail_pad;
  if (p.TI >= 2) {
    const int NU = 4 * UH / p.epi_warps;
    const size_t pb = 256 * (size_t)NU;
    p.npb = (fixed + p.epi_warps * 2 * pb + 4 * p.stage_bytes <= 232448) ? 2 : 1;
    p.ep_bytes = p.epi_warps * p.npb * pb;
    fixed += p.ep_bytes;
  }
  if (!pick_ring(fixed, p.stage_bytes, n_issuers, H / RK, &p.stages, &p.ni)) return p;
  // TMA-issuing lanes of the producer warp (they split the ring's stages; nl | stages).  As many as
  // issuers by default; measured exceptions (3-4 % each): two interleaved tiles do better with more lanes
  // (B=2048: 2.55 -> 2.46 ms, B=1024: 1.89 -> 1.78 ms), a single tile on a six-stage ring with fewer
  // (H=1024: 3.89 -> 3.75 ms).
  p.nl = p.ni;
  if (p.TI == 1) p.nl = p.stages == 6 ? 2 : 4;
  if (p.TI == 2) p.nl = UH == 32 ? 2 : 4;
  if (p.stages % p.nl != 0 || p.nl > H / RK) p.nl = p.ni;
  p.smem = fixed + (size_t)p.stages * p.stage_bytes;
  p.n_flags = (size_t)(d.seq_len + 1) * p.nbt;
  p.off_flags = sizeof(Control);
  p.ws_bytes = p.off_flags + round_up(p.n_flags * sizeof(int), 256);
  p.ok = true;
  return p;
}

struct FwdParams {
  int T, B, H;
  int nbt, nh, nb_par, ntl;
  int stages;
  int ni;                   // MMA-issuing warps in use
  int nl;                   // TMA-issuing lanes of the producer warp (nl divides the ring depth)
  int ws;                   // 1: the Wh slice streamed through the ring instead of resident
  int hb;                   // bytes of the h rows in a ring stage
  int stage_bytes;
  int fmt;
  int no_arrive;
  int inference;            // skip the stores that only backward needs
  int flag_target;          // arrivals that complete a flag: nh CTAs per batch tile
  int npb;                  // TMA landing buffers per epilogue warp (interleaved tiles)
  int ep_bytes;             // bytes of the epilogue's TMA buffers (between the weights and the ring)
  unsigned long long limit_ns;
  Control* ctl;
  int* flags;
  void* ifgo;               // [T,B,4H] in/out
  void* out;                // [T+1,B,H]
  void* cell;               // [T+1,B,H]
};

// Position in a CTA's sequence of work items, which every role walks in the same order:
//   for chunk (TI tiles) : for step in [0, steps) : for j in [0, TI) : tile pb + (chunk*TI + j)*nb_par
// (tiles past the last one are skipped).  next() moves to the following existing item.
template <int TI>
struct ItemCursor {
  int ch, t, j;
  __device__ __forceinline__ void init() { ch = 0; t = 0; j = -1; }
  __device__ __forceinline__ bool next(int pb, int nb_par, int nbt, int n_chunks, int steps) {
    for (;;) {
      if (++j == TI) { j = 0; if (++t == steps) { t = 0; ++ch; } }
      if (ch >= n_chunks) return false;
      if (pb + (ch * TI + j) * nb_par < nbt) return true;
    }
  }
  __device__ __forceinline__ int tile(int pb, int nb_par) const { return pb + (ch * TI + j) * nb_par; }
};

// UH: hidden units per CTA (16 or 32).  TI: batch tiles interleaved per CTA (1, 2 or 4).
// Warps: 1 TMA producer, NACC MMA issuers, with interleaved tiles one publisher warp, 8 epilogue
// warps - at most 12 (3 per SM sub-partition), which leaves 168 registers per thread; a 13th would cap
// them at 128.  The epilogue must not spill.
template <int UH, int TI, typename T16>
__global__ void __launch_bounds__(32 * (UH == 16 && TI >= 2 ? 12 : 11), 1)
fwd_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmH,
           const __grid_constant__ CUtensorMap tmP, const FwdParams p) {
  constexpr int N = 4 * UH;
  // One tile in flight: plain stores of h, the release behind them, then what only backward needs (the release waits for
  // every store of the SM that is under way).  TMA stores that the warps wait for in front of the release cost 0.1 to
  // 0.3 us a step more (H = 1536, B = 128: 8.8 -> 8.6; H = 1088, B = 200: 7.8 -> 7.5).
  // Interleaved tiles are throughput bound, and there the epilogue's row-strided 16-byte global
  // accesses (a thread owns a batch row: 32 sectors per warp instruction) were the bottleneck: the
  // projected pre-activations come in as TMA boxes through shared memory, one set of buffers per
  // epilogue warp (tmP: ifgo as {unit, row, gate, step}), and the final pre-activations go out from
  // the same buffers (16 units per thread: coalesced plain stores; 8 units: a TMA box): eight of the
  // twelve 16-byte accesses a thread makes per 8 units.  h keeps its direct stores (they are what
  // the step hand-off orders) and so do the cell rows (a buffer for them would cost a ring stage).
  constexpr bool TMAEP = (TI >= 2);
  // Epilogue warps: two warpgroups that split the CTA's units (8 or 16 per thread, free of spills).
  constexpr int EW = 8;
  constexpr int NU = 4 * UH / EW;                   // units per epilogue thread
  constexpr int NV = NU / 8;                        // 16-byte pieces per operand per thread
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int H = p.H;
  const int KC = H / RK;                            // K chunks
  uint8_t* w_s = smem;                              // [KC][N rows][128 B]
  const int R_STAGES = p.stages;
  const int SB = p.stage_bytes;                     // h chunk (16 KB) [+ Wh chunk when streamed]
  uint8_t* ep_s = smem + (p.ws ? 0 : (size_t)KC * N * 128);   // epilogue TMA buffers (interleaved tiles)
  const int HB = p.hb;                                    // h rows of a stage; a streamed Wh chunk follows them
  uint8_t* a_s = ep_s + p.ep_bytes;                       // [stages][h chunk | optional Wh chunk]
  uint64_t* bars = reinterpret_cast<uint64_t*>(a_s + (size_t)R_STAGES * SB);
  uint64_t* full = bars;                            // [R_MAX_STAGES]
  uint64_t* empty = bars + R_MAX_STAGES;            // [R_MAX_STAGES]
  uint64_t* acc_full = bars + 2 * R_MAX_STAGES;     // [2]
  uint64_t* acc_empty = acc_full + 2;               // [2]
  uint64_t* w_full = acc_empty + 2;                 // [1]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(w_full + 1);
  volatile int* dead = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int* pub_cnt = const_cast<int*>(dead) + 1;        // [4] arrivals of the epilogue warps, by item index mod 4
  uint64_t* pub_bar = reinterpret_cast<uint64_t*>(pub_cnt + 4);   // [4] item stored? by item index mod 4
  uint64_t* pre_full = pub_bar + 4;                 // [8 epilogue warps][2] landing buffer filled

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ht = blockIdx.x % p.nh, pb = blockIdx.x / p.nh;
  // NACC warps issue MMAs concurrently, each for whole chunks into its own TMEM accumulator, and the epilogue adds them
  // up: a thread issues one every 55 clocks at best, but loses some hundred to every chunk's barriers.
  // With interleaved tiles the epilogue warps are the bottleneck and the release that publishes an item
  // stalls its thread for a memory round trip, so a PUBLISHER warp does the releasing (and the proxy
  // fence of the hand-off): the epilogue warps only arrive on a CTA-local barrier after storing h.
  constexpr bool PUBLISHER = (TI >= 2);
  constexpr int NACC = UH == 32 ? 1 : 2;   // issuer warps / partial accumulators
  constexpr int FIRST_EPI = 1 + NACC + (PUBLISHER ? 1 : 0);   // first epilogue warp
  // Columns per item buffer (NACC * N <= 256).  Interleaved tiles pack the two buffers into the first
  // 256 columns and keep the tiles' cell rows (fp32, a column per unit) in the columns behind them.
  constexpr int ACC_STRIDE = (TI >= 2) ? NACC * N : 256;
  constexpr int C_BASE = 2 * ACC_STRIDE;
  static_assert(TI == 1 || C_BASE + TI * UH <= 512, "cell rows do not fit the tensor memory");
  constexpr uint32_t TMEM_COLS = 512;
  const int nacc = p.ni;                             // accumulators / issuers / TMA lanes in use

  if (threadIdx.x == 0) {
    // full[s] is armed (arrive + expected bytes) for its first use here and re-armed by the MMA issuer
    // that consumed it for every later use, which keeps that work out of the latency-bound TMA producer loop
    for (int s = 0; s < R_STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(&acc_full[a], nacc); mbar_init(&acc_empty[a], EW); }
    mbar_init(w_full, 1);
    *dead = 0;
    for (int i = 0; i < 4; ++i) pub_cnt[i] = 0;
    for (int i = 0; i < 4; ++i) mbar_init(&pub_bar[i], EW);
    for (int i = 0; i < 16; ++i) mbar_init(&pre_full[i], 1);
    fence_mbar_init();
    for (int s = 0; s < R_STAGES; ++s) mbar_expect_tx(&full[s], SB);
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmH);
    if (TMAEP) tma_prefetch_desc(&tmP);
  }
  if (warp == 1) tmem_alloc(tmem_slot, TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  WaitCtx wc{dead, p.ctl, p.limit_ns, -1, (int)blockIdx.x};

  // Work items of this CTA, in the order every role walks them:
  //   for chunk (TI tiles) : for t in [0,T) : for j in [0,TI) : (t, bt = pb + (chunk*TI + j) * nb_par)
  const int n_chunks = (p.ntl + TI - 1) / TI;

  if (warp == 0) {
    // ---------------------------------------------------------------- TMA producer
    // One thread needs a few hundred clocks per cp.async.bulk.tensor issue, so p.ni lanes issue in
    // lockstep, each owning the ring stages congruent to its lane index.
    if (lane == 0 && !p.ws) {
      // resident Wh slice: rows (gate g, unit ht*UH + u), K chunks of [N][64]
      mbar_expect_tx(w_full, (uint32_t)((size_t)KC * N * 128));
      for (int kc = 0; kc < KC; ++kc) tma_load_3d(w_s + (size_t)kc * N * 128, &tmW, w_full, kc * RK, ht * UH, 0);
    }
    int gs = 0;                // ring position of the current item's chunk 0
    uint32_t gph = 0;
    bool ok = true;
    // With interleaved tiles an item's arrival counter is usually complete long before its turn, and
    // what costs is the round trip of looking: lane 31 reads the NEXT item's counter while the other
    // lanes issue the current item's loads, and lane 0 only spins when that early look found it incomplete.
    ItemCursor<TI> nx;
    nx.init();
    bool nx_valid = nx.next(pb, p.nb_par, p.nbt, n_chunks, p.T);   // the first item itself
    int early = 0;             // lane 31: early reading of the next item's counter
    for (int ch = 0; ch < n_chunks && ok; ++ch) {
      for (int t = 0; t < p.T && ok; ++t) {
        for (int j = 0; j < TI && ok; ++j) {
          const int bt = pb + (ch * TI + j) * p.nb_par;
          if (bt >= p.nbt) continue;
          // what lane 31 read for this item while the previous item's loads were being issued
          const int early_now = (TI >= 2) ? __shfl_sync(0xffffffffu, early, 31) : 0;
          if (TI >= 2) nx_valid = nx_valid && nx.next(pb, p.nb_par, p.nbt, n_chunks, p.T);
          bool lane_ok = true;
          // One tile in flight: the wait for each issuing lane's first ring stage (half a thousand clocks
          // even when the stage is long free) is taken BEFORE the counter, off the step's chain.
          const int nl = p.nl;                 // TMA-issuing lanes: lane l owns the ring stages == l (mod nl)
          const int kc_first = (lane + nl - gs % nl) % nl;
          if (TI == 1 && lane < nl && kc_first < KC) {
            int s = gs + kc_first;
            uint32_t ph = gph;
            while (s >= R_STAGES) { s -= R_STAGES; ph ^= 1; }
            lane_ok = mbar_wait(&empty[s], ph ^ 1, wc);
          }
          if (t > 0) {   // h[t] of this batch tile complete: every epilogue warp of every hidden tile arrived
            int seen = 1;
            if (lane == 0 && !(TI >= 2 && early_now >= p.flag_target)) {
              wc.d0 = t; wc.d1 = bt;
              seen = wait_flag_ge(&p.flags[(size_t)t * p.nbt + bt], p.flag_target, p.ctl, p.limit_ns, t, bt) ? 1 : 0;
            }
            seen = __shfl_sync(0xffffffffu, seen, 0);
            __syncwarp();      // (a shuffle orders no memory: the issuing lanes come behind the acquire)
            if (!seen) { *dead = 1; ok = false; break; }
            // a proxy fence between the peers' arrivals (interleaved tiles: their plain stores, fenced by their publisher
            // warps) and this warp's TMA reads
            if (!PUBLISHER) fence_proxy_async_global();
          }
          const int row0 = bt * RB;
          if (lane < nl && lane_ok) {
            // this lane owns ring stages == lane (mod nl): the item's chunks that land there
            for (int kc = kc_first; kc < KC; kc += nl) {
              int s = gs + kc;
              uint32_t ph = gph;
              while (s >= R_STAGES) { s -= R_STAGES; ph ^= 1; }
              if (!(TI == 1 && kc == kc_first) && !mbar_wait(&empty[s], ph ^ 1, wc)) { lane_ok = false; break; }
              tma_load_3d(a_s + (size_t)s * SB, &tmH, &full[s], kc * RK, row0, t);
              if (p.ws) tma_load_3d(a_s + (size_t)s * SB + HB, &tmW, &full[s], kc * RK, ht * UH, 0);
            }
          } else if (TI >= 2 && lane == 31) {
            // (the other arm of the same branch: the issuing lanes do not wait for this read)
            early = 0;
            if (nx_valid && nx.t > 0) early = ld_acquire_gpu(&p.flags[(size_t)nx.t * p.nbt + nx.tile(pb, p.nb_par)]);
          }
          if (__any_sync(0xffffffffu, !lane_ok)) { ok = false; break; }
          gs += KC;
          while (gs >= R_STAGES) { gs -= R_STAGES; gph ^= 1; }
        }
      }
    }
  } else if (PUBLISHER && warp == 1 + NACC) {
    // ---------------------------------------------------------------- publisher
    // Walks the items in the epilogue's order; when all epilogue warps have stored an item's h rows
    // (their arrival on pub_bar is a CTA-scope release, this wait the acquire), the proxy fence of the
    // hand-off and one release at GPU scope count this CTA in on the item's arrival counter.  An
    // epilogue warp can be at most four items ahead (it needs the counters this thread completes),
    // so four barriers never mix items.
    if (lane == 0) {
      int k = 0;
      bool ok = true;
      for (int ch = 0; ch < n_chunks && ok; ++ch) {
        for (int t = 0; t < p.T && ok; ++t) {
          for (int j = 0; j < TI && ok; ++j) {
            const int bt = pb + (ch * TI + j) * p.nb_par;
            if (bt >= p.nbt) continue;
            wc.d0 = t; wc.d1 = bt;
            if (!mbar_wait(&pub_bar[k & 3], (uint32_t)(k >> 2) & 1u, wc)) { ok = false; break; }
            fence_proxy_async_global();
            if (!p.no_arrive) red_release_gpu_add(&p.flags[(size_t)(t + 1) * p.nbt + bt], 1);
            ++k;
          }
        }
      }
    }
  } else if (warp < 1 + NACC) {
    // ---------------------------------------------------------------- MMA issuers
    const int x = warp - 1;                 // accumulator / K-slice index of this issuer
    if (elect_one()) {                      // (a thread chosen by `elect` issues an MMA every 55 clocks, by lane == 0 every 74)
      constexpr uint64_t descK = smem_desc_base(16, 1024);
      const uint32_t idesc = instr_desc(p.fmt, 0, 0, RB, N);
      // issuer x owns WHOLE chunks (kc = x, x+NACC, ...): four MMAs and one commit per chunk
      bool ok = (x < nacc) && (p.ws || mbar_wait(w_full, 0, wc));
      int gs = 0;
      uint32_t gph = 0;
      uint32_t acc_ph[2] = {0, 0};
      int it = 0;
      const uint32_t w_addr = smem_u32(w_s);
      for (int ch = 0; ch < n_chunks && ok; ++ch) {
        for (int t = 0; t < p.T && ok; ++t) {
          for (int j = 0; j < TI && ok; ++j) {
            const int bt = pb + (ch * TI + j) * p.nb_par;
            if (bt >= p.nbt) continue;
            const int a = it & 1;
            ++it;
            if (!mbar_wait(&acc_empty[a], acc_ph[a] ^ 1, wc)) { ok = false; break; }
            acc_ph[a] ^= 1;
            tc_fence_after();
            const uint32_t d_tmem = tmem_base + a * ACC_STRIDE + x * N;
            uint32_t acc_on = 0;   // first MMA of the item overwrites this issuer's accumulator
            for (int kc = (x + nacc - gs % nacc) % nacc; kc < KC; kc += nacc) {
              int s = gs + kc;
              uint32_t ph = gph;
              while (s >= R_STAGES) { s -= R_STAGES; ph ^= 1; }
              if (!mbar_wait_spin(&full[s], ph, wc)) { ok = false; break; }
              // arm the stage's next use: R_STAGES chunks further on (chunks wrap around within an item)
              mbar_expect_tx(&full[s], SB);
              tc_fence_after();
              const uint32_t sa = smem_u32(a_s + (size_t)s * SB);
              const uint32_t sb = p.ws ? sa + HB : w_addr + (uint32_t)kc * N * 128;
#pragma unroll
              for (int k = 0; k < RK / 16; ++k)
                umma_f16(d_tmem, smem_desc(descK, sa + k * 32), smem_desc(descK, sb + k * 32), idesc,
                         (k > 0) ? 1u : acc_on);
              acc_on = 1;
              umma_commit(&empty[s]);
            }
            if (ok) umma_commit(&acc_full[a]);
            gs += KC;
            while (gs >= R_STAGES) { gs -= R_STAGES; gph ^= 1; }
          }
        }
      }
    }
  } else if constexpr (TMAEP) {
    // ---------------------------------------------------------------- epilogue, interleaved tiles
    // thread = (batch row, NU units), worked in passes of 8 units.  Each warp owns `npb` landing
    // buffers [4 gates][32 rows][NU units]: rows of 16 bytes lie back to back, rows of 32 bytes carry
    // the 32-byte swizzle, so the 32 lanes' 16-byte pieces of one gate fall into different banks.
    // Lane 0 issues the warp's TMA loads (`npb` items ahead) and stores.
    constexpr int PB_BYTES = 256 * NU, NPIECE = NU / 8;
    const int ew = warp - FIRST_EPI;
    const int q = warp & 3;                 // TMEM lane quarter this warp may read
    const int ug = ew >> 2;
    const int row_in_tile = q * 32 + lane;
    const int unit0 = ht * UH + ug * NU;
    const int npb = p.npb;
    uint8_t* pbuf = ep_s + (size_t)ew * npb * PB_BYTES;
    uint64_t* pfull = pre_full + 2 * ew;
    T16* out = reinterpret_cast<T16*>(p.out);
    T16* cell = reinterpret_cast<T16*>(p.cell);
    auto c_off = [&](int v) { return (NU == 16) ? lane * 32 + ((v ^ ((lane >> 2) & 1)) * 16) : lane * 16; };
    auto p_off = [&](int g, int v) { return g * (64 * NU) + c_off(v); };
    // the load cursor runs `npb` items ahead of the item being worked on (lane 0 only)
    ItemCursor<TI> lc;
    lc.init();
    bool lc_valid = lc.next(pb, p.nb_par, p.nbt, n_chunks, p.T);
    int n_loaded = 0;
    auto issue_load = [&]() {
      if (!lc_valid) return;
      const int b = (npb == 2) ? (n_loaded & 1) : 0;
      mbar_expect_tx(&pfull[b], PB_BYTES);
      tma_load_4d(pbuf + (size_t)b * PB_BYTES, &tmP, &pfull[b], unit0, lc.tile(pb, p.nb_par) * RB + q * 32, 0, lc.t);
      ++n_loaded;
      lc_valid = lc.next(pb, p.nb_par, p.nbt, n_chunks, p.T);
    };
    if (lane == 0)
      for (int i = 0; i < npb; ++i) issue_load();
    int it = 0;                             // items consumed
    bool ok = true;
    // cell rows of this thread's (row, NU units) for tile slot j: tensor-memory columns behind the accumulators
    const uint32_t c_taddr = tmem_base + C_BASE + (uint32_t(q * 32) << 16) + ug * NU;
    for (int ch = 0; ch < n_chunks && ok; ++ch) {
#pragma unroll
      for (int j = 0; j < TI; ++j) {
        const int bt = pb + (ch * TI + j) * p.nb_par;
        const int row = bt * RB + row_in_tile;
#pragma unroll
        for (int v = 0; v < NPIECE; ++v) {
          float c0[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) c0[u] = 0.f;
          if (bt < p.nbt && row < p.B) unpack8<T16>(ldg16(cell + (size_t)row * H + unit0 + 8 * v), c0);
          uint32_t cr[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) cr[u] = __float_as_uint(c0[u]);
          tmem_st_32x8(c_taddr + j * UH + 8 * v, cr);
        }
      }
      tmem_st_wait();
      for (int t = 0; t < p.T && ok; ++t) {
#pragma unroll
        for (int j = 0; j < TI; ++j) {
          const int bt = pb + (ch * TI + j) * p.nb_par;
          if (bt >= p.nbt) continue;
          const int a = it & 1;
          const uint32_t a_ph = (uint32_t)(it >> 1) & 1u;
          const int b = (npb == 2) ? (it & 1) : 0;
          const uint32_t b_ph = (npb == 2) ? ((uint32_t)(it >> 1) & 1u) : ((uint32_t)it & 1u);
          ++it;
          const int row = bt * RB + row_in_tile;
          const bool row_ok = row < p.B;
          wc.d0 = t; wc.d1 = bt;
          if (!mbar_wait(&acc_full[a], a_ph, wc)) { ok = false; break; }
          if (!mbar_wait(&pfull[b], b_ph, wc)) { ok = false; break; }
          tc_fence_after();
          const uint32_t taddr = tmem_base + a * ACC_STRIDE + (uint32_t(q * 32) << 16) + ug * NU;
          uint8_t* pbb = pbuf + (size_t)b * PB_BYTES;
          const size_t o1 = ((size_t)(t + 1) * p.B + row) * H + unit0;
#pragma unroll
          for (int v = 0; v < NPIECE; ++v) {
            float pa[4][8];
            uint32_t cr[8];
            tmem_ld_32x8(c_taddr + j * UH + 8 * v, cr);
#pragma unroll
            for (int g = 0; g < 4; ++g) {
              uint32_t acc[NACC][8];
#pragma unroll
              for (int x = 0; x < NACC; ++x) tmem_ld_32x8(taddr + x * N + g * UH + 8 * v, acc[x]);
              tmem_ld_wait();
#pragma unroll
              for (int u = 0; u < 8; ++u) {
                float s0 = __uint_as_float(acc[0][u]);
#pragma unroll
                for (int x = 1; x < NACC; ++x)
                  if (x < nacc) s0 += __uint_as_float(acc[x][u]);
                pa[g][u] = s0;
              }
            }
            if (v == NPIECE - 1) {
              // the accumulator is in registers: hand the TMEM buffer back to the MMA warps
              tc_fence_before();
              __syncwarp();
              if (lane == 0) mbar_arrive(&acc_empty[a]);
            }
#pragma unroll
            for (int g = 0; g < 4; ++g) {
              const uint4 pw4 = *reinterpret_cast<const uint4*>(pbb + p_off(g, v));
              const uint32_t w[4] = {pw4.x, pw4.y, pw4.z, pw4.w};
#pragma unroll
              for (int u = 0; u < 4; ++u) {
                const float2 f2 = cvt2<T16>(w[u]);
                pa[g][2 * u] += f2.x;
                pa[g][2 * u + 1] += f2.y;
              }
            }
            float hv[8], cv[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
              const float cn = sigmoid_fast(pa[1][u]) * __uint_as_float(cr[u]) + sigmoid_fast(pa[0][u]) * tanh_fast(pa[2][u]);
              cv[u] = cn;
              cr[u] = __float_as_uint(cn);
              hv[u] = sigmoid_fast(pa[3][u]) * tanh_fast(cn);
            }
            tmem_st_32x8(c_taddr + j * UH + 8 * v, cr);
            if (row_ok) store8<T16>(out + o1 + 8 * v, hv);
            // final pre-activations back in place (16-bit, as stored)
#pragma unroll
            for (int g = 0; g < 4; ++g)
              *reinterpret_cast<uint4*>(pbb + p_off(g, v)) =
                  make_uint4(pk2<T16>(pa[g][0], pa[g][1]), pk2<T16>(pa[g][2], pa[g][3]), pk2<T16>(pa[g][4], pa[g][5]),
                             pk2<T16>(pa[g][6], pa[g][7]));
            if (row_ok && (!p.inference || t == p.T - 1)) store8<T16>(cell + o1 + 8 * v, cv);
          }
          tmem_st_wait();
          // publish h[t+1] first (it is all the peers wait for): the publisher warp fences and releases
          __syncwarp();
          if (lane == 0) mbar_arrive(&pub_bar[(it - 1) & 3]);
          // then the final pre-activations leave the landing buffer, and the box of the item `npb` ahead is
          // fetched into it
          if constexpr (NU == 16) {
            // Plain stores, NOT a TMA store: an SM's TMA unit writes only ~29 B/clk and the stores queue in
            // front of the h loads (measured: 8 such boxes per item cut a concurrent h stream from 71 to
            // 33 B/clk).  Two lanes cover a row's 32 bytes, so a warp instruction writes 16 full sectors:
            // instruction k = (gate k/2, rows 16*(k%2) ...), lane = (row, 16-byte piece).
            if (!p.inference) {
              T16* gbase = reinterpret_cast<T16*>(p.ifgo) + ((size_t)t * p.B + (size_t)bt * RB + q * 32) * (4 * (size_t)H) + unit0;
              const int r_lo = lane >> 1, v = lane & 1;
#pragma unroll
              for (int k = 0; k < 8; ++k) {
                const int g = k >> 1, r = (k & 1) * 16 + r_lo;
                const uint4 w = *reinterpret_cast<const uint4*>(pbb + g * (64 * NU) + r * 32 + ((v ^ ((r >> 2) & 1)) * 16));
                if (bt * RB + q * 32 + r < p.B) stg16(gbase + (size_t)r * (4 * (size_t)H) + (size_t)g * H + v * 8, w);
              }
            }
            fence_proxy_async_smem();      // the buffer's reads come before the next box is written into it
            __syncwarp();
            if (lane == 0) issue_load();
          } else {
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              const int row0 = bt * RB + q * 32;
              if (!p.inference) tma_store_4d(&tmP, pbb, unit0, row0, 0, t);
              tma_store_commit();
              tma_store_wait_read<0>();
              issue_load();
            }
          }
          __syncwarp();
        }
      }
    }
    if (lane == 0) tma_store_wait<0>();
  } else {
    // ---------------------------------------------------------------- epilogue
    // thread = (batch row, NU units): warpgroup `ug` takes the ug-th group of NU of the CTA's UH units
    const int ew = warp - FIRST_EPI;
    const int q = warp & 3;                 // TMEM lane quarter this warp may read
    const int ug = ew >> 2;
    const int row_in_tile = q * 32 + lane;
    const int unit0 = ht * UH + ug * NU;
    const size_t H4 = 4 * (size_t)H;
    T16* ifgo = reinterpret_cast<T16*>(p.ifgo);
    T16* out = reinterpret_cast<T16*>(p.out);
    T16* cell = reinterpret_cast<T16*>(p.cell);
    int it = 0;                             // items consumed: TMEM buffer it & 1, on its (it >> 1)-th use
    bool ok = true;
    for (int ch = 0; ch < n_chunks && ok; ++ch) {
      float c[TI][NU];
      uint4 pre[4 * NV];                    // projected pre-activations of the NEXT item: 4 gates x NU units
      // initial cell state of this chunk's tiles
#pragma unroll
      for (int j = 0; j < TI; ++j) {
        const int bt = pb + (ch * TI + j) * p.nb_par;
        const int row = bt * RB + row_in_tile;
#pragma unroll
        for (int u = 0; u < NU; ++u) c[j][u] = 0.f;
        if (bt < p.nbt && row < p.B) {
#pragma unroll
          for (int v = 0; v < NV; ++v) unpack8<T16>(ldg16(cell + (size_t)row * H + unit0 + 8 * v), &c[j][8 * v]);
        }
      }
      auto load_pre = [&](int t, int bt) {
        const int row = bt * RB + row_in_tile;
        if (t < p.T && bt < p.nbt && row < p.B) {
          const T16* src = ifgo + ((size_t)t * p.B + row) * H4 + unit0;
#pragma unroll
          for (int g = 0; g < 4; ++g)
#pragma unroll
            for (int v = 0; v < NV; ++v) pre[g * NV + v] = ldg16(src + (size_t)g * H + 8 * v);
        }
      };
      load_pre(0, pb + (ch * TI) * p.nb_par);   // pre-activations of the first item
      for (int t = 0; t < p.T && ok; ++t) {
#pragma unroll
        for (int j = 0; j < TI; ++j) {
          const int bt = pb + (ch * TI + j) * p.nb_par;
          if (bt >= p.nbt) continue;
          const int a = it & 1;
          const uint32_t a_ph = (uint32_t)(it >> 1) & 1u;
          ++it;
          const int row = bt * RB + row_in_tile;
          const bool row_ok = row < p.B;
          wc.d0 = t; wc.d1 = bt;
          if (!mbar_wait(&acc_full[a], a_ph, wc)) { ok = false; break; }
          tc_fence_after();
          const uint32_t taddr = tmem_base + a * ACC_STRIDE + (uint32_t(q * 32) << 16) + ug * NU;
          // accumulator read-out (the issuers' partial sums, GG gates per wait: 64 values in flight), gate maths, h store; the final pre-activations are saved after the release
          constexpr int GG = 4;
          const size_t o1 = ((size_t)(t + 1) * p.B + row) * H + unit0;
          T16* gdst = ifgo + ((size_t)t * p.B + row) * H4 + unit0;
          float pa[4][NU];
#pragma unroll
          for (int g0 = 0; g0 < 4; g0 += GG) {
            uint32_t v[GG][NACC][NU];
#pragma unroll
            for (int g = 0; g < GG; ++g)
#pragma unroll
              for (int x = 0; x < NACC; ++x) tmem_ld_cols<NU>(taddr + x * N + (g0 + g) * UH, v[g][x]);
            tmem_ld_wait();
#pragma unroll
            for (int g = 0; g < GG; ++g)
#pragma unroll
              for (int u = 0; u < NU; ++u) {
                float s0 = __uint_as_float(v[g][0][u]);
#pragma unroll
                for (int x = 1; x < NACC; ++x)
                  if (x < nacc) s0 += __uint_as_float(v[g][x][u]);
                pa[g0 + g][u] = s0;
              }
          }
          // the accumulator is in registers: hand the TMEM buffer back to the MMA warps
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&acc_empty[a]);
#pragma unroll
          for (int g = 0; g < 4; ++g)
#pragma unroll
            for (int v = 0; v < NV; ++v) {
              const uint4 pw4 = pre[g * NV + v];
              const uint32_t w[4] = {pw4.x, pw4.y, pw4.z, pw4.w};
#pragma unroll
              for (int u = 0; u < 4; ++u) {
                const float2 f2 = cvt2<T16>(w[u]);
                pa[g][8 * v + 2 * u] += f2.x;
                pa[g][8 * v + 2 * u + 1] += f2.y;
              }
            }
          float hv[NU];
#pragma unroll
          for (int u = 0; u < NU; ++u) {
            const float cn = sigmoid_fast(pa[1][u]) * c[j][u] + sigmoid_fast(pa[0][u]) * tanh_fast(pa[2][u]);
            c[j][u] = cn;
            hv[u] = sigmoid_fast(pa[3][u]) * tanh_fast(cn);
          }
          if (row_ok) {
#pragma unroll
            for (int v = 0; v < NV; ++v) store8<T16>(out + o1 + 8 * v, &hv[8 * v]);
          }
          // publish h[t+1] first (it is all the peers wait for): one arrival per CTA and item, by the last epilogue warp
          // whose rows are stored (a warp can be at most two items ahead of another, so four counters never mix items)
          __syncwarp();
          if (lane == 0 && (smem_count_arrive(&pub_cnt[it & 3]) & (EW - 1)) == EW - 1 && !p.no_arrive)
            red_release_gpu_add(&p.flags[(size_t)(t + 1) * p.nbt + bt], 1);
          __syncwarp();
          // only now (after the release: a fence would otherwise wait for these loads) fetch the NEXT
          // item's projected pre-activations; they land while the peers run their step
          {
            int nj = j + 1, nt = t;
            if (nj == TI || pb + (ch * TI + nj) * p.nb_par >= p.nbt) { nj = 0; nt = t + 1; }
            load_pre(nt, pb + (ch * TI + nj) * p.nb_par);
            // the item after that: only pull its lines into L2 (a 32-byte sector covers both
            // warpgroups' pieces when each takes 16 bytes, so one of them asks)
            int fj = nj + 1, ft = nt;
            if (fj == TI || pb + (ch * TI + fj) * p.nb_par >= p.nbt) { fj = 0; ft = nt + 1; }
            const int fbt = pb + (ch * TI + fj) * p.nb_par;
            const int frow = fbt * RB + row_in_tile;
            if (ft < p.T && fbt < p.nbt && frow < p.B && (NV == 2 || ug == 0)) {
              const T16* src = ifgo + ((size_t)ft * p.B + frow) * H4 + unit0;
#pragma unroll
              for (int g = 0; g < 4; ++g) prefetch_l2(src + (size_t)g * H);
            }
          }
          // off the critical path: final pre-activations and c[t+1], saved for backward (inference: only the last cell
          // state is needed, as c_n)
          if (row_ok && (!p.inference || t == p.T - 1)) {
#pragma unroll
            for (int v = 0; v < NV; ++v) store8<T16>(cell + o1 + 8 * v, &c[j][8 * v]);
          }
          if (row_ok && !p.inference) {
#pragma unroll
            for (int g = 0; g < 4; ++g)
#pragma unroll
              for (int v = 0; v < NV; ++v) store8<T16>(gdst + (size_t)g * H + 8 * v, &pa[g][8 * v]);
          }
        }
      }
    }
  }
  // ---------------------------------------------------------------- teardown
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

template <int UH, int TI, typename T16>
static int launch_fwd_t(const RecPlan& pl, const CUtensorMap& tw, const CUtensorMap& th, const CUtensorMap& tp,
                        FwdParams& p, cudaStream_t st) {
  auto kern = fwd_kernel<UH, TI, T16>;
  BLSTM_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pl.smem));
  void* args[] = {(void*)&tw, (void*)&th, (void*)&tp, (void*)&p};
  BLSTM_CUDA_OK(cudaLaunchCooperativeKernel((void*)kern, dim3(pl.grid), dim3(pl.threads), args, pl.smem, st));
  count_launch();
  return BLSTM_OK;
}


// =====================================================================================
// Backward (replaces lstm_persistent_seq_bwd, fastlstm/kernels.py:1201-1409)
//
// dh_{t-1}[B,H] = d_ifgo[t][B,4H] x Wh[4H,H] has K = 4H.  A cluster of four CTAs owns 64
// output units of one batch tile; CTA r of the cluster takes gate r's K range (H rows of
// Wh, resident in shared memory as an N-major operand) and streams the matching H columns
// of d_ifgo[t] through TMA.  Each CTA ends a step with a partial [128 x 64] fp32 product in
// TMEM; the four partials are reduce-scattered through distributed shared memory by ROWS (a
// warp reads one 32-row quarter of the accumulator anyway; each CTA receives three 8 KB slices)
// so that CTA r finishes with dh of rows [32r, 32r+32) of the tile for all 64 units - whose gate
// maths it then does: thread = row x 8 units, a warp = 4 rows x 64 units, so every global access
// of the gate maths moves whole 128-byte lines.  (A split by units left 16-unit rows: 32-byte
// pieces that went through TMA boxes, whose stores had to complete before a hand-off: T=256, B=4096,
// H=512 took 9.5 ms a launch, 8.1 this way; T=256, B=256, H=768 2.36 -> 1.91; T=512, B=256, H=1024
// 5.1 -> 4.5; T=1024, B=32, H=2048 11.3 -> 10.5.  Bound by the hand-off chain of a step.)  dc is
// carried in fp32 registers, d_ifgo[t-1] is published with the same per-(step, batch tile)
// arrival counters as in the forward kernel.
// =====================================================================================
constexpr int DB_PARTS = 1024;            // row groups of the bias-gradient column sum
constexpr int XROW_BYTES = 128;           // one row of half a slice: 32 fp32; its 16-byte pieces are XOR-swizzled
constexpr int XSLOT_BYTES = 2 * 32 * XROW_BYTES;  // one exchanged slice: 2 halves x 32 rows x 32 fp32 = 8 KB

struct BwdPlan {
  bool ok;
  int nug, nbt, nb_par, ntl, TI, grid, threads, stages, ni, nl, ws, alias;
  int hb;                   // bytes of the d_ifgo rows in a ring stage (128 rows, or a single smaller tile's own)
  size_t w_bytes, recv_bytes, stage_bytes, smem;
  size_t off_flags, n_flags, off_db, ws_bytes;
};

// CTAs of the backward kernel that can be resident at once.  Clusters of four do not tile every GPC
// without a remainder: a B200 with 148 SMs holds 33 of them, 132 CTAs (asked of the occupancy
// calculator once per process, for the kernel's largest shared-memory footprint; defined behind the kernel).
static int bwd_cta_capacity();

static BwdPlan make_bwd_plan(const blstm_desc& d) {
  BwdPlan p{};
  p.ok = false;
  if (d.flags & BLSTM_FLAG_FORCE_GENERIC) return p;
  if (d.dtype != BLSTM_F16 && d.dtype != BLSTM_BF16) return p;
  const int H = d.hidden_size, B = d.batch;
  if (H % 64 != 0 || H < 64 || H > 2048) return p;
  p.nbt = cdiv(B, RB);
  p.nug = H / 64;
  const int per_tile = p.nug * 4;
  const int sms = std::min(plan_sm_count(), bwd_cta_capacity()) / ((d.flags & BLSTM_FLAG_HALF_DEVICE) ? 2 : 1);
  if (per_tile > sms) return p;
  p.nb_par = sms / per_tile;
  if (p.nb_par > p.nbt) p.nb_par = p.nbt;
  p.ntl = cdiv(p.nbt, p.nb_par);
  // Batch tiles interleaved per CTA.  Their only per-tile state is the carries in registers: the
  // exchange buffers below are indexed by item parity, not by tile.
  p.TI = p.ntl >= 3 ? 4 : p.ntl >= 2 ? 2 : 1;
  p.grid = p.nb_par * per_tile;
  p.threads = 0;                          // set below
  p.w_bytes = (size_t)H * 128;
  p.ws = p.w_bytes > 128 * 1024 ? 1 : 0;                   // stream the Wh slice through the ring
  p.hb = (p.nbt == 1 ? (int)round_up((size_t)B, 8) : RB) * 128;
  p.stage_bytes = p.hb + (p.ws ? 8192 : 0);
  // (a stage that holds fewer than 128 rows is still READ as 128 rows by the MMA: the ring is followed by
  //  enough shared memory for the last stage's read to stay inside the allocation)
  const size_t tail_pad = p.stage_bytes < (size_t)R_STAGE_BYTES ? R_STAGE_BYTES - p.stage_bytes : 0;
  // Streamed means all of it (the depth of the ring is worth more than the bytes a resident part saves:
  // H=2048 measured 12.5 ms with 18 of 32 chunks resident against 11.5 ms with none).
  const size_t wres = p.ws ? 0 : p.w_bytes;
  // Cluster exchange: receive slots (4 CTAs x 8 KB, this CTA's own among them) and send staging (3 x 8 KB), one
  // set.  With interleaved tiles a CTA tells the cluster when it has consumed an item's slices, and nobody
  // stages or ships the next item before all four have said so (`consumed` in the kernel).
  p.recv_bytes = (size_t)(4 + 3) * XSLOT_BYTES;
  if (1024 + wres + p.recv_bytes + 1024 + 3 * p.stage_bytes > 232448 && p.TI >= 2)
    p.TI = 1;                                               // not enough room to interleave tiles
  size_t fixed = 1024 + wres + p.recv_bytes + 1024 + tail_pad;  // 1024: barriers and counters behind the ring
  // warps: 1 producer + 2 MMA issuers + a publisher (idle unless tiles are interleaved) + 2 epilogue warpgroups = 12
  // (3 per SM sub-partition, 168 registers each); a 13th warp would cap every thread at 128 registers.
  const int n_issuers = 2;
  p.threads = 32 * 12;
  if (!pick_ring(fixed, p.stage_bytes, n_issuers, H / RK, &p.stages, &p.ni)) return p;
  // One tile in flight and a shallow ring (H = 768, 1024: the resident weights leave four stages, or two):
  // the ring is idle while an item's slices cross the cluster, so the exchange buffers are laid over
  // its first stages and the ring gets their 56 KB.  A peer may then write a slice only after this
  // CTA has finished the item's MMAs, which each CTA tells its peers (see `rdy` in the kernel).
  p.alias = 0;
  if (p.TI == 1 && p.stages < 6) {
    int st2 = 0, ni2 = 0;
    const size_t fixed2 = 1024 + wres + 1024 + tail_pad;
    if (pick_ring(fixed2, p.stage_bytes, n_issuers, H / RK, &st2, &ni2) && st2 > p.stages &&
        (size_t)st2 * p.stage_bytes >= p.recv_bytes) {
      p.alias = 1; p.stages = st2; p.ni = ni2; fixed = fixed2;
    }
  }
  // TMA-issuing lanes of the producer warp (nl | stages): four interleaved tiles do better with four
  // (B=4096, H=512: 8.5 -> 8.1 ms), a single tile on a six-stage ring with two (H=1024: 5.33 -> 5.22 ms)
  p.nl = p.ni;
  if (p.TI == 4) p.nl = 4;
  if (p.TI == 1) p.nl = p.stages == 6 ? 2 : 4;
  if (p.stages % p.nl != 0 || p.nl > H / RK) p.nl = p.ni;
  p.smem = fixed + (size_t)p.stages * p.stage_bytes;
  p.n_flags = (size_t)d.seq_len * p.nbt;
  p.off_flags = sizeof(Control);
  p.off_db = p.off_flags + round_up(p.n_flags * sizeof(int), 256);
  p.ws_bytes = p.off_db + round_up((size_t)std::max(DB_PARTS, p.nb_par * 32) * 4 * H * sizeof(float), 256);
  p.ok = true;
  return p;
}

struct BwdParams {
  int T, B, H;
  int nbt, nug, nb_par, ntl;
  int stages;
  int ni;
  int nl;                   // TMA-issuing lanes of the producer warp (nl divides the ring depth)
  int ws;                   // 1: the Wh slice streamed through the ring instead of resident
  int hb;                   // bytes of the d_ifgo rows in a ring stage
  int stage_bytes;
  int fmt;
  int no_arrive;
  int flag_target;          // arrivals that complete a flag: H/16 CTAs per batch tile
  int alias;                // 1: exchange buffers laid over the first ring stages (one tile in flight)
  unsigned long long limit_ns;
  Control* ctl;
  int* flags;               // [T][nbt]: arrivals for d_ifgo[t]
  const void* dout;         // [T,B,H]
  const void* dh_n;         // [B,H] or null
  const void* dc_n;         // [B,H] or null
  const void* ifgo;         // [T,B,4H]
  const void* cell;         // [T+1,B,H]
  void* d_ifgo;             // [T,B,4H]
  void* dh0;                // [B,H]
  void* dc0;                // [B,H]
  float* db_part;           // [nb_par * 32][4H] bias-gradient partial sums (one row per CTA group and four rows of its tiles), or null
};

template <int TI, typename T16>
__global__ void __launch_bounds__(384, 1)
bwd_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmG, const BwdParams p) {
  // Warps: 0 = TMA producer, then NACC MMA issuers, then (interleaved tiles only) one PUBLISHER warp,
  // then 8 epilogue warps from warp 4 on - 12 in all either way.
  // With interleaved tiles the epilogue warps are the bottleneck, and the release that publishes an
  // item stalls its thread for a memory round trip: there a thread of its own does the releasing
  // (the epilogue warps only arrive on a CTA-local barrier after their stores), which costs one issuer.
  constexpr bool PUBLISHER = (TI >= 2);
  constexpr int N = 64, NACC = 2, ACC_STRIDE = 256;   // NACC: MMA issuer warps
  constexpr int FIRST_EPI = 4;
  constexpr int ITEM_WARPS = 8;                   // epilogue warps, all working on every item
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int H = p.H;
  const int KC = H / RK;
  const int R_STAGES = p.stages;
  uint8_t* w_s = smem;                                        // [KC][64 k rows][128 B]
  const int SB = p.stage_bytes;                               // d_ifgo chunk (16 KB) [+ Wh chunk when streamed]
  const int HB = p.hb;                                        // d_ifgo rows of a stage; a streamed Wh chunk follows
  uint8_t* recv = smem + (p.ws ? 0 : (size_t)KC * 8192);      // [4 senders][2 halves][32 rows][128 B]
  uint8_t* stage = recv + (size_t)4 * XSLOT_BYTES;            // [3 receivers][2 halves][32 rows][128 B]
  uint8_t* a_s = p.alias ? recv : stage + (size_t)3 * XSLOT_BYTES;   // ring (over the exchange buffers if aliased)
  uint64_t* bars = reinterpret_cast<uint64_t*>(a_s + (size_t)R_STAGES * SB);
  uint64_t* full = bars;
  uint64_t* empty = bars + R_MAX_STAGES;
  uint64_t* acc_full = bars + 2 * R_MAX_STAGES;
  uint64_t* acc_empty = acc_full + 2;
  uint64_t* w_full = acc_empty + 2;
  uint64_t* xchg = w_full + 1;                                // slices of an item complete
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(xchg + 1);
  volatile int* dead = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int* pub_cnt = const_cast<int*>(dead) + 1;        // [4] arrivals of the epilogue warps, by item index mod 4
  uint64_t* pub_bar = reinterpret_cast<uint64_t*>(pub_cnt + 4);   // [4] item stored? by item index mod 4
  uint64_t* rdy = pub_bar + 4;                                 // aliased buffers: the 3 peers' issuers are done with their MMAs
  uint64_t* consumed = rdy + 1;                                // interleaved tiles: the cluster's four CTAs read an item's slices
  uint64_t* taken = consumed + 1;                              // ... this CTA's eight warps did

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t r = cluster_ctarank();                       // gate whose K range this CTA owns
  const int cid = blockIdx.x >> 2;
  const int ugc = cid % p.nug, pb = cid / p.nug;
  constexpr uint32_t TMEM_COLS = 512;
  const int nacc = p.ni;                             // accumulators / issuers / TMA lanes in use

  if (threadIdx.x == 0) {
    // full[s] is armed (arrive + expected bytes) for its first use here and re-armed by the MMA issuer
    // that consumed it for every later use, which keeps that work out of the latency-bound TMA producer loop
    for (int s = 0; s < R_STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(&acc_full[a], nacc); mbar_init(&acc_empty[a], ITEM_WARPS); }
    mbar_init(w_full, 1);
    mbar_init(xchg, 3);                             // one expect_tx arrival + tx bytes, and the two warps of the own quarter
    *dead = 0;
    for (int i = 0; i < 4; ++i) pub_cnt[i] = 0;
    for (int i = 0; i < 4; ++i) mbar_init(&pub_bar[i], ITEM_WARPS);
    mbar_init(rdy, 3 * nacc);
    mbar_init(consumed, 4);
    mbar_init(taken, ITEM_WARPS);
    fence_mbar_init();
    for (int s = 0; s < R_STAGES; ++s) mbar_expect_tx(&full[s], SB);
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmG);
  }
  if (warp == 1) tmem_alloc(tmem_slot, TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  cluster_sync_all();                 // peers' barriers exist before anyone arrives on them remotely
  const uint32_t tmem_base = *tmem_slot;
  WaitCtx wc{dead, p.ctl, p.limit_ns, -1, (int)blockIdx.x};
  const int n_chunks = (p.ntl + TI - 1) / TI;
  const int T = p.T;

  // Items of a chunk: for s in [0,T] : for j in [0,TI).  Item (s,j) first (s > 0) forms
  // dh = d_ifgo[T-s] x Wh for its tile, then (s < T) does the gate maths of step t = T-1-s.
  if (warp == 0) {
    // ---------------------------------------------------------------- TMA producer
    if (lane == 0 && !p.ws) {
      mbar_expect_tx(w_full, (uint32_t)((size_t)KC * 8192));
      for (int kc = 0; kc < KC; ++kc)
        tma_load_2d(w_s + (size_t)kc * 8192, &tmW, w_full, ugc * 64, (int)r * H + kc * RK);
    }
    int gs = 0;
    uint32_t gph = 0;
    bool ok = true;
    // With interleaved tiles an item's arrival counter is usually complete long before its turn, and
    // what costs is the round trip of looking: lane 31 reads the NEXT item's counter while the other
    // lanes issue the current item's loads, and lane 0 only spins when that early look found it incomplete.
    ItemCursor<TI> nx;
    nx.init();
    bool nx_valid = nx.next(pb, p.nb_par, p.nbt, n_chunks, T);   // the first item itself
    int early = 0;             // lane 31: early reading of the next item's counter
    for (int ch = 0; ch < n_chunks && ok; ++ch) {
      for (int st = 1; st <= T && ok; ++st) {
        const int tg = T - st;      // timestep whose d_ifgo is streamed
        for (int j = 0; j < TI && ok; ++j) {
          const int bt = pb + (ch * TI + j) * p.nb_par;
          if (bt >= p.nbt) continue;
          const int early_now = (TI >= 2) ? __shfl_sync(0xffffffffu, early, 31) : 0;
          if (TI >= 2) nx_valid = nx_valid && nx.next(pb, p.nb_par, p.nbt, n_chunks, T);
          int seen = 1;
          if (lane == 0 && !(TI >= 2 && early_now >= p.flag_target)) {
            wc.d0 = tg; wc.d1 = bt;
            seen = wait_flag_ge(&p.flags[(size_t)tg * p.nbt + bt], p.flag_target, p.ctl, p.limit_ns, tg, bt) ? 1 : 0;
          }
          seen = __shfl_sync(0xffffffffu, seen, 0);
          __syncwarp();      // (a shuffle orders no memory: the issuing lanes come behind the acquire)
          if (!seen) { *dead = 1; ok = false; break; }
          // a proxy fence between the peers' arrivals (interleaved tiles: their plain stores, fenced by their publisher
          // warps) and the TMA reads below
          if (!PUBLISHER) fence_proxy_async_global();
          const int row0 = bt * RB, col0 = (int)r * H;
          bool lane_ok = true;
          const int nl = p.nl;                 // TMA-issuing lanes: lane l owns the ring stages == l (mod nl)
          if (lane < nl) {
            // this lane owns ring stages == lane (mod nl): the item's chunks that land there
            for (int kc = (lane + nl - gs % nl) % nl; kc < KC; kc += nl) {
              int s = gs + kc;
              uint32_t ph = gph;
              while (s >= R_STAGES) { s -= R_STAGES; ph ^= 1; }
              if (!mbar_wait(&empty[s], ph ^ 1, wc)) { lane_ok = false; break; }
              tma_load_3d(a_s + (size_t)s * SB, &tmG, &full[s], col0 + kc * RK, row0, tg);
              if (p.ws) tma_load_2d(a_s + (size_t)s * SB + HB, &tmW, &full[s], ugc * 64, col0 + kc * RK);
            }
          } else if (TI >= 2 && lane == 31) {
            // (the other arm of the same branch: the issuing lanes do not wait for this read)
            early = 0;
            if (nx_valid) early = ld_acquire_gpu(&p.flags[(size_t)(T - 1 - nx.t) * p.nbt + nx.tile(pb, p.nb_par)]);
          }
          if (__any_sync(0xffffffffu, !lane_ok)) { ok = false; break; }
          gs += KC;
          while (gs >= R_STAGES) { gs -= R_STAGES; gph ^= 1; }
        }
      }
    }
  } else if (PUBLISHER && warp == 1 + NACC) {
    // ---------------------------------------------------------------- publisher
    // Walks the items in the epilogue's order.  When all eight epilogue warps have read an item's slices, one fence at
    // cluster scope and an arrival per CTA tell the cluster (a release by every warp stalls them 0.7 k clocks and more).  When
    // all eight have stored an item's d_ifgo rows (their arrival on pub_bar is a CTA-scope release, this wait the
    // acquire), one release at GPU scope counts this CTA in on the item's arrival counter.  An epilogue warp can
    // be at most four items ahead of the slowest (it needs the counters this thread completes), so
    // four barriers never mix items; and it needs this thread's arrival for an item before it reads the next one's slices.
    if (lane == 0) {
      int k = 0, it = 0;
      bool ok = true;
      for (int ch = 0; ch < n_chunks && ok; ++ch) {
        for (int st = 0; st <= T && ok; ++st) {
          for (int j = 0; j < TI && ok; ++j) {
            const int bt = pb + (ch * TI + j) * p.nb_par;
            if (bt >= p.nbt) continue;
            wc.d0 = T - 1 - st; wc.d1 = bt;
            if (st > 0) {
              if (!mbar_wait(taken, (uint32_t)it & 1u, wc)) { ok = false; break; }
              ++it;
              fence_acq_rel_cluster();
#pragma unroll
              for (int dst = 0; dst < 4; ++dst) mbar_arrive_remote_relaxed(mapa_shared(smem_u32(consumed), dst));
            }
            if (st == T) continue;
            if (!mbar_wait(&pub_bar[k & 3], (uint32_t)(k >> 2) & 1u, wc)) { ok = false; break; }
            // the generic->async proxy fence of the hand-off runs here, on the causality path between
            // the epilogue warps' stores (ordered before this thread by the barrier) and the release
            fence_proxy_async_global();
            if (!p.no_arrive) red_release_gpu_add(&p.flags[(size_t)(T - 1 - st) * p.nbt + bt], 1);
            ++k;
          }
        }
      }
    }
  } else if (warp < 1 + NACC) {
    // ---------------------------------------------------------------- MMA issuers (own whole chunks)
    const int x = warp - 1;
    if (elect_one()) {
      constexpr uint64_t descA = smem_desc_base(16, 1024);       // d_ifgo tile, K-major
      constexpr uint64_t descB = smem_desc_base(8192, 1024);     // Wh chunk, N-major (64 units wide)
      const uint32_t idesc = instr_desc(p.fmt, 0, 1, RB, N);
      bool ok = (x < nacc) && (p.ws || mbar_wait(w_full, 0, wc));
      int gs = 0;
      uint32_t gph = 0;
      uint32_t acc_ph[2] = {0, 0};
      int it = 0;
      const uint32_t w_addr = smem_u32(w_s);
      for (int ch = 0; ch < n_chunks && ok; ++ch) {
        for (int st = 1; st <= T && ok; ++st) {
          for (int j = 0; j < TI && ok; ++j) {
            const int bt = pb + (ch * TI + j) * p.nb_par;
            if (bt >= p.nbt) continue;
            const int a = it & 1;
            ++it;
            if (!mbar_wait(&acc_empty[a], acc_ph[a] ^ 1, wc)) { ok = false; break; }
            acc_ph[a] ^= 1;
            tc_fence_after();
            const uint32_t d_tmem = tmem_base + a * ACC_STRIDE + x * N;
            uint32_t acc_on = 0;
            for (int kc = (x + nacc - gs % nacc) % nacc; kc < KC; kc += nacc) {
              int s = gs + kc;
              uint32_t ph = gph;
              while (s >= R_STAGES) { s -= R_STAGES; ph ^= 1; }
              if (!mbar_wait_spin(&full[s], ph, wc)) { ok = false; break; }
              // arm the stage's next use: R_STAGES chunks further on (chunks wrap around within an item)
              mbar_expect_tx(&full[s], SB);
              tc_fence_after();
              const uint32_t sa = smem_u32(a_s + (size_t)s * SB);
              const uint32_t sb = p.ws ? sa + HB : w_addr + (uint32_t)kc * 8192;
#pragma unroll
              for (int k = 0; k < RK / 16; ++k)
                umma_f16(d_tmem, smem_desc(descA, sa + k * 32), smem_desc(descB, sb + k * 2048), idesc,
                         (k > 0) ? 1u : acc_on);
              acc_on = 1;
              umma_commit(&empty[s]);
            }
            if (ok) umma_commit(&acc_full[a]);
            // aliased: once these MMAs have read it the ring, and the exchange buffers laid over it, is idle until the
            // next item: the three peers may write their slices
            if (TI == 1 && ok && p.alias) umma_commit_multicast(rdy, (uint16_t)(0xF ^ (1u << r)));
            gs += KC;
            while (gs >= R_STAGES) { gs -= R_STAGES; gph ^= 1; }
          }
        }
      }
    }
  } else if (warp >= FIRST_EPI) {
    // ---------------------------------------------------------------- epilogue: two warpgroups
    constexpr int NU = 8;                        // units per thread
    const int ew = warp - FIRST_EPI;
    // accumulator read-out: thread = row `lane` of quarter q, units 32g .. 32g+31
    const int g = ew >> 2, q = warp & 3;
    // gate maths: thread = row grow of this CTA's quarter r, units gu .. gu+7 of the cluster's 64
    const int grow = ew * 4 + (lane >> 3), gu = (lane & 7) * 8;
    const int row_in_tile = (int)r * 32 + grow;
    const int unit0 = ugc * 64 + gu;
    const size_t H4 = 4 * (size_t)H;
    const T16* ifgo = reinterpret_cast<const T16*>(p.ifgo);
    const T16* cell = reinterpret_cast<const T16*>(p.cell);
    const T16* dout = reinterpret_cast<const T16*>(p.dout);
    T16* dg = reinterpret_cast<T16*>(p.d_ifgo);
    // where the accumulator's pieces go: this CTA's own receive slot, or the staging slot of CTA q
    // (a slot is two halves of 32 rows x 32 units, one per warpgroup, so that every warp ships its own 4 KB)
    uint8_t* put = (q == (int)r ? recv + (size_t)r * XSLOT_BYTES : stage + (size_t)(q < (int)r ? q : q - 1) * XSLOT_BYTES) + g * (XSLOT_BYTES / 2);
    // a half's row is 128 bytes; piece k lies at k XOR row XOR half: conflict-free for the writers (32 rows, one piece)
    // and for the readers (a row's even, then odd pieces of both halves)
    const int half = (lane >> 2) & 1;
    const uint8_t* get = recv + half * (XSLOT_BYTES / 2) + grow * XROW_BYTES;
    const int get_x = (grow & 7) ^ half;
    // Bias gradient (replaces the reduction of fastlstm/lstm.py:497 and a separate pass over d_ifgo):
    // every thread adds the d_ifgo values it stores - as stored, i.e. rounded - to 32 fp32 sums of its
    // own (4 gates x 8 units) that live in the tensor-memory columns behind the accumulators, one
    // 32-column block per warpgroup; after the last step the four rows of a warp are added up with
    // shuffles and its first eight lanes write the warp's partial sums.
    constexpr int DB_COL = 192;                  // NACC * N <= 192 columns per accumulator buffer are in use
    const uint32_t db_taddr = tmem_base + DB_COL + g * 32 + (uint32_t(q * 32) << 16);
    const bool want_db = p.db_part != nullptr;
    if (want_db) {
      uint32_t z[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) z[u] = 0u;
#pragma unroll
      for (int k = 0; k < 4; ++k) tmem_st_32x8(db_taddr + 8 * k, z);
      tmem_st_wait();
    }
    int it = 0;                 // MMA items consumed so far: TMEM buffer it & 1, on its (it >> 1)-th use
    int pub_it = 0;             // gate-maths items published so far
    bool ok = true;
    for (int ch = 0; ch < n_chunks && ok; ++ch) {
      // dc and c[t+1] are carried per interleaved tile; dh is rebuilt from the accumulator in every item, so one
      // copy serves all tiles (its first value, the gradient of h_n, is fetched in the tile's first item)
      float dc[TI][NU], dhc[NU];
      uint4 cn[TI];      // c[t+1] of the tile's next item
      uint4 pf[6];       // next item's inputs: gates i,f,g,o, c[t], dout[t]
#pragma unroll
      for (int j = 0; j < TI; ++j) {
        const int bt = pb + (ch * TI + j) * p.nb_par;
        const int row = bt * RB + row_in_tile;
        const bool rok = bt < p.nbt && row < p.B;
        cn[j] = make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int u = 0; u < NU; ++u) dc[j][u] = 0.f;
        if (rok) {
          cn[j] = ldg16(cell + ((size_t)T * p.B + row) * H + unit0);
          if (p.dc_n) unpack8<T16>(ldg16(reinterpret_cast<const T16*>(p.dc_n) + (size_t)row * H + unit0), dc[j]);
        }
      }
      auto prefetch = [&](int t, int bt) {
        const int row = bt * RB + row_in_tile;
        if (bt < p.nbt && row < p.B) {
          const size_t m = (size_t)t * p.B + row;
          const T16* gsrc = ifgo + m * H4 + unit0;
#pragma unroll
          for (int k = 0; k < 4; ++k) pf[k] = ldg16(gsrc + (size_t)k * H);
          pf[4] = ldg16(cell + m * H + unit0);
          pf[5] = ldg16(dout + m * H + unit0);
        }
      };
      // two items ahead the same lines are only pulled into L2: lane k of a row's eight asks for the k-th of its six
      auto prefetch_far = [&](int t, int bt) {
        const int row = bt * RB + row_in_tile, k = lane & 7;
        if (k < 6 && bt < p.nbt && row < p.B) {
          const size_t m = (size_t)t * p.B + row;
          prefetch_l2(k < 4 ? ifgo + m * H4 + (size_t)k * H + ugc * 64 : (k == 4 ? cell : dout) + m * H + ugc * 64);
        }
      };
      // Everything in the gate maths that does not depend on dh is worked out ahead of the accumulator:
      //   dh = dout + dh_carry;  dcv = dh*fA + dc;  d_i = dcv*fBi;  d_f = dcv*fBf;  d_g = dcv*fBg;
      //   d_o = dh*fBo;  dc' = dcv*fSf
      // With one tile in flight that happens as soon as the prefetched inputs land (the warps would
      // only wait for the next accumulator); with interleaved tiles it fills the cluster exchange.
      constexpr bool USE_FACTORS = (TI <= 2);
      constexpr bool EARLY_FACTORS = (TI == 1);
      constexpr int NF = USE_FACTORS ? NU : 1;
      float fA[NF], fBi[NF], fBf[NF], fBg[NF], fBo[NF], fSf[NF], fDd[NF];
      // (c1: c[t+1] of the item; its c[t] takes its place for the tile's next one)
      auto factors = [&](uint4& c1v) {
        if constexpr (USE_FACTORS) {
          const uint32_t wi[4] = {pf[0].x, pf[0].y, pf[0].z, pf[0].w};
          const uint32_t wf[4] = {pf[1].x, pf[1].y, pf[1].z, pf[1].w};
          const uint32_t wg[4] = {pf[2].x, pf[2].y, pf[2].z, pf[2].w};
          const uint32_t wo[4] = {pf[3].x, pf[3].y, pf[3].z, pf[3].w};
          const uint32_t w1[4] = {c1v.x, c1v.y, c1v.z, c1v.w};
          const uint32_t w0[4] = {pf[4].x, pf[4].y, pf[4].z, pf[4].w};
          const uint32_t wd[4] = {pf[5].x, pf[5].y, pf[5].z, pf[5].w};
#pragma unroll
          for (int w = 0; w < 4; ++w) {
            const float2 pi = cvt2<T16>(wi[w]), pff = cvt2<T16>(wf[w]), pg = cvt2<T16>(wg[w]), po = cvt2<T16>(wo[w]);
            const float2 c1 = cvt2<T16>(w1[w]), c0 = cvt2<T16>(w0[w]), dd = cvt2<T16>(wd[w]);
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const int u = 2 * w + e;
              const float si = sigmoid_fast(e ? pi.y : pi.x), sf = sigmoid_fast(e ? pff.y : pff.x);
              const float so = sigmoid_fast(e ? po.y : po.x);
              const float tg = tanh_fast(e ? pg.y : pg.x), tc = tanh_fast(e ? c1.y : c1.x);
              fA[u] = so * (1.f - tc * tc);
              fBi[u] = tg * si * (1.f - si);
              fBf[u] = (e ? c0.y : c0.x) * sf * (1.f - sf);
              fBg[u] = si * (1.f - tg * tg);
              fBo[u] = tc * so * (1.f - so);
              fSf[u] = sf;
              fDd[u] = e ? dd.y : dd.x;
            }
          }
          c1v = pf[4];
        }
      };
      prefetch(T - 1, pb + (ch * TI) * p.nb_par);
      if (USE_FACTORS && EARLY_FACTORS) factors(cn[0]);
      for (int st = 0; st <= T && ok; ++st) {
#pragma unroll
        for (int j = 0; j < TI; ++j) {
          const int bt = pb + (ch * TI + j) * p.nb_par;
          if (bt >= p.nbt) continue;
          const int row = bt * RB + row_in_tile;
          const bool row_ok = row < p.B;
          if (st > 0) {
            // ---- dh = (sum over the cluster's four K ranges of) d_ifgo[T-st] x Wh
            const int a = it & 1;
            const uint32_t a_ph = (uint32_t)(it >> 1) & 1u;
            // one set of exchange buffers: its barriers change phase with every item
            const uint32_t x_ph = (uint32_t)it & 1u;
            ++it;
            wc.d0 = T - st; wc.d1 = bt;
            if (!mbar_wait(&acc_full[a], a_ph, wc)) { ok = false; break; }
            if constexpr (TI >= 2) {
              // the previous item's slices have been read by the whole cluster (so the staging below overwrites
              // nothing a copy still reads, and the receive slots are free again)
              if (it > 1 && !mbar_wait_cluster(consumed, (uint32_t)it & 1u, wc)) { ok = false; break; }
            }
            if (ew == 0 && lane == 0) {
              // what this CTA is about to receive (nothing for a quarter without rows)
              mbar_expect_tx(xchg, bt * RB + (int)r * 32 < p.B ? 3 * XSLOT_BYTES : 0);
            }
            tc_fence_after();
            const bool q_ok = bt * RB + q * 32 < p.B;       // quarter q has rows
            const uint32_t taddr = tmem_base + a * ACC_STRIDE + (uint32_t(q * 32) << 16) + g * 32;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              // the issuers' partial accumulators for 16 units: NACC loads, ONE wait
              uint32_t v[NACC][16];
#pragma unroll
              for (int xx = 0; xx < NACC; ++xx) tmem_ld_32x16(taddr + xx * N + h * 16, v[xx]);
              tmem_ld_wait();
#pragma unroll
              for (int c4 = 0; c4 < 4; ++c4) {
                float sum[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                  float a0 = __uint_as_float(v[0][4 * c4 + u]);
                  if (nacc > 1) a0 += __uint_as_float(v[1][4 * c4 + u]);
                  sum[u] = a0;
                }
                *reinterpret_cast<float4*>(put + lane * XROW_BYTES + (((h * 4 + c4) ^ (lane & 7) ^ g) << 4)) = make_float4(sum[0], sum[1], sum[2], sum[3]);
              }
            }
            tc_fence_before();
            fence_proxy_async_smem();                 // staged slices -> visible to the bulk-copy engine
            __syncwarp();
            if (lane == 0) {
              mbar_arrive(&acc_empty[a]);
              if (q == (int)r) mbar_arrive(xchg);
              else if (q_ok && (!p.alias || mbar_wait_cluster(rdy, x_ph, wc)))       // aliased: every peer's ring is idle
                dsmem_bulk_copy(mapa_shared(smem_u32(recv) + r * XSLOT_BYTES + g * (XSLOT_BYTES / 2), q), put, XSLOT_BYTES / 2,
                                mapa_shared(smem_u32(xchg), q));
            }
            __syncwarp();
            if (USE_FACTORS && !EARLY_FACTORS && st < T) factors(cn[j]);       // fills the wait for the peers' slices
            if (!mbar_wait_cluster(xchg, x_ph, wc)) { ok = false; break; }
#pragma unroll
            for (int u = 0; u < NU; ++u) dhc[u] = 0.f;
#pragma unroll
            for (int s = 0; s < 4; ++s)
#pragma unroll
              for (int o = 0; o < 2; ++o) {
                const float4 v = *reinterpret_cast<const float4*>(get + s * XSLOT_BYTES + (((2 * (lane & 3) + o) ^ get_x) << 4));
                dhc[4 * o] += v.x;
                dhc[4 * o + 1] += v.y;
                dhc[4 * o + 2] += v.z;
                dhc[4 * o + 3] += v.w;
              }
            if constexpr (TI >= 2) {
              // this warp has read the item's slices: the publisher tells the cluster once all eight have
              __syncwarp();
              if (lane == 0) mbar_arrive(taken);
            }
          }
          if (st == 0) {
#pragma unroll
            for (int u = 0; u < NU; ++u) dhc[u] = 0.f;
            if (row_ok && p.dh_n) unpack8<T16>(ldg16(reinterpret_cast<const T16*>(p.dh_n) + (size_t)row * H + unit0), dhc);
          }
          if (st < T) {
            // ---- gate maths of step t for this thread's row and 8 units, two per packed word
            const int t = T - 1 - st;
            uint32_t qi[4], qf[4], qg[4], qo[4];
            if constexpr (USE_FACTORS) {
              if (!EARLY_FACTORS && st == 0) factors(cn[j]);            // later items computed them during the exchange
#pragma unroll
              for (int w = 0; w < 4; ++w) {
                float r_[2][4];
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                  const int u = 2 * w + e;
                  const float dh = fDd[u] + dhc[u];
                  const float dcv = fmaf(dh, fA[u], dc[j][u]);
                  r_[e][0] = dcv * fBi[u];
                  r_[e][1] = dcv * fBf[u];
                  r_[e][2] = dcv * fBg[u];
                  r_[e][3] = dh * fBo[u];
                  dc[j][u] = dcv * fSf[u];
                }
                qi[w] = pk2<T16>(r_[0][0], r_[1][0]);
                qf[w] = pk2<T16>(r_[0][1], r_[1][1]);
                qg[w] = pk2<T16>(r_[0][2], r_[1][2]);
                qo[w] = pk2<T16>(r_[0][3], r_[1][3]);
              }
            } else {
              // four interleaved tiles leave no registers for the factors: all of the maths here
              const uint32_t wi[4] = {pf[0].x, pf[0].y, pf[0].z, pf[0].w};
              const uint32_t wf[4] = {pf[1].x, pf[1].y, pf[1].z, pf[1].w};
              const uint32_t wg[4] = {pf[2].x, pf[2].y, pf[2].z, pf[2].w};
              const uint32_t wo[4] = {pf[3].x, pf[3].y, pf[3].z, pf[3].w};
              const uint32_t w1[4] = {cn[j].x, cn[j].y, cn[j].z, cn[j].w};
              const uint32_t w0[4] = {pf[4].x, pf[4].y, pf[4].z, pf[4].w};
              const uint32_t wd[4] = {pf[5].x, pf[5].y, pf[5].z, pf[5].w};
              cn[j] = pf[4];
#pragma unroll
              for (int w = 0; w < 4; ++w) {
                const float2 pi = cvt2<T16>(wi[w]), pff = cvt2<T16>(wf[w]), pg = cvt2<T16>(wg[w]), po = cvt2<T16>(wo[w]);
                const float2 c1 = cvt2<T16>(w1[w]), c0 = cvt2<T16>(w0[w]), dd = cvt2<T16>(wd[w]);
                float r_[2][4];
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                  const int u = 2 * w + e;
                  const float si = sigmoid_fast(e ? pi.y : pi.x), sf = sigmoid_fast(e ? pff.y : pff.x);
                  const float so = sigmoid_fast(e ? po.y : po.x);
                  const float tg = tanh_fast(e ? pg.y : pg.x), tc = tanh_fast(e ? c1.y : c1.x);
                  const float dh = (e ? dd.y : dd.x) + dhc[u];
                  const float dcv = fmaf(dh * so, 1.f - tc * tc, dc[j][u]);
                  r_[e][0] = dcv * (tg * si * (1.f - si));
                  r_[e][1] = dcv * ((e ? c0.y : c0.x) * sf * (1.f - sf));
                  r_[e][2] = dcv * (si * (1.f - tg * tg));
                  r_[e][3] = dh * (tc * so * (1.f - so));
                  dc[j][u] = dcv * sf;
                }
                qi[w] = pk2<T16>(r_[0][0], r_[1][0]);
                qf[w] = pk2<T16>(r_[0][1], r_[1][1]);
                qg[w] = pk2<T16>(r_[0][2], r_[1][2]);
                qo[w] = pk2<T16>(r_[0][3], r_[1][3]);
              }
            }
            if (row_ok) {
              T16* dstp = dg + ((size_t)t * p.B + row) * H4 + unit0;
              stg16(dstp, make_uint4(qi[0], qi[1], qi[2], qi[3]));
              stg16(dstp + (size_t)H, make_uint4(qf[0], qf[1], qf[2], qf[3]));
              stg16(dstp + 2 * (size_t)H, make_uint4(qg[0], qg[1], qg[2], qg[3]));
              stg16(dstp + 3 * (size_t)H, make_uint4(qo[0], qo[1], qo[2], qo[3]));
            }
            // publish d_ifgo[t] rows of this warp, then (after the release) fetch the next item's inputs: one arrival per
            // CTA and item, by the publisher warp (interleaved tiles) or the last epilogue warp whose rows are stored
            // (a warp can be at most four items ahead of another - the maths-only items that open a chunk - so four
            // counters never mix items)
            __syncwarp();
            if (lane == 0) {
              if constexpr (PUBLISHER) {
                mbar_arrive(&pub_bar[pub_it & 3]);
              } else {
                const bool pub = (smem_count_arrive(&pub_cnt[pub_it & 3]) & (ITEM_WARPS - 1)) == ITEM_WARPS - 1;
                if (pub && !p.no_arrive) red_release_gpu_add(&p.flags[(size_t)t * p.nbt + bt], 1);
              }
            }
            __syncwarp();
            ++pub_it;
            {
              int nj = j + 1, ns = st;
              if (nj == TI || pb + (ch * TI + nj) * p.nb_par >= p.nbt) { nj = 0; ns = st + 1; }
              if (ns < T) prefetch(T - 1 - ns, pb + (ch * TI + nj) * p.nb_par);
              int fj = nj + 1, fs = ns;
              if (fj == TI || pb + (ch * TI + fj) * p.nb_par >= p.nbt) { fj = 0; fs = ns + 1; }
              if (fs < T) prefetch_far(T - 1 - fs, pb + (ch * TI + fj) * p.nb_par);
            }
            // bias-gradient sums: after the publication, off the hand-off chain
            if (want_db) {   // warp-uniform: tensor-memory loads and stores need the whole warp; rows past B add 0
              const uint32_t* qs[4] = {qi, qf, qg, qo};
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                uint32_t acc[8];
                tmem_ld_32x8(db_taddr + 8 * k, acc);
                tmem_ld_wait();
#pragma unroll
                for (int w = 0; w < 4; ++w) {
                  const float2 f2 = cvt2<T16>(qs[k][w]);
                  acc[2 * w] = __float_as_uint(__uint_as_float(acc[2 * w]) + (row_ok ? f2.x : 0.f));
                  acc[2 * w + 1] = __float_as_uint(__uint_as_float(acc[2 * w + 1]) + (row_ok ? f2.y : 0.f));
                }
                tmem_st_32x8(db_taddr + 8 * k, acc);
              }
              tmem_st_wait();
            }
            if (USE_FACTORS && EARLY_FACTORS && st + 1 < T) factors(cn[0]);
          } else if (row_ok) {
            // ---- after the last step: the carries are the gradients of the initial state
            store8<T16>(reinterpret_cast<T16*>(p.dh0) + (size_t)row * H + unit0, dhc);
            store8<T16>(reinterpret_cast<T16*>(p.dc0) + (size_t)row * H + unit0, dc[j]);
          }
        }
      }
    }
    if (want_db) {
      float* dst = p.db_part + (((size_t)pb * 4 + r) * ITEM_WARPS + ew) * H4 + unit0;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        uint32_t acc[8];
        tmem_ld_32x8(db_taddr + 8 * k, acc);
        tmem_ld_wait();
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          float v = __uint_as_float(acc[u]);
          v += __shfl_xor_sync(0xffffffffu, v, 8);
          v += __shfl_xor_sync(0xffffffffu, v, 16);
          if (lane < 8) dst[(size_t)k * H + u] = v;
        }
      }
    }
  }
  // ---------------------------------------------------------------- teardown
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
  cluster_sync_all();   // no CTA leaves while a peer may still write into its shared memory
}

// Column sums of d_ifgo [rows, cols] (16-bit) over gridDim.y interleaved row groups -> part[gridDim.y][cols].
// HBM-bound (the whole d_ifgo is read once): a thread owns 8 adjacent columns (one 16-byte load per
// row, a warp covers 512 contiguous bytes) and keeps 8 row loads in flight.
template <typename T16>
__global__ void __launch_bounds__(128) colsum_kernel(const T16* __restrict__ g, int rows, int cols, float* __restrict__ part) {
  const int col = (blockIdx.x * 128 + threadIdx.x) * 8;
  if (col >= cols) return;
  float s[8];
  const int DB = gridDim.y;
#pragma unroll
  for (int u = 0; u < 8; ++u) s[u] = 0.f;
  const T16* src = g + col;
  int rr = blockIdx.y;
  for (; rr + 7 * DB < rows; rr += 8 * DB) {
    uint4 v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = ldg16(src + (size_t)(rr + i * DB) * cols);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint32_t w[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
#pragma unroll
      for (int u = 0; u < 4; ++u) { const float2 f = cvt2<T16>(w[u]); s[2 * u] += f.x; s[2 * u + 1] += f.y; }
    }
  }
  for (; rr < rows; rr += DB) {
    const uint4 v = ldg16(src + (size_t)rr * cols);
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int u = 0; u < 4; ++u) { const float2 f = cvt2<T16>(w[u]); s[2 * u] += f.x; s[2 * u + 1] += f.y; }
  }
  float* dst = part + (size_t)blockIdx.y * cols + col;
  *reinterpret_cast<float4*>(dst) = make_float4(s[0], s[1], s[2], s[3]);
  *reinterpret_cast<float4*>(dst + 4) = make_float4(s[4], s[5], s[6], s[7]);
}

static int bwd_cta_capacity() {
  static std::atomic<int> cached{0};
  int c = cached.load(std::memory_order_relaxed);
  if (c > 0) return c;
  int cap = 132;
  DeviceInfo di;
  if (get_device_info(&di) == BLSTM_OK && di.sm_count > 0) {
    cap = di.sm_count * 132 / 148 / 4 * 4;
    auto kern = bwd_kernel<1, __half>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448) == cudaSuccess) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(di.sm_count / 4 * 4);
      cfg.blockDim = dim3(384);
      cfg.dynamicSmemBytes = 232448;
      cudaLaunchAttribute attr;
      attr.id = cudaLaunchAttributeClusterDimension;
      attr.val.clusterDim.x = 4;
      attr.val.clusterDim.y = 1;
      attr.val.clusterDim.z = 1;
      cfg.attrs = &attr;
      cfg.numAttrs = 1;
      int mc = 0;
      if (cudaOccupancyMaxActiveClusters(&mc, kern, &cfg) == cudaSuccess && mc > 0) cap = mc * 4;
    }
    (void)cudaGetLastError();
  }
  cached.store(cap, std::memory_order_relaxed);
  return cap;
}

template <int TI, typename T16>
static int launch_bwd_t(const BwdPlan& pl, const CUtensorMap& tw, const CUtensorMap& tg, BwdParams& p, cudaStream_t st) {
  return launch_coresident(bwd_kernel<TI, T16>, pl.grid, pl.threads, pl.smem, 4, st, tw, tg, p);
}

}  // namespace sm100

using namespace sm100;

int sm100_plan_family(const blstm_desc& d, int phase) {
  if (small_plan(d, phase).ok) return BLSTM_FAMILY_SMALL_BATCH;
  if (resident_plan(d, phase).ok || tiles_plan(d, phase).ok || fwd_tiles_plan(d, phase).ok) return BLSTM_FAMILY_RESIDENT;
  return (phase == BLSTM_PHASE_BWD ? make_bwd_plan(d).ok : make_plan(d, phase).ok) ? BLSTM_FAMILY_BATCH_TILES : BLSTM_FAMILY_NONE;
}
int sm100_plan_turns(const blstm_desc& d, int phase) {
  const SmallPlan p = small_plan(d, phase);
  return p.ok ? p.nch : 0;
}
int sm100_plan_beside(const blstm_desc& d, int phase) {
  const SmallPlan p = small_plan(d, phase);
  return p.ok ? resident_clusters(p.nc) / p.ncl : 0;
}
bool sm100_recurrence_supported(const blstm_desc& d, int phase) { return sm100_plan_family(d, phase) != BLSTM_FAMILY_NONE; }
size_t sm100_recurrence_workspace(const blstm_desc& d, int phase) {
  const SmallPlan sp = small_plan(d, phase);
  if (sp.ok) return small_workspace(d, sp, phase);
  if (const ResPlan rp = resident_plan(d, phase); rp.ok) return rp.ws_bytes;
  if (const TilesPlan tp = tiles_plan(d, phase); tp.ok) return tp.ws_bytes;
  if (const FwdTilesPlan fp = fwd_tiles_plan(d, phase); fp.ok) return fp.ws_bytes;
  return phase == BLSTM_PHASE_BWD ? make_bwd_plan(d).ws_bytes : make_plan(d, phase).ws_bytes;
}

size_t sm100_recurrence_control(const blstm_desc& d, int phase) {
  if (small_plan(d, phase).ok) return sizeof(Control);
  if (const ResPlan rp = resident_plan(d, phase); rp.ok) return rp.off_db;
  if (const TilesPlan tp = tiles_plan(d, phase); tp.ok) return tp.off_db;
  if (const FwdTilesPlan fp = fwd_tiles_plan(d, phase); fp.ok) return fp.ws_bytes;
  return phase == BLSTM_PHASE_BWD ? make_bwd_plan(d).off_db : make_plan(d, phase).ws_bytes;
}

int sm100_plan_detail(const blstm_desc& d, int phase, char* buf, size_t n) {
  const SmallPlan sp = small_plan(d, phase);
  if (sp.ok) return small_plan_detail(d, sp, phase, buf, n);
  if (const ResPlan rp = resident_plan(d, phase); rp.ok) return resident_plan_detail(rp, phase, buf, n);
  if (const TilesPlan tp = tiles_plan(d, phase); tp.ok) return tiles_plan_detail(tp, buf, n);
  if (const FwdTilesPlan fp = fwd_tiles_plan(d, phase); fp.ok) return fwd_tiles_plan_detail(fp, buf, n);
  if (phase == BLSTM_PHASE_BWD) {
    const BwdPlan p = make_bwd_plan(d);
    if (!p.ok) return 0;
    return snprintf(buf, n, "sm100 bwd cluster=4 units_per_cluster=64 TI=%d grid=%d threads=%d stages=%d issuers=%d "
                    "loaders=%d rows_per_stage=%d wh=%s alias=%d smem=%zu", p.TI, p.grid, p.threads, p.stages, p.ni, p.nl,
                    p.hb / 128, p.ws ? "streamed" : "resident", p.alias, p.smem);
  }
  const RecPlan p = make_plan(d, phase);
  if (!p.ok) return 0;
  return snprintf(buf, n, "sm100 fwd UH=%d TI=%d grid=%d threads=%d stages=%d issuers=%d loaders=%d rows_per_stage=%d wh=%s smem=%zu",
                  p.UH, p.TI, p.grid, p.threads, p.stages, p.ni, p.nl, p.hb / 128, p.ws ? "streamed" : "resident", p.smem);
}

int sm100_fwd_recurrence(const blstm_desc& d, void* ifgo, const void* Wh, void* out, void* cell, void* ws,
                         size_t ws_bytes, cudaStream_t st) {
  const SmallPlan sp = small_plan(d, BLSTM_PHASE_FWD);
  if (sp.ok) return small_fwd_recurrence(d, sp, ifgo, Wh, out, cell, ws, st);
  if (const ResPlan rp = resident_plan(d, BLSTM_PHASE_FWD); rp.ok) {
    if (ws_bytes < rp.ws_bytes) return BLSTM_E_WORKSPACE;
    return resident_fwd_recurrence(d, rp, ifgo, Wh, out, cell, ws, st);
  }
  if (const FwdTilesPlan fp = fwd_tiles_plan(d, BLSTM_PHASE_FWD); fp.ok) {
    if (ws_bytes < fp.ws_bytes) return BLSTM_E_WORKSPACE;
    return fwd_tiles_recurrence(d, fp, ifgo, Wh, out, cell, ws, st);
  }
  const RecPlan pl = make_plan(d, BLSTM_PHASE_FWD);
  if (!pl.ok) return BLSTM_E_UNSUPPORTED;
  if (ws_bytes < pl.ws_bytes) return BLSTM_E_WORKSPACE;
  DeviceInfo di;
  int rc = get_device_info(&di);
  if (rc) return rc;
  if (!di.coop || pl.grid > di.sm_count) return BLSTM_E_NOT_CORESIDENT;
  const int H = d.hidden_size, B = d.batch, T = d.seq_len;
  CUtensorMap tw, th;
  {  // Wh [4H,H] as {k, unit row, gate}
    uint64_t dims[3] = {(uint64_t)H, (uint64_t)H, 4};
    uint64_t str[2] = {(uint64_t)H * 2, (uint64_t)H * H * 2};
    uint32_t box[3] = {RK, (uint32_t)pl.UH, 4};
    rc = encode_tensor_map(&tw, Wh, 3, dims, str, box);
    if (rc) return rc;
  }
  {  // out [T+1,B,H] as {k, batch row, t}: rows past B are zero-filled, never another timestep
    uint64_t dims[3] = {(uint64_t)H, (uint64_t)B, (uint64_t)(T + 1)};
    uint64_t str[2] = {(uint64_t)H * 2, (uint64_t)B * H * 2};
    uint32_t box[3] = {RK, (uint32_t)(pl.hb / 128), 1};
    rc = encode_tensor_map(&th, out, 3, dims, str, box);
    if (rc) return rc;
  }
  CUtensorMap tp;
  {
    const int NU = 4 * pl.UH / pl.epi_warps;
    if (pl.TI == 1) {
      tp = th;         // (not used)
    } else {  // ifgo [T,B,4H] as {unit, batch row, gate, t}: a box is one warp's 4 gates x 32 rows x NU units;
       // the box's inner extent equals the swizzle span (32 bytes) or is a single 16-byte piece (none)
      uint64_t dims[4] = {(uint64_t)H, (uint64_t)B, 4, (uint64_t)T};
      uint64_t str[3] = {(uint64_t)4 * H * 2, (uint64_t)H * 2, (uint64_t)B * 4 * H * 2};
      uint32_t box[4] = {(uint32_t)NU, 32, 4, 1};
      rc = encode_tensor_map(&tp, ifgo, 4, dims, str, box, 2, NU == 16 ? 32 : 0);
      if (rc) return rc;
    }
  }
  FwdParams p;
  p.npb = pl.npb;
  p.ep_bytes = (int)pl.ep_bytes;
  p.T = T; p.B = B; p.H = H;
  p.nbt = pl.nbt; p.nh = pl.nh; p.nb_par = pl.nb_par; p.ntl = pl.ntl;
  p.stages = pl.stages;
  p.ni = pl.ni;
  p.nl = pl.nl;
  p.ws = pl.ws;
  p.hb = pl.hb;
  p.stage_bytes = (int)pl.stage_bytes;
  p.fmt = d.dtype == BLSTM_BF16 ? 1 : 0;
  p.no_arrive = (d.flags & BLSTM_FLAG_TEST_NO_ARRIVE) ? 1 : 0;
  p.inference = (d.flags & BLSTM_FLAG_INFERENCE) ? 1 : 0;
  p.flag_target = pl.nh;            // one arrival per CTA and item
  p.limit_ns = d.wait_limit_us > 0 ? (unsigned long long)d.wait_limit_us * 1000ull : kDefaultWaitNs;
  p.ctl = reinterpret_cast<Control*>(ws);
  p.flags = reinterpret_cast<int*>(static_cast<char*>(ws) + pl.off_flags);
  p.ifgo = ifgo; p.out = out; p.cell = cell;
  const bool bf = d.dtype == BLSTM_BF16;
#define BLSTM_FWD_CASE(U, I)                                                                         \
  if (pl.UH == U && pl.TI == I)                                                                      \
    return bf ? launch_fwd_t<U, I, __nv_bfloat16>(pl, tw, th, tp, p, st)                             \
              : launch_fwd_t<U, I, __half>(pl, tw, th, tp, p, st);
  BLSTM_FWD_CASE(16, 1)
  BLSTM_FWD_CASE(16, 2)
  BLSTM_FWD_CASE(16, 4)
  BLSTM_FWD_CASE(32, 2)
  BLSTM_FWD_CASE(32, 4)
#undef BLSTM_FWD_CASE
  return BLSTM_E_UNSUPPORTED;
}

int sm100_bwd_recurrence(const blstm_desc& d, const void* dout, const void* dh_n, const void* dc_n,
                         const void* ifgo, const void* cell, const void* Wh, void* d_ifgo, void* dh0, void* dc0,
                         float* db, void* ws, size_t ws_bytes, cudaStream_t st) {
  const SmallPlan sp = small_plan(d, BLSTM_PHASE_BWD);
  if (sp.ok) return small_bwd_recurrence(d, sp, dout, dh_n, dc_n, ifgo, cell, Wh, d_ifgo, dh0, dc0, db, ws, st);
  if (const ResPlan rp = resident_plan(d, BLSTM_PHASE_BWD); rp.ok) {
    if (ws_bytes < rp.ws_bytes) return BLSTM_E_WORKSPACE;
    return resident_bwd_recurrence(d, rp, dout, dh_n, dc_n, ifgo, cell, Wh, d_ifgo, dh0, dc0, db, ws, st);
  }
  if (const TilesPlan tp = tiles_plan(d, BLSTM_PHASE_BWD); tp.ok) {
    if (ws_bytes < tp.ws_bytes) return BLSTM_E_WORKSPACE;
    return tiles_bwd_recurrence(d, tp, dout, dh_n, dc_n, ifgo, cell, Wh, d_ifgo, dh0, dc0, db, ws, st);
  }
  const BwdPlan pl = make_bwd_plan(d);
  if (!pl.ok) return BLSTM_E_UNSUPPORTED;
  if (ws_bytes < pl.ws_bytes) return BLSTM_E_WORKSPACE;
  DeviceInfo di;
  int rc = get_device_info(&di);
  if (rc) return rc;
  if (!di.coop || pl.grid > di.sm_count) return BLSTM_E_NOT_CORESIDENT;
  const int H = d.hidden_size, B = d.batch, T = d.seq_len;
  CUtensorMap tw, tg;
  {  // Wh [4H,H] row-major: rows are K (gate-major), columns the output units (N-major operand)
    uint64_t dims[2] = {(uint64_t)H, (uint64_t)4 * H};
    uint64_t str[1] = {(uint64_t)H * 2};
    uint32_t box[2] = {64, 64};
    rc = encode_tensor_map(&tw, Wh, 2, dims, str, box);
    if (rc) return rc;
  }
  {  // d_ifgo [T,B,4H] as {k, batch row, t}
    uint64_t dims[3] = {(uint64_t)4 * H, (uint64_t)B, (uint64_t)T};
    uint64_t str[2] = {(uint64_t)4 * H * 2, (uint64_t)B * 4 * H * 2};
    uint32_t box[3] = {RK, (uint32_t)(pl.hb / 128), 1};
    rc = encode_tensor_map(&tg, d_ifgo, 3, dims, str, box);
    if (rc) return rc;
  }
  BwdParams p;
  p.T = T; p.B = B; p.H = H;
  p.nbt = pl.nbt; p.nug = pl.nug; p.nb_par = pl.nb_par; p.ntl = pl.ntl; p.stages = pl.stages; p.ni = pl.ni;
  p.nl = pl.nl;
  p.ws = pl.ws; p.hb = pl.hb; p.stage_bytes = (int)pl.stage_bytes;
  p.alias = pl.alias;
  p.fmt = d.dtype == BLSTM_BF16 ? 1 : 0;
  p.no_arrive = (d.flags & BLSTM_FLAG_TEST_NO_ARRIVE) ? 1 : 0;
  p.flag_target = H / 16;           // one arrival per CTA and item
  p.limit_ns = d.wait_limit_us > 0 ? (unsigned long long)d.wait_limit_us * 1000ull : kDefaultWaitNs;
  p.ctl = reinterpret_cast<Control*>(ws);
  p.flags = reinterpret_cast<int*>(static_cast<char*>(ws) + pl.off_flags);
  p.dout = dout; p.dh_n = dh_n; p.dc_n = dc_n; p.ifgo = ifgo; p.cell = cell;
  p.d_ifgo = d_ifgo; p.dh0 = dh0; p.dc0 = dc0;
  p.db_part = db ? reinterpret_cast<float*>(static_cast<char*>(ws) + pl.off_db) : nullptr;
  const bool bf = d.dtype == BLSTM_BF16;
  if (pl.TI == 1)      rc = bf ? launch_bwd_t<1, __nv_bfloat16>(pl, tw, tg, p, st) : launch_bwd_t<1, __half>(pl, tw, tg, p, st);
  else if (pl.TI == 2) rc = bf ? launch_bwd_t<2, __nv_bfloat16>(pl, tw, tg, p, st) : launch_bwd_t<2, __half>(pl, tw, tg, p, st);
  else                 rc = bf ? launch_bwd_t<4, __nv_bfloat16>(pl, tw, tg, p, st) : launch_bwd_t<4, __half>(pl, tw, tg, p, st);
  if (rc) return rc;
  if (db) return reduce_db(p.db_part, pl.nb_par * 32, 4 * H, db, st);
  return BLSTM_OK;
}

int sm100_bias_grad(const blstm_desc& d, const void* d_ifgo, float* db, void* ws, size_t ws_bytes, cudaStream_t st) {
  // as many partial rows as the backward recurrence's workspace has room for, behind the control block
  const int rows = d.seq_len * d.batch, cols = 4 * d.hidden_size;
  const int parts = (int)std::min<size_t>(DB_PARTS, (ws_bytes - sizeof(Control)) / (cols * sizeof(float)));
  if (parts < 1) return BLSTM_E_WORKSPACE;
  float* part = reinterpret_cast<float*>(static_cast<char*>(ws) + sizeof(Control));
  dim3 grid(cdiv(cols, 1024), parts);
  if (d.dtype == BLSTM_BF16) colsum_kernel<__nv_bfloat16><<<grid, 128, 0, st>>>((const __nv_bfloat16*)d_ifgo, rows, cols, part);
  else                       colsum_kernel<__half><<<grid, 128, 0, st>>>((const __half*)d_ifgo, rows, cols, part);
  BLSTM_CUDA_OK(cudaGetLastError());
  count_launch();
  return reduce_db(part, parts, cols, db, st);
}

}  // namespace blstm
