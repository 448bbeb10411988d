// fp32 recurrences inside one cluster (FFMA: the tolerance of 1e-5 forbids TF32).  Small and mid-size hidden sizes, where
// the grid-wide kernels of generic.cu hand every step over through L2 counters (9 us a step forward, 25 us backward at
// H = 128) and read the weights from shared or global memory for every product.
// (Replaces persistent_fwd_kernel and lstm_persistent_seq_bwd, fastlstm/kernels.py:414-663 and :1201-1409, for fp32.)
//
// As in sm100_small.cu: a cluster of NC CTAs owns a few batch rows and all hidden units, the weights stay in registers
// for the whole sequence, a step's results reach the peers by st.async on their mbarriers, nothing crosses clusters.
// Rows are worked in chunks of R (1, 2, 4 or 8) with barriers of their own.  Two warps (backward) or four (forward)
// that do nothing else move pre-activations, states and gradients between global memory and a ring of item slots
// (H is any number here, so no TMA); the slot's results go out over the same places its inputs came in.
// Measured (B200, us per step, grid-wide kernels before): forward H = 128, B = 16: 9.1 -> 0.95; H = 257, B = 44: 16.5 -> 1.9;
// H = 64, B = 1024: 7.3 -> 4.1; backward 25.7 -> 1.6, 48.9 -> 3.2, 15.8 -> 9.8.
#include <algorithm>

#include "cluster_util.cuh"
#include "generic.cuh"
#include "f32_cluster.cuh"

namespace blstm {
namespace sm100 {

struct F32Params {
  int T, B, H;
  int nc, rows, nch;        // CTAs per cluster, batch rows per cluster, chunks per cluster
  int no_arrive, inference;
  unsigned long long limit_ns;
  Control* ctl;
  const float* Wh;
  float* ifgo;              // forward: in/out; backward: in
  float* out;               // forward
  float* cell;              // forward: out; backward: in
  const float* dout;
  const float* dh_n;        // or null
  const float* dc_n;        // or null
  float* d_ifgo;
  float* dh0;
  float* dc0;
  float* db_part;           // [clusters][4H] or null
};

constexpr int F_SLOTS = 4;

// Adds up `v` of the 2^L lanes that differ in lane bits MASK, MASK/2, ...; halves the rows at every level while there
// are two or more, so that a lane ends with the rows its bits select.
template <int N, int R, int MASK, int LAST>
__device__ __forceinline__ void reduce_rows(float (&v)[N][R], int lane) {
  if constexpr (MASK >= LAST) {
    if constexpr (R >= 2) {
      float k[N][R / 2];
      const bool up = (lane & MASK) != 0;
#pragma unroll
      for (int n = 0; n < N; ++n)
#pragma unroll
        for (int r = 0; r < R / 2; ++r) {
          const float mine = up ? v[n][R / 2 + r] : v[n][r], other = up ? v[n][r] : v[n][R / 2 + r];
          k[n][r] = mine + __shfl_xor_sync(0xffffffffu, other, MASK);
        }
      reduce_rows<N, R / 2, MASK / 2, LAST>(k, lane);
#pragma unroll
      for (int n = 0; n < N; ++n)
#pragma unroll
        for (int r = 0; r < R / 2; ++r) v[n][r] = k[n][r];
    } else {
#pragma unroll
      for (int n = 0; n < N; ++n) v[n][0] += __shfl_xor_sync(0xffffffffu, v[n][0], MASK);
      reduce_rows<N, R, MASK / 2, LAST>(v, lane);
    }
  }
}

// =====================================================================================
// Forward.  Warp = 4 units x 8 K slices: lane 8u+s multiplies k = 32j + 4s .. 4s+3 (j < KJ) of unit u's four gate rows -
// 16 KJ weights in registers - with the R rows of h, which a warp reads as one 128-byte broadcast per row and j; the
// slices are added up by shuffles that leave lane 8u+s with row s.  A CTA owns 32 units.
//   warps 0-7 computing, warps 8-11 global traffic.  Bound by FFMA (KJ R 16 per step and warp, two warps a scheduler)
//   and the exchange.
// =====================================================================================
template <int KJ, int R, bool CL>
__global__ void __launch_bounds__(384, 1) f32_fwd_kernel(const F32Params p) {
  constexpr int U = 32, S = F_SLOTS, P = U + 4;                 // P: slot row pitch (8 rows x 4 units: 32 banks)
  constexpr int HP = 32 * KJ;                                   // h row pitch
  constexpr int SLOT = 6 * R * P;                               // [i f g o h c][row][P]
  extern __shared__ __align__(16) float sm[];
  const int H = p.H, T = p.T, B = p.B;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = CL ? (int)cluster_ctarank() : 0;
  const int cl = CL ? blockIdx.x / p.nc : blockIdx.x;
  const int row0 = cl * p.rows, rows = min(p.rows, B - row0);
  const int nch = rows > 0 ? (rows + R - 1) / R : 0;
  const int cta0 = rank * U;

  float* slots = sm;                                            // [S][SLOT]
  float* h_s = slots + S * SLOT;                                // [chunk][parity][R][HP]
  float* c_s = h_s + p.nch * 2 * R * HP;                        // [chunk][8 warps][32 lanes]
  uint64_t* hbar = reinterpret_cast<uint64_t*>(c_s + p.nch * 256);   // [chunk][parity]
  uint64_t* full = hbar + 2 * SB_MAX_CHUNKS;                    // [S]
  uint64_t* staged = full + S;                                  // [S]
  volatile int* dead = reinterpret_cast<volatile int*>(staged + S);

  if (threadIdx.x == 0) {
    *dead = 0;
    for (int i = 0; i < 2 * nch; ++i) mbar_init(&hbar[i], CL ? 1 : 8);
    for (int i = 0; i < S; ++i) { mbar_init(&full[i], 4); mbar_init(&staged[i], 8); }
    fence_mbar_init();
    if (CL)
      for (int i = 0; i < 2 * nch; ++i) mbar_expect_tx(&hbar[i], p.nc * U * 4 * min(R, rows - (i >> 1) * R));
  }
  for (int i = threadIdx.x; i < p.nch * 2 * R * HP; i += blockDim.x) {
    const int k = i % HP, r = i / HP, row = (r / (2 * R)) * R + r % R;
    h_s[i] = ((r / R) % 2 == 0 && row < rows && k < H) ? p.out[(size_t)(row0 + row) * H + k] : 0.f;
  }
  __syncthreads();
  if (CL) cluster_sync_all();

  if (warp >= 8) {
    // ---------------------------------------------------------------- global traffic: items in the order (t, chunk)
    regs_dec<40>();
    constexpr int NL = (4 * R * U + 127) / 128;
    const int tid = threadIdx.x - 256, n = nch * T;
    const int x = cta0 + lane;                                  // (32 units: a warp instruction moves one row of one part)
    auto fetch = [&](int k, float (&v)[NL]) {
      const int t = k / nch, ch = k - t * nch;
#pragma unroll
      for (int i = 0; i < NL; ++i) {
        const int e = (tid >> 5) + 4 * i, g = e / R, r = ch * R + e % R;
        v[i] = (e < 4 * R && k < n && r < rows && x < H) ? p.ifgo[(((size_t)t * B + row0 + r) * 4 + g) * H + x] : 0.f;
      }
    };
    auto put = [&](int k, const float (&v)[NL]) {
      if (k >= n) return;
      float* sl = slots + (k % S) * SLOT;
#pragma unroll
      for (int i = 0; i < NL; ++i) {
        const int e = (tid >> 5) + 4 * i;
        if (e < 4 * R) sl[e * P + lane] = v[i];
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&full[k % S]);
    };
    float v[NL];
    for (int k = 0; k < S; ++k) { fetch(k, v); put(k, v); }
    for (int k = 0; k < n; ++k) {
      fetch(k + S, v);
      const int t = k / nch, ch = k - t * nch;
      if (!wait_inline(&staged[k % S], (uint32_t)(k / S) & 1u, dead, p.ctl, p.limit_ns, t, cl)) break;
      const float* sl = slots + (k % S) * SLOT;
      for (int e = tid >> 5; e < 6 * R; e += 4) {
        const int g = e / R, r = ch * R + e % R;
        if (r >= rows || x >= H) continue;
        const float o = sl[e * P + lane];
        const size_t o1 = ((size_t)(t + 1) * B + row0 + r) * H + x;
        if (g == 4) p.out[o1] = o;
        else if (g == 5) { if (!p.inference || t == T - 1) p.cell[o1] = o; }
        else if (!p.inference) p.ifgo[(((size_t)t * B + row0 + r) * 4 + g) * H + x] = o;
      }
      put(k + S, v);
    }
  } else {
    // ---------------------------------------------------------------- computing
    regs_inc<232>();
    const int u = lane >> 3, s = lane & 7;
    const int unit = cta0 + warp * 4 + u;
    float w[KJ][4][4];                                          // [j][k][gate]
#pragma unroll
    for (int j = 0; j < KJ; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          const int k = 32 * j + 4 * s + i;
          w[j][i][g] = (unit < H && k < H) ? p.Wh[((size_t)g * H + unit) * H + k] : 0.f;
        }
    const int row = R == 8 ? s : R == 4 ? s >> 1 : R == 2 ? s >> 2 : 0;      // the row the reduction leaves here
    const bool own = R == 8 || (R == 4 && !(s & 1)) || (R == 2 && !(s & 3)) || s == 0;   // one lane of those that have it
    for (int ch = 0; ch < nch; ++ch)
      c_s[ch * 256 + threadIdx.x] = (unit < H && ch * R + row < rows) ? p.cell[(size_t)(row0 + ch * R + row) * H + unit] : 0.f;
    // this lane sends row `srow`'s four units of the warp to CTAs u, u+4, ...
    const int srow = s;
    uint32_t peer[4];
    const uint32_t sbase = smem_u32(sm), hoff = smem_u32(h_s) - sbase, boff = smem_u32(hbar) - sbase;
#pragma unroll
    for (int i = 0; i < 4; ++i) peer[i] = CL ? mapa_shared(sbase, min(u + 4 * i, p.nc - 1)) : sbase;
    const int srclane = R == 8 ? srow : R == 4 ? 2 * srow : R == 2 ? 4 * srow : 0;
    for (int t = 0, k = 0; t < T; ++t) {
      bool ok = true;
      for (int ch = 0; ch < nch; ++ch, ++k) {
        const int par = t & 1;
        float* sl = slots + (k % S) * SLOT;
        if (!wait_inline(&full[k % S], (uint32_t)(k / S) & 1u, dead, p.ctl, p.limit_ns, t, cl)) { ok = false; break; }
        float pre[4];
#pragma unroll
        for (int g = 0; g < 4; ++g) pre[g] = sl[(g * R + row) * P + warp * 4 + u];
        if (t > 0) {
          uint64_t* bar = &hbar[2 * ch + par];
          if (!wait_inline(bar, (uint32_t)((t - 1) >> 1) & 1u, dead, p.ctl, p.limit_ns, t, cl)) { ok = false; break; }
          if (CL && threadIdx.x == 0 && t + 2 < T) mbar_expect_tx(bar, p.nc * U * 4 * min(R, rows - ch * R));
        }
        float acc[4][R] = {};
        const float* hb = h_s + (size_t)(ch * 2 + par) * R * HP + 4 * s;
#pragma unroll
        for (int j = 0; j < KJ; ++j)
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const float4 h4 = *reinterpret_cast<const float4*>(hb + r * HP + 32 * j);
            const float hh[4] = {h4.x, h4.y, h4.z, h4.w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
              for (int g = 0; g < 4; ++g) acc[g][r] = fmaf(hh[i], w[j][i][g], acc[g][r]);
          }
        reduce_rows<4, R, 4, 1>(acc, lane);
        float a[4];
#pragma unroll
        for (int g = 0; g < 4; ++g) a[g] = acc[g][0] + pre[g];
        const float c = sigmoid_acc(a[1]) * c_s[ch * 256 + threadIdx.x] + sigmoid_acc(a[0]) * tanh_acc(a[2]);
        const float h = sigmoid_acc(a[3]) * tanh_acc(c);
        float4 hv;
        hv.x = __shfl_sync(0xffffffffu, h, srclane);
        hv.y = __shfl_sync(0xffffffffu, h, 8 + srclane);
        hv.z = __shfl_sync(0xffffffffu, h, 16 + srclane);
        hv.w = __shfl_sync(0xffffffffu, h, 24 + srclane);
        if (srow < R && ch * R + srow < rows && t + 1 < T && !p.no_arrive) {
          const uint32_t ho = hoff + (uint32_t)(((ch * 2 + (par ^ 1)) * R + srow) * HP + cta0 + warp * 4) * 4;
          const uint4 hw = make_uint4(__float_as_uint(hv.x), __float_as_uint(hv.y), __float_as_uint(hv.z), __float_as_uint(hv.w));
          if (CL) {
            const uint32_t bo = boff + (uint32_t)(2 * ch + (par ^ 1)) * 8;
#pragma unroll
            for (int i = 0; i < 4; ++i)
              if (u + 4 * i < p.nc) st_async16(peer[i] + ho, hw, peer[i] + bo);
          } else if (u == 0) {
            st_shared16(sbase + ho, hw);
          }
        }
        if (!CL) {
          __syncwarp();
          if (lane == 0) mbar_arrive(&hbar[2 * ch + (par ^ 1)]);
        }
        c_s[ch * 256 + threadIdx.x] = c;
        if (own) {
          float* o = sl + row * P + warp * 4 + u;
#pragma unroll
          for (int g = 0; g < 4; ++g) o[g * R * P] = a[g];
          o[4 * R * P] = h;
          o[5 * R * P] = c;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&staged[k % S]);
      }
      if (!ok) break;
    }
  }
  __syncthreads();
  if (CL) cluster_sync_all();
}

// =====================================================================================
// Backward.  The product dh[t-1] = d_ifgo[t] x Wh is split by K as in the 16-bit kernel: a CTA multiplies the d_ifgo of
// its own U units (U rows of each gate) into partial sums for all H units and sends them to their owners, who add the
// NC sources up in a fixed order.  Warp = 8 quads of output units x 4 gates: lane 4q+g multiplies gate g's U rows of
// its quad - 4 U weights in registers - and the gates are added up by shuffles that leave every lane some rows of the
// quad: 16 bytes to send per row.  The same warps do the gate maths of the CTA's units before the product.
// PW: product warps (32 output units each); two more warps move the global traffic.
// =====================================================================================
template <int U, int PW, int R, bool CL>
__global__ void __launch_bounds__(384, 1) f32_bwd_kernel(const F32Params p) {
  constexpr int S = F_SLOTS;
  constexpr int SLOT = 6 * R * U;                               // [i f g o c dout][row][U]
  constexpr int DG = U * R + 4;                                 // one gate of the product's operand (+4: the gates' banks)
  constexpr int NT = 32 * PW;
  constexpr int NI = (U * R + NT - 1) / NT;                     // gate-maths items per thread
  extern __shared__ __align__(16) float sm[];
  const int H = p.H, T = p.T, B = p.B;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = CL ? (int)cluster_ctarank() : 0;
  const int cl = CL ? blockIdx.x / p.nc : blockIdx.x;
  const int row0 = cl * p.rows, rows = min(p.rows, B - row0);
  const int nch = rows > 0 ? (rows + R - 1) / R : 0;
  const int cta0 = rank * U;

  float* slots = sm;                                            // [S][SLOT]
  float* dg_s = slots + S * SLOT;                               // [2][4][DG]: [gate][unit][row]
  float* x_s = dg_s + 2 * 4 * DG;                               // [chunk][parity][source][R][U]
  float* st_s = x_s + (size_t)p.nch * 2 * p.nc * R * U;         // [chunk][dc | c][NI][NT]
  uint64_t* xbar = reinterpret_cast<uint64_t*>(st_s + (size_t)p.nch * 2 * NI * NT);   // [chunk][parity]
  uint64_t* full = xbar + 2 * SB_MAX_CHUNKS;
  uint64_t* staged = full + S;
  uint64_t* dfull = staged + S;                                 // [2] d_ifgo operand written
  volatile int* dead = reinterpret_cast<volatile int*>(dfull + 2);
  const int quads = max(0, min(U, H - cta0) + 3) / 4;           // unit quads of this CTA that exist
  auto expect = [&](int ch) { return p.nc * quads * 16 * min(R, rows - ch * R); };

  if (threadIdx.x == 0) {
    *dead = 0;
    for (int i = 0; i < 2 * nch; ++i) mbar_init(&xbar[i], CL ? 1 : PW);
    for (int i = 0; i < S; ++i) { mbar_init(&full[i], 2); mbar_init(&staged[i], PW); }
    for (int i = 0; i < 2; ++i) mbar_init(&dfull[i], PW);
    fence_mbar_init();
    if (CL)
      for (int i = 0; i < 2 * nch; ++i) mbar_expect_tx(&xbar[i], expect(i >> 1));
  }
  for (int i = threadIdx.x; i < 2 * 4 * DG + p.nch * 2 * p.nc * R * U; i += blockDim.x) dg_s[i] = 0.f;
  __syncthreads();
  if (CL) cluster_sync_all();

  if (warp >= 10) {
    // ---------------------------------------------------------------- global traffic: items in the order (step, chunk)
    constexpr int NL = (6 * R * U + 63) / 64;
    const int tid = threadIdx.x - 320, n = nch * T;
    auto fetch = [&](int k, float (&v)[NL]) {
      const int st = k / nch, ch = k - st * nch, t = T - 1 - st;
#pragma unroll
      for (int i = 0; i < NL; ++i) {
        const int e = tid + 64 * i, x = cta0 + e % U, g = e / (U * R), r = ch * R + (e / U) % R;
        float o = 0.f;
        if (e < 6 * R * U && k < n && r < rows && x < H) {
          const size_t m = (size_t)t * B + row0 + r;
          o = g == 4 ? p.cell[m * H + x] : g == 5 ? p.dout[m * H + x] : p.ifgo[(m * 4 + g) * H + x];
        }
        v[i] = o;
      }
    };
    auto put = [&](int k, const float (&v)[NL]) {
      if (k >= n) return;
      float* sl = slots + (k % S) * SLOT;
#pragma unroll
      for (int i = 0; i < NL; ++i)
        if (tid + 64 * i < 6 * R * U) sl[tid + 64 * i] = v[i];
      __syncwarp();
      if (lane == 0) mbar_arrive(&full[k % S]);
    };
    float v[NL];
    for (int k = 0; k < S; ++k) { fetch(k, v); put(k, v); }
    for (int k = 0; k < n; ++k) {
      fetch(k + S, v);
      const int st = k / nch, ch = k - st * nch, t = T - 1 - st;
      if (!wait_inline(&staged[k % S], (uint32_t)(k / S) & 1u, dead, p.ctl, p.limit_ns, t, cl)) break;
      const float* sl = slots + (k % S) * SLOT;
      for (int e = tid; e < 4 * R * U; e += 64) {
        const int x = cta0 + e % U, g = e / (U * R), r = ch * R + (e / U) % R;
        if (r < rows && x < H) p.d_ifgo[(((size_t)t * B + row0 + r) * 4 + g) * H + x] = sl[e];
      }
      put(k + S, v);
    }
  } else if (warp < PW) {
    // ---------------------------------------------------------------- gate maths and product
    const int g = lane & 3, quad = warp * 8 + (lane >> 2);
    const int unit0 = quad * 4;                                 // output units unit0 .. unit0+3
    float w[U][4];
#pragma unroll
    for (int k = 0; k < U; ++k)
#pragma unroll
      for (int i = 0; i < 4; ++i)
        w[k][i] = (cta0 + k < H && unit0 + i < H) ? p.Wh[((size_t)g * H + cta0 + k) * H + unit0 + i] : 0.f;
    const uint32_t sbase = smem_u32(sm), xoff = smem_u32(x_s) - sbase, boff = smem_u32(xbar) - sbase;
    const int owner = unit0 / U;
    const bool there = unit0 < H && !p.no_arrive;
    const uint32_t pbase = CL ? mapa_shared(sbase, min(owner, p.nc - 1)) : sbase;
    const uint32_t dst = pbase + xoff + (uint32_t)(rank * R * U + unit0 - owner * U) * 4;
    for (int ch = 0; ch < nch; ++ch)
#pragma unroll
      for (int i = 0; i < NI; ++i) {
        const int e = threadIdx.x + i * NT, x = cta0 + e % U, r = ch * R + e / U;
        const bool in = e < U * R && r < rows && x < H;
        float* s2 = st_s + (size_t)(ch * 2 * NI + i) * NT + threadIdx.x;
        s2[0] = (in && p.dc_n) ? p.dc_n[(size_t)(row0 + r) * H + x] : 0.f;
        s2[NI * NT] = in ? p.cell[((size_t)T * B + row0 + r) * H + x] : 0.f;
      }
    auto gather = [&](int st, int ch, int e) {
      const float* src = x_s + ((size_t)(ch * 2 + ((st - 1) & 1)) * p.nc * R * U) + e;
      float d = 0.f;
#pragma unroll 4
      for (int s = 0; s < p.nc; ++s) d += src[(size_t)s * R * U];
      return d;
    };
    float db[NI][4] = {};
    bool ok = true;
    int k = 0;
    for (int st = 0; st < T && ok; ++st) {
      for (int ch = 0; ch < nch; ++ch, ++k) {
        const int par = k & 1;
        float* sl = slots + (k % S) * SLOT;
        if (!wait_inline(&full[k % S], (uint32_t)(k / S) & 1u, dead, p.ctl, p.limit_ns, T - 1 - st, cl)) { ok = false; break; }
        // what does not depend on dh
        float so[NI], tc[NI], fI[NI], fF[NI], fG[NI], sf[NI], c0[NI], dd[NI];
#pragma unroll
        for (int i = 0; i < NI; ++i) {
          const int e = threadIdx.x + i * NT;
          if (e >= U * R) continue;
          const float si = sigmoid_acc(sl[e]), tg = tanh_acc(sl[2 * R * U + e]);
          sf[i] = sigmoid_acc(sl[R * U + e]);
          so[i] = sigmoid_acc(sl[3 * R * U + e]);
          c0[i] = sl[4 * R * U + e];
          dd[i] = sl[5 * R * U + e];
          tc[i] = tanh_acc(st_s[(size_t)(ch * 2 * NI + NI + i) * NT + threadIdx.x]);
          fI[i] = tg * si * (1.f - si);
          fF[i] = c0[i] * sf[i] * (1.f - sf[i]);
          fG[i] = si * (1.f - tg * tg);
        }
        if (st > 0) {
          uint64_t* bar = &xbar[2 * ch + ((st - 1) & 1)];
          if (!wait_inline(bar, (uint32_t)((st - 1) >> 1) & 1u, dead, p.ctl, p.limit_ns, T - 1 - st, cl)) { ok = false; break; }
          if (CL && threadIdx.x == 0 && st + 1 < T) mbar_expect_tx(bar, expect(ch));
        }
#pragma unroll
        for (int i = 0; i < NI; ++i) {
          const int e = threadIdx.x + i * NT;
          if (e >= U * R) continue;
          const int r = ch * R + e / U, x = cta0 + e % U;
          float dh = 0.f;
          if (st > 0) dh = gather(st, ch, e);
          else if (p.dh_n && r < rows && x < H) dh = p.dh_n[(size_t)(row0 + r) * H + x];
          dh += dd[i];
          float* s2 = st_s + (size_t)(ch * 2 * NI + i) * NT + threadIdx.x;
          const float dc = fmaf(dh * so[i], 1.f - tc[i] * tc[i], s2[0]);
          const float q[4] = {dc * fI[i], dc * fF[i], dc * fG[i], dh * tc[i] * so[i] * (1.f - so[i])};
          s2[0] = dc * sf[i];
          s2[NI * NT] = c0[i];
          const bool in = r < rows && x < H;
#pragma unroll
          for (int gg = 0; gg < 4; ++gg) {
            dg_s[(par * 4 + gg) * DG + (e % U) * R + e / U] = q[gg];
            sl[gg * R * U + e] = q[gg];
            if (in) db[i][gg] += q[gg];
          }
        }
        __syncwarp();
        if (lane == 0) { mbar_arrive(&dfull[par]); mbar_arrive(&staged[k % S]); }
        // every warp's d_ifgo of this item (buffer `par` is written again two items on, when all warps have read this one:
        // they have passed the next item's barrier by then)
        if (!wait_inline(&dfull[par], (uint32_t)(k >> 1) & 1u, dead, p.ctl, p.limit_ns, T - 1 - st, cl)) { ok = false; break; }
        float acc[4][R] = {};
        const float* da = dg_s + (par * 4 + g) * DG;
#pragma unroll
        for (int kk = 0; kk < U; ++kk) {
          float d[R];
          if constexpr (R >= 4) {
#pragma unroll
            for (int r4 = 0; r4 < R / 4; ++r4) {
              const float4 f = *reinterpret_cast<const float4*>(da + kk * R + 4 * r4);
              d[4 * r4] = f.x; d[4 * r4 + 1] = f.y; d[4 * r4 + 2] = f.z; d[4 * r4 + 3] = f.w;
            }
          } else if constexpr (R == 2) {
            const float2 f = *reinterpret_cast<const float2*>(da + kk * 2);
            d[0] = f.x; d[1] = f.y;
          } else {
            d[0] = da[kk];
          }
#pragma unroll
          for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int r = 0; r < R; ++r) acc[i][r] = fmaf(d[r], w[kk][i], acc[i][r]);
        }
        reduce_rows<4, R, 2, 1>(acc, lane);
        // this lane's rows: R = 8: two (2g', 2g'+1), 4: one, 2: one (lanes with bit 0 clear send), 1: one (lane g = 0 sends)
        constexpr int NR = R == 8 ? 2 : 1;
        const int r0 = R == 8 ? ((g >> 1) * 4 + (g & 1) * 2) : R == 4 ? g : R == 2 ? g >> 1 : 0;
        const bool sends = there && (R >= 4 || (R == 2 ? !(g & 1) : g == 0));
        const uint32_t buf = (uint32_t)((ch * 2 + (st & 1)) * p.nc) * R * U * 4, bo = boff + (uint32_t)(2 * ch + (st & 1)) * 8;
#pragma unroll
        for (int i = 0; i < NR; ++i)
          if (sends && ch * R + r0 + i < rows) {
            const uint4 v = make_uint4(__float_as_uint(acc[0][i]), __float_as_uint(acc[1][i]), __float_as_uint(acc[2][i]), __float_as_uint(acc[3][i]));
            const uint32_t a = dst + buf + (uint32_t)(r0 + i) * U * 4;
            if (CL) st_async16(a, v, pbase + bo); else st_shared16(a, v);
          }
        if (!CL) {
          __syncwarp();
          if (lane == 0) mbar_arrive(&xbar[2 * ch + (st & 1)]);
        }
      }
    }
    // ---- gradients of the initial states, bias gradient
    for (int ch = 0; ch < nch && ok; ++ch) {
      if (!wait_inline(&xbar[2 * ch + ((T - 1) & 1)], (uint32_t)((T - 1) >> 1) & 1u, dead, p.ctl, p.limit_ns, -1, cl)) break;
#pragma unroll
      for (int i = 0; i < NI; ++i) {
        const int e = threadIdx.x + i * NT, r = ch * R + e / U, x = cta0 + e % U;
        if (e >= U * R || r >= rows || x >= H) continue;
        p.dh0[(size_t)(row0 + r) * H + x] = gather(T, ch, e);
        p.dc0[(size_t)(row0 + r) * H + x] = st_s[(size_t)(ch * 2 * NI + i) * NT + threadIdx.x];
      }
    }
    if (p.db_part && nch > 0) {
      // rows of a unit lie in different threads: add them up in shared memory (the operand buffers are free: every
      // warp is past its last product once all have arrived here)
      asm volatile("bar.sync 1, %0;" ::"n"(NT) : "memory");
#pragma unroll
      for (int i = 0; i < NI; ++i) {
        const int e = threadIdx.x + i * NT;
        if (e < U * R)
#pragma unroll
          for (int gg = 0; gg < 4; ++gg) dg_s[gg * DG + (e % U) * R + e / U] = db[i][gg];
      }
      asm volatile("bar.sync 1, %0;" ::"n"(NT) : "memory");
      for (int i = threadIdx.x; i < 4 * U; i += NT) {
        const int gg = i / U, x = i % U;
        float v = 0.f;
#pragma unroll
        for (int r = 0; r < R; ++r) v += dg_s[gg * DG + x * R + r];
        if (cta0 + x < H) p.db_part[(size_t)cl * 4 * H + (size_t)gg * H + cta0 + x] = v;
      }
    }
  }
  __syncthreads();
  if (CL) cluster_sync_all();
}

// ---------------------------------------------------------------- plans and launches
// Units per CTA and K groups by the hidden size alone: a row's results do not depend on the batch.
F32Plan f32_plan(const blstm_desc& d, int phase) {
  F32Plan p{};
  if (d.dtype != BLSTM_F32 || (d.flags & (BLSTM_FLAG_FORCE_GENERIC | BLSTM_FLAG_NO_CLUSTER)) || d.hidden_size > 320) return p;
  const int H = d.hidden_size, B = d.batch;
  // 32 units per CTA, except backward past H = 256: ten product warps leave 168 registers a thread, room for 4 x 24 weights
  p.U = (phase == BLSTM_PHASE_BWD && H > 256) ? 24 : 32;
  p.nc = cdiv(H, p.U);
  if (p.nc == 1 && (d.flags & BLSTM_FLAG_TEST_NO_ARRIVE)) return p;      // (no wait that could run out)
  const int cap = d.flags & BLSTM_FLAG_HALF_DEVICE ? (resident_clusters(p.nc) + 1) / 2 : resident_clusters(p.nc);   // (a hint: clusters are independent)
  const int per = cdiv(B, std::min(cap, B));
  p.R = per >= 5 ? 8 : per >= 3 ? 4 : per;
  p.nch = cdiv(per, p.R);
  p.rows = p.R * p.nch;
  p.ncl = cdiv(B, p.rows);
  p.kj = cdiv(H, 32);
  if (p.kj == 5 || p.kj == 7) ++p.kj;
  p.pw = H <= 32 ? 1 : H <= 64 ? 2 : H <= 128 ? 4 : H <= 256 ? 8 : 10;
  if (phase == BLSTM_PHASE_FWD) {
    p.smem = 4 * ((size_t)F_SLOTS * 6 * p.R * 36 + (size_t)p.nch * 2 * p.R * 32 * p.kj + (size_t)p.nch * 256) + 512;
  } else {
    const int ni = cdiv(p.U * p.R, 32 * p.pw);
    p.smem = 4 * ((size_t)F_SLOTS * 6 * p.R * p.U + 2 * 4 * (p.U * p.R + 4) + (size_t)p.nch * 2 * p.nc * p.R * p.U +
                  (size_t)p.nch * 2 * ni * 32 * p.pw) + 512;
  }
  // Up to 32 units one warp does all of a CTA's backward work: one chunk of at most 4 rows (8 rows take 8 us a step, the
  // grid-wide kernel 4 to 9).
  const int most = phase == BLSTM_PHASE_BWD && H <= 32 ? 1 : SB_MAX_CHUNKS;
  p.ok = p.nch <= most && (most > 1 || p.R <= 4) && p.smem <= 232448;
  return p;
}

template <int KJ>
static int f32_fwd_r(const F32Plan& pl, const F32Params& p, cudaStream_t st) {
  const int grid = pl.ncl * pl.nc;
#define BLSTM_F32_FWD(RR) \
  if (pl.R == RR) return launch_clusters(f32_fwd_kernel<KJ, RR, (KJ > 1)>, grid, 384, pl.smem, pl.nc, st, p);
  BLSTM_F32_FWD(1)
  BLSTM_F32_FWD(2)
  BLSTM_F32_FWD(4)
  BLSTM_F32_FWD(8)
#undef BLSTM_F32_FWD
  return BLSTM_E_UNSUPPORTED;
}

template <int U, int PW>
static int f32_bwd_r(const F32Plan& pl, const F32Params& p, cudaStream_t st) {
  const int grid = pl.ncl * pl.nc;
#define BLSTM_F32_BWD(RR) \
  if (pl.R == RR) return launch_clusters(f32_bwd_kernel<U, PW, RR, (PW > 1)>, grid, 384, pl.smem, pl.nc, st, p);
  BLSTM_F32_BWD(1)
  BLSTM_F32_BWD(2)
  BLSTM_F32_BWD(4)
  BLSTM_F32_BWD(8)
#undef BLSTM_F32_BWD
  return BLSTM_E_UNSUPPORTED;
}

static F32Params f32_params(const blstm_desc& d, const F32Plan& pl, void* ws) {
  F32Params p{};
  p.T = d.seq_len; p.B = d.batch; p.H = d.hidden_size;
  p.nc = pl.nc; p.rows = pl.rows; p.nch = pl.nch;
  p.no_arrive = (d.flags & BLSTM_FLAG_TEST_NO_ARRIVE) ? 1 : 0;
  p.inference = (d.flags & BLSTM_FLAG_INFERENCE) ? 1 : 0;
  p.limit_ns = d.wait_limit_us > 0 ? (unsigned long long)d.wait_limit_us * 1000ull : kDefaultWaitNs;
  p.ctl = reinterpret_cast<Control*>(ws);
  return p;
}

}  // namespace sm100

using namespace sm100;

size_t f32_workspace(const blstm_desc& d, const F32Plan& pl, int phase) {
  return sizeof(Control) + (phase == BLSTM_PHASE_BWD ? round_up((size_t)pl.ncl * 4 * d.hidden_size * sizeof(float), 256) : 0);
}

int f32_fwd_recurrence(const blstm_desc& d, const F32Plan& pl, void* ifgo, const void* Wh, void* out, void* cell, void* ws,
                       cudaStream_t st) {
  F32Params p = f32_params(d, pl, ws);
  p.Wh = (const float*)Wh; p.ifgo = (float*)ifgo; p.out = (float*)out; p.cell = (float*)cell;
  switch (pl.kj) {
    case 1: return f32_fwd_r<1>(pl, p, st);
    case 2: return f32_fwd_r<2>(pl, p, st);
    case 3: return f32_fwd_r<3>(pl, p, st);
    case 4: return f32_fwd_r<4>(pl, p, st);
    case 6: return f32_fwd_r<6>(pl, p, st);
    case 8: return f32_fwd_r<8>(pl, p, st);
    case 9: return f32_fwd_r<9>(pl, p, st);
    case 10: return f32_fwd_r<10>(pl, p, st);
  }
  return BLSTM_E_UNSUPPORTED;
}

int f32_bwd_recurrence(const blstm_desc& d, const F32Plan& pl, const void* dout, const void* dh_n, const void* dc_n,
                       const void* ifgo, const void* cell, const void* Wh, void* d_ifgo, void* dh0, void* dc0, float* db,
                       void* ws, cudaStream_t st) {
  F32Params p = f32_params(d, pl, ws);
  p.Wh = (const float*)Wh; p.ifgo = (float*)ifgo; p.cell = (float*)cell;
  p.dout = (const float*)dout; p.dh_n = (const float*)dh_n; p.dc_n = (const float*)dc_n;
  p.d_ifgo = (float*)d_ifgo; p.dh0 = (float*)dh0; p.dc0 = (float*)dc0;
  p.db_part = db ? reinterpret_cast<float*>(static_cast<char*>(ws) + sizeof(Control)) : nullptr;
  int rc = BLSTM_E_UNSUPPORTED;
  if (pl.U == 24) rc = f32_bwd_r<24, 10>(pl, p, st);
  else if (pl.pw == 1) rc = f32_bwd_r<32, 1>(pl, p, st);
  else if (pl.pw == 2) rc = f32_bwd_r<32, 2>(pl, p, st);
  else if (pl.pw == 4) rc = f32_bwd_r<32, 4>(pl, p, st);
  else rc = f32_bwd_r<32, 8>(pl, p, st);
  if (rc) return rc;
  return db ? reduce_db(p.db_part, pl.ncl, 4 * d.hidden_size, db, st) : BLSTM_OK;
}

}  // namespace blstm
