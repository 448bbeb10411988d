// Plans and launchers of the recurrences whose weights stay on the chip (16-bit, large hidden sizes).
#pragma once
#include "common.cuh"

namespace blstm {
namespace sm100 {

constexpr int RES_MIN_H = 256;         // (smaller sizes have the small-batch kernels or several 128-row tiles a CTA)

struct ResPlan {
  bool ok;
  int ks, own, mt, ng;      // CTAs per cluster (parts of K); of these, owners of batch rows; M tiles; groups of rows
  int ti, rows, N;          // tiles per group, in turn; batch rows of a tile; N of the MMAs
  int kc_total, kcm, nt;    // chunks of K; most of a CTA; of these in tensor memory
  int x_bytes;
  int ni;                   // MMA issuers
  int group;                // chunks at once
  int grid;
  size_t smem, off_db, ws_bytes;
};

ResPlan resident_plan(const blstm_desc& d, int phase);

// ... backward, for batches of several tiles per group
struct TilesPlan {
  bool ok;
  int mt, ng, nbt, N;       // M tiles; groups; batch tiles; their rows
  int kc, nt, w_col;        // K chunks of a CTA; of these in tensor memory, from which column on
  int s2, group;            // ring stages per issuer; chunks of a stage
  int grid;
  size_t smem, off_db, ws_bytes;
};

TilesPlan tiles_plan(const blstm_desc& d, int phase);

// ... and forward, for batches of several 32-row tiles per group
struct FwdTilesPlan {
  bool ok;
  int mt, ng, nbt;          // M tiles; groups; batch tiles
  int kc, nt, w_col, group; // K chunks; of these in tensor memory, from which column on; at once
  int grid;
  size_t smem, ws_bytes;
};

FwdTilesPlan fwd_tiles_plan(const blstm_desc& d, int phase);

}  // namespace sm100

int resident_fwd_recurrence(const blstm_desc& d, const sm100::ResPlan& pl, void* ifgo, const void* Wh, void* out, void* cell, void* ws,
                            cudaStream_t st);
int resident_bwd_recurrence(const blstm_desc& d, const sm100::ResPlan& pl, const void* dout, const void* dh_n, const void* dc_n,
                            const void* ifgo, const void* cell, const void* Wh, void* d_ifgo, void* dh0, void* dc0, float* db,
                            void* ws, cudaStream_t st);
int tiles_bwd_recurrence(const blstm_desc& d, const sm100::TilesPlan& pl, const void* dout, const void* dh_n, const void* dc_n,
                         const void* ifgo, const void* cell, const void* Wh, void* d_ifgo, void* dh0, void* dc0, float* db, void* ws,
                         cudaStream_t st);
int fwd_tiles_recurrence(const blstm_desc& d, const sm100::FwdTilesPlan& pl, void* ifgo, const void* Wh, void* out, void* cell, void* ws,
                         cudaStream_t st);
int fwd_tiles_plan_detail(const sm100::FwdTilesPlan& pl, char* buf, size_t n);
int tiles_plan_detail(const sm100::TilesPlan& pl, char* buf, size_t n);
int resident_plan_detail(const sm100::ResPlan& pl, int phase, char* buf, size_t n);

}  // namespace blstm
