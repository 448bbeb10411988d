// Plans and launchers of the small-batch recurrences (16-bit; clusters that hold the weights and exchange a step's
// results through distributed shared memory).
#pragma once
#include "common.cuh"

namespace blstm {
namespace sm100 {

struct SmallPlan {
  bool ok;                  // the kernels cover the shape and are the faster ones for it
  int nc, gc;               // CTAs per cluster; groups of 8 hidden units per CTA
  int ks;                   // K steps of 16 (an even number)
  int kr;                   // K steps whose weights live in registers
  int rows, ncl;            // batch rows per cluster, clusters
  int nch;                  // chunks of 8 rows per cluster
  int rpl, kspl, slots;     // forward: replicas of the gc warps, K parts, item slots of the ring
  int mgroups, mpw;         // backward: M tiles worked at once, M tiles per warp
  int nparts;               // backward: rows of bias-gradient partial sums
  int threads, grid;
  size_t smem;
};

struct SmallFwdParams {
  int T, B, H;
  int nc, gc, ks, rows, nch, rpl, slots;
  int no_arrive, inference;
  unsigned long long limit_ns;
  Control* ctl;
  const void* Wh;
  const void* out;          // [T+1,B,H]: slot 0 (the other steps are written through the tensor maps)
  const void* cell;         // [T+1,B,H]: slot 0
};

struct SmallBwdParams {
  int T, B, H;
  int nc, gc, rows, nch, mgroups;
  int no_arrive;
  unsigned long long limit_ns;
  Control* ctl;
  const void* dh_n;         // [B,H] or null
  const void* dc_n;         // [B,H] or null
  const void* cell;         // [T+1,B,H]: slot T
  const void* Wh;
  void* dh0;                // [B,H]
  void* dc0;                // [B,H]
  float* db_part;           // [clusters][4H] or null
};

SmallPlan small_plan(const blstm_desc& d, int phase);

}  // namespace sm100

size_t small_workspace(const blstm_desc& d, const sm100::SmallPlan& pl, int phase);
int small_fwd_recurrence(const blstm_desc& d, const sm100::SmallPlan& pl, void* ifgo, const void* Wh, void* out, void* cell,
                         void* ws, cudaStream_t st);
int small_bwd_recurrence(const blstm_desc& d, const sm100::SmallPlan& pl, const void* dout, const void* dh_n, const void* dc_n,
                         const void* ifgo, const void* cell, const void* Wh, void* d_ifgo, void* dh0, void* dc0,
                         float* db, void* ws, cudaStream_t st);
int small_plan_detail(const blstm_desc& d, const sm100::SmallPlan& pl, int phase, char* buf, size_t n);

}  // namespace blstm
