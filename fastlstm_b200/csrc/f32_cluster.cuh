// Plan and launchers of the fp32 recurrences inside one cluster.
#pragma once
#include "common.cuh"

namespace blstm {
namespace sm100 {

struct F32Plan {
  bool ok;
  int U, nc;                // hidden units per CTA, CTAs per cluster
  int R, nch, rows, ncl;    // rows per chunk, chunks and rows per cluster, clusters
  int kj, pw;               // forward: groups of 32 K steps; backward: product warps
  size_t smem;
};

F32Plan f32_plan(const blstm_desc& d, int phase);

}  // namespace sm100

size_t f32_workspace(const blstm_desc& d, const sm100::F32Plan& pl, int phase);
int f32_fwd_recurrence(const blstm_desc& d, const sm100::F32Plan& pl, void* ifgo, const void* Wh, void* out, void* cell,
                       void* ws, cudaStream_t st);
int f32_bwd_recurrence(const blstm_desc& d, const sm100::F32Plan& pl, const void* dout, const void* dh_n, const void* dc_n,
                       const void* ifgo, const void* cell, const void* Wh, void* d_ifgo, void* dh0, void* dc0, float* db,
                       void* ws, cudaStream_t st);

}  // namespace blstm
