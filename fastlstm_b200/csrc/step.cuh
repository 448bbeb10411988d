// Launcher of the single-timestep layer kernel.
#pragma once
#include "common.cuh"

namespace blstm {

bool step_supported(const blstm_desc& d);
int step_fwd(const blstm_desc& d, const void* x, const void* h0, const void* c0, const void* Wx, const void* Wh, const void* bx,
             const void* bh, void* out, void* cell, void* ifgo, Control* ctl, cudaStream_t st);

}  // namespace blstm
