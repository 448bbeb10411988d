// Helpers of the recurrences that run inside one cluster: remote stores that complete an mbarrier, bounded waits without
// a call, register shares.
#pragma once

#include <cstdlib>

#include "sm100_common.cuh"

namespace blstm {
namespace sm100 {

constexpr int SB_MAX_CHUNKS = 16;      // row chunks per cluster
constexpr int SB_MAX_SLOTS = 32;       // item slots of a ring

__device__ __forceinline__ void st_async16(uint32_t addr, uint4 v, uint32_t bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1,%2,%3,%4}, [%5];"
               ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "r"(bar) : "memory");
}
__device__ __forceinline__ void st_shared16(uint32_t addr, uint4 v) {
  asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
// Bounded mbarrier wait, inlined on purpose: a call on the waiting path would spill the weight fragments around it.
__device__ __forceinline__ bool wait_inline(uint64_t* bar, uint32_t parity, volatile int* dead, Control* ctl,
                                            unsigned long long limit_ns, int d0, int d1) {
  if (mbar_try_wait_cluster(bar, parity)) return true;
  unsigned spins = 0;
  unsigned long long t0 = 0;
  while (!mbar_try_wait_cluster(bar, parity)) {
    if ((++spins & 63u) != 0u) continue;
    if (*dead || ld_relaxed_gpu(&ctl->abort) != 0) { *dead = 1; return false; }
    const unsigned long long now = globaltimer_ns();
    if (t0 == 0) t0 = now;
    if (now - t0 > limit_ns) {
      *dead = 1;
      record_timeout(ctl, d0, d1);
      return false;
    }
  }
  return true;
}
template <int N> __device__ __forceinline__ void regs_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N> __device__ __forceinline__ void regs_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }

// Clusters of nc CTAs that can be resident at once, one CTA per SM.
int resident_clusters(int nc);

// Launches `kern` on clusters of nc CTAs.
template <typename Kern, typename... Args>
inline int launch_clusters(Kern kern, int grid, int threads, size_t smem, int nc, cudaStream_t st, const Args&... args) {
  BLSTM_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  if (nc > 8) BLSTM_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = nc;
  attr.val.clusterDim.y = 1;
  attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = nc > 1 ? 1 : 0;
  BLSTM_CUDA_OK(cudaLaunchKernelEx(&cfg, kern, args...));
  count_launch();
  return BLSTM_OK;
}

// Launches `kern` on clusters of nc CTAs that wait for one another across clusters: the whole grid has to be resident at
// once.  FASTLSTM_B200_NO_COOP=1 drops the cooperative attribute (profilers that replay kernels refuse a cooperative
// cluster launch); co-residency then rests on the occupancy check alone.
template <typename Kern, typename... Args>
inline int launch_coresident(Kern kern, int grid, int threads, size_t smem, int nc, cudaStream_t st, const Args&... args) {
  BLSTM_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attrs[2];
  attrs[0].id = cudaLaunchAttributeClusterDimension;
  attrs[0].val.clusterDim.x = nc;
  attrs[0].val.clusterDim.y = 1;
  attrs[0].val.clusterDim.z = 1;
  attrs[1].id = cudaLaunchAttributeCooperative;
  attrs[1].val.cooperative = 1;
  cfg.attrs = attrs;
  static const bool no_coop = [] { const char* e = getenv("FASTLSTM_B200_NO_COOP"); return e && e[0] == '1'; }();
  cfg.numAttrs = no_coop ? 1 : 2;
  int max_clusters = 0;
  BLSTM_CUDA_OK(cudaOccupancyMaxActiveClusters(&max_clusters, kern, &cfg));
  if (max_clusters * nc < grid) return BLSTM_E_NOT_CORESIDENT;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kern, args...);
  if (cfg.numAttrs == 2 && (e == cudaErrorNotSupported || e == cudaErrorCooperativeLaunchTooLarge)) {
    // Only when the driver refuses the cooperative + cluster combination as such is the cooperative
    // attribute dropped (co-residency then rests on the occupancy check above); any other launch error
    // is reported as it is.
    (void)cudaGetLastError();
    cfg.numAttrs = 1;
    e = cudaLaunchKernelEx(&cfg, kern, args...);
  }
  BLSTM_CUDA_OK(e);
  count_launch();
  return BLSTM_OK;
}

}  // namespace sm100
}  // namespace blstm
