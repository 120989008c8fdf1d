// Definition of launch_dense (dense_launch.cuh), included by the files that instantiate it.
#pragma once

#include "../runtime/host_common.h"
#include "dense_launch.cuh"

#include <atomic>

namespace fluxb {
extern std::atomic<uint64_t> g_launches;

template <class Cfg>
int launch_dense(const DenseGemmParams& p, int grid, cudaStream_t stream, bool coop) {
  constexpr int kThreads = Cfg::THREADS;
  static bool configured[64] = {false};
  int dev = 0;
  FLUXB_CUDA_OK(cudaGetDevice(&dev));
  if (dev >= 64 || !configured[dev]) {
    FLUXB_CUDA_OK(cudaFuncSetAttribute(dense_gemm_kernel<Cfg>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES));
    if (dev < 64) configured[dev] = true;
  }
  {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid, 1, 1);
    cfg.blockDim = dim3(kThreads, 1, 1);
    cfg.dynamicSmemBytes = Cfg::SMEM_BYTES;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int na = 0;
    if constexpr (Cfg::CG == 2) {
      attr[na].id = cudaLaunchAttributeClusterDimension;
      attr[na].val.clusterDim.x = 2;
      attr[na].val.clusterDim.y = 1;
      attr[na].val.clusterDim.z = 1;
      ++na;
    }
    if (coop) {
      attr[na].id = cudaLaunchAttributeCooperative;
      attr[na].val.cooperative = 1;
      ++na;
    }
    cfg.attrs = attr;
    cfg.numAttrs = na;
    FLUXB_CUDA_OK(cudaLaunchKernelEx(&cfg, dense_gemm_kernel<Cfg>, p));
  }
  FLUXB_CUDA_OK(cudaGetLastError());
  g_launches.fetch_add(1, std::memory_order_relaxed);
  note_gemm({FLUXB_KERNEL_PERSISTENT, Cfg::BM, Cfg::BN, Cfg::CG, 1 << p.split_shift, coop ? 1 : 0});
  return kOk;
}

}  // namespace fluxb

#define FLUXB_DENSE_INSTANCE(...) \
  template int fluxb::launch_dense<fluxb::DenseCfg<__VA_ARGS__>>(const fluxb::DenseGemmParams&, int, cudaStream_t, bool)
