// Launcher of one dense-kernel variant. The definition and its instantiations live in dense_inst_*.cu (a few
// variants per file, so that a rebuild compiles them side by side); everybody else sees the declaration.
#pragma once

#include "../sm100/gemm_dense.cuh"

#include <cuda_runtime.h>

namespace fluxb {

// coop: the launch carries the cooperative attribute, so the grid only starts when all of its CTAs
// can be resident together (and the launch fails, instead of waiting forever inside the kernel, when
// they never can). Every launch whose CTAs wait for one another or for peers asks for it.
template <class Cfg>
int launch_dense(const DenseGemmParams& p, int grid, cudaStream_t stream, bool coop);

}  // namespace fluxb
