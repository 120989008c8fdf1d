// Split-K launches of the dense GEMM entry points (dense_skinny.cu).
#pragma once

#include "../include/fluxb.h"
#include "../sm100/gemm_skinny.cuh"

namespace fluxb {

struct SkinnyShape {
  int32_t bn, tiles, splits;
};

// `d` carries the checked operands of the call, `a` the pointers and pitches its tensor maps are made from.
int dense_skinny(const DenseGemmParams& d, const SkinnyShape& s, const fluxb_dense_args_t* a, void* out, int64_t ldd,
                 cudaStream_t stream);

}  // namespace fluxb

// The rule (exported for its tests): see dense_skinny.cu
extern "C" int fluxb_skinny_shape(int32_t M, int32_t N, int32_t k_blocks, int32_t blockscale, int32_t sms,
                                  int32_t* bn, int32_t* tiles, int32_t* splits);
