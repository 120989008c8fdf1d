// Launches of the split-K kernel (gemm_skinny.cuh): tensor maps, ring depth, cluster size.
#include "dense_skinny.h"

#include "../runtime/host_common.h"

#include <atomic>
#include <cstring>

namespace fluxb {
extern std::atomic<uint64_t> g_launches;

namespace {

template <class Cfg>
int launch_skinny(const SkinnyParams& p, int grid, cudaStream_t stream) {
  static bool configured[64] = {false};
  int dev = 0;
  FLUXB_CUDA_OK(cudaGetDevice(&dev));
  if (dev >= 64 || !configured[dev]) {
    FLUXB_CUDA_OK(cudaFuncSetAttribute(skinny_gemm_kernel<Cfg>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       Cfg::SMEM_BYTES));
    if (dev < 64) configured[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid, 1, 1);
  cfg.blockDim = dim3(Cfg::THREADS, 1, 1);
  cfg.dynamicSmemBytes = Cfg::SMEM_BYTES;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = p.splits;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = p.splits > 1 ? 1 : 0;
  FLUXB_CUDA_OK(cudaLaunchKernelEx(&cfg, skinny_gemm_kernel<Cfg>, p));
  FLUXB_CUDA_OK(cudaGetLastError());
  g_launches.fetch_add(1, std::memory_order_relaxed);
  note_gemm({FLUXB_KERNEL_SPLIT_K, 128, Cfg::BN, 1, p.splits, 0});
  return kOk;
}

template <class Cfg>
int run_skinny(SkinnyParams& p, const SkinnyShape& s, const fluxb_dense_args_t* a, cudaStream_t stream) {
  constexpr bool in16 = Cfg::KIND == 0;
  const CUtensorMapDataType in_dt = in16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_UINT8;
  p.a_rows = (p.M < 128 ? p.M + 7 : 128) & ~7;
  p.stages = Cfg::RING_BYTES / Cfg::stage_bytes(p.a_rows);
  if (p.stages > Cfg::MAX_STAGES) p.stages = Cfg::MAX_STAGES;
  p.splits = s.splits;
  int rc;
  {
    uint64_t dims[2] = {static_cast<uint64_t>(p.K), static_cast<uint64_t>(p.M)};
    uint64_t str[1] = {static_cast<uint64_t>(a->lda) * Cfg::ELT};
    uint32_t box[2] = {Cfg::BK, static_cast<uint32_t>(p.a_rows)};
    if ((rc = encode_tmap(&p.tm_a, in_dt, 2, a->a, dims, str, box, Swz::B128))) return rc;
  }
  {
    uint64_t dims[2] = {static_cast<uint64_t>(p.b_kn ? p.N : p.K), static_cast<uint64_t>(p.b_kn ? p.K : p.N)};
    uint64_t str[1] = {static_cast<uint64_t>(a->ldb) * Cfg::ELT};
    uint32_t box[2] = {p.b_kn ? 64u : Cfg::BK, static_cast<uint32_t>(p.b_kn ? Cfg::BK : Cfg::BN)};
    if ((rc = encode_tmap(&p.tm_b, in_dt, 2, a->b, dims, str, box, Swz::B128))) return rc;
  }
  return launch_skinny<Cfg>(p, s.tiles * s.splits, stream);
}

}  // namespace

int dense_skinny(const DenseGemmParams& d, const SkinnyShape& s, const fluxb_dense_args_t* a, void* out, int64_t ldd,
                 cudaStream_t stream) {
  SkinnyParams p;
  memset(&p, 0, sizeof(p));
  p.M = d.M;
  p.N = d.N;
  p.K = d.K;
  p.m_tiles = (d.M + 127) / 128;
  p.b_kn = d.b_kn;
  p.ab_fmt = d.ab_fmt;
  p.out_f16 = d.out_f16;
  p.act = d.act;
  p.scale_flags = d.scale_flags;
  p.timeout_ns = d.timeout_ns;
  p.status = d.status;
  p.bias = d.bias;
  p.bias_row_stride = d.bias_row_stride;
  p.scale_a = d.scale_a;
  p.scale_b = d.scale_b;
  p.sa = d.sa;
  p.sb = d.sb;
  p.d = reinterpret_cast<uint16_t*>(out);
  p.ldd = ldd;
  if (a->blockscale) return run_skinny<SkinnyCfg<64, 1, true>>(p, s, a, stream);
  if (a->in_dtype == FLUXB_INT8)
    return s.bn == 64 ? run_skinny<SkinnyCfg<64, 2>>(p, s, a, stream) : run_skinny<SkinnyCfg<128, 2>>(p, s, a, stream);
  if (a->in_dtype == FLUXB_BF16 || a->in_dtype == FLUXB_FP16)
    return s.bn == 64 ? run_skinny<SkinnyCfg<64, 0>>(p, s, a, stream) : run_skinny<SkinnyCfg<128, 0>>(p, s, a, stream);
  return s.bn == 64 ? run_skinny<SkinnyCfg<64, 1>>(p, s, a, stream) : run_skinny<SkinnyCfg<128, 1>>(p, s, a, stream);
}

}  // namespace fluxb

using namespace fluxb;

// Which plain GEMMs run on the split-K kernel, and how: bn = 0 (none), 64 or 128 columns per tile, splits CTAs
// per tile. k_blocks: 128-byte blocks along K; blockscale as in fluxb_dense_args_t. Times in us inside a graph,
// weights from memory, persistent kernel -> this one:
//  * up to 64 rows, always: 16 x 4096 x 16384 110 -> 30, 16 x 16384 x 4096 36 -> 28, 16 x 65536 x 2048 66 -> 48,
//    64 x 12288 x 4096 int8 19.5 -> 16.3, 1 x 4096 x 4096 32 -> 12. 128 columns: 64 repeat the rows of A more often.
//  * more rows, as long as the 64-column tiles fit the chip twice: 128 x 4096 x 4096 32 -> 16, 1024 x 2048 x 8192
//    63 -> 38, 300 x 1024 x 8192 58 -> 20. (1000 x 3000 x 5000, 376 tiles: 54 on the persistent kernel, 66 here.)
//    64 columns balance better, but once they fill the chip without a split, two K halves of 128 columns read
//    less: 2048 x 1024 x 4096 27 -> 23, from 49 k-blocks on. 64 / 128 columns, geometric means over 65 - 2048 rows in
//    all types: 32 k-blocks 0.91, 40 0.95, 48 0.98, 64 1.04, 96 1.08 (128 x 16384 x 4096 int8 17.8 / 20.8, where the
//    persistent kernel takes 17.8).
//  * block scales: 64 columns (the fp32 row of a thread stays in registers): 48 x 3584 x 8192 46 -> 15,
//    1024 x 2048 x 8192 46 -> 37; 64 x 24576 x 4096, 384 tiles: 31 on the persistent kernel, 37 here.
// Splits: to one CTA per SM wherever four k-blocks are left each, on to two per SM only with 16 left each (8192
// columns x 2048 fp8: 2 splits 8.5, 4 splits 10.0); eight were never faster than four.
extern "C" int fluxb_skinny_shape(int32_t M, int32_t N, int32_t k_blocks, int32_t blockscale, int32_t sms,
                                  int32_t* bn, int32_t* tiles, int32_t* splits) {
  FLUXB_REQUIRE(M > 0 && N > 0 && k_blocks > 0 && sms > 0 && bn && tiles && splits, "split-K arguments");
  *bn = *tiles = *splits = 0;
  if (blockscale > 1) return kOk;
  const int64_t mt = (M + 127) / 128;
  const int64_t t64 = mt * ((N + 63) / 64), t128 = mt * ((N + 127) / 128);
  if ((blockscale != 0 || M > 64) && t64 > 2 * sms) return kOk;
  int w = (blockscale != 0 || M > 64) ? 64 : 128;
  if (w == 64 && blockscale == 0 && t64 > sms && k_blocks > 48) w = 128;
  const int64_t t = w == 64 ? t64 : t128;
  int s = 1;
  while (s < 4 && 2 * s * t <= 2 * sms && k_blocks >= (2 * s * t <= sms ? 8 : 32) * s) s *= 2;
  *bn = w;
  *tiles = static_cast<int32_t>(t);
  *splits = s;
  return kOk;
}
