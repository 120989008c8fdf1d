// Split-K GEMM for problems whose output tiles do not fill the chip: D[M,N] = A[M,K] * B[N,K]^T.
//
// Such calls (a few tokens against a whole weight matrix) are bound by streaming the weight, and what the
// persistent kernel lacks there is bytes in flight: one CTA per output tile leaves SMs without work, and its
// 128-row A stages are mostly padding. Here a cluster of S CTAs shares one 128 x BN output tile, each CTA
// accumulating its own K range in its own TMEM; the S fp32 partial tiles meet in distributed shared memory,
// where every CTA adds its share of the tile in rank order (the same sum on every run), applies scales, bias
// and activation and stores 16-byte pieces. Two CTAs fit an SM, so one streams while the other starts or ends.
// A stage holds only the rows that exist (rounded up to 8): the MMA still reads 128 rows, the rest of
// them whatever lies behind in the ring (inside this CTA's shared memory), and those rows of D are never read.
//
//   warps 0..3  epilogue (TMEM lane quadrant = warp); block-scaled: they also promote every k-block
//   warp 4      TMA producer
//   warp 5      MMA issuer
#pragma once

#include "gemm_dense.cuh"

namespace fluxb {

struct SkinnyParams {
  CUtensorMap tm_a;              // A [M, K], box {BK, a_rows}
  CUtensorMap tm_b;              // B [N, K], box {BK, BN}; b_kn: B [K, N], box {64, BK}
  int32_t M, N, K;
  int32_t m_tiles;               // row tiles of 128, innermost in the grid
  int32_t a_rows;                // rows of an A stage: min(M, 128) rounded up to 8
  int32_t stages, splits;        // ring depth; CTAs per cluster
  int32_t b_kn, ab_fmt, out_f16, act;
  uint32_t scale_flags;          // as in DenseGemmParams
  uint64_t timeout_ns;
  Status* status;
  const void* bias;
  int64_t bias_row_stride;
  const float* scale_a;
  const float* scale_b;
  const float* sa;               // block scales: [ceil(M/128), K/128, 128] and [N/128, K/128]
  const float* sb;
  uint16_t* d;
  int64_t ldd;
};

template <int BN_, int KIND_, bool BS_ = false>
struct SkinnyCfg {
  static constexpr int BN = BN_, KIND = KIND_;
  static constexpr bool BS = BS_;
  static constexpr int ELT = KIND_ == 0 ? 2 : 1;
  static constexpr int BK = 128 / ELT, UMMA_K = 32 / ELT;
  static constexpr int THREADS = 192;
  static constexpr int B_BYTES = BN_ * 128;
  static constexpr int ACC_BUFS = BS_ ? 4 : 1;           // block-scaled: a fresh accumulator per k-block
  static constexpr int TMEM_COLS = BN_ * ACC_BUFS;       // 64 .. 256: two CTAs share the 512 columns
  static_assert(TMEM_COLS <= 256, "two CTAs per SM");
  static constexpr int PITCH = BN_ * 4 + 16;             // bytes per row of the staged fp32 tile (odd in 16-byte units)
  static constexpr int MAX_STAGES = 16;
  static constexpr int BAR_BYTES = 512;
  static constexpr int SMEM_BYTES = 112 * 1024;          // two CTAs per SM
  static constexpr int RING_BYTES = SMEM_BYTES - BAR_BYTES - 1024;
  static_assert(RING_BYTES >= 128 * PITCH, "the staged tile reuses the ring");
  __host__ __device__ static constexpr int stage_bytes(int a_rows) { return a_rows * 128 + B_BYTES; }
};

template <class Cfg>
__global__ void __launch_bounds__(Cfg::THREADS, 2) skinny_gemm_kernel(const __grid_constant__ SkinnyParams p) {
  constexpr int BN = Cfg::BN, BK = Cfg::BK;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = ptx::smem_u32(smem_raw);
  const uint32_t pad = (1024u - (raw_addr & 1023u)) & 1023u;
  const uint32_t smem_base = raw_addr + pad;
  const uint32_t bar_base = smem_base + Cfg::RING_BYTES;
  uint8_t* bar_ptr = smem_raw + pad + Cfg::RING_BYTES;
  // all A stages, then all B stages: an A tile read past its rows stays inside the ring
  const int a_bytes = p.a_rows * 128;
  const uint32_t b_base = smem_base + p.stages * a_bytes;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (Cfg::MAX_STAGES + s); };
  auto tfull_bar = [&](int a) { return bar_base + 8u * (2 * Cfg::MAX_STAGES + a); };
  auto tempty_bar = [&](int a) { return bar_base + 8u * (2 * Cfg::MAX_STAGES + Cfg::ACC_BUFS + a); };
  constexpr int kWords = 8 * (2 * Cfg::MAX_STAGES + 2 * Cfg::ACC_BUFS);
  static_assert(kWords + 8 <= Cfg::BAR_BYTES, "barrier block too small");
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(bar_ptr + kWords);
  volatile uint32_t* abort_word = tmem_slot + 1;

  const int warp = ptx::warp_index(), lane = threadIdx.x & 31;
  const int S = p.splits;
  const int rank = S > 1 ? static_cast<int>(ptx::cluster_ctarank()) : 0;
  const int tile = blockIdx.x / S;
  const int m0 = (tile % p.m_tiles) * 128, n0 = (tile / p.m_tiles) * BN;
  const int rows = min(128, p.M - m0);
  const int k_blocks = (p.K + BK - 1) / BK;
  const int kb0 = static_cast<int>(static_cast<int64_t>(k_blocks) * rank / S);
  const int kb1 = static_cast<int>(static_cast<int64_t>(k_blocks) * (rank + 1) / S);

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) {
      ptx::mbar_init(full_bar(s), 1);
      ptx::mbar_init(empty_bar(s), 1);
    }
    for (int a = 0; a < Cfg::ACC_BUFS; ++a) {
      ptx::mbar_init(tfull_bar(a), 1);
      ptx::mbar_init(tempty_bar(a), 4);
    }
    *abort_word = 0;
    ptx::fence_mbar_init();
  }
  if (warp == 4 && lane == 0) {
    ptx::prefetch_tmap(&p.tm_a);
    ptx::prefetch_tmap(&p.tm_b);
  }
  if (warp == 5) {
    ptx::tmem_alloc<1>(ptx::smem_u32(const_cast<uint32_t*>(tmem_slot)), Cfg::TMEM_COLS);
    ptx::tmem_relinquish<1>();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  WaitCtx wc{p.status, abort_word, p.timeout_ns};

  uint32_t facc[Cfg::BS ? BN : 1];   // block-scaled: this thread's row of the tile, fp32
  if (warp == 4) {
    // (the whole warp walks the k-blocks, one elected lane issues)
    const bool b_kn = Cfg::KIND == 0 && p.b_kn != 0;
    int stage = 0;
    uint32_t phase = 0;
    for (int kb = kb0; kb < kb1; ++kb) {
      if (!mbar_wait_warp(wc, empty_bar(stage), phase ^ 1u, kSiteSmemEmpty)) break;
      const uint32_t sb = b_base + stage * Cfg::B_BYTES;
      if (ptx::elect_one()) {
        ptx::mbar_arrive_expect_tx(full_bar(stage), static_cast<uint32_t>(a_bytes + Cfg::B_BYTES));
        if (b_kn) {
#pragma unroll
          for (int j = 0; j < BN / 64; ++j)
            ptx::tma_load_2d(sb + j * (BK * 128), &p.tm_b, full_bar(stage), n0 + j * 64, kb * BK);
        } else {
          ptx::tma_load_2d(sb, &p.tm_b, full_bar(stage), kb * BK, n0);
        }
        ptx::tma_load_2d(smem_base + stage * a_bytes, &p.tm_a, full_bar(stage), kb * BK, m0);
      }
      __syncwarp();
      if (++stage == p.stages) {
        stage = 0;
        phase ^= 1u;
      }
    }
  } else if (warp == 5) {
    const bool b_kn = Cfg::KIND == 0 && p.b_kn != 0;
    const uint32_t bstep = b_kn ? static_cast<uint32_t>(Cfg::UMMA_K * 128) >> 4 : 2u;
    const uint32_t idesc = ptx::umma_idesc(p.ab_fmt, p.ab_fmt, 128, BN, 0, b_kn ? 1u : 0u, Cfg::KIND == 2 ? 2u : 1u);
    int stage = 0;
    uint32_t phase = 0;
    for (int kb = kb0; kb < kb1; ++kb) {
      const uint32_t n = static_cast<uint32_t>(kb - kb0);
      const uint32_t buf = n % Cfg::ACC_BUFS;
      if (Cfg::BS && !mbar_wait_warp(wc, tempty_bar(buf), ((n / Cfg::ACC_BUFS) & 1u) ^ 1u, kSiteTmemEmpty)) break;
      if (!mbar_wait_warp(wc, full_bar(stage), phase, kSiteSmemFull)) break;
      ptx::tc_fence_after();
      const uint64_t adesc = ptx::umma_desc_k_sw128(smem_base + stage * a_bytes);
      const uint32_t sb = b_base + stage * Cfg::B_BYTES;
      const uint64_t bdesc = b_kn ? ptx::umma_desc_mn_sw128(sb, BK * 128, 1024) : ptx::umma_desc_k_sw128(sb);
      if (ptx::elect_one()) {
#pragma unroll
        for (int k = 0; k < BK / Cfg::UMMA_K; ++k)
          ptx::umma_ss<1, Cfg::KIND>(tmem_base + buf * BN, adesc + 2u * k, bdesc + bstep * k, idesc,
                                     (k != 0 || (!Cfg::BS && n != 0)) ? 1u : 0u);
        ptx::umma_commit(empty_bar(stage));
        if constexpr (Cfg::BS) ptx::umma_commit(tfull_bar(buf));
      }
      __syncwarp();
      if (++stage == p.stages) {
        stage = 0;
        phase ^= 1u;
      }
    }
    if constexpr (!Cfg::BS) {
      if (ptx::elect_one()) ptx::umma_commit(tfull_bar(0));
      __syncwarp();
    }
  } else {
    const bool live = warp * 32 < rows;            // some row of this quadrant exists
    const uint32_t lane_base = tmem_base + (static_cast<uint32_t>(warp * 32) << 16);
    const uint32_t my_row = smem_base + (warp * 32 + lane) * Cfg::PITCH;
    if constexpr (Cfg::BS) {
      // every k-block's partial product times its scales into fp32 registers; the scales of four k-blocks are
      // fetched while the four before them are multiplied
      constexpr int G = 4;
      const int kbs = k_blocks;
      const float* sa_ptr = p.sa + static_cast<int64_t>(m0 >> 7) * kbs * 128 + warp * 32 + lane;
      const float* sb_ptr = p.sb + static_cast<int64_t>(n0 >> 7) * kbs;
      float csa[G], csb[G], nsa[G], nsb[G];
      auto load_scales = [&](int kb, float* dsa, float* dsb) {
#pragma unroll
        for (int i = 0; i < G; ++i) {
          const int kk = kb + i < kb1 ? kb + i : kb1 - 1;
          dsa[i] = sa_ptr[static_cast<int64_t>(kk) * 128];
          dsb[i] = sb_ptr[kk];
        }
      };
#pragma unroll
      for (int j = 0; j < BN; ++j) facc[j] = 0u;
      load_scales(kb0, csa, csb);
      for (int kg = kb0; kg < kb1; kg += G) {
        load_scales(kg + G, nsa, nsb);
#pragma unroll
        for (int i = 0; i < G; ++i) {
          if (kg + i >= kb1) break;
          const uint32_t n = static_cast<uint32_t>(kg + i - kb0);
          const uint32_t buf = n % Cfg::ACC_BUFS;
          mbar_wait(wc, tfull_bar(buf), (n / Cfg::ACC_BUFS) & 1u, kSiteTmemFull);
          __syncwarp();
          ptx::tc_fence_after();
          const float sc = csa[i] * csb[i];
          if (live) {
#pragma unroll
            for (int c = 0; c < BN; c += 32) {
              uint32_t r[32];
              ptx::tmem_ld_32x32b_x32(lane_base + buf * BN + c, r);
              ptx::tmem_ld_wait();
#pragma unroll
              for (int j = 0; j < 32; ++j)
                facc[c + j] = __float_as_uint(fmaf(__uint_as_float(r[j]), sc, __uint_as_float(facc[c + j])));
            }
          }
          ptx::tc_fence_before();
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive_relaxed(tempty_bar(buf));
        }
#pragma unroll
        for (int i = 0; i < G; ++i) {
          csa[i] = nsa[i];
          csb[i] = nsb[i];
        }
      }
    } else {
      mbar_wait(wc, tfull_bar(0), 0u, kSiteTmemFull);
      __syncwarp();
      ptx::tc_fence_after();
      if (live) {
        // the ring is free: the partial tile goes there, one row per thread
#pragma unroll
        for (int c = 0; c < BN; c += 32) {
          uint32_t r[32];
          ptx::tmem_ld_32x32b_x32(lane_base + c, r);
          ptx::tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; j += 4)
            ptx::st_shared_v4_f32(my_row + (c + j) * 4, make_float4(__uint_as_float(r[j]), __uint_as_float(r[j + 1]),
                                                                    __uint_as_float(r[j + 2]), __uint_as_float(r[j + 3])));
        }
      }
      ptx::tc_fence_before();
    }
  }
  if (*abort_word) {
    // a wait gave up: let copies and MMAs in flight land before this CTA's shared memory and TMEM go away
    const uint64_t t0 = ptx::globaltimer_ns();
    while (ptx::globaltimer_ns() - t0 < 200000ull) __nanosleep(2000);
  }
  if constexpr (Cfg::BS) {
    // (a warp that promoted its last k-block may be ahead of the others, but that block was the last to be
    // multiplied: nothing of the ring is read any more)
    if (warp < 4 && warp * 32 < rows) {
      const uint32_t my_row = smem_base + (warp * 32 + lane) * Cfg::PITCH;
#pragma unroll
      for (int c = 0; c < BN; c += 4)
        ptx::st_shared_v4_f32(my_row + c * 4, make_float4(__uint_as_float(facc[c]), __uint_as_float(facc[c + 1]),
                                                          __uint_as_float(facc[c + 2]), __uint_as_float(facc[c + 3])));
    }
  }
  __syncwarp();
  if (S > 1) ptx::cluster_sync();
  else __syncthreads();
  if (warp == 5) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc<1>(tmem_base, Cfg::TMEM_COLS);
  }

  // ---- sum of the partial tiles, 8 columns of one row at a time, dealt out over the cluster
  const bool f16 = p.out_f16 != 0;
  const bool sa_vec = (p.scale_flags & 1u) != 0u, sb_vec = (p.scale_flags & 2u) != 0u;
  const bool scaled = p.scale_a != nullptr || p.scale_b != nullptr;
  float alpha = 1.f;
  if (p.scale_a != nullptr && !sa_vec) alpha *= *p.scale_a;
  if (p.scale_b != nullptr && !sb_vec) alpha *= *p.scale_b;
  const uint16_t* bias = reinterpret_cast<const uint16_t*>(p.bias);
  const int units = rows * (BN / 8);
  for (int u = rank * Cfg::THREADS + static_cast<int>(threadIdx.x); u < units; u += S * Cfg::THREADS) {
    const int r = u / (BN / 8), col = n0 + (u % (BN / 8)) * 8;
    if (col >= p.N) continue;                       // (N is a multiple of 8)
    const uint32_t addr = smem_base + r * Cfg::PITCH + (u % (BN / 8)) * 32;
    float v[8];
    if constexpr (Cfg::KIND == 2) {
      int32_t acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};    // s32 partial sums: exact in any order
#pragma unroll 4
      for (int s = 0; s < S; ++s) {
        const uint32_t a = ptx::mapa_u32(addr, s);
        const uint4 x = ptx::ld_cluster_v4(a), y = ptx::ld_cluster_v4(a + 16);
        acc[0] += static_cast<int32_t>(x.x), acc[1] += static_cast<int32_t>(x.y);
        acc[2] += static_cast<int32_t>(x.z), acc[3] += static_cast<int32_t>(x.w);
        acc[4] += static_cast<int32_t>(y.x), acc[5] += static_cast<int32_t>(y.y);
        acc[6] += static_cast<int32_t>(y.z), acc[7] += static_cast<int32_t>(y.w);
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = __int2float_rn(acc[j]);
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = 0.f;
#pragma unroll 4
      for (int s = 0; s < S; ++s) {
        const uint32_t a = ptx::mapa_u32(addr, s);
        const uint4 x = ptx::ld_cluster_v4(a), y = ptx::ld_cluster_v4(a + 16);
        v[0] += __uint_as_float(x.x), v[1] += __uint_as_float(x.y);
        v[2] += __uint_as_float(x.z), v[3] += __uint_as_float(x.w);
        v[4] += __uint_as_float(y.x), v[5] += __uint_as_float(y.y);
        v[6] += __uint_as_float(y.z), v[7] += __uint_as_float(y.w);
      }
    }
    const int row = m0 + r;
    if (scaled) {
      float ar = alpha;
      if (sa_vec) ar *= p.scale_a[row];
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] *= sb_vec ? ar * p.scale_b[col + j] : ar;
    }
    if (bias != nullptr) {
      const uint16_t* b = bias + (p.bias_row_stride ? row * p.bias_row_stride : 0) + col;
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] += ptx::half_bits_to_float(b[j], f16);
    }
    if (p.act != 0) {
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = ptx::activate(v[j], p.act);
    }
    uint4 o;
    o.x = ptx::pack_half2(f16, v[0], v[1]);
    o.y = ptx::pack_half2(f16, v[2], v[3]);
    o.z = ptx::pack_half2(f16, v[4], v[5]);
    o.w = ptx::pack_half2(f16, v[6], v[7]);
    ptx::st_global_v4(p.d + static_cast<int64_t>(row) * p.ldd + col, o);
  }
  __syncwarp();
  if (S > 1) ptx::cluster_sync();                   // the others may still be reading this CTA's partial tile
}

}  // namespace fluxb
