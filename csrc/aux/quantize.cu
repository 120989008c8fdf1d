// Block-scaled FP8 quantisation: 1x128 (per row, per 128 columns) and 128x128 blocks, each with
// an optional second output for the transposed matrix, in one pass over the input.
//
//   scale     = 448 / max(amax, eps)       (e4m3; 57344 for e5m2), 1 if the block is all zero
//   q         = saturate_to_fp8(x * scale)
//   scale_inv = 1 / scale                  (what is stored)
//
// 1x128 layout: q [M,K], scale_inv [ceil(M/128), ceil(K/128), 128] (row inside the block last);
// the transposed output is a separate quantisation of x^T with its own 1x128 blocks, i.e. one
// scale per column of x per 128 rows: q_t [K,M], scale_inv_t [ceil(K/128), ceil(M/128), 128].
// 128x128 layout: scale_inv [ceil(M/128), ceil(K/128)], q_t = transpose(q),
// scale_inv_t [ceil(K/128), ceil(M/128)].
// Reference: src/quantization/quantization.cu (ComputeScale :306-362, kernels :428-1193) and
// src/quantization/ths_op/quantization.cc:75-172.
#include "../include/fluxb.h"
#include "../runtime/host_common.h"

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>

#include <atomic>
#include <type_traits>

namespace fluxb {
extern std::atomic<uint64_t> g_launches;

namespace {

constexpr int kTile = 128;
constexpr int kThreads = 256;

__device__ __forceinline__ float compute_scale(float amax, float eps, float fp8_max) {
  const float a = fmaxf(amax, eps);
  if (a == 0.f) return 1.f;
  const float s = fp8_max / a;
  if (isinf(s)) return 3.3895313892515355e38f;  // largest finite bf16: the clamp of the reference
  return s;
}

// ---------------------------------------------------------------------------------------------
// Fast path for 16-bit inputs and whole 128 x 128 tiles: the tile lives in registers. A thread owns
// 4 consecutive rows x 8 columns (16 bytes per row) in each of two passes over the 32 row groups,
// so that a half-warp reads one 256-byte row segment per instruction; row maxima are reduced by
// shuffles, column maxima through a small shared array; q leaves as 8-byte stores (128 contiguous
// bytes per row), q^T is transposed through a swizzled shared tile (a thread's 4 rows of one column
// are one 32-bit word) and leaves as 16-byte stores. 16384 x 8192 bf16, 1x128: 90 us with the transpose, 68 without, both
// 0.92 of the copy rate, so memory bounds it; 108 and 82 with the row maxima as a butterfly, bound by instruction issue.
// ---------------------------------------------------------------------------------------------
template <bool BF16>
__device__ __forceinline__ uint32_t habs2_bits(uint32_t v) {
  return v & 0x7FFF7FFFu;
}
template <bool BF16>
__device__ __forceinline__ uint32_t hmax2_bits(uint32_t a, uint32_t b) {
  // operands are non-negative 16-bit floats: their order is the order of their bit patterns
  uint32_t r;
  asm("max.u16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
template <bool BF16>
__device__ __forceinline__ float h_lo(uint32_t v) {
  if constexpr (BF16) return __uint_as_float(v << 16);
  else return __half2float(__ushort_as_half(static_cast<unsigned short>(v & 0xFFFFu)));
}
template <bool BF16>
__device__ __forceinline__ float h_hi(uint32_t v) {
  if constexpr (BF16) return __uint_as_float(v & 0xFFFF0000u);
  else return __half2float(__ushort_as_half(static_cast<unsigned short>(v >> 16)));
}
__device__ __forceinline__ uint32_t cvt_fp8x2(float lo, float hi, bool e5m2) {
  return static_cast<uint32_t>(
      __nv_cvt_float2_to_fp8x2(make_float2(lo, hi), __NV_SATFINITE, e5m2 ? __NV_E5M2 : __NV_E4M3));
}

// Maxima of eight rows over the 16 lanes that share them: each step of the exchange halves the rows a lane still
// holds, so that lane l ends with row (l >> 1) & 7 (eight shuffles instead of 32), and a row's scale is divided out by
// two lanes instead of sixteen. 8192 x 8192 bf16, 1x128: 43.8 -> 33.6 us (6.0 TB/s), with the transpose 58.5 -> 48.1.
template <class Max>
__device__ __forceinline__ uint32_t max_rows8(uint32_t (&m)[8], int lane, Max&& vmax) {
#pragma unroll
  for (int half = 4; half > 0; half >>= 1) {
    const bool up = (lane & (2 * half)) != 0;
#pragma unroll
    for (int j = 0; j < half; ++j) {
      const uint32_t send = up ? m[j] : m[j + half], keep = up ? m[j + half] : m[j];
      m[j] = vmax(keep, __shfl_xor_sync(0xffffffffu, send, 2 * half));
    }
  }
  return vmax(m[0], __shfl_xor_sync(0xffffffffu, m[0], 1));
}

template <bool BF16, bool SQUARE>
__global__ void __launch_bounds__(kThreads) quant_tile_kernel(
    const uint16_t* __restrict__ x, int64_t ldx, uint8_t* __restrict__ q, uint8_t* __restrict__ qt,
    float* __restrict__ sinv, float* __restrict__ sinv_t, int M, int K, float eps, int e5m2,
    int64_t batch_stride_x, int64_t batch_stride_q, int64_t batch_stride_s) {
  __shared__ uint32_t colred[kThreads / 32][64];         // packed column maxima per warp
  __shared__ float col_scale[kTile];
  __shared__ float red[kThreads / 32];
  __shared__ __align__(16) uint32_t tile_t[kTile * 32];   // q^T tile: 128 rows (columns of x) x 128 bytes, swizzled
  const int kb = blockIdx.x, mb = blockIdx.y, bz = blockIdx.z;
  const int MB = gridDim.y, KB = gridDim.x;
  x += bz * batch_stride_x;
  q += bz * batch_stride_q;
  if (qt) qt += bz * batch_stride_q;
  sinv += bz * batch_stride_s;
  if (sinv_t) sinv_t += bz * batch_stride_s;
  const int row0 = mb * kTile, col0 = kb * kTile;
  const float fp8_max = e5m2 ? 57344.f : 448.f;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int chunk = lane & 15;                  // 8-column chunk of the tile
  const bool e5 = e5m2 != 0;

  // ---- load: pass `it`, row group g = it * 16 + warp * 2 + lane / 16, rows 4g .. 4g + 3
  uint4 v[2][4];
#pragma unroll
  for (int it = 0; it < 2; ++it) {
    const int g = it * 16 + warp * 2 + (lane >> 4);
#pragma unroll
    for (int r = 0; r < 4; ++r)
      v[it][r] = *reinterpret_cast<const uint4*>(x + static_cast<int64_t>(row0 + 4 * g + r) * ldx + col0 + chunk * 8);
  }
  // ---- maxima: per row (over the 16 lanes that share it) and per column pair (over this thread's rows)
  uint32_t rm[8];                               // row 4 * it + r of this thread
  uint32_t cm[4] = {0u, 0u, 0u, 0u};
#pragma unroll
  for (int it = 0; it < 2; ++it)
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const uint32_t a0 = habs2_bits<BF16>(v[it][r].x), a1 = habs2_bits<BF16>(v[it][r].y);
      const uint32_t a2 = habs2_bits<BF16>(v[it][r].z), a3 = habs2_bits<BF16>(v[it][r].w);
      cm[0] = hmax2_bits<BF16>(cm[0], a0);
      cm[1] = hmax2_bits<BF16>(cm[1], a1);
      cm[2] = hmax2_bits<BF16>(cm[2], a2);
      cm[3] = hmax2_bits<BF16>(cm[3], a3);
      rm[4 * it + r] = hmax2_bits<BF16>(hmax2_bits<BF16>(a0, a1), hmax2_bits<BF16>(a2, a3));
    }
  if (qt != nullptr || SQUARE) {
#pragma unroll
    for (int w = 0; w < 4; ++w) cm[w] = hmax2_bits<BF16>(cm[w], __shfl_xor_sync(0xffffffffu, cm[w], 16));
    if (lane < 16) {
#pragma unroll
      for (int w = 0; w < 4; ++w) colred[warp][chunk * 4 + w] = cm[w];
    }
  }
  float tile_scale = 1.f;
  if constexpr (SQUARE) {
    __syncthreads();
    // one scale for the tile: maximum over all packed column maxima
    uint32_t m = 0u;
    if (tid < 64) {
#pragma unroll
      for (int w = 0; w < kThreads / 32; ++w) m = hmax2_bits<BF16>(m, colred[w][tid]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = hmax2_bits<BF16>(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (lane == 0) red[warp] = fmaxf(h_lo<BF16>(m), h_hi<BF16>(m));
    __syncthreads();
    const float amax = fmaxf(red[0], red[1]);
    tile_scale = compute_scale(amax, eps, fp8_max);
    if (tid == 0) {
      sinv[mb * KB + kb] = 1.f / tile_scale;
      if (sinv_t) sinv_t[kb * MB + mb] = 1.f / tile_scale;
    }
  }
  float row_scale = 1.f;                        // of row (lane >> 1) & 7
  if constexpr (!SQUARE) {
    const uint32_t m = max_rows8(rm, lane, [](uint32_t a, uint32_t b) { return hmax2_bits<BF16>(a, b); });
    row_scale = compute_scale(fmaxf(h_lo<BF16>(m), h_hi<BF16>(m)), eps, fp8_max);
    const int k = (lane >> 1) & 7;
    if ((lane & 1) == 0)
      sinv[(static_cast<int64_t>(mb) * KB + kb) * kTile + 4 * ((k >> 2) * 16 + warp * 2 + (lane >> 4)) + (k & 3)] =
          1.f / row_scale;
  }
  // ---- q: one scale per row (or the tile's), 8 bytes per thread and row
#pragma unroll
  for (int it = 0; it < 2; ++it) {
    const int g = it * 16 + warp * 2 + (lane >> 4);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      float scale = tile_scale;
      if constexpr (!SQUARE) scale = __shfl_sync(0xffffffffu, row_scale, (lane & 16) | ((4 * it + r) << 1));
      const uint32_t w[4] = {v[it][r].x, v[it][r].y, v[it][r].z, v[it][r].w};
      uint2 o;
      o.x = cvt_fp8x2(h_lo<BF16>(w[0]) * scale, h_hi<BF16>(w[0]) * scale, e5) |
            (cvt_fp8x2(h_lo<BF16>(w[1]) * scale, h_hi<BF16>(w[1]) * scale, e5) << 16);
      o.y = cvt_fp8x2(h_lo<BF16>(w[2]) * scale, h_hi<BF16>(w[2]) * scale, e5) |
            (cvt_fp8x2(h_lo<BF16>(w[3]) * scale, h_hi<BF16>(w[3]) * scale, e5) << 16);
      *reinterpret_cast<uint2*>(q + static_cast<int64_t>(row0 + 4 * g + r) * K + col0 + chunk * 8) = o;
    }
  }
  if (qt == nullptr) return;
  // ---- q^T: one scale per column (or the tile's)
  if constexpr (!SQUARE) {
    __syncthreads();
    if (tid < 64) {
      uint32_t m = 0u;
#pragma unroll
      for (int w = 0; w < kThreads / 32; ++w) m = hmax2_bits<BF16>(m, colred[w][tid]);
      const float s0 = compute_scale(h_lo<BF16>(m), eps, fp8_max), s1 = compute_scale(h_hi<BF16>(m), eps, fp8_max);
      col_scale[2 * tid] = s0;
      col_scale[2 * tid + 1] = s1;
      float* st = sinv_t + (static_cast<int64_t>(kb) * MB + mb) * kTile + 2 * tid;
      st[0] = 1.f / s0;
      st[1] = 1.f / s1;
    }
    __syncthreads();
  }
  // a thread's 4 rows of one column are one word of row c of the transposed tile; word g of row c
  // sits at (g ^ swizzle(c)) so that the lanes of a warp hit different banks
#pragma unroll
  for (int it = 0; it < 2; ++it) {
    const int g = it * 16 + warp * 2 + (lane >> 4);
    uint32_t w[4][4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      w[r][0] = v[it][r].x;
      w[r][1] = v[it][r].y;
      w[r][2] = v[it][r].z;
      w[r][3] = v[it][r].w;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int c = chunk * 8 + j;
      const float scale = SQUARE ? tile_scale : col_scale[c];
      float f[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) f[r] = ((j & 1) ? h_hi<BF16>(w[r][j >> 1]) : h_lo<BF16>(w[r][j >> 1])) * scale;
      const uint32_t word = cvt_fp8x2(f[0], f[1], e5) | (cvt_fp8x2(f[2], f[3], e5) << 16);
      tile_t[c * 32 + (g ^ ((chunk * 4) & 31))] = word;
    }
  }
  __syncthreads();
  // rows of q^T: 8 x 16 bytes each
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int idx = tid + k * kThreads;          // 0 .. 1023
    const int c = idx >> 3, part = idx & 7;      // row of q^T, 16-byte piece
    const int phys = (part * 4) ^ (((c >> 3) * 4) & 31);
    const uint4 o = *reinterpret_cast<const uint4*>(&tile_t[c * 32 + phys]);
    *reinterpret_cast<uint4*>(qt + static_cast<int64_t>(col0 + c) * M + row0 + part * 16) = o;
  }
}

// ---------------------------------------------------------------------------------------------
// Any other shape, pitch or alignment, and fp32 inputs: the same register tile with guards. What is outside
// the matrix reads as zero, so the scales of the rows and columns that pad the last blocks are those of
// zeros. Maxima ignore NaN. An 8-column chunk is read with 16-byte loads where the row pitch and the base
// allow them, elsewhere with the widest loads its row allows; q leaves as 8-byte stores where K allows them. Rows whose
// start may be on any byte (q with K % 8 != 0, q^T with M % 8 != 0) are written from the shared tile, half a warp per
// row, in aligned 8-byte stores and one byte per lane for the two ends.
// Bound by instruction issue, not by memory: 5000 x 8192 bf16, 1x128 with the transpose, takes 37 us (4.4 TB/s); 44 us
// with a butterfly and sixteen divisions per row, 70 us with one thread per column for the column maxima and byte
// stores of q^T, 73 us with fp32 maxima and every row of q^T through the word writer (2.7 instructions per cycle and SM
// in all of these). Rows that start on any element, 5001 x 8191 bf16: 63 us with the transpose, 45 without (126 and 87 with
// element loads and a warp per row of 4-byte stores; 87 and 66 with a shared tile read and written element by element);
// few rows, 33 x 4096, 128 x 128 with the transpose: 4.2 us (7.2; 4.6).
// ---------------------------------------------------------------------------------------------
template <typename T>
struct Chunk8 {      // 8 consecutive elements of a row, as they are in memory
  static constexpr bool BF16 = std::is_same<T, __nv_bfloat16>::value;
  static constexpr int NW = 4;                 // words; maxima are taken on pairs
  uint32_t w[NW];
  __device__ __forceinline__ uint32_t abs_word(int i) const { return w[i] & 0x7FFF7FFFu; }
  static __device__ __forceinline__ uint32_t vmax(uint32_t a, uint32_t b) {   // NaN in one operand: the other
    uint32_t r;
    if constexpr (BF16) asm("max.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    else asm("max.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
  }
  static __device__ __forceinline__ float column(uint32_t m, int c) { return (c & 1) ? h_hi<BF16>(m) : h_lo<BF16>(m); }
  static __device__ __forceinline__ float row(uint32_t m) { return fmaxf(h_lo<BF16>(m), h_hi<BF16>(m)); }
  __device__ __forceinline__ void zero() { w[0] = w[1] = w[2] = w[3] = 0u; }
  __device__ __forceinline__ void load_vec(const T* p) {
    const uint4 v = *reinterpret_cast<const uint4*>(p);
    w[0] = v.x, w[1] = v.y, w[2] = v.z, w[3] = v.w;
  }
  __device__ __forceinline__ void load_any(const T* p) {      // 8 elements on any element boundary
    const uintptr_t a = reinterpret_cast<uintptr_t>(p);
    if ((a & 7) == 0) {
      const uint2 lo = reinterpret_cast<const uint2*>(p)[0], hi = reinterpret_cast<const uint2*>(p)[1];
      w[0] = lo.x, w[1] = lo.y, w[2] = hi.x, w[3] = hi.y;
    } else if ((a & 3) == 0) {
#pragma unroll
      for (int j = 0; j < 4; ++j) w[j] = reinterpret_cast<const uint32_t*>(p)[j];
    } else {
      const uint16_t* h = reinterpret_cast<const uint16_t*>(p);
      const uint32_t* m = reinterpret_cast<const uint32_t*>(h + 1);
      const uint32_t m0 = m[0], m1 = m[1], m2 = m[2];
      w[0] = h[0] | (m0 << 16);
      w[1] = __funnelshift_r(m0, m1, 16);
      w[2] = __funnelshift_r(m1, m2, 16);
      w[3] = (m2 >> 16) | (static_cast<uint32_t>(h[7]) << 16);
    }
  }
  __device__ __forceinline__ void load_some(const T* p, int n) {
    zero();
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (j < n) w[j >> 1] |= static_cast<uint32_t>(reinterpret_cast<const uint16_t*>(p)[j]) << (16 * (j & 1));
  }
  __device__ __forceinline__ float get(int j) const {
    return (j & 1) ? h_hi<BF16>(w[j >> 1]) : h_lo<BF16>(w[j >> 1]);
  }
};
template <>
struct Chunk8<float> {
  static constexpr int NW = 8;
  float w[NW];
  __device__ __forceinline__ uint32_t abs_word(int i) const { return __float_as_uint(fabsf(w[i])); }
  static __device__ __forceinline__ uint32_t vmax(uint32_t a, uint32_t b) {
    return __float_as_uint(fmaxf(__uint_as_float(a), __uint_as_float(b)));
  }
  static __device__ __forceinline__ float column(uint32_t m, int) { return __uint_as_float(m); }
  static __device__ __forceinline__ float row(uint32_t m) { return __uint_as_float(m); }
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int j = 0; j < 8; ++j) w[j] = 0.f;
  }
  __device__ __forceinline__ void load_vec(const float* p) {
    const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
    w[0] = a.x, w[1] = a.y, w[2] = a.z, w[3] = a.w;
    w[4] = b.x, w[5] = b.y, w[6] = b.z, w[7] = b.w;
  }
  __device__ __forceinline__ void load_any(const float* p) {
    if ((reinterpret_cast<uintptr_t>(p) & 7) == 0) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 v = reinterpret_cast<const float2*>(p)[j];
        w[2 * j] = v.x, w[2 * j + 1] = v.y;
      }
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) w[j] = p[j];
    }
  }
  __device__ __forceinline__ void load_some(const float* p, int n) {
    zero();
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (j < n) w[j] = p[j];
  }
  __device__ __forceinline__ float get(int j) const { return w[j]; }
};

// A row of a 128 x 128-byte shared tile (word i at i ^ swz) -> n bytes at dst, any alignment; half a warp, l = 0 .. 15.
// What lies between the first and the last 8-byte boundary leaves as aligned 8-byte stores, each put together from three
// words of the tile; the at most 14 bytes around it as one byte per lane.
__device__ __forceinline__ void store_tile_row(const uint32_t* tile_row, int swz, uint8_t* dst, int n, int l) {
  const int head = min(n, static_cast<int>((0 - reinterpret_cast<uintptr_t>(dst)) & 7));
  const int body = (n - head) >> 3, tail = (n - head) & 7;
  if (l < body) {
    const int o = head + 8 * l, k = o >> 2, s = 8 * (o & 3);
    // (o + 7 <= 127: word k + 2 is beyond the row only where s is 0 and nothing of it is used)
    const uint32_t w0 = tile_row[k ^ swz], w1 = tile_row[(k + 1) ^ swz], w2 = tile_row[((k + 2) & 31) ^ swz];
    *reinterpret_cast<uint2*>(dst + o) = make_uint2(__funnelshift_r(w0, w1, s), __funnelshift_r(w1, w2, s));
  }
  if (l < head + tail) {
    const int b = l < head ? l : n - head - tail + l;
    dst[b] = static_cast<uint8_t>(tile_row[(b >> 2) ^ swz] >> (8 * (b & 3)));
  }
}

template <typename T, bool SQUARE>
__global__ void __launch_bounds__(kThreads, sizeof(T) == 2 ? 3 : 2) quant_ragged_kernel(
    const T* __restrict__ x, int64_t ldx, uint8_t* __restrict__ q, uint8_t* __restrict__ qt,
    float* __restrict__ sinv, float* __restrict__ sinv_t, int M, int K, float eps, int e5m2,
    int64_t batch_stride_x, int64_t batch_stride_q, int64_t batch_stride_s) {
  __shared__ __align__(16) uint32_t colred[kThreads / 32][16 * Chunk8<T>::NW];   // column maxima per warp
  __shared__ float col_scale[kTile];
  __shared__ float red[kThreads / 32];
  __shared__ __align__(16) uint32_t tile[kTile * 32];     // q or q^T: 128 rows x 128 bytes
  const int kb = blockIdx.x, mb = blockIdx.y, bz = blockIdx.z;
  const int MB = gridDim.y, KB = gridDim.x;
  x += bz * batch_stride_x;
  q += bz * batch_stride_q;
  if (qt) qt += bz * batch_stride_q;
  sinv += bz * batch_stride_s;
  if (sinv_t) sinv_t += bz * batch_stride_s;
  const int row0 = mb * kTile, col0 = kb * kTile;
  const int rows = min(kTile, M - row0), cols = min(kTile, K - col0);
  const float fp8_max = e5m2 ? 57344.f : 448.f;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int chunk = lane & 15;
  const bool e5 = e5m2 != 0;
  const int ncol = min(8, cols - chunk * 8);              // columns of this thread's chunk inside the matrix
  const bool vec_x = ldx % (16 / static_cast<int>(sizeof(T))) == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0;
  const bool vec_q = (K & 7) == 0 && (reinterpret_cast<uintptr_t>(q) & 7) == 0;
  const bool vec_qt = (M & 15) == 0 && (reinterpret_cast<uintptr_t>(qt) & 15) == 0 && rows == kTile;
  const bool vec8_qt = (M & 7) == 0 && (reinterpret_cast<uintptr_t>(qt) & 7) == 0;

  // ---- load: pass `it`, row group g = it * 16 + warp * 2 + lane / 16, rows 4g .. 4g + 3
  Chunk8<T> v[2][4];
  auto load = [&](auto&& whole) {
#pragma unroll
    for (int it = 0; it < 2; ++it)
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int row = 4 * (it * 16 + warp * 2 + (lane >> 4)) + r;
        const T* src = x + static_cast<int64_t>(row0 + row) * ldx + col0 + chunk * 8;
        if (row < rows && ncol == 8) whole(v[it][r], src);
        else if (row < rows) v[it][r].load_some(src, ncol);
        else v[it][r].zero();
      }
  };
  if (vec_x) load([](Chunk8<T>& c, const T* p) { c.load_vec(p); });
  else load([](Chunk8<T>& c, const T* p) { c.load_any(p); });
  // ---- maxima
  using C = Chunk8<T>;
  constexpr int NW = C::NW;
  uint32_t rm[8];                               // row 4 * it + r of this thread
  uint32_t cm[NW];
#pragma unroll
  for (int j = 0; j < NW; ++j) cm[j] = 0u;
#pragma unroll
  for (int it = 0; it < 2; ++it)
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      uint32_t m = 0u;
#pragma unroll
      for (int j = 0; j < NW; ++j) {
        const uint32_t w = v[it][r].abs_word(j);
        m = C::vmax(m, w);
        cm[j] = C::vmax(cm[j], w);
      }
      rm[4 * it + r] = m;
    }
  float tile_scale = 1.f;
  if constexpr (SQUARE) {
    float m = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) m = fmaxf(m, C::row(rm[k]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (lane == 0) red[warp] = m;
    __syncthreads();
    float amax = red[0];
#pragma unroll
    for (int w = 1; w < kThreads / 32; ++w) amax = fmaxf(amax, red[w]);
    tile_scale = compute_scale(amax, eps, fp8_max);
    if (tid == 0) {
      sinv[mb * KB + kb] = 1.f / tile_scale;
      if (sinv_t) sinv_t[kb * MB + mb] = 1.f / tile_scale;
    }
  } else if (qt != nullptr) {
#pragma unroll
    for (int j = 0; j < NW; ++j) cm[j] = C::vmax(cm[j], __shfl_xor_sync(0xffffffffu, cm[j], 16));
    if (lane < 16) {
#pragma unroll
      for (int j = 0; j < NW; j += 4)
        *reinterpret_cast<uint4*>(&colred[warp][chunk * NW + j]) = make_uint4(cm[j], cm[j + 1], cm[j + 2], cm[j + 3]);
    }
  }
  float row_scale = 1.f;                        // of row (lane >> 1) & 7
  if constexpr (!SQUARE) {
    const uint32_t m = max_rows8(rm, lane, [](uint32_t a, uint32_t b) { return C::vmax(a, b); });
    row_scale = compute_scale(C::row(m), eps, fp8_max);
    const int k = (lane >> 1) & 7;
    if ((lane & 1) == 0)
      sinv[(static_cast<int64_t>(mb) * KB + kb) * kTile + 4 * ((k >> 2) * 16 + warp * 2 + (lane >> 4)) + (k & 3)] =
          1.f / row_scale;
  }
  // ---- q
#pragma unroll
  for (int it = 0; it < 2; ++it) {
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int row = 4 * (it * 16 + warp * 2 + (lane >> 4)) + r;
      float scale = tile_scale;
      if constexpr (!SQUARE) scale = __shfl_sync(0xffffffffu, row_scale, (lane & 16) | ((4 * it + r) << 1));
      const C& c = v[it][r];
      uint2 o;
      o.x = cvt_fp8x2(c.get(0) * scale, c.get(1) * scale, e5) | (cvt_fp8x2(c.get(2) * scale, c.get(3) * scale, e5) << 16);
      o.y = cvt_fp8x2(c.get(4) * scale, c.get(5) * scale, e5) | (cvt_fp8x2(c.get(6) * scale, c.get(7) * scale, e5) << 16);
      if (!vec_q) *reinterpret_cast<uint2*>(&tile[row * 32 + chunk * 2]) = o;
      else if (row < rows && ncol == 8)
        *reinterpret_cast<uint2*>(q + static_cast<int64_t>(row0 + row) * K + col0 + chunk * 8) = o;
    }
  }
  if (!vec_q) {
    __syncthreads();
    for (int r = tid >> 4; r < rows; r += kThreads / 16)
      store_tile_row(&tile[r * 32], 0, q + static_cast<int64_t>(row0 + r) * K + col0, cols, lane & 15);
  }
  if (qt == nullptr) return;
  // ---- q^T (the barrier also ends the reading of a staged q)
  __syncthreads();
  if constexpr (!SQUARE) {
    if (tid < kTile) {
      uint32_t m = 0u;
#pragma unroll
      for (int w = 0; w < kThreads / 32; ++w) m = C::vmax(m, colred[w][NW == 8 ? tid : tid >> 1]);
      const float s = compute_scale(C::column(m, tid), eps, fp8_max);
      col_scale[tid] = s;
      sinv_t[(static_cast<int64_t>(kb) * MB + mb) * kTile + tid] = 1.f / s;
    }
    __syncthreads();
  }
  // a thread's 4 rows of one column are one word of row c of the transposed tile; word g of row c
  // sits at g ^ swizzle(c) so that the lanes of a warp hit different banks
#pragma unroll
  for (int it = 0; it < 2; ++it) {
    const int g = it * 16 + warp * 2 + (lane >> 4);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int c = chunk * 8 + j;
      const float scale = SQUARE ? tile_scale : col_scale[c];
      tile[c * 32 + (g ^ ((chunk * 4) & 31))] =
          cvt_fp8x2(v[it][0].get(j) * scale, v[it][1].get(j) * scale, e5) |
          (cvt_fp8x2(v[it][2].get(j) * scale, v[it][3].get(j) * scale, e5) << 16);
    }
  }
  __syncthreads();
  if (vec_qt) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int idx = tid + k * kThreads;
      const int c = idx >> 3, part = idx & 7;
      if (c < cols)
        *reinterpret_cast<uint4*>(qt + static_cast<int64_t>(col0 + c) * M + row0 + part * 16) =
            *reinterpret_cast<const uint4*>(&tile[c * 32 + ((part * 4) ^ (((c >> 3) * 4) & 31))]);
    }
  } else if (vec8_qt) {
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int idx = tid + k * kThreads;
      const int c = idx >> 4, part = idx & 15;
      if (c < cols && part * 8 < rows)
        *reinterpret_cast<uint2*>(qt + static_cast<int64_t>(col0 + c) * M + row0 + part * 8) =
            *reinterpret_cast<const uint2*>(&tile[c * 32 + ((part * 2) ^ (((c >> 3) * 4) & 31))]);
    }
  } else {
    for (int c = tid >> 4; c < cols; c += kThreads / 16)
      store_tile_row(&tile[c * 32], ((c >> 3) * 4) & 31, qt + static_cast<int64_t>(col0 + c) * M + row0, rows, lane & 15);
  }
}

template <typename T, bool SQUARE>
int launch_quant(const void* x, int64_t ldx, void* q, void* qt, float* sinv, float* sinv_t, int M,
                 int K, int batch, float eps, int e5m2, cudaStream_t stream) {
  if constexpr (sizeof(T) == 2) {
    // whole tiles, 16-byte aligned rows everywhere: the register-tile kernel
    const bool aligned = M % kTile == 0 && K % kTile == 0 && ldx % 8 == 0 &&
                         ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(q) |
                           reinterpret_cast<uintptr_t>(qt)) & 15) == 0;
    if (aligned) {
      constexpr bool kBf16 = std::is_same<T, __nv_bfloat16>::value;
      dim3 grid(K / kTile, M / kTile, batch);
      const int64_t sstride = SQUARE ? static_cast<int64_t>(M / kTile) * (K / kTile)
                                     : static_cast<int64_t>(M / kTile) * (K / kTile) * kTile;
      quant_tile_kernel<kBf16, SQUARE><<<grid, kThreads, 0, stream>>>(
          reinterpret_cast<const uint16_t*>(x), ldx, reinterpret_cast<uint8_t*>(q), reinterpret_cast<uint8_t*>(qt),
          sinv, sinv_t, M, K, eps, e5m2, static_cast<int64_t>(M) * ldx, static_cast<int64_t>(M) * K, sstride);
      FLUXB_CUDA_OK(cudaGetLastError());
      g_launches.fetch_add(1, std::memory_order_relaxed);
      return kOk;
    }
  }
  const int MB = (M + kTile - 1) / kTile, KB = (K + kTile - 1) / kTile;
  dim3 grid(KB, MB, batch);
  const int64_t sstride = SQUARE ? static_cast<int64_t>(MB) * KB : static_cast<int64_t>(MB) * KB * kTile;
  quant_ragged_kernel<T, SQUARE><<<grid, kThreads, 0, stream>>>(
      reinterpret_cast<const T*>(x), ldx, reinterpret_cast<uint8_t*>(q),
      reinterpret_cast<uint8_t*>(qt), sinv, sinv_t, M, K, eps, e5m2,
      static_cast<int64_t>(M) * ldx, static_cast<int64_t>(M) * K, sstride);
  FLUXB_CUDA_OK(cudaGetLastError());
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return kOk;
}

}  // namespace
}  // namespace fluxb

using namespace fluxb;

extern "C" int fluxb_quantize_blockwise(const void* x, int64_t ldx, int in_dtype, void* q, void* qt,
                                        float* scale_inv, float* scale_inv_t, int M, int K,
                                        int batch, int square, float eps, int out_dtype,
                                        void* stream) {
  FLUXB_REQUIRE(x && q && scale_inv && M > 0 && K > 0 && batch > 0, "quantize arguments");
  FLUXB_REQUIRE((qt == nullptr) == (scale_inv_t == nullptr), "transposed output and scale go together");
  FLUXB_REQUIRE(out_dtype == FLUXB_FP8_E4M3 || out_dtype == FLUXB_FP8_E5M2, "fp8 output type");
  const int e5m2 = out_dtype == FLUXB_FP8_E5M2;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
#define FLUXB_QUANT(T)                                                                           \
  return square ? launch_quant<T, true>(x, ldx, q, qt, scale_inv, scale_inv_t, M, K, batch, eps, \
                                        e5m2, s)                                                 \
                : launch_quant<T, false>(x, ldx, q, qt, scale_inv, scale_inv_t, M, K, batch, eps, \
                                         e5m2, s)
  switch (in_dtype) {
    case FLUXB_BF16: FLUXB_QUANT(__nv_bfloat16);
    case FLUXB_FP16: FLUXB_QUANT(__half);
    case FLUXB_FP32: FLUXB_QUANT(float);
    default: return fail(kErrUnsupported, "quantize input must be bf16, fp16 or fp32");
  }
#undef FLUXB_QUANT
}
