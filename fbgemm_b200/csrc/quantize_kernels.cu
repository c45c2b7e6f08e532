// Row-wise quantizers that build the fused rows the lookups read: the step
// before the hot path.  The arithmetic follows the scalar reference so that the
// produced bytes are identical:
//   8-bit + fp32 scale,bias  src/QuantUtils.cc:677-718
//   N-bit + fp16 scale,bias  src/QuantUtils.cc:534-611
// (fp32 subtract, fp32 multiply by the inverse scale, round half to even).
//
// Bound by memory: 4 bytes read per column, 1/4 to 1 written.  The vector form
// (rows of whole, aligned float4s, up to 1024 columns) therefore reads a row
// once, into registers - 8, 16 or 32 lanes per row, several rows per lane group
// in flight - and stores the codes of four columns at a time; the row-by-row form
// with a second pass over the row and byte stores took 248 us for 1 M x 128
// columns (8-bit), where the memory needs 99 us.  Other widths keep that form.
#include <cuda_fp16.h>

#include "internal.h"

namespace fbgemm_b200 {

namespace {

constexpr int kQuantThreads = 256;

__device__ __forceinline__ void warp_min_max(const float* row, int cols, int lane, float* mn, float* mx) {
  float lo = __ldg(row), hi = lo;  // every lane seeds with element 0
  for (int c = lane; c < cols; c += 32) {
    const float v = __ldg(row + c);
    lo = fminf(lo, v);
    hi = fmaxf(hi, v);
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, d));
    hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, d));
  }
  *mn = lo;
  *mx = hi;
}

// Rows are only byte-aligned in general: write a 32-bit word byte by byte.
__device__ __forceinline__ void store_u32_bytes(uint8_t* dst, uint32_t v) {
  dst[0] = (uint8_t)(v & 0xffu);
  dst[1] = (uint8_t)((v >> 8) & 0xffu);
  dst[2] = (uint8_t)((v >> 16) & 0xffu);
  dst[3] = (uint8_t)(v >> 24);
}

// Scale, bias and codes of one row from its minimum and maximum.
template <int BITS, bool FP32_SB>
struct Coder {
  float mn, inv;
  uint32_t sb[FP32_SB ? 2 : 1];  // scale, bias as they are stored

  __device__ __forceinline__ void init(float lo, float hi) {
    if constexpr (FP32_SB) {
      mn = lo;
      const float range = __fsub_rn(hi, lo);
      sb[0] = __float_as_uint(__fdiv_rn(range, 255.0f));
      sb[1] = __float_as_uint(lo);
      inv = __fdiv_rn(255.0f, __fadd_rn(range, 1e-8f));
    } else {
      constexpr int QMAX = (1 << BITS) - 1;
      // the bias is stored as fp16: round the minimum first
      const __half mn_h = __float2half_rn(lo);
      mn = __half2float(mn_h);
      const float range = __fsub_rn(hi, mn);
      // The scale is stored as fp16 too; quantize with the value a reader will see.
      __half scale_h = __float2half_rn(range == 0.f ? 1.0f : __fdiv_rn(range, (float)QMAX));
      float scale = __half2float(scale_h);
      if (scale == 0.f) {
        scale = 1.0f;
        scale_h = __ushort_as_half((unsigned short)0x3C00);
      }
      inv = __fdiv_rn(1.0f, scale);
      if (isinf(inv)) {
        inv = 1.0f;
        scale_h = __ushort_as_half((unsigned short)0x3C00);
      }
      sb[0] = (uint32_t)__half_as_ushort(scale_h) | ((uint32_t)__half_as_ushort(mn_h) << 16);
    }
  }
  __device__ __forceinline__ uint32_t code(float x) const {
    const int q = __float2int_rn(__fmul_rn(__fsub_rn(x, mn), inv));
    if constexpr (FP32_SB) {
      return (uint32_t)q & 0xffu;
    } else {
      return (uint32_t)max(0, min(q, (1 << BITS) - 1));
    }
  }
};

// Rows of whole, aligned float4s.  LPR lanes per row, NV float4s per lane, R
// rows per lane group, all their loads issued before the first use.
template <int BITS, bool FP32_SB, int LPR, int NV, int R>
__global__ void __launch_bounds__(kQuantThreads)
quantize_vector_kernel(const float* __restrict__ in, int64_t rows, int cols, uint8_t* __restrict__ out) {
  const int gl = threadIdx.x % LPR;
  const int64_t group = (int64_t)blockIdx.x * (kQuantThreads / LPR) + threadIdx.x / LPR;
  const int64_t groups = (int64_t)gridDim.x * (kQuantThreads / LPR);
  const int n4 = cols >> 2;
  const int data_bytes = cols * BITS / 8;
  const int64_t pitch = data_bytes + (FP32_SB ? 8 : 4);
  float4 v[R][NV];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int64_t row = min(group + r * groups, rows - 1);
    const float4* x = reinterpret_cast<const float4*>(in + row * cols);
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int k = gl + i * LPR;
      v[r][i] = __ldcs(x + (k < n4 ? k : 0));  // lanes beyond the row repeat its first columns
    }
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    float lo = v[r][0].x, hi = lo;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      lo = fminf(fminf(lo, fminf(v[r][i].x, v[r][i].y)), fminf(v[r][i].z, v[r][i].w));
      hi = fmaxf(fmaxf(hi, fmaxf(v[r][i].x, v[r][i].y)), fmaxf(v[r][i].z, v[r][i].w));
    }
#pragma unroll
    for (int d = LPR / 2; d > 0; d >>= 1) {
      lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, d));
      hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, d));
    }
    const int64_t row = group + r * groups;
    if (row >= rows) {
      continue;
    }
    Coder<BITS, FP32_SB> coder;
    coder.init(lo, hi);
    uint8_t* o = out + row * pitch;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int k = gl + i * LPR;
      if (k < n4) {
        const uint32_t c = coder.code(v[r][i].x) | (coder.code(v[r][i].y) << BITS) | (coder.code(v[r][i].z) << (2 * BITS)) |
            (coder.code(v[r][i].w) << (3 * BITS));
        if constexpr (BITS == 8) {
          reinterpret_cast<uint32_t*>(o)[k] = c;
        } else if constexpr (BITS == 4) {
          reinterpret_cast<uint16_t*>(o)[k] = (uint16_t)c;
        } else {
          o[k] = (uint8_t)c;
        }
      }
    }
    if (gl < (FP32_SB ? 2 : 1)) {
      uint8_t* s = o + data_bytes + 4 * gl;
      const uint32_t w = coder.sb[FP32_SB ? gl : 0];
      if constexpr (BITS == 8) {
        *reinterpret_cast<uint32_t*>(s) = w;
      } else if constexpr (BITS == 4) {
        reinterpret_cast<uint16_t*>(s)[0] = (uint16_t)w;
        reinterpret_cast<uint16_t*>(s)[1] = (uint16_t)(w >> 16);
      } else {
        store_u32_bytes(s, w);
      }
    }
  }
}

// Any width and alignment, row by row: one warp per row, whole bytes per lane.
template <int BITS, bool FP32_SB>
__global__ void __launch_bounds__(kQuantThreads)
quantize_row_kernel(const float* __restrict__ in, int64_t rows, int cols, uint8_t* __restrict__ out) {
  constexpr int EPB = 8 / BITS;
  const int lane = threadIdx.x & 31;
  const int64_t row = (int64_t)blockIdx.x * (kQuantThreads / 32) + (threadIdx.x >> 5);
  if (row >= rows) {
    return;
  }
  const int data_bytes = cols / EPB;
  const float* x = in + row * cols;
  uint8_t* o = out + row * ((int64_t)data_bytes + (FP32_SB ? 8 : 4));
  float mn, mx;
  warp_min_max(x, cols, lane, &mn, &mx);
  Coder<BITS, FP32_SB> coder;
  coder.init(mn, mx);
  if (lane < (FP32_SB ? 2 : 1)) {
    store_u32_bytes(o + data_bytes + 4 * lane, coder.sb[FP32_SB ? lane : 0]);
  }
  for (int b = lane; b < data_bytes; b += 32) {
    uint32_t packed = 0;
#pragma unroll
    for (int e = 0; e < EPB; ++e) {
      packed |= coder.code(__ldg(x + b * EPB + e)) << (e * BITS);
    }
    o[b] = (uint8_t)packed;
  }
}

// The vector form where rows are whole float4s and codes can be stored four columns at a time.
template <int BITS, bool FP32_SB>
cudaError_t launch_quantize(const float* in, int64_t rows, int cols, uint8_t* out, cudaStream_t s) {
  const bool vector = cols % 4 == 0 && cols <= 1024 && reinterpret_cast<uintptr_t>(in) % 16 == 0 &&
      reinterpret_cast<uintptr_t>(out) % (BITS == 8 ? 4 : BITS == 4 ? 2 : 1) == 0;
  const int rows_per_block = !vector ? kQuantThreads / 32
      : cols <= 32                   ? kQuantThreads / 8 * 4
      : cols <= 64                   ? kQuantThreads / 16 * 4
      : cols <= 128                  ? kQuantThreads / 32 * 4
      : cols <= 256                  ? kQuantThreads / 32 * 2
                                     : kQuantThreads / 32;
  const int64_t blocks = (rows + rows_per_block - 1) / rows_per_block;
  if (blocks <= 0 || blocks > 0x7fffffffLL) {
    return cudaErrorInvalidValue;
  }
  void (*fn)(const float*, int64_t, int, uint8_t*) = !vector ? quantize_row_kernel<BITS, FP32_SB>
      : cols <= 32                                           ? quantize_vector_kernel<BITS, FP32_SB, 8, 1, 4>
      : cols <= 64                                           ? quantize_vector_kernel<BITS, FP32_SB, 16, 1, 4>
      : cols <= 128                                          ? quantize_vector_kernel<BITS, FP32_SB, 32, 1, 4>
      : cols <= 256                                          ? quantize_vector_kernel<BITS, FP32_SB, 32, 2, 2>
      : cols <= 512                                          ? quantize_vector_kernel<BITS, FP32_SB, 32, 4, 1>
                                                             : quantize_vector_kernel<BITS, FP32_SB, 32, 8, 1>;
  fn<<<(unsigned)blocks, kQuantThreads, 0, s>>>(in, rows, cols, out);
  g_launch_count.fetch_add(1, std::memory_order_relaxed);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_quantize_8bit(const float* in, int64_t rows, int cols, uint8_t* out, cudaStream_t s) {
  return launch_quantize<8, true>(in, rows, cols, out, s);
}

cudaError_t launch_quantize_nbit(int bit_rate, const float* in, int64_t rows, int cols, uint8_t* out, cudaStream_t s) {
  switch (bit_rate) {
    case 8: return launch_quantize<8, false>(in, rows, cols, out, s);
    case 4: return launch_quantize<4, false>(in, rows, cols, out, s);
    case 2: return launch_quantize<2, false>(in, rows, cols, out, s);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace fbgemm_b200
