// Row-wise quantizers that build the fused rows the lookups read: the step
// before the hot path.  The arithmetic follows the scalar reference so that the
// produced bytes are identical:
//   8-bit + fp32 scale,bias  src/QuantUtils.cc:677-718
//   N-bit + fp16 scale,bias  src/QuantUtils.cc:534-611
// (fp32 subtract, fp32 multiply by the inverse scale, round half to even).
//
// Bound by memory: 4 bytes read per column, 1/4 to 1 written.  Rows follow one
// another without gaps, so a block takes 16 KB of them as one stretch of bytes,
// whatever their width: 16-byte asynchronous copies bring them to shared memory,
// groups of 4 to 32 lanes (launch_quantize) quantize row by row from there into the bytes
// of the fused rows, and those leave as 16-byte stores of whole sectors.  8 blocks
// per SM keep 128 KB on their way.  A warp per row that read its row twice and
// stored single bytes took 248 us for 1 M x 128 columns (8-bit), rows held in
// registers and stored by words 129 us, this 101 us
// (a pass of the public call takes 119); memory needs 99 us.
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

__device__ __forceinline__ void copy_async(void* smem, const void* global, int bytes) {
  const uint32_t dst = (uint32_t)__cvta_generic_to_shared(smem);
  if (bytes == 16) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(global) : "memory");
  } else {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(global) : "memory");
  }
}

// Block b quantizes rows b * per_block onwards, which start 16-byte aligned on both sides if the tables do.  LPR lanes per row.
template <int BITS, bool FP32_SB, int LPR>
__global__ void __launch_bounds__(kQuantThreads)
quantize_block_kernel(const float* __restrict__ in, int64_t rows, int cols, uint8_t* __restrict__ out, int per_block) {
  extern __shared__ __align__(16) float smem[];
  constexpr int EPB = 8 / BITS;
  const int data_bytes = cols / EPB;
  const int pitch = data_bytes + (FP32_SB ? 8 : 4);
  const int64_t row0 = (int64_t)blockIdx.x * per_block;
  const int n = (int)min((int64_t)per_block, rows - row0);
  const float* x = in + row0 * cols;
  uint8_t* o = out + row0 * pitch;
  uint8_t* coded = reinterpret_cast<uint8_t*>(smem + (int64_t)per_block * cols);

  const int values = n * cols;
  int done = 0;
  if (reinterpret_cast<uintptr_t>(x) % 16 == 0) {
    done = values & ~3;
    for (int i = 4 * threadIdx.x; i < done; i += 4 * kQuantThreads) {
      copy_async(smem + i, x + i, 16);
    }
  }
  for (int i = done + threadIdx.x; i < values; i += kQuantThreads) {
    copy_async(smem + i, x + i, 4);
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();

  const int gl = threadIdx.x % LPR;
  const unsigned mask = LPR == 32 ? 0xffffffffu : ((1u << (LPR % 32)) - 1u) << (threadIdx.x % 32 / LPR * LPR);
  for (int r = threadIdx.x / LPR; r < n; r += kQuantThreads / LPR) {
    const float* row = smem + r * cols;
    uint8_t* c = coded + r * pitch;
    float lo = row[0], hi = lo;
    if (cols % 4 == 0) {
      for (int k = gl; k < cols / 4; k += LPR) {
        const float4 v = reinterpret_cast<const float4*>(row)[k];
        lo = fminf(fminf(lo, fminf(v.x, v.y)), fminf(v.z, v.w));
        hi = fmaxf(fmaxf(hi, fmaxf(v.x, v.y)), fmaxf(v.z, v.w));
      }
    } else {
      for (int k = gl; k < cols; k += LPR) {
        lo = fminf(lo, row[k]);
        hi = fmaxf(hi, row[k]);
      }
    }
#pragma unroll
    for (int d = LPR / 2; d > 0; d >>= 1) {
      lo = fminf(lo, __shfl_xor_sync(mask, lo, d));
      hi = fmaxf(hi, __shfl_xor_sync(mask, hi, d));
    }
    Coder<BITS, FP32_SB> coder;
    coder.init(lo, hi);
    if (cols % 4 == 0) {
      for (int k = gl; k < cols / 4; k += LPR) {
        const float4 v = reinterpret_cast<const float4*>(row)[k];
        const uint32_t four =
            coder.code(v.x) | (coder.code(v.y) << BITS) | (coder.code(v.z) << (2 * BITS)) | (coder.code(v.w) << (3 * BITS));
        if constexpr (BITS == 8) {
          reinterpret_cast<uint32_t*>(c)[k] = four;
        } else if constexpr (BITS == 4) {
          reinterpret_cast<uint16_t*>(c)[k] = (uint16_t)four;
        } else {
          c[k] = (uint8_t)four;
        }
      }
    } else {
      for (int b = gl; b < data_bytes; b += LPR) {
        uint32_t packed = 0;
#pragma unroll
        for (int e = 0; e < EPB; ++e) {
          packed |= coder.code(row[b * EPB + e]) << (e * BITS);
        }
        c[b] = (uint8_t)packed;
      }
    }
    if (gl < (FP32_SB ? 2 : 1)) {
      store_u32_bytes(c + data_bytes + 4 * gl, coder.sb[FP32_SB ? gl : 0]);
    }
  }
  __syncthreads();

  const int bytes = n * pitch;
  int copied = 0;
  if (reinterpret_cast<uintptr_t>(o) % 16 == 0) {
    copied = bytes & ~15;
    for (int i = 16 * threadIdx.x; i < copied; i += 16 * kQuantThreads) {
      *reinterpret_cast<uint4*>(o + i) = *reinterpret_cast<const uint4*>(coded + i);
    }
  }
  for (int i = copied + threadIdx.x; i < bytes; i += kQuantThreads) {
    o[i] = coded[i];
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

// By blocks of about 16 KB of whole rows that start on 16-byte boundaries on both sides; rows too wide for that row by
// row.  Lanes per row: as many as give every lane of the block a row to work on, so that narrow rows share a warp and
// its divisions and exchanges (4 M rows of 32 columns: 169 us with 8 lanes per row, 136 with 4).
template <int BITS, bool FP32_SB>
cudaError_t launch_quantize(const float* in, int64_t rows, int cols, uint8_t* out, cudaStream_t s) {
  constexpr int kBlockBytes = 16384;
  const int pitch = (int)((int64_t)cols * BITS / 8) + (FP32_SB ? 8 : 4);
  int step = 1;  // rows after which both sides are back on a 16-byte boundary
  while ((int64_t)step * pitch % 16 != 0 || (int64_t)step * cols % 4 != 0) {
    step *= 2;
  }
  const bool by_blocks = (int64_t)step * cols * 4 <= 2 * kBlockBytes;
  int per_block = kQuantThreads / 32;
  if (by_blocks) {
    per_block = kBlockBytes / (4 * cols) / step * step;
    per_block = per_block < step ? step : per_block > 512 ? 512 : per_block;
  }
  const int64_t blocks = (rows + per_block - 1) / per_block;
  if (blocks <= 0 || blocks > 0x7fffffffLL) {
    return cudaErrorInvalidValue;
  }
  if (by_blocks) {
    const int smem = per_block * (4 * cols + pitch);  // 44 KB at most: 32 KB and its codes, or 16 KB and theirs
    (per_block >= 64         ? quantize_block_kernel<BITS, FP32_SB, 4>
         : per_block > 16 ? quantize_block_kernel<BITS, FP32_SB, 8>
         : per_block > 8  ? quantize_block_kernel<BITS, FP32_SB, 16>
                          : quantize_block_kernel<BITS, FP32_SB, 32>)
        <<<(unsigned)blocks, kQuantThreads, smem, s>>>(in, rows, cols, out, per_block);
  } else {
    quantize_row_kernel<BITS, FP32_SB><<<(unsigned)blocks, kQuantThreads, 0, s>>>(in, rows, cols, out);
  }
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
