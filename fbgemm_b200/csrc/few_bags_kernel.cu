// The pooled lookup of a handful of bags in one quantized table: a block per
// bag and 128 columns.
//
// A launch of few bags is a chain of trips to memory and nothing else: with a
// warp per bag (bag_kernel.cuh) a bag of 100 rows takes the chain index -> scale
// and row four times over, a dozen rows in flight.  Here every thread resolves a
// row, all rows of the bag (up to kRows at a time) are copied to shared memory
// at once, asynchronously, and a thread per column adds them up from there:
// offsets, indices, rows, one trip each.  10 bags of 100 rows, 8-bit D = 64 at
// 4 M rows: 11.1 / 4.6 us per launch, 23.4 / 15.6 called and awaited.
//
// Arithmetic as in the scalar reference, per column and in index order:
// acc = fma(w*scale, q, acc + w*bias).  Skipped rows (pruned, -1, out of range)
// take part with scale and bias 0, which leaves a sum as it is (no sum is ever -0).
#include "bag_kernel.cuh"

namespace fbgemm_b200 {
namespace bag {

namespace {

constexpr int kRows = kFewThreads;     // resolved at a time, one per thread
constexpr int kPitch = kFewColumns;    // bytes of a row in shared memory, at most

// The rows, where asynchronous copies (of four bytes and more) cannot take them: in units of T, as many lanes a row as it
// has units, eight loads of each lane's issued before the first is stored.
template <typename T, int PITCH>
__device__ __forceinline__ void copy_units(const uint8_t* const* at, uint8_t (*to)[PITCH], int rows, int tile_at, int bytes) {
  constexpr int kInFlight = 8;
  const int units = (bytes + (int)sizeof(T) - 1) / (int)sizeof(T);
  const int log_lanes = units <= 8 ? 3 : units <= 16 ? 4 : 5;
  const int unit = threadIdx.x & ((1 << log_lanes) - 1), step = kFewThreads >> log_lanes;
  for (int u = unit; u < units; u += 32) {
    for (int r0 = threadIdx.x >> log_lanes; r0 < rows; r0 += kInFlight * step) {
      T v[kInFlight];
#pragma unroll
      for (int k = 0; k < kInFlight; ++k) {
        const int r = r0 + k * step;
        const uint8_t* row = r < rows ? at[r] : nullptr;
        v[k] = row ? __ldg(reinterpret_cast<const T*>(row + tile_at) + u) : (T)0;
      }
#pragma unroll
      for (int k = 0; k < kInFlight; ++k) {
        const int r = r0 + k * step;
        if (r < rows) {
          reinterpret_cast<T*>(to[r])[u] = v[k];
        }
      }
    }
  }
}

template <int FMT>
__global__ void __launch_bounds__(kFewThreads) few_bags_kernel(const __grid_constant__ BagCall c) {
  constexpr int kPitchBytes = kPitch * FMT / 8;
  constexpr int kWords = kPitchBytes / 4;  // of a row: 32, 16 or 8
  __shared__ __align__(16) uint8_t rows_s[kRows][kPitchBytes];
  __shared__ const uint8_t* at_s[kRows];
  __shared__ float2 sb_s[kRows];
  __shared__ long long sums_s[kFewThreads / 32];
  const BagTable& p = c.t;
  const int tid = threadIdx.x;
  const int64_t bag = blockIdx.x;
  const bool idx64 = p.flags & kIdx64;
  const bool off64 = p.flags & kOff64;
  const bool half_sb = FMT != kInt8 || (p.flags & kSbFirst);
  const int tile_at = blockIdx.y * kPitchBytes;
  const int bytes = min(p.data_bytes - tile_at, kPitchBytes);  // of this tile
  wait_for_previous_launch();

  int64_t start;
  int len;
  if (p.flags & kLengths) {
    long long sum = 0;  // of the bags before this one
    for (int64_t i = tid; i < bag; i += kFewThreads) {
      sum += max((int)load_int(p.offsets, i, off64), 0);  // the reference narrows to 32 bits too
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
      sum += __shfl_xor_sync(0xffffffffu, sum, d);
    }
    if (tid % 32 == 0) {
      sums_s[tid / 32] = sum;
    }
    len = max((int)load_int(p.offsets, bag, off64), 0);
    __syncthreads();
    start = 0;
#pragma unroll
    for (int i = 0; i < kFewThreads / 32; ++i) {
      start += sums_s[i];
    }
    if (bag + 1 == p.bags && tid == 0 && blockIdx.y == 0 && start + len != p.index_size) {  // `return current == index_size`
      report(p.status, FBGEMM_B200_STATUS_SIZE_MISMATCH, p.bags, start + len, p.index_size);
    }
  } else {
    const bool rebase = !(p.flags & kAbsOffsets);
    const int64_t base = rebase ? load_int(p.offsets, 0, off64) : 0;
    const int64_t o0 = load_int(p.offsets, bag, off64), o1 = load_int(p.offsets, bag + 1, off64);
    if (rebase && bag == 0 && tid == 0 && blockIdx.y == 0) {
      const int64_t total = load_int(p.offsets, p.bags, off64) - base;
      if (total != p.index_size) {
        report(p.status, FBGEMM_B200_STATUS_SIZE_MISMATCH, p.bags, total, p.index_size);
      }
    }
    start = o0 - base;
    len = (int)(o1 - o0);
  }
  if (len < 0 || start < 0 || start + len > p.index_size) {  // never read past the caller's arrays
    if (tid == 0) {
      report(p.status, FBGEMM_B200_STATUS_BAG_OVERRUN, bag, start, len < 0 ? 0 : len);
    }
    start = len = 0;
  }

  // Whole words: the last one may run into scale and bias behind the payload, but not beyond the row.
  const bool by_words = few_by_words(p);
  const bool by_halves = few_by_halves(p);
  const int col = blockIdx.y * kPitch + tid;
  float acc = 0.f;
  for (int c0 = 0; c0 < len; c0 += kRows) {
    const int n = min(len - c0, kRows);
    // The row's address first, so that the copies start; its scale and bias arrive meanwhile.
    bool keep = false;
    float w = 1.f;
    uint32_t sb_lo = 0, sb_hi = 0;
    if (tid < n) {
      const int64_t pos = start + c0 + tid;
      int64_t id = load_int(p.indices, pos, idx64);
      keep = id >= 0 && id < p.data_size;
      if (!keep && !(id == -1 && (p.flags & kSbFirst))) {
        report(p.status, FBGEMM_B200_STATUS_BAD_INDEX, bag, pos, (int32_t)id);
      }
      if (p.flags & kWeighted) {
        w = __ldg(p.weights + (p.flags & kPositional ? (int64_t)(c0 + tid) : pos));
      }
      if ((p.flags & kPruned) && keep) {
        id = __ldg(p.cit + id);
        keep = id >= 0;
      }
      const uint8_t* row = keep ? p.data + id * p.stride : nullptr;
      at_s[tid] = row;
      if (keep) {
        sb_lo = load_u32(row + p.sb_off, p.sb_align);
        if (!half_sb) {
          sb_hi = load_u32(row + p.sb_off + 4, p.sb_align);
        }
      }
    }
    if (by_words) {
      __syncwarp();  // each warp copies the rows that its threads found (the block's rows, after a barrier, 0.7 us longer)
      const int first = tid / 32 * 32, last = min(n, first + 32), word = tid % kWords;
      for (int r = first + tid % 32 / kWords; r < last; r += 32 / kWords) {
        const uint8_t* row = at_s[r];
        if (row && 4 * word < bytes) {
          const uint32_t to = (uint32_t)__cvta_generic_to_shared(&rows_s[r][4 * word]);
          asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(to), "l"(row + tile_at + 4 * word) : "memory");
        }
      }
    } else {
      __syncthreads();
      if (by_halves) {
        copy_units<uint16_t, kPitchBytes>(at_s, rows_s, n, tile_at, bytes);
      } else {
        copy_units<uint8_t, kPitchBytes>(at_s, rows_s, n, tile_at, bytes);
      }
    }
    if (tid < n) {
      float scale = half_sb ? __half2float(__ushort_as_half((unsigned short)(sb_lo & 0xffffu))) : __uint_as_float(sb_lo);
      float bias = half_sb ? __half2float(__ushort_as_half((unsigned short)(sb_lo >> 16))) : __uint_as_float(sb_hi);
      if ((p.flags & kWeighted) && keep) {
        scale = __fmul_rn(w, scale);
        bias = __fmul_rn(w, bias);
      }
      sb_s[tid] = make_float2(scale, bias);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    if (tid < kPitch && col < p.cols) {
#pragma unroll 8
      for (int r = 0; r < n; ++r) {
        const float2 sb = sb_s[r];
        const uint32_t byte = rows_s[r][tid * FMT / 8];
        const uint32_t q = FMT == 8 ? byte : (byte >> (tid * FMT % 8)) & ((1u << (FMT % 8)) - 1u);
        // q as a float, exactly: planted in the mantissa of 2^23
        const float x = __fsub_rn(__uint_as_float(q | 0x4b000000u), 8388608.f);
        acc = __fmaf_rn(sb.x, x, __fadd_rn(acc, sb.y));
      }
    }
    __syncthreads();  // the rows are overwritten by the next ones
  }

  if (tid < kPitch && col < p.cols) {
    if ((p.flags & kNormalize) && len != 0) {
      acc = __fmul_rn(acc, __fdiv_rn(1.f, (float)len));
    }
    char* row = static_cast<char*>(p.out) + bag * p.out_pitch;
    if (p.flags & (kOutHalf | kOutBf16)) {
      reinterpret_cast<uint16_t*>(row)[col] = (uint16_t)to_16bit(acc, p.flags & kOutBf16);
    } else {
      reinterpret_cast<float*>(row)[col] = acc;
    }
  }
}

}  // namespace

BagFn few_bags(int fmt) {
  return fmt == kInt8 ? few_bags_kernel<kInt8> : fmt == kInt4 ? few_bags_kernel<kInt4> : few_bags_kernel<kInt2>;
}

}  // namespace bag
}  // namespace fbgemm_b200
