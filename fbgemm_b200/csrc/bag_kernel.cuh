// The pooled lookup: one lane group (a warp, or a half or quarter of one) per
// bag and column tile.
//
// Arithmetic as in the scalar reference (src/RefImplementations.cc:1290-1346,
// :1427-1541, :1617-1688, :1746-1822 of FBGEMM), so fp32 results are bit-equal:
// per output column, rows strictly in index order,
//     acc = fma(w*scale, q, acc + w*bias)
// two columns at a time with the packed fp32 instructions of sm_100
// (add.rn.f32x2, fma.rn.f32x2), which round each half like the scalar forms;
// sums are kept scaled by a power of two (see kDown).
//
// What bounds a lookup is the chain offsets -> index -> row of every bag and
// instruction issue, not bytes.  Hence the layout:
//  * The columns of a row are spread over the lane group, 1 to 16 bytes of
//    payload per lane.  A row in flight costs a lane one or two registers, so
//    4 or 8 rows of a bag are in flight with a full set of warps on the SM, 8 or
//    12 in the deep form (rows_ahead).
//  * Everything that is per row and not per column is done ONCE per row, by the
//    lane that owns the row in the walk over the bag's indices (one index per
//    lane at a time, coalesced): index load, range check, pruning map, weight,
//    scale and bias load, their conversion and weighting.  The results go
//    through shared memory: where the row lies, and ready for the packed
//    instructions {scale, scale of the second column, bias, bias} (see Places) -
//    one 16-byte broadcast load per row.
//  * Rows that an index does not name (pruned, -1, out of range) drop out of
//    that queue by ballot and popcount, so the row loop knows no skipped rows.
//  * Row loads are issued ahead of the arithmetic, four rows at a time.
#pragma once

#include <cuda_fp16.h>

#include <type_traits>

#include "internal.h"

namespace fbgemm_b200 {
namespace bag {

constexpr int kWarps = 4;
constexpr int kThreads = kWarps * 32;

using u64 = unsigned long long;

__device__ __forceinline__ u64 pack2(float lo, float hi) {
  u64 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(u64 v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ u64 add2(u64 a, u64 b) {
  u64 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ u64 mul2(u64 a, u64 b) {
  u64 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ u64 fma2(u64 a, u64 b, u64 c) {
  u64 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

__device__ __forceinline__ int64_t load_int(const void* p, int64_t i, bool is64) {
  return is64 ? (int64_t)__ldg(reinterpret_cast<const long long*>(p) + i)
              : (int64_t)__ldg(reinterpret_cast<const int*>(p) + i);
}

// Inlined: a call in the row walk would put the kernel's registers under the calling convention.
__device__ __forceinline__ void report(int32_t* st, int code, int64_t bag, int64_t pos, int64_t val) {
  if (atomicCAS(st, 0, code) == 0) {
    st[1] = (int32_t)bag;
    st[2] = (int32_t)pos;
    st[3] = (int32_t)val;
  }
}

// fp32 -> fp16 (round to nearest even, cpu_float2half_rn) or bf16 the way the
// reference does it: (bits + 0x8000) >> 16 (cpu_float2bfloat16,
// include/fbgemm/FloatConversion.h:312-315).
__device__ __forceinline__ uint32_t to_16bit(float v, bool bf16) {
  return bf16 ? (__float_as_uint(v) + 0x8000u) >> 16 : (uint32_t)__half_as_ushort(__float2half_rn(v));
}

// VB payload bytes of one row, as loaded by one lane.
template <int VB>
struct Bytes {
  uint32_t w[VB < 4 ? 1 : VB / 4];
  __device__ __forceinline__ void load(const uint8_t* p) {
    if constexpr (VB == 1) {
      w[0] = __ldg(p);
    } else if constexpr (VB == 2) {
      w[0] = __ldg(reinterpret_cast<const unsigned short*>(p));
    } else if constexpr (VB == 4) {
      w[0] = __ldg(reinterpret_cast<const uint32_t*>(p));
    } else if constexpr (VB == 8) {
      const uint2 v = __ldg(reinterpret_cast<const uint2*>(p));
      w[0] = v.x;
      w[1] = v.y;
    } else {
      const uint4 v = __ldg(reinterpret_cast<const uint4*>(p));
      w[0] = v.x;
      w[1] = v.y;
      w[2] = v.z;
      w[3] = v.w;
    }
  }
};

// Row formats.  Quantized rows are named by their bit width.
enum : int { kInt8 = 8, kInt4 = 4, kInt2 = 2, kF32 = 32, kF16 = 16, kBf16 = 17, kFp8 = 9 };
__host__ __device__ constexpr bool is_quantized(int fmt) { return fmt <= 8; }
__host__ __device__ constexpr int column_bits(int fmt) { return fmt == kBf16 ? 16 : fmt == kFp8 ? 8 : fmt; }

// Integer -> float without an instruction of its own.  Fewer than 25 bits that
// lie at bit p of a register and up are, read as fp32, the number q * 2^(p - 149)
// (subnormal, or of the least exponent, which has the same spacing): one logic
// instruction cuts a column out where it lies (8-bit: one byte permute takes it
// to bit 0), and the scale makes up for the power of two.  So that such a scale
// is an fp32 number the sums are kept as multiples of 2^-kDown of themselves:
//     acc' = fma(scale * 2^(149 - p - kDown), q * 2^(p - 149), acc' + bias * 2^-kDown)
// and brought back by an exact multiplication at the end.  Every step rounds as
// the unscaled one does where neither form leaves fp32's normal range, which holds
// for all rows whose weighted scale and bias are zero or of magnitude 2^-68
// (3e-21) to 2^36 (7e10): all values are then multiples of 2^-91 (2^-149 scaled:
// exact where subnormal) and, over 2^31 positions, below 2^76.  A bag with a row
// of other values (infinite ones, NaN and weights of 1e-30 among them) is pooled
// once more, unscaled (pool_again).  kDown moves those 104 powers of two up and
// down: weights that decay, and softmax weights, are small far more often than
// embeddings are large.
// Before, each column's bits were planted in the mantissa of a power of two that
// a packed addition then subtracted.  One row of 8 columns a lane, issue cycles of
// a scheduler, rows and scales in shared memory: 8-bit 22.0 / 18.0, 4-bit 25.1 / 19.4.
// 64 mixed tables of 16 384 bags 1135 / 1069 us, 8 4-bit tables of 65 536 bags 635 / 610.
constexpr int kDown = 58;
constexpr float kSumUp = (float)(1ull << kDown);                                    // 2^kDown
constexpr float kBiasDown = 1.f / kSumUp;
constexpr float kScaleUp = (float)(1ull << 60) * (float)(1ull << (89 - kDown));     // 2^(149 - kDown)
constexpr int kLeast = kDown - 126, kMost = kDown - 22;                             // powers of two of the range

// Whether a weighted scale or bias is one that the scaled sums are not made for.
__device__ __forceinline__ bool out_of_scale(float x) {
  const uint32_t magnitude = __float_as_uint(x) << 1;
  return magnitude != 0 && magnitude - ((uint32_t)(127 + kLeast) << 24) >= ((uint32_t)(kMost - kLeast) << 24);
}

// Where column K of a chunk of COLS columns lies: kPlaces columns are cut out of
// one shifted word, each with a scale of its own.
template <int BITS, int COLS>
struct Places {
  static constexpr int kPlaces = BITS == 8 ? 1 : COLS >= 8 ? 4 : 2;
  template <int K>
  __device__ __forceinline__ static float value(const uint32_t* w) {
    constexpr int at = K * BITS % 32;
    constexpr int shift = at / (kPlaces * BITS) * (kPlaces * BITS);
    const uint32_t x = w[K * BITS / 32];
    if constexpr (BITS == 8) {
      return __uint_as_float(COLS == 1 ? x : __byte_perm(x, 0u, 0x4440u | (at / 8)));
    } else {
      return __uint_as_float((x >> shift) & (((1u << BITS) - 1u) << (at - shift)));
    }
  }
};

// How FP8 widens to fp32.
template <int FMT, int COLS>
struct Constants {
  __device__ __forceinline__ void init(const BagTable&) {}
};
// FP8 -> fp32 as Float8ToFloat_ref (src/RefImplementations.cc:184-215): the seven low bits shifted into fp32's
// exponent and mantissa, times 2^(127 - bias), sign OR-ed in.
template <int COLS>
struct Constants<kFp8, COLS> {
  float mult;
  int shift;
  __device__ __forceinline__ void init(const BagTable& p) {
    mult = __uint_as_float((uint32_t)(254 - p.fp8_exponent_bias) << 23);
    shift = 24 - (8 - p.fp8_exponent_bits);
  }
};

// The columns a lane owns of a row: CPL chunks of VB payload bytes, chunk c at
// byte (c * G + lane) * VB of the tile.  acc[] holds them as fp32 pairs: the
// columns of a chunk in order, or (where a chunk is one column) the columns of
// two chunks.
template <int FMT, int VB, int CPL>
struct Cols {
  static constexpr int BITS = column_bits(FMT);
  static constexpr int kPerChunk = VB * 8 / BITS;
  static constexpr int kPairs = kPerChunk * CPL / 2;
  static_assert(kPerChunk * CPL % 2 == 0, "whole pairs");
  static constexpr bool kQuantized = is_quantized(FMT);
  static constexpr bool kHalfSb = FMT != kInt8;  // 8-bit rows: only with scale and bias first
  using M = Constants<FMT, kPerChunk>;

  // Column k of an unquantized chunk.
  __device__ __forceinline__ static float value(const M& m, const uint32_t* w, int k) {
    const uint32_t x = w[k * BITS / 32] >> (k * BITS % 32);
    if constexpr (FMT == kF32) {
      return __uint_as_float(x);
    } else if constexpr (FMT == kF16) {
      return __half2float(__ushort_as_half((unsigned short)(x & 0xffffu)));
    } else if constexpr (FMT == kBf16) {
      return __uint_as_float(x << 16);
    } else {
      const float mag = __fmul_rn(__uint_as_float((x & 0x7fu) << m.shift), m.mult);
      return __uint_as_float(__float_as_uint(mag) | ((x & 0x80u) << 24));
    }
  }
  using P = Places<BITS, kPerChunk>;
  template <int K>
  __device__ __forceinline__ static void pool_chunk(u64* acc, const uint32_t* w, u64 s2, u64 further, u64 b2) {
    if constexpr (K < kPerChunk) {
      const u64 q = pack2(P::template value<K>(w), P::template value<K + 1>(w));
      acc[K / 2] = fma2(K % P::kPlaces < 2 ? s2 : further, q, add2(acc[K / 2], b2));
      pool_chunk<K + 2>(acc, w, s2, further, b2);
    }
  }
  // One row.  Quantized: acc' = fma(scale', q, acc' + bias'), `s2` the scales of the columns at places 0 and 1;
  // otherwise acc = fma(w, x, acc) with w in `s2` (src/RefImplementations.cc:1347-1424, :1543-1615).
  __device__ __forceinline__ static void pool(const M& m, u64 (&acc)[kPairs], const Bytes<VB> (&d)[CPL], u64 s2, u64 b2) {
    if constexpr (!is_quantized(FMT)) {
#pragma unroll
      for (int i = 0; i < kPairs; ++i) {
        constexpr int n = kPerChunk;
        const float lo = value(m, d[2 * i / n].w, 2 * i % n);
        const float hi = value(m, d[(2 * i + 1) / n].w, (2 * i + 1) % n);
        acc[i] = fma2(s2, pack2(lo, hi), acc[i]);
      }
    } else if constexpr (kPerChunk == 1) {
#pragma unroll
      for (int c = 0; c < CPL; c += 2) {
        const u64 q = pack2(P::template value<0>(d[c].w), P::template value<0>(d[c + 1].w));
        acc[c / 2] = fma2(s2, q, add2(acc[c / 2], b2));
      }
    } else {
      // the scales of places 2 and 3 (one multiplication instead of two shifts more)
      constexpr float down = 1.f / (1 << (2 * BITS % 32));
      const u64 further = P::kPlaces > 2 ? mul2(s2, pack2(down, down)) : s2;
#pragma unroll
      for (int c = 0; c < CPL; ++c) {
        pool_chunk<0>(acc + c * kPerChunk / 2, d[c].w, s2, further, b2);
      }
    }
  }
  // The same unscaled, column by column (pool_again).
  __device__ __forceinline__ static void pool_unscaled(float (&acc)[2 * kPairs], const Bytes<VB> (&d)[CPL], float scale,
                                                       float bias) {
#pragma unroll
    for (int k = 0; k < 2 * kPairs; ++k) {
      const int bit = k % kPerChunk * BITS;
      const uint32_t q = (d[k / kPerChunk].w[bit / 32] >> (bit % 32)) & ((1u << (BITS % 32)) - 1u);
      acc[k] = __fmaf_rn(scale, (float)q, __fadd_rn(acc[k], bias));
    }
  }
};

// Four little-endian bytes at p, whose address is a multiple of `align`.
__device__ __forceinline__ uint32_t load_u32(const uint8_t* p, int align) {
  if (align >= 4) {
    return __ldg(reinterpret_cast<const uint32_t*>(p));
  }
  if (align == 2) {
    const unsigned short* h = reinterpret_cast<const unsigned short*>(p);
    return (uint32_t)__ldg(h) | ((uint32_t)__ldg(h + 1) << 16);
  }
  return (uint32_t)__ldg(p) | ((uint32_t)__ldg(p + 1) << 8) | ((uint32_t)__ldg(p + 2) << 16) |
      ((uint32_t)__ldg(p + 3) << 24);
}

// Store N consecutive columns of an output row, all of them inside the row, at
// an address that is a multiple of `align` bytes or of the N columns' size.
template <int N>
__device__ __forceinline__ void store_f32(float* o, const float* v, int align) {
  if (N >= 4 && align >= 16) {
#pragma unroll
    for (int i = 0; i + 4 <= N; i += 4) {
      *reinterpret_cast<float4*>(o + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
    }
  } else if (N >= 2 && align >= 8) {
#pragma unroll
    for (int i = 0; i + 2 <= N; i += 2) {
      *reinterpret_cast<float2*>(o + i) = make_float2(v[i], v[i + 1]);
    }
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      o[i] = v[i];
    }
  }
}
template <int N>
__device__ __forceinline__ void store_u16(uint16_t* o, const uint32_t* h, int align) {
  if (N >= 8 && align >= 16) {
#pragma unroll
    for (int i = 0; i + 8 <= N; i += 8) {
      *reinterpret_cast<uint4*>(o + i) = make_uint4(h[i] | (h[i + 1] << 16), h[i + 2] | (h[i + 3] << 16),
                                                    h[i + 4] | (h[i + 5] << 16), h[i + 6] | (h[i + 7] << 16));
    }
  } else if (N >= 4 && align >= 8) {
#pragma unroll
    for (int i = 0; i + 4 <= N; i += 4) {
      *reinterpret_cast<uint2*>(o + i) = make_uint2(h[i] | (h[i + 1] << 16), h[i + 2] | (h[i + 3] << 16));
    }
  } else if (N >= 2 && align >= 4) {
#pragma unroll
    for (int i = 0; i + 2 <= N; i += 2) {
      *reinterpret_cast<uint32_t*>(o + i) = h[i] | (h[i + 1] << 16);
    }
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      o[i] = (uint16_t)h[i];
    }
  }
}

template <int N>
__device__ __forceinline__ void store_columns(const BagTable& p, char* row, int col0, const float* v) {
  const int left = p.cols - col0;
  if (p.flags & (kOutHalf | kOutBf16)) {
    const bool bf16 = p.flags & kOutBf16;
    uint16_t* o = reinterpret_cast<uint16_t*>(row) + col0;
    uint32_t h[N];
    if (!bf16 && N % 2 == 0) {
#pragma unroll
      for (int i = 0; i + 1 < N; i += 2) {
        const __half2 two = __floats2half2_rn(v[i], v[i + 1]);  // one instruction for both
        const uint32_t bits = *reinterpret_cast<const uint32_t*>(&two);
        h[i] = bits & 0xffffu;
        h[i + 1] = bits >> 16;
      }
    } else {
#pragma unroll
      for (int i = 0; i < N; ++i) {
        h[i] = to_16bit(v[i], bf16);
      }
    }
    if (left >= N) {
      store_u16<N>(o, h, p.out_align);
    } else {
#pragma unroll
      for (int i = 0; i < N; ++i) {
        if (i < left) {
          o[i] = (uint16_t)h[i];
        }
      }
    }
  } else {
    float* o = reinterpret_cast<float*>(row) + col0;
    if (left >= N) {
      store_f32<N>(o, v, p.out_align);
    } else {
#pragma unroll
      for (int i = 0; i < N; ++i) {
        if (i < left) {
          o[i] = v[i];
        }
      }
    }
  }
}

// Where rows lie: byte offsets from row 0, in 32 bits where the table allows
// (WIDE = false: one 32-bit addition per row and chunk, 10 % of the instructions
// less than 64-bit addresses), else in 64.
template <bool WIDE>
using Row = typename std::conditional<WIDE, unsigned long long, uint32_t>::type;

// Where a lane finds its chunks of a row; lanes whose chunk lies beyond the
// payload read chunk 0 instead and do not store.  OWN (one chunk a lane): where
// row 0 has the lane's chunk is an address of its own, opaque to the compiler,
// which otherwise adds row, chunk and table up anew for every row (three
// instructions instead of two).  It costs a register or two: see own_address.
template <int VB, int CPL, int G, bool WIDE, bool OWN>
struct LaneData {
  static_assert(!OWN || CPL == 1, "one address");
  const uint8_t* first;
  uint32_t at[CPL];  // from there
  __device__ __forceinline__ void init(const uint8_t* data, int tile_at, int gl, int data_bytes) {
    first = data;
#pragma unroll
    for (int c = 0; c < CPL; ++c) {
      const int a = tile_at + (c * G + gl) * VB;
      at[c] = a < data_bytes ? a : 0;
    }
    if constexpr (OWN) {
      asm volatile("mov.b64 %0, %1;" : "=l"(first) : "l"(data + at[0]));
    }
  }
  // Chunk c of the row whose payload starts at `row`.
  __device__ __forceinline__ const uint8_t* chunk(const uint8_t* row, const uint8_t* data, int c) const {
    return OWN ? first + (row - data) : row + at[c];
  }
  __device__ __forceinline__ void load(Bytes<VB> (&d)[CPL], Row<WIDE> row) const {
#pragma unroll
    for (int c = 0; c < CPL; ++c) {
      d[c].load(OWN ? first + row : first + (Row<WIDE>)(row + at[c]));
    }
  }
};

// Queue of a warp: the rows that its lanes found, in index order.
template <bool WIDE>
struct __align__(16) Queue {
  Row<WIDE> row[32];
  ulonglong2 sb[32];  // {scale of place 0, of place 1}, {bias, bias}; {weight, weight} of unquantized rows
};

// What a kernel is compiled for.
//  kLean  bags by offsets, weights per index, every index a row of the table
//  kFull  besides: -1 as a pruned index, no_bag, positional
//         weights, lengths in place of offsets
//  kMapped  besides: pruning maps (their part, unused, cost 64 table-batched tables 4 %, 3000 bags by lengths 2 %)
//  kWide  the same where positions, bags (31 bits) or row offsets (32) need more
// The lean form saves the queue's compaction and half of the tests, a tenth of
// the time of 65536 bags of 30 rows (8-bit D = 128 76.4 against 83.6 us).
enum : int { kLean = 0, kFull = 1, kWide = 2, kMapped = 3 };

// Groups of four rows whose loads are issued ahead of the arithmetic.  Measured on 65536 bags of 30 rows: with half
// warps per bag none is best for 4-bit rows (67.9 against 69.4 us at D = 128), one for 8- and 2-bit rows (82 against
// 102 us, 66 against 68); quarter warps want none, whole warps one.  Launches whose warps are all resident with more
// registers each (kDeep) take one more with whole warps.
__host__ __device__ constexpr int rows_ahead(int fmt, int g, bool deep) {
  return g == 32 ? (deep ? 2 : 1) : deep ? 1 : g == 16 && (fmt == kInt8 || fmt == kInt2) ? 1 : 0;
}

// Whether lanes keep an address of their own: kernels whose rows in flight leave registers for it.  us per call without /
// with: 8-bit 10 000 bags 13.0 / 12.5, pruned 2-bit 8192 bags 9.7 / 9.5, fp16 D = 64 1500 bags 3.15 / 2.92, 8 4-bit tables
// of 65 536 bags 616 / 605, 64 mixed ones of 16 384 1128 / 1121.  Beyond the line: 8-bit D = 128 on half warps of 40
// registers, 65 536 bags of 64 rows, 94.2 / 98.9; in the deep form fp32 D = 128 4000 bags 7.9 / 8.5, 8-bit D = 256 by lengths
// 1500 bags 5.7 / 6.3 (their rows in flight spill); several chunks a lane (8-bit D = 257, 4007 bags of 15 rows) 20.9 / 23.7.
__host__ __device__ constexpr bool own_address(int fmt, int vb, int cpl, int g, int mode, bool deep) {
  const int bytes_in_flight = vb * (rows_ahead(fmt, g, deep) + 1);
  const int most = deep ? (is_quantized(fmt) && mode != kLean ? 16 : 24) : is_quantized(fmt) && mode == kLean ? 8 : 0;
  return cpl == 1 && bytes_in_flight <= most;
}

// The stream's next launch may be set up while this one drains; it waits here until all results of this one are there.
__device__ __forceinline__ void wait_for_previous_launch() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void let_next_launch_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Where a bag starts, from the lengths alone (kLengths): the block adds up those of all bags before its own, coalesced
// and from L2, then every lane those between.
template <int G>
__device__ __forceinline__ void bag_from_lengths(const BagTable& p, int64_t first, int64_t bag, int64_t& start, int& length) {
  __shared__ long long sums[kWarps];
  const bool is64 = p.flags & kOff64;
  auto at = [&](int64_t i) {
    const int v = (int)load_int(p.offsets, i, is64);  // the reference narrows to 32 bits too
    return v < 0 ? 0 : v;
  };
  long long sum = 0;
#pragma unroll 4
  for (int64_t i = threadIdx.x; i < first; i += kThreads) {
    sum += at(i);
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    sum += __shfl_xor_sync(0xffffffffu, sum, d);
  }
  if (threadIdx.x % 32 == 0) {
    sums[threadIdx.x / 32] = sum;
  }
  __syncthreads();
  sum = 0;
#pragma unroll
  for (int i = 0; i < kWarps; ++i) {
    sum += sums[i];
  }
  if (first + kWarps * (32 / G) >= p.bags && threadIdx.x == 0) {  // the last block: `return current == index_size`
    long long total = sum;
    for (int64_t i = first; i < p.bags; ++i) {
      total += at(i);
    }
    if (total != p.index_size) {
      report(p.status, FBGEMM_B200_STATUS_SIZE_MISMATCH, p.bags, total, p.index_size);
    }
  }
  for (int64_t i = first; i < bag && i < p.bags; ++i) {
    sum += at(i);
  }
  start = sum;
  length = bag < p.bags ? at(bag) : 0;
}

// A bag pooled once more from its first position, one row at a time, with 64-bit row addresses and unscaled sums, where
// * its row-wise sparse map names rows beyond 32-bit offsets (several short maps may share one large table).  Rare, so it
//   costs the other bags one comparison per mapped row and no registers (11.3 us before and after for 8192 bags of 30
//   rows, 2-bit D = 128), where 64-bit addresses for every pruned table would cost each of their rows the wide form's
//   extra instructions;
// * a row's weighted scale or bias is out_of_scale.  A chain of two or three loads per row: a launch with one such bag of 20
//   rows takes 5 us longer, one whose weights are all 1e-30 two to three times as long (us, weights of 1 / 1e-30 and, while
//   the range was 2^-52 to 2^52, 1e-16 too: 8-bit 10 000 bags of 20 rows 10.1 / 20.5, 4-bit 4096 ragged bags 7.3 / 22.7,
//   2-bit pruned 8192 bags 9.2 / 30.0, 8 4-bit tables of 16 384 bags 142 / 424, 64 mixed ones of 512 49 / 83).  Kept small:
//   its instructions arrive with the first bag that needs them.  Four rows at a time 4096 ragged bags of which one is such
//   take 17.6 us instead of 14.5.
template <class C, int VB, int CPL, class Lane>
__device__ __forceinline__ void pool_again(const BagTable& p, const typename C::M& constants, const Lane& lane_data,
                                           int64_t start, int len, u64 (&acc)[C::kPairs]) {
  float sum[2 * C::kPairs];
#pragma unroll
  for (int k = 0; k < 2 * C::kPairs; ++k) {
    sum[k] = 0.f;
  }
#pragma unroll
  for (int k = 0; k < C::kPairs; ++k) {
    acc[k] = 0ull;
  }
#pragma unroll 1
  for (int c = 0; c < len; ++c) {
    int64_t idx = load_int(p.indices, start + c, p.flags & kIdx64);
    if (idx < 0 || idx >= p.data_size) {
      continue;
    }
    if (p.flags & kPruned) {
      const int32_t m = __ldg(p.cit + idx);
      if (m < 0) {
        continue;
      }
      idx = m;
    }
    const uint8_t* row = p.data + (uint64_t)idx * (uint64_t)p.stride;
    const float w = p.flags & kWeighted ? __ldg(p.weights + (p.flags & kPositional ? (int64_t)c : start + c)) : 1.f;
    Bytes<VB> d[CPL];
#pragma unroll
    for (int i = 0; i < CPL; ++i) {
      d[i].load(lane_data.chunk(row, p.data, i));
    }
    if constexpr (C::kQuantized) {
      const uint8_t* sb = row + p.sb_off;
      const uint32_t lo = load_u32(sb, p.sb_align);
      float scale, bias;
      if (C::kHalfSb || (p.flags & kSbFirst)) {
        scale = __half2float(__ushort_as_half((unsigned short)(lo & 0xffffu)));
        bias = __half2float(__ushort_as_half((unsigned short)(lo >> 16)));
      } else {
        scale = __uint_as_float(lo);
        bias = __uint_as_float(load_u32(sb + 4, p.sb_align));
      }
      if (p.flags & kWeighted) {
        scale = __fmul_rn(w, scale);
        bias = __fmul_rn(w, bias);
      }
      C::pool_unscaled(sum, d, scale, bias);
    } else {
      C::pool(constants, acc, d, pack2(w, w), 0ull);
    }
  }
  if constexpr (C::kQuantized) {
#pragma unroll
    for (int k = 0; k < C::kPairs; ++k) {
      acc[k] = pack2(sum[2 * k], sum[2 * k + 1]);
    }
  }
}

// One block's work on table `p`: bags block * kWarps * (32 / G) onwards, columns of tile `tile` of the row.
template <int FMT, int VB, int CPL, int G, int MODE, bool kDeep>
__device__ __forceinline__ void pool_bags(const BagTable& p, void* const* peers, uint32_t block, int tile,
                                          Queue<MODE == kWide> (&queues)[kWarps]) {
  constexpr bool WIDE = MODE == kWide, FULL = MODE != kLean, MAPS = WIDE || MODE == kMapped;
  constexpr int kAhead = rows_ahead(FMT, G, kDeep);
  using C = Cols<FMT, VB, CPL>;
  using Pos = typename std::conditional<WIDE, int64_t, int32_t>::type;  // bags and positions
  constexpr int kTileBytes = G * VB * CPL;
  constexpr unsigned kGroupMask = G == 32 ? 0xffffffffu : (1u << (G % 32)) - 1u;
  constexpr bool kQuantized = is_quantized(FMT);
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int gl = lane % G;
  const int grp = lane / G;
  Row<WIDE>* q_row = queues[warp].row + grp * G;
  ulonglong2* q_sb = queues[warp].sb + grp * G;
  const bool idx64 = p.flags & kIdx64;
  const bool off64 = p.flags & kOff64;
  const bool weighted = p.flags & kWeighted;
  const bool positional = FULL && (p.flags & kPositional);
  const bool pruned = MAPS && (p.flags & kPruned);
  const bool no_bag = FULL && (p.flags & kNoBag);
  const bool by_lengths = FULL && (p.flags & kLengths);
  const bool minus_one_skips = FULL && FMT != kFp8 && (p.flags & (kSbFirst | kNoBag)) == kSbFirst;
  const bool half_sb = FMT != kInt8 || (p.flags & kSbFirst);

  const Pos bag = (Pos)block * (kWarps * (32 / G)) + warp * (32 / G) + grp;
  LaneData<VB, CPL, G, WIDE, own_address(FMT, VB, CPL, G, MODE, kDeep)> lane_data;
  lane_data.init(p.data, tile * kTileBytes, gl, p.data_bytes);
  const uint8_t* sb_data = p.data + p.sb_off;
  typename C::M constants;
  constants.init(p);
  wait_for_previous_launch();

  Pos pos = 0;  // of this lane's next candidate: one in every G indices of the bag
  int len = 0;
  {
    int64_t start = 0;
    int bag_len = 0;
    if (by_lengths) {
      bag_from_lengths<G>(p, (int64_t)block * (kWarps * (32 / G)), bag, start, bag_len);
    } else {
      // rebasing to offsets[0] (the functor's convention) unless the offsets are absolute
      const bool rebase = !(p.flags & (kNoBag | kAbsOffsets));
      const int64_t off_base = rebase ? load_int(p.offsets, 0, off64) : 0;
      if (block == 0 && threadIdx.x == 0 && rebase) {
        // `return current == index_size` of the reference
        const int64_t total = load_int(p.offsets, p.bags, off64) - off_base;
        if (total != p.index_size) {
          report(p.status, FBGEMM_B200_STATUS_SIZE_MISMATCH, p.bags, total, p.index_size);
        }
      }
      if (bag < (Pos)p.bags) {
        // no_bag: output row m is the single row indices[m]
        const int64_t o0 = no_bag ? bag : load_int(p.offsets, bag, off64);
        const int64_t o1 = no_bag ? (int64_t)bag + 1 : load_int(p.offsets, (int64_t)bag + 1, off64);
        start = o0 - off_base;
        bag_len = (int)(o1 - o0);  // the reference narrows to 32 bits too
      }
    }
    // Offsets that step backwards: the reference, which walks the index array
    // with a running position, ends up past index_size and returns false.
    if (bag_len < 0 || start < 0 || start + bag_len > p.index_size) {
      if (gl == 0) {
        report(p.status, FBGEMM_B200_STATUS_BAG_OVERRUN, bag, start, bag_len < 0 ? 0 : bag_len);
      }
      start = bag_len = 0;  // never read past the caller's arrays
    }
    pos = (Pos)start + gl;
    len = bag_len;
  }
  // Uniform to the compiler too (a redux result, unlike a shuffle's): the row loop then branches without
  // reconvergence barriers and keeps its constants in uniform registers (2-bit D = 256 107 against 127 us).
  const int longest = (int)__reduce_max_sync(0xffffffffu, (unsigned)len);

  u64 acc[C::kPairs];
#pragma unroll
  for (int k = 0; k < C::kPairs; ++k) {
    acc[k] = 0ull;  // (+0.f, +0.f)
  }

  auto fetch = [&](int c) -> uint2 {
    uint2 r = make_uint2(0u, 0u);
    if (c < len) {
      if (idx64) {
        r = __ldg(static_cast<const uint2*>(p.indices) + pos);
      } else {
        r.x = __ldg(static_cast<const uint32_t*>(p.indices) + pos);
      }
    }
    return r;
  };
  uint2 raw = fetch(gl);
  bool again = false;  // a row of this lane's lies beyond 32-bit offsets, or is out_of_scale
#pragma unroll 1
  for (int c0 = 0; c0 < longest; c0 += G) {
    const int c = c0 + gl;
    const bool in_bag = c < len;
    float w = 1.f;
    if (weighted && in_bag) {
      w = __ldg(p.weights + (positional ? (Pos)c : pos));
    }
    bool keep;
    if constexpr (WIDE) {
      const long long v = idx64 ? (long long)(((u64)raw.y << 32) | raw.x) : (long long)(int)raw.x;
      keep = in_bag && (u64)v < (u64)p.data_size;
    } else {
      keep = in_bag && raw.y == 0 && raw.x < p.limit;
    }
    Row<WIDE> id = 0;
    if (keep) {
      id = raw.x;
      if constexpr (WIDE) {
        id |= (u64)raw.y << 32;
      }
    }
    if (in_bag && !keep && !(minus_one_skips && raw.x == 0xffffffffu && (!idx64 || raw.y == 0xffffffffu))) {
      report(p.status, FBGEMM_B200_STATUS_BAD_INDEX, bag, pos, (int32_t)raw.x);
    }
    if (pruned && keep) {
      const int32_t m = __ldg(p.cit + id);
      keep = m >= 0;
      id = keep ? (uint32_t)m : 0u;
      if constexpr (!WIDE) {
        // a table larger than its map: below, with 64-bit row addresses
        again = again || (keep && id >= p.map_limit);
        keep = keep && id < p.map_limit;
        id = keep ? id : 0u;
      }
    }
    pos += G;
    raw = fetch(c + G);  // the next stretch's, on its way during this one's arithmetic

    // Where this lane's row goes in the queue, how many rows the group has, and the most that a group of the warp has.
    // Slots behind a group's rows hold row 0 with scale and bias 0, which leave every sum as it is (x + 0 = x, and no
    // sum is ever -0), so that groups of four rows need no special case for the last one.
    int at = gl, count = len - c0, most = min(longest - c0, G);
    bool gaps = FULL;
    if constexpr (!FULL && !kQuantized) {
      gaps = __any_sync(0xffffffffu, in_bag && !keep);  // an index out of range pools nothing
    }
    if (gaps) {
      // kept rows to the front of the queue in order, the other lanes' slots behind them
      const unsigned ballot = __ballot_sync(0xffffffffu, keep);
      const unsigned kept = G == 32 ? ballot : (ballot >> (grp * G)) & kGroupMask;
      const unsigned below = (1u << gl) - 1u;
      count = __popc(kept);
      at = keep ? __popc(kept & below) : count + __popc(~kept & below);
      most = count;
      if constexpr (G < 32) {
#pragma unroll
        for (int g = 0; g < 32 / G; ++g) {
          most = max(most, __popc((ballot >> (g * G)) & kGroupMask));
        }
      }
    }
    uint32_t sb_lo = 0, sb_hi = 0;
    const Row<WIDE> row_at = id * (Row<WIDE>)p.stride;
    q_row[at] = row_at;
    if (kQuantized && keep) {
      const uint8_t* s = sb_data + row_at;
      if (half_sb) {
        sb_lo = load_u32(s, p.sb_align);
      } else if (p.sb_align >= 8) {
        const uint2 v = __ldg(reinterpret_cast<const uint2*>(s));
        sb_lo = v.x;
        sb_hi = v.y;
      } else {
        sb_lo = load_u32(s, p.sb_align);
        sb_hi = load_u32(s + 4, p.sb_align);
      }
    }
    __syncwarp();

    // The row loop, four rows at a time, the loads kAhead groups ahead of the arithmetic.
    Bytes<VB> d[kAhead + 1][4][CPL];
    auto load = [&](Bytes<VB> (&to)[4][CPL], int r) {
      if constexpr (WIDE) {
        const ulonglong2 ab = *reinterpret_cast<const ulonglong2*>(q_row + r);
        const ulonglong2 cd = *reinterpret_cast<const ulonglong2*>(q_row + r + 2);
        lane_data.load(to[0], ab.x);
        lane_data.load(to[1], ab.y);
        lane_data.load(to[2], cd.x);
        lane_data.load(to[3], cd.y);
      } else {
        const uint4 rows = *reinterpret_cast<const uint4*>(q_row + r);
        lane_data.load(to[0], rows.x);
        lane_data.load(to[1], rows.y);
        lane_data.load(to[2], rows.z);
        lane_data.load(to[3], rows.w);
      }
    };
#pragma unroll
    for (int g = 0; g < kAhead; ++g) {
      if (4 * g < most) {
        load(d[g], 4 * g);
      }
    }
    if constexpr (kQuantized) {
      float scale, bias;
      if (half_sb) {
        scale = __half2float(__ushort_as_half((unsigned short)(sb_lo & 0xffffu)));
        bias = __half2float(__ushort_as_half((unsigned short)(sb_lo >> 16)));
      } else {
        scale = __uint_as_float(sb_lo);
        bias = __uint_as_float(sb_hi);
      }
      if (weighted && keep) {
        scale = __fmul_rn(w, scale);
        bias = __fmul_rn(w, bias);
      }
      again = again || out_of_scale(scale) || out_of_scale(bias);
      scale = __fmul_rn(scale, kScaleUp);
      bias = __fmul_rn(bias, kBiasDown);
      const float next = FMT == kInt8 ? scale : __fmul_rn(scale, 1.f / (1 << (FMT % 32)));  // of place 1
      q_sb[at] = make_ulonglong2(pack2(scale, next), pack2(bias, bias));
    } else {
      q_sb[at].x = pack2(w, w);
    }
    __syncwarp();
#pragma unroll 1
    for (int r0 = 0; r0 < most; r0 += 4 * (kAhead + 1)) {
#pragma unroll
      for (int g = 0; g <= kAhead; ++g) {
        const int r = r0 + 4 * g;
        if (g > 0 && r >= most) {
          break;
        }
        if (r + 4 * kAhead < most) {
          load(d[(g + kAhead) % (kAhead + 1)], r + 4 * kAhead);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          if (MAPS && kDeep && u == 2 && r + 2 >= most) {
            break;  // half of a stretch's rows are gone: the last group is often half empty (4-bit D = 128, 13.8 / 12.1 us)
          }
          if constexpr (kQuantized) {
            const ulonglong2 s = q_sb[r + u];
            C::pool(constants, acc, d[g][u], s.x, s.y);
          } else if (r + u < count) {  // (row 0 times 0 is no harmless addition when its values may be infinite)
            C::pool(constants, acc, d[g][u], q_sb[r + u].x, 0ull);
          }
        }
      }
    }
    __syncwarp();  // the queue is rewritten by the next stretch
  }

  constexpr bool kAgain = kQuantized || (MAPS && !WIDE);
  // Pooled again before the row is stored; with eight bytes a lane and whole warps of the lean deep form after it, and stored
  // again: the walk's code is better with it there.  us, before / after the store: 8-bit D = 256, 590 bags of 16 rows
  // 4.17 / 3.88, 1500 of 20 rows 5.59 / 5.28; D = 512, 100 bags of 16 rows 4.09 / 3.79; D = 1024, 1100 bags of 2 rows
  // 4.13 / 3.82.  (8-bit D = 64 3.32 / 3.36, pruned D = 256 4.59 / 4.71; the 40-register forms spill, 4-bit D = 128, 15 000
  // bags 12.6 / 16.5.)
  constexpr bool kAgainLast = kAgain && kDeep && G == 32 && VB == 8 && MODE == kLean;
  float up = kQuantized ? kSumUp : 1.f;  // from the scaled sums to the pooled row
  unsigned lanes = 0;                    // of the group's, those that met a row for pool_again
  if constexpr (kAgain) {
    lanes = __ballot_sync(0xffffffffu, again);
  }
  auto pool_anew = [&] {
    if (lanes != 0 && ((lanes >> (grp * G)) & kGroupMask)) {
      pool_again<C, VB, CPL>(p, constants, lane_data, pos - gl - (Pos)((longest + G - 1) / G * G), len, acc);
      up = 1.f;
    }
  };
  if constexpr (kAgain && !kAgainLast) {
    pool_anew();
  }

  if constexpr (!kDeep) {
    let_next_launch_start();  // (small launches gain nothing from it: 8.1 against 7.6 us for 4096 ragged bags)
  }
  if (bag >= (Pos)p.bags) {
    return;
  }
#pragma unroll 1
  for (;;) {
    int bag_len = 0;
    if (p.flags & kNormalize) {
      bag_len = by_lengths ? (int)load_int(p.offsets, bag, off64)
                           : (int)(load_int(p.offsets, (int64_t)bag + 1, off64) - load_int(p.offsets, bag, off64));
    }
    if (kQuantized || bag_len != 0) {
      // (exact but for the mean's own rounding: a power of two, and no sum is near either end of the range)
      const float by = bag_len != 0 ? __fmul_rn(__fdiv_rn(1.f, (float)bag_len), up) : up;
      const u64 by2 = pack2(by, by);
#pragma unroll
      for (int k = 0; k < C::kPairs; ++k) {
        acc[k] = mul2(acc[k], by2);
      }
    }
    char* row;
    if (p.num_peers > 0) {
      const int64_t d = bag / p.bags_per_peer;
      row = static_cast<char*>(peers[d]) + (bag - d * p.bags_per_peer) * p.out_pitch;
    } else {
      row = static_cast<char*>(p.out) + bag * p.out_pitch;
    }
    float v[2 * C::kPairs];
#pragma unroll
    for (int k = 0; k < C::kPairs; ++k) {
      unpack2(acc[k], v[2 * k], v[2 * k + 1]);
    }
#pragma unroll
    for (int c = 0; c < CPL; ++c) {
      const int col = tile * (kTileBytes * 8 / C::BITS) + (c * G + gl) * C::kPerChunk;
      if (col < p.cols) {
        store_columns<C::kPerChunk>(p, row, col, v + c * C::kPerChunk);
      }
    }
    if (!kAgainLast || lanes == 0) {
      return;
    }
    pool_anew();
    lanes = 0;
  }
}

// 12 blocks of 4 warps per SM, i.e. 40 registers: a lookup waits for memory, and resident warps are what hides it.
// 65536 bags of 30 rows took 82 / 112 / 77 us (8-bit D = 128, 4-bit D = 256, 4-bit D = 128) against 95 / 144 / 121 us
// with the 60 to 100 registers the compiler takes when left alone; 16 blocks (32 registers) were no better.
constexpr int kBlocksPerSm = 12;

// One table per launch: its parameters travel in constant memory, blockIdx.y is the column tile.
struct BagCall {
  BagTable t;
  void* peers[FBGEMM_B200_MAX_PEERS];
};

template <int FMT, int VB, int CPL, int G, int MODE>
__global__ void __launch_bounds__(kThreads, kBlocksPerSm) bag_kernel(const __grid_constant__ BagCall c) {
  __shared__ Queue<MODE == kWide> queues[kWarps];
  pool_bags<FMT, VB, CPL, G, MODE, false>(c.t, c.peers, blockIdx.x, blockIdx.y, queues);
}

// The same for launches whose warps are all resident with 56 registers each:
// residency costs nothing there, so they go into more rows in flight per bag.
// 10 bags of 100 rows (8-bit D = 64) 7.7 against 8.7 us, 10 000 bags of 20 rows
// (8-bit D = 128, half warps) 11.6 against 13.9 us.
constexpr int kDeepBlocksPerSm = 9;
template <int FMT, int VB, int CPL, int G, int MODE>
__global__ void __launch_bounds__(kThreads, kDeepBlocksPerSm) bag_kernel_deep(const __grid_constant__ BagCall c) {
  __shared__ Queue<MODE == kWide> queues[kWarps];
  pool_bags<FMT, VB, CPL, G, MODE, true>(c.t, c.peers, blockIdx.x, blockIdx.y, queues);
}

// The compiled combinations of row format, payload bytes per lane and chunk,
// chunks per lane and lanes per bag.  Whole warps (32 lanes) for every format
// and alignment, wide rows in several tiles; half and quarter warps for the
// narrow rows of large batches (see pick_variant in bag_dispatch.cu).
#define FBGEMM_B200_BAG_VARIANTS_8(X)                                                                       \
  X(kInt8, 2, 1, 16) X(kInt8, 1, 2, 16) X(kInt8, 4, 1, 16) X(kInt8, 8, 1, 16) X(kInt8, 4, 2, 16)              \
  X(kInt8, 2, 1, 32) X(kInt8, 1, 2, 32) X(kInt8, 4, 1, 32) X(kInt8, 2, 2, 32) X(kInt8, 1, 4, 32)              \
  X(kInt8, 8, 1, 32) X(kInt8, 4, 2, 32)
#define FBGEMM_B200_BAG_VARIANTS_4(X)                                                                       \
  X(kInt4, 2, 1, 8) X(kInt4, 4, 1, 8) X(kInt4, 1, 1, 16) X(kInt4, 2, 1, 16) X(kInt4, 4, 1, 16)                \
  X(kInt4, 1, 1, 32) X(kInt4, 2, 1, 32) X(kInt4, 1, 2, 32) X(kInt4, 4, 1, 32) X(kInt4, 2, 2, 32) X(kInt4, 1, 4, 32)
#define FBGEMM_B200_BAG_VARIANTS_2(X)                                                                       \
  X(kInt2, 2, 1, 8) X(kInt2, 1, 1, 16) X(kInt2, 2, 1, 16)                                                     \
  X(kInt2, 1, 1, 32) X(kInt2, 2, 1, 32) X(kInt2, 1, 2, 32)
#define FBGEMM_B200_BAG_VARIANTS_PLAIN(X)                                                                   \
  X(kF32, 16, 1, 32) X(kF32, 8, 1, 32) X(kF32, 4, 2, 32)                                                      \
  X(kF16, 8, 1, 32) X(kF16, 4, 1, 32) X(kF16, 2, 2, 32)                                                       \
  X(kBf16, 8, 1, 32) X(kBf16, 4, 1, 32) X(kBf16, 2, 2, 32)                                                    \
  X(kFp8, 4, 1, 32) X(kFp8, 2, 1, 32) X(kFp8, 1, 2, 32)
#define FBGEMM_B200_BAG_VARIANTS(X) \
  FBGEMM_B200_BAG_VARIANTS_8(X) FBGEMM_B200_BAG_VARIANTS_4(X) FBGEMM_B200_BAG_VARIANTS_2(X) FBGEMM_B200_BAG_VARIANTS_PLAIN(X)

// Behind a pruning map, and when launches on other streams fill the chip: 16 columns a lane, which want the deep form's
// registers (the other forms would spill).
#define FBGEMM_B200_BAG_VARIANTS_DEEP_MAPPED(X) X(kInt2, 4, 1, 8)

#define FBGEMM_B200_BAG_ID(FMT, VB, CPL, G) id_##FMT##_##VB##_##CPL##_##G,
enum VariantId : int {
  FBGEMM_B200_BAG_VARIANTS(FBGEMM_B200_BAG_ID) FBGEMM_B200_BAG_VARIANTS_DEEP_MAPPED(FBGEMM_B200_BAG_ID) kVariants
};
#undef FBGEMM_B200_BAG_ID

// Several tables per launch (what the reference's multi-table caller does with
// a loop of functor calls, fbgemm_gpu/codegen/inference/embedding_forward_quantized_cpu_template.cpp:343-473):
// unit u - one column tile of one table - owns the blocks [first_block[u],
// first_block[u + 1]), whatever the tables' row formats.  The units arrive by
// value, in constant memory; a block finds its own by bisection.
constexpr int kMaxUnits = 128, kMaxTables = 64;
struct BagUnits {
  int32_t count;
  int32_t first_block[kMaxUnits + 1];
  struct Unit {
    uint8_t variant, table;
    uint16_t tile;
  } unit[kMaxUnits];
  BagTable t[kMaxTables];
  void* peers[kMaxTables][FBGEMM_B200_MAX_PEERS];
};
static_assert(kVariants <= 256, "a variant is a byte");
static_assert(sizeof(BagUnits) < 32764, "one kernel argument");

template <int MODE>
__global__ void __launch_bounds__(kThreads, kBlocksPerSm) bag_units_kernel(const __grid_constant__ BagUnits a) {
  __shared__ Queue<MODE == kWide> queues[kWarps];
  int lo = 0, hi = a.count;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if ((int)blockIdx.x >= a.first_block[mid]) {
      lo = mid;
    } else {
      hi = mid;
    }
  }
  const BagUnits::Unit u = a.unit[lo];
  const BagTable& t = a.t[u.table];
  const uint32_t block = blockIdx.x - a.first_block[lo];
  switch (u.variant) {
#define FBGEMM_B200_BAG_CASE(FMT, VB, CPL, G)                                   \
  case id_##FMT##_##VB##_##CPL##_##G:                                                  \
    pool_bags<FMT, VB, CPL, G, MODE, false>(t, a.peers[u.table], block, u.tile, queues); \
    break;
    FBGEMM_B200_BAG_VARIANTS(FBGEMM_B200_BAG_CASE)
#undef FBGEMM_B200_BAG_CASE
  }
}

using BagFn = void (*)(const BagCall);

// A handful of bags in one quantized table (few_bags_kernel.cu): a block per bag and kFewColumns columns.
constexpr int kFewThreads = 256, kFewColumns = 128;
BagFn few_bags(int fmt);
// Whether it copies rows in words of four bytes (the last one may run into scale and bias behind the payload, but not
// beyond the row) or in smaller units.
__host__ __device__ __forceinline__ bool few_by_words(const BagTable& t) {
  return t.data_align >= 4 && (t.data_bytes % 4 == 0 || t.sb_off > 0);
}
// Of those, by halves where rows allow it.
__host__ __device__ __forceinline__ bool few_by_halves(const BagTable& t) {
  return t.data_align >= 2 && (t.data_bytes % 2 == 0 || t.sb_off > 0);
}
// Units that a row's widest tile takes.
inline int few_units(const BagTable& t, int fmt) {
  const int bytes = t.data_bytes < kFewColumns * fmt / 8 ? t.data_bytes : kFewColumns * fmt / 8;
  return few_by_halves(t) ? (bytes + 1) / 2 : bytes;
}

constexpr int kDeepForms = 4;             // kDeepForms + form: its deep form (there is none of kWide)
constexpr int kForms = 2 * kDeepForms;
using BagUnitsFn = void (*)(const BagUnits);

}  // namespace bag

// The single-table kernels by variant id and form; one translation unit per
// group of formats (bag_kernel_*.cu).
void bag_kernels_8(bag::BagFn (*fn)[bag::kForms]);
void bag_kernels_4(bag::BagFn (*fn)[bag::kForms]);
void bag_kernels_2(bag::BagFn (*fn)[bag::kForms]);
void bag_kernels_plain(bag::BagFn (*fn)[bag::kForms]);
bag::BagUnitsFn bag_units_lean();
bag::BagUnitsFn bag_units_full();
bag::BagUnitsFn bag_units_mapped();
bag::BagUnitsFn bag_units_wide();

}  // namespace fbgemm_b200
