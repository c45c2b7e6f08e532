// Index remapping of table-batched pruned tables: sparse index -> dense index
// (or -1 for a pruned row) through a per-table open-addressing hash map or a
// per-table array, run by a table-batched caller before the lookup.
//
// Reference: pruned_hashmap_lookup_{un}weighted_cpu and pruned_array_lookup_cpu,
// fbgemm_gpu/codegen/inference/embedding_forward_quantized_cpu_template.cpp:524-601,
// :605-659; hash :102-120 (MurmurHash3 finalisers); the reference's CUDA forms
// (embedding_forward_quantized_split_lookup.cu:20-160) give a warp to every
// bag.  Here a thread owns one POSITION of the index array, so the work per
// thread does not depend on how ragged the bags are and index loads and result
// stores are coalesced; the thread finds its table by bisection over the T+1
// table starts offsets[t*B] (staged in shared memory when they fit) and then
// probes alone (see pruned_hashmap_kernel for what happens to long probe sequences).
//
// The reference's probe loop has no end on a full table that lacks the key;
// here it stops after `capacity` slots with -1, so no launch can spin.
#include "internal.h"
#include "position_tables.cuh"

namespace fbgemm_b200 {

namespace {

constexpr int kThreads = 256;
constexpr int kPerThread = 4;  // positions per thread, array form

__device__ __forceinline__ int64_t load_int(const void* p, int64_t i, bool is64) {
  return is64 ? (int64_t)__ldg(reinterpret_cast<const long long*>(p) + i)
              : (int64_t)__ldg(reinterpret_cast<const int*>(p) + i);
}

__device__ __forceinline__ void store_int(void* p, int64_t i, int64_t v, bool is64) {
  if (is64) {
    static_cast<long long*>(p)[i] = v;
  } else {
    static_cast<int*>(p)[i] = (int)v;
  }
}

__device__ __forceinline__ uint32_t hash32(uint32_t h) {
  h ^= h >> 16;
  h *= 0x85ebca6bu;
  h ^= h >> 13;
  h *= 0xc2b2ae35u;
  h ^= h >> 16;
  return h;
}

__device__ __forceinline__ uint64_t hash64(uint64_t k) {
  k ^= k >> 33;
  k *= 0xff51afd7ed558ccdULL;
  k ^= k >> 33;
  k *= 0xc4ceb9fe1a85ec53ULL;
  k ^= k >> 33;
  return k;
}

struct PrunedArgs {
  const void* indices;
  const void* offsets;
  const void* map;            // hash table ([.][2]) or remapping array
  const int64_t* map_offsets; // [T + 1]
  void* dense;
  int32_t* status;
  int64_t index_size;
  int32_t T;
  int32_t B;
  int32_t index64;
  int32_t map64;
};

__device__ __forceinline__ void report(const PrunedArgs& a, int code, int64_t table, int64_t pos, int64_t value) {
  if (atomicCAS(a.status, 0, code) == 0) {
    a.status[1] = (int32_t)table;
    a.status[2] = (int32_t)pos;
    a.status[3] = (int32_t)value;
  }
}

// The array form, and tables without a map: one load per position.
__global__ void __launch_bounds__(kThreads) pruned_array_kernel(const PrunedArgs a) {
  __shared__ int64_t starts_s[kSharedStarts];
  const int64_t* starts = stage_table_starts(a, starts_s);
  const int64_t base = ((int64_t)blockIdx.x * kPerThread) * kThreads + threadIdx.x;
#pragma unroll
  for (int i = 0; i < kPerThread; ++i) {
    const int64_t k = base + (int64_t)i * kThreads;
    if (k >= a.index_size) {
      break;
    }
    const int t = table_of(a, starts, k);
    if (t < 0) {
      continue;
    }
    const int64_t idx = load_int(a.indices, k, a.index64);
    const int64_t map_start = __ldg(a.map_offsets + t);
    const int64_t capacity = __ldg(a.map_offsets + t + 1) - map_start;
    int64_t dense = -1;
    if (capacity <= 0) {
      dense = idx;
    } else if (idx < 0 || idx >= capacity) {
      report(a, FBGEMM_B200_STATUS_BAD_INDEX, t, k, idx);
    } else {
      dense = load_int(a.map, map_start + idx, a.map64);
    }
    store_int(a.dense, k, dense, a.index64);
  }
}

template <bool MAP64>
__device__ __forceinline__ void load_slot(const void* slots, int64_t at, int64_t& key, int64_t& value) {
  if constexpr (MAP64) {
    const longlong2 kv = __ldg(reinterpret_cast<const longlong2*>(slots) + at);
    key = kv.x;
    value = kv.y;
  } else {
    const int2 kv = __ldg(reinterpret_cast<const int2*>(slots) + at);
    key = kv.x;
    value = kv.y;
  }
}

// One 32-byte sector of a map: four 8-byte slots or two 16-byte ones.
template <bool MAP64>
struct Sector {
  static constexpr int kSlotBytes = MAP64 ? 16 : 8;
  static constexpr int kSlots = 32 / kSlotBytes;
  uint32_t w[8];

  // Slots [lo, hi) of the sector are slots `first` .. of the table; the others
  // are loaded along with them where the whole sector belongs to the maps.
  __device__ __forceinline__ void load(const char* p, const char* maps, const char* maps_end, const char* slots, int64_t first,
                                       int lo, int hi) {
    if (p >= maps && p + 32 <= maps_end) {
      asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
          : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7])
          : "l"(p));
      return;
    }
#pragma unroll
    for (int j = 0; j < kSlots; ++j) {
      int64_t key = 0, value;
      if (j >= lo && j < hi) {
        load_slot<MAP64>(slots, first + j - lo, key, value);
      }
      w[j * kSlotBytes / 4] = (uint32_t)key;
      w[j * kSlotBytes / 4 + 1] = (uint32_t)(key >> 32);
    }
  }

  // Bit j: slot j of [lo, hi) holds the key or nothing.
  __device__ __forceinline__ uint32_t ends(int64_t idx, int lo, int hi) const {
    uint32_t m = 0;
    // an index that an 8-byte slot cannot hold ends at the empty slots alone
    const int idx32 = idx == (int64_t)(int32_t)idx ? (int)idx : -1;
#pragma unroll
    for (int j = 0; j < kSlots; ++j) {
      bool end;
      if constexpr (MAP64) {
        const int64_t key = (int64_t)(((uint64_t)w[4 * j + 1] << 32) | w[4 * j]);
        end = key == -1 || key == idx;
      } else {
        end = (int)w[2 * j] == -1 || (int)w[2 * j] == idx32;
      }
      m |= end ? 1u << j : 0u;
    }
    return m & ((1u << hi) - (1u << lo));
  }
};

// A probe sequence that its first slots did not end.
struct alignas(16) Walk {
  const char* slots;
  int64_t idx;
  uint32_t slot, capacity;
  uint32_t left;  // slots not yet seen
  uint32_t at;    // position, from the block's first one
};

constexpr int kHashPer = 2;  // positions per thread, hash-map form
constexpr int kWalkLanes = 8;  // lanes that walk one long sequence together
constexpr int kHashTables = 1024;  // what a block keeps of the tables, 32 bytes each, fits in shared memory below this

// The hash-map form, two phases.  First a thread per position: table, index,
// hash, and the first two sectors of its probe sequence (at least five 8-byte
// slots), which end most of them.  Then the sequences left over, put in line by
// warp, are walked by kWalkLanes lanes each, a sector per lane and step.
// At a load factor of 0.8 a hit walks 3 slots on average and a miss 13, some of
// them a hundred, and a warp that walks 32 sequences a thread each goes on until
// the longest ends, with 8 of 32 lanes active: bound by instructions (63 % of the
// issue slots, 2100 instructions per warp) while DRAM stood at 12 %.
// 2.0 M positions over 16 tables of 2.4 M 8-byte slots at that load, half of the
// keys present: 171 us a thread per sequence, 170 with two sectors at a time,
// 75 in two phases (16-byte slots 202 and 105; 4-byte indices 159 and 74).  One
// and four positions per thread: 82 and 88 us; four lanes per walk: 78.
// The remainder by the capacity is Barrett's, with a reciprocal that each block
// works out per table; it is exact: the quotient comes out at most one too small.
template <bool MAP64>
__global__ void __launch_bounds__(kThreads) pruned_hashmap_kernel(const PrunedArgs a) {
  using S = Sector<MAP64>;
  extern __shared__ int64_t tables_s[];
  __shared__ Walk walks[kThreads / 32][32 * kHashPer];
  const bool staged = a.T < kHashTables;
  int64_t* const starts = staged ? tables_s : nullptr;  // [T + 1]
  int64_t* const firsts = tables_s + a.T + 1;           // [T] each
  int64_t* const capacities = firsts + a.T;
  uint64_t* const reciprocals = reinterpret_cast<uint64_t*>(capacities + a.T);
  const int64_t block_at = (int64_t)blockIdx.x * kThreads * kHashPer;
  int64_t idx[kHashPer];
#pragma unroll
  for (int i = 0; i < kHashPer; ++i) {
    const int64_t k = block_at + i * kThreads + threadIdx.x;
    idx[i] = k < a.index_size ? load_int(a.indices, k, a.index64) : 0;
  }
  if (staged) {
    for (int t = threadIdx.x; t <= a.T; t += kThreads) {
      starts[t] = table_start(a, static_cast<const int64_t*>(nullptr), t);
      if (t < a.T) {
        const int64_t first = __ldg(a.map_offsets + t), capacity = __ldg(a.map_offsets + t + 1) - first;
        firsts[t] = first;
        capacities[t] = capacity;
        reciprocals[t] = capacity > 0 ? ~0ULL / (uint64_t)capacity : 0;
      }
    }
    __syncthreads();
  }
  const char* const map = static_cast<const char*>(a.map);
  const char* const maps = map + __ldg(a.map_offsets) * S::kSlotBytes;
  const char* const maps_end = map + __ldg(a.map_offsets + a.T) * S::kSlotBytes;
  const int lane = threadIdx.x & 31;
  Walk* const line = walks[threadIdx.x >> 5];
  int in_line = 0;
  int t = -1;
#pragma unroll
  for (int i = 0; i < kHashPer; ++i) {
    const int64_t k = block_at + i * kThreads + threadIdx.x;
    if (k >= a.index_size) {
      t = -1;
    } else if (t < 0 || k >= table_start(a, starts, t + 1)) {
      t = table_of(a, starts, k);
    }
    bool open = false;
    Walk w;
    if (t >= 0) {
      const int64_t first = staged ? firsts[t] : __ldg(a.map_offsets + t);
      const int64_t capacity = staged ? capacities[t] : __ldg(a.map_offsets + t + 1) - first;
      w.slots = map + first * S::kSlotBytes;
      w.idx = idx[i];
      if (capacity <= 0) {
        store_int(a.dense, k, idx[i], a.index64);  // a table without a map keeps its indices
      } else {
        const uint64_t h = a.index64 ? hash64((uint64_t)idx[i]) : (uint64_t)hash32((uint32_t)idx[i]);
        uint64_t slot;
        if (staged) {
          slot = h - __umul64hi(h, reciprocals[t]) * (uint64_t)capacity;
          slot -= slot >= (uint64_t)capacity ? (uint64_t)capacity : 0;
        } else {
          slot = h % (uint64_t)capacity;
        }
        if (capacity > 0x7fffffffLL) {
          // a table of 2^31 slots or more: walked here, with 64-bit slot arithmetic
          int64_t dense = -1;
          for (int64_t probes = 0; probes < capacity; ++probes) {
            int64_t key, value;
            load_slot<MAP64>(w.slots, (int64_t)slot, key, value);
            if (key == -1 || key == idx[i]) {
              dense = key == -1 ? -1 : value;
              break;
            }
            slot = (int64_t)slot + 1 == capacity ? 0 : slot + 1;
          }
          store_int(a.dense, k, dense, a.index64);
        } else {
          w.slot = (uint32_t)slot;
          w.capacity = (uint32_t)capacity;
          const char* here = w.slots + (int64_t)w.slot * S::kSlotBytes;
          const char* sector = reinterpret_cast<const char*>(reinterpret_cast<uintptr_t>(here) & ~(uintptr_t)31);
          const int off = (int)(here - sector) / S::kSlotBytes;
          const int n = (int)min(w.capacity - w.slot, (uint32_t)(2 * S::kSlots - off));
          const int end0 = min(off + n, S::kSlots), end1 = max(off + n - S::kSlots, 0);
          S s0, s1;
          s0.load(sector, maps, maps_end, w.slots, w.slot, off, end0);
          s1.load(sector + 32, maps, maps_end, w.slots, (int64_t)w.slot + S::kSlots - off, 0, end1);
          const uint32_t m = s0.ends(w.idx, off, end0) | s1.ends(w.idx, 0, end1) << S::kSlots;
          if (m != 0) {
            int64_t key, value;
            load_slot<MAP64>(w.slots, (int64_t)w.slot + __ffs(m) - 1 - off, key, value);
            store_int(a.dense, k, key == -1 ? -1 : value, a.index64);
          } else if ((uint32_t)n >= w.capacity) {
            store_int(a.dense, k, -1, a.index64);  // a full table without the key
          } else {
            w.slot = w.slot + n == w.capacity ? 0 : w.slot + n;
            w.left = w.capacity - n;
            w.at = i * kThreads + threadIdx.x;
            open = true;
          }
        }
      }
    }
    const uint32_t opens = __ballot_sync(~0u, open);
    if (open) {
      line[in_line + __popc(opens & ((1u << lane) - 1))] = w;
    }
    in_line += __popc(opens);
  }
  __syncwarp();

  constexpr int kWalks = 32 / kWalkLanes;
  constexpr uint32_t kLanes = kWalkLanes == 32 ? ~0u : (1u << kWalkLanes) - 1;
  const int group = lane / kWalkLanes, gl = lane % kWalkLanes;
  Walk w;
  bool walking = group < in_line;
  if (walking) {
    w = line[group];
  }
  int next = kWalks;  // first sequence in line that no lanes have taken
  while (__any_sync(~0u, walking)) {
    uint32_t m = 0;
    int64_t first = 0;
    int off = 0, lo = 0;
    if (walking) {
      const char* here = w.slots + (int64_t)w.slot * S::kSlotBytes;
      const char* sector = reinterpret_cast<const char*>(reinterpret_cast<uintptr_t>(here) & ~(uintptr_t)31);
      off = (int)(here - sector) / S::kSlotBytes;
      lo = gl == 0 ? off : 0;
      // slots from this sector's first one to the table's end
      const int64_t room = (int64_t)w.capacity - w.slot + off - gl * S::kSlots;
      const int hi = (int)max((int64_t)lo, min(room, (int64_t)S::kSlots));
      first = (int64_t)w.slot - off + gl * S::kSlots;
      if (hi > lo) {
        S s;
        s.load(sector + gl * 32, maps, maps_end, w.slots, first + lo, lo, hi);
        m = s.ends(w.idx, lo, hi);
      }
    }
    const uint32_t ended = (__ballot_sync(~0u, m != 0) >> (group * kWalkLanes)) & kLanes;
    if (walking) {
      if (ended != 0) {
        if (gl == __ffs(ended) - 1) {
          int64_t key, value;
          load_slot<MAP64>(w.slots, first + __ffs(m) - 1, key, value);
          store_int(a.dense, block_at + w.at, key == -1 ? -1 : value, a.index64);
        }
        walking = false;
      } else {
        const uint32_t n = min((uint32_t)(kWalkLanes * S::kSlots - off), w.capacity - w.slot);
        if (n >= w.left) {
          if (gl == 0) {
            store_int(a.dense, block_at + w.at, -1, a.index64);  // a full table without the key
          }
          walking = false;
        } else {
          w.left -= n;
          w.slot = w.slot + n == w.capacity ? 0 : w.slot + n;
        }
      }
    }
    if (next < in_line) {
      const uint32_t idle = __ballot_sync(~0u, !walking && gl == 0);
      const int mine = next + __popc(idle & ((1u << (group * kWalkLanes)) - 1));
      if (!walking && mine < in_line) {
        w = line[mine];
        walking = true;
      }
      next += __popc(idle);
    }
  }
}

// Filling the hash map on the device.  The reference only inserts on the host, one key after the
// other; here every position claims the first free slot of its probe sequence with a compare-and-swap
// on the key, so the slots a cluster's keys end up in depend on the order the threads arrive in - the
// table differs from the host-built one byte for byte but every lookup gives the same answer (a key
// sits within its probe sequence, before the first empty slot).  Positions whose dense index is -1
// are not inserted, as in the reference; a table without a free slot is reported.
template <bool MAP64>
__global__ void __launch_bounds__(kThreads) pruned_hashmap_insert_kernel(const PrunedArgs a, const void* dense_indices) {
  __shared__ int64_t starts_s[kSharedStarts];
  const int64_t* starts = stage_table_starts(a, starts_s);
  const int64_t k = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  const int t = k < a.index_size ? table_of(a, starts, k) : -1;
  if (t < 0) {
    return;
  }
  const int64_t dense = load_int(dense_indices, k, a.index64);
  const int64_t map_start = __ldg(a.map_offsets + t);
  const int64_t capacity = __ldg(a.map_offsets + t + 1) - map_start;
  if (dense == -1 || capacity <= 0) {
    return;
  }
  const int64_t idx = load_int(a.indices, k, a.index64);
  const uint64_t h = a.index64 ? hash64((uint64_t)idx) : (uint64_t)hash32((uint32_t)idx);
  int64_t slot = (int64_t)(h % (uint64_t)capacity);
  for (int64_t probes = 0; probes < capacity; ++probes) {
    const int64_t at = 2 * (map_start + slot);
    int64_t seen;
    if constexpr (MAP64) {
      unsigned long long* keys = static_cast<unsigned long long*>(const_cast<void*>(a.map));
      seen = (int64_t)atomicCAS(keys + at, ~0ULL, (unsigned long long)idx);
      if (seen == -1 || seen == idx) {
        reinterpret_cast<long long*>(keys)[at + 1] = dense;
        return;
      }
    } else {
      int* keys = static_cast<int*>(const_cast<void*>(a.map));
      seen = atomicCAS(keys + at, -1, (int)idx);
      if (seen == -1 || seen == (int)idx) {
        keys[at + 1] = (int)dense;
        return;
      }
    }
    slot = slot + 1 == capacity ? 0 : slot + 1;
  }
  report(a, FBGEMM_B200_STATUS_TABLE_FULL, t, k, idx);
}

}  // namespace

cudaError_t launch_pruned_lookup(
    bool hashmap,
    int32_t T,
    int32_t B,
    const void* indices,
    const void* offsets,
    int index_bytes,
    int64_t index_size,
    const void* map,
    int map_bytes,
    const int64_t* map_offsets,
    void* dense_indices,
    int32_t* status,
    cudaStream_t stream) {
  if (index_size == 0) {
    return cudaSuccess;
  }
  PrunedArgs a{};
  a.indices = indices;
  a.offsets = offsets;
  a.map = map;
  a.map_offsets = map_offsets;
  a.dense = dense_indices;
  a.status = status;
  a.index_size = index_size;
  a.T = T;
  a.B = B;
  a.index64 = index_bytes == 8;
  a.map64 = map_bytes == 8;
  const int64_t per_block = (int64_t)kThreads * (hashmap ? kHashPer : kPerThread);
  const int64_t blocks = (index_size + per_block - 1) / per_block;
  if (blocks > 0x7fffffffLL) {
    return cudaErrorInvalidValue;
  }
  const size_t shared = hashmap && T < kHashTables ? (4 * (size_t)T + 1) * sizeof(int64_t) : 0;
  if (!hashmap) {
    pruned_array_kernel<<<(unsigned)blocks, kThreads, 0, stream>>>(a);
  } else if (a.map64) {
    pruned_hashmap_kernel<true><<<(unsigned)blocks, kThreads, shared, stream>>>(a);
  } else {
    pruned_hashmap_kernel<false><<<(unsigned)blocks, kThreads, shared, stream>>>(a);
  }
  g_launch_count.fetch_add(1, std::memory_order_relaxed);
  return cudaGetLastError();
}

}  // namespace fbgemm_b200

namespace fbgemm_b200 {

cudaError_t launch_pruned_hashmap_insert(
    int32_t T,
    int32_t B,
    const void* indices,
    const void* dense_indices,
    const void* offsets,
    int index_bytes,
    int64_t index_size,
    void* hash_table,
    int hash_bytes,
    const int64_t* hash_table_offsets,
    int32_t* status,
    cudaStream_t stream) {
  if (index_size == 0) {
    return cudaSuccess;
  }
  PrunedArgs a{};
  a.indices = indices;
  a.offsets = offsets;
  a.map = hash_table;
  a.map_offsets = hash_table_offsets;
  a.status = status;
  a.index_size = index_size;
  a.T = T;
  a.B = B;
  a.index64 = index_bytes == 8;
  a.map64 = hash_bytes == 8;
  const int64_t blocks = (index_size + kThreads - 1) / kThreads;
  if (blocks > 0x7fffffffLL) {
    return cudaErrorInvalidValue;
  }
  if (a.map64) {
    pruned_hashmap_insert_kernel<true><<<(unsigned)blocks, kThreads, 0, stream>>>(a, dense_indices);
  } else {
    pruned_hashmap_insert_kernel<false><<<(unsigned)blocks, kThreads, 0, stream>>>(a, dense_indices);
  }
  g_launch_count.fetch_add(1, std::memory_order_relaxed);
  return cudaGetLastError();
}

}  // namespace fbgemm_b200
