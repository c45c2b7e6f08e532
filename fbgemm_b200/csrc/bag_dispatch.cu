// Which bag kernel (bag_kernel.cuh) takes a lookup, and how many tables go into
// one launch.
#include <algorithm>
#include <atomic>
#include <vector>

#include "bag_kernel.cuh"
#include "few_bags_rule.h"

namespace fbgemm_b200 {

namespace {

struct VariantInfo {
  int fmt, vb, cpl, g;
  bool deep_mapped;  // compiled in the deep form with a pruning map alone
};
constexpr VariantInfo kVariantInfo[] = {
#define INFO(FMT, VB, CPL, G) {bag::FMT, VB, CPL, G, false},
#define INFO_DEEP_MAPPED(FMT, VB, CPL, G) {bag::FMT, VB, CPL, G, true},
    FBGEMM_B200_BAG_VARIANTS(INFO) FBGEMM_B200_BAG_VARIANTS_DEEP_MAPPED(INFO_DEEP_MAPPED)
#undef INFO
#undef INFO_DEEP_MAPPED
};

// Largest power of two, 16 at most, that divides v.
int alignment_of(uint64_t v) {
  return v % 16 == 0 ? 16 : v % 8 == 0 ? 8 : v % 4 == 0 ? 4 : v % 2 == 0 ? 2 : 1;
}

int format_of(const SpmdmParams& p, int bit_rate) {
  switch (p.in_kind) {
    case FBGEMM_B200_IN_QUANTIZED: return bit_rate;
    case FBGEMM_B200_IN_F32: return bag::kF32;
    case FBGEMM_B200_IN_F16: return bag::kF16;
    case FBGEMM_B200_IN_BF16: return bag::kBf16;
    default: return bag::kFp8;
  }
}

void bag_table_of(const SpmdmParams& p, BagTable* t) {
  t->data = p.table + p.data_row_off;
  t->indices = p.indices;
  t->offsets = p.offsets;
  t->weights = p.weights;
  t->cit = p.cit;
  t->out = p.out;
  t->status = p.status;
  t->data_size = p.data_size;
  t->bags = p.output_size;
  t->index_size = p.index_size;
  const int esize = (p.flags & (kOutHalf | kOutBf16)) ? 2 : 4;
  t->out_pitch = p.output_stride * esize;
  t->bags_per_peer = p.bags_per_peer;
  t->sb_off = p.sb_row_off - p.data_row_off;
  t->stride = p.input_stride;
  t->cols = p.block_size;
  t->data_bytes = p.data_bytes;
  t->flags = p.flags;
  // a 32-bit index is negative from 2^31 on
  t->limit = (uint32_t)std::min<int64_t>(p.data_size, (p.flags & kIdx64) ? 0xffffffffLL : 0x80000000LL);
  t->map_limit = (uint32_t)(0xffffffffull / (uint64_t)p.input_stride);
  const uint64_t sb = reinterpret_cast<uintptr_t>(p.table + p.sb_row_off) | (uint64_t)p.input_stride;
  t->sb_align = (int16_t)std::min(8, alignment_of(sb));
  uint64_t o = (uint64_t)t->out_pitch;
  for (int i = 0; i < p.num_peers; ++i) {
    o |= reinterpret_cast<uintptr_t>(p.peer_out[i]);
  }
  if (p.num_peers <= 0) {
    o |= reinterpret_cast<uintptr_t>(p.out);
  }
  t->num_peers = p.num_peers;
  t->out_align = (int16_t)alignment_of(o);
  t->fp8_exponent_bits = (int16_t)p.fp8_exponent_bits;
  t->fp8_exponent_bias = (int16_t)p.fp8_exponent_bias;
  t->data_align = (int16_t)alignment_of(reinterpret_cast<uintptr_t>(t->data) | (uint64_t)t->stride);
}

// The form of a table's kernel.  (A row-wise sparse call says how many rows its
// map has, not how many its table holds, which may be more: see pool_again.)
int form_of(const BagTable& t) {
  const bool wide = (unsigned __int128)t.data_size * (uint64_t)t.stride > 0xffffffffull || t.bags > 0x7fffff00LL ||
      t.index_size > 0x7fffff00LL;
  const bool options = t.flags & (kSbFirst | kNoBag | kPositional | kLengths);
  return wide ? bag::kWide : t.flags & kPruned ? bag::kMapped : options || t.data_size == 0 ? bag::kFull : bag::kLean;
}

// The current device's SMs.
int64_t sm_count() {
  constexpr int kDevices = 64;
  static std::atomic<int> counts[kDevices];
  int device = 0, n = 0;
  if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= kDevices) {
    return 148;
  }
  n = counts[device].load(std::memory_order_relaxed);
  if (n == 0) {
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || n <= 0) {
      return 148;
    }
    counts[device].store(n, std::memory_order_relaxed);
  }
  return n;
}

// Warps that are resident on `sms` SMs at a time, and blocks of the deep form.
int64_t resident_warps(int64_t sms) {
  return sms * bag::kBlocksPerSm * bag::kWarps;
}
int64_t deep_fit(int64_t sms) {
  return sms * bag::kDeepBlocksPerSm;
}

// Whole warps per bag while every bag on the chip finds a resident warp: the
// fewer lanes share a bag, the longer its rows take, and nothing else is there
// to run.  Beyond that narrow rows take half warps (one and the same walk serves
// two bags), the narrowest quarter warps.  Measured, us, on bags of 30 rows at
// 12 M rows: 4-bit D = 64, 4096 bags 7.0 / 8.9 / 10.9 with 32 / 16 / 8 lanes;
// 8192 bags 11.6 / 10.0 / 12.2; 65536 bags 61.8 / 51.9 / 48.7.  4-bit D = 128,
// 65536 bags 80.9 / 72.8 / 78.3.  Wider rows always want whole warps.  Quarter
// warps from 8 bags per resident warp on: 33000 bags of 2-bit D = 64 take 39.5 us
// with them and 33.6 without, 4-bit 40.4 and 38.7, 64 mixed tables of 512 bags
// 53.3 and 50.6; 100000 bags of 4-bit D = 64 86.5 and 91.9.
//
// Launches on other streams (launch_history.h) are on the chip too, but a quarter
// of their bags counts against whole warps: a small launch spends most of its
// time in start-up and drain.  us per call on 1, 2, 4, 8, 16 streams with
// 32 / 16 / 8 lanes, 4-bit D = 64, 4096 bags of 30 rows at 10 M rows:
//   10.2 / 13.1 / 17.6,  5.7 / 7.1 / 9.2,  4.4 / 4.4 / 5.3,  4.4 / 3.5 / 3.8,  4.0 / 3.3 / 3.2
// (by its own size alone every such launch took whole warps and the deep form,
// 5.0 us from four streams on).  Behind a pruning map quarter warps pay from 4
// bags per resident warp on, 8192 bags of 2-bit D = 128 at 20 M rows, 2, 4 and 16
// streams: 8.5 / 9.6 / 10.8,  8.3 / 8.9 / 7.6,  7.9 / 8.6 / 7.1.
// Bags that a launch and those beside it keep on the chip at a time.
int64_t bags_at_a_time(int64_t bags, int64_t beside) {
  return bags + beside / 4;
}

int64_t blocks_of(int64_t bags, int variant) {
  const int64_t per_block = (int64_t)bag::kWarps * (32 / kVariantInfo[variant].g);
  return (bags + per_block - 1) / per_block;
}

// `bags` in the launch, `beside` in those on other streams; `single`: one table's launch.
int pick_variant(const BagTable& t, int fmt, int64_t bags, int64_t beside, bool single, int64_t sms, int* tiles) {
  const int align = t.data_align;
  const bool mapped = t.flags & kPruned;
  const int64_t resident = resident_warps(sms);
  const int64_t quarter_warps_from = (mapped && beside > 0 ? 4 : 8) * resident;
  const int least_g = bags_at_a_time(bags, beside) <= resident ? 32 : bags + beside <= quarter_warps_from ? 16 : 8;
  int best = -1;
  double best_cost = 0;
  for (int i = 0; i < bag::kVariants; ++i) {
    const VariantInfo& v = kVariantInfo[i];
    if (v.fmt != fmt || v.vb > align || v.g < least_g) {
      continue;
    }
    if (v.deep_mapped && !(single && form_of(t) == bag::kMapped && blocks_of(bags, i) <= 2 * deep_fit(sms))) {
      continue;
    }
    // the last chunk may run into scale,bias behind the payload, but not beyond the row
    if (t.data_bytes % v.vb != 0 && !(bag::is_quantized(fmt) && t.sb_off > 0 && v.vb <= 4)) {
      continue;
    }
    const int tile = v.vb * v.cpl * v.g;
    const int n = (t.data_bytes + tile - 1) / tile;
    if (n > 1 && v.g < 32) {
      continue;
    }
    // Instructions per row: what a row costs besides its columns, its loads, and per column of a lane one that cuts it out,
    // half a packed addition and half a packed multiply-add (unquantized rows, whose conversions differ, 2.5 in all).  Half
    // an instruction more where four chunks a lane make the rows in flight spill, and for a few bags, whose warps do not
    // fill the chip and rather have more tiles.  us with 2.5 throughout / so: 8-bit D = 150 (two tiles of 4 columns a lane
    // for three of 2), 4007, 15 000 and 60 000 bags 9.4 / 9.6, 30.5 / 27.5, 120 / 103, 700 bags if they did too 5.6 / 6.0;
    // 8-bit D = 301 (five tiles of 2 for three of 4), 700, 1500, 4007 and 15 000 bags 9.1 / 6.4, 12.2 / 12.4, 18.9 / 16.0,
    // 71 / 59; 4-bit D = 802 (seven for four), 700 and 15 000 bags 10.0 / 7.3, 119 / 89.
    const double cols = (double)v.vb * v.cpl * 8 / bag::column_bits(fmt);
    const double per_column = !bag::is_quantized(fmt) ? 2.5 : 2.0 + (v.cpl >= 4 ? 0.5 : 0.0) + (bags + beside <= 8 * sms ? 0.5 : 0.0);
    const double cost = n * (6.0 + 1.5 * v.cpl + per_column * cols) * v.g;
    if (best < 0 || cost < best_cost) {
      best = i;
      best_cost = cost;
      *tiles = n;
    }
  }
  return best;
}

bag::BagFn single_kernel(int variant, int form) {
  struct All {
    bag::BagFn fn[bag::kVariants][bag::kForms] = {};
    All() {
      bag_kernels_8(fn);
      bag_kernels_4(fn);
      bag_kernels_2(fn);
      bag_kernels_plain(fn);
    }
  };
  static const All all;
  return all.fn[variant][form];
}

// The launch may be set up while the stream's previous one drains: the kernels
// wait for its results themselves (griddepcontrol.wait).  0.3 to 0.6 us less
// between launches of 4 to 12 us.
template <typename Arg>
cudaError_t launch(void (*fn)(Arg), dim3 grid, const Arg& arg, cudaStream_t stream, int threads = bag::kThreads) {
  cudaLaunchAttribute overlap{};
  overlap.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  overlap.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3((unsigned)threads);
  cfg.stream = stream;
  cfg.attrs = &overlap;
  cfg.numAttrs = 1;
  g_launch_count.fetch_add(1, std::memory_order_relaxed);
  return cudaLaunchKernelEx(&cfg, fn, arg);
}

}  // namespace

cudaError_t launch_bags(const SpmdmParams& p, int bit_rate, cudaStream_t stream) {
  bag::BagCall c;
  bag_table_of(p, &c.t);
  for (int i = 0; i < p.num_peers; ++i) {
    c.peers[i] = p.peer_out[i];
  }
  const int64_t sms = sm_count();
  int tiles = 0;
  const int fmt = format_of(p, bit_rate);
  const int v = pick_variant(c.t, fmt, p.output_size, p.bags_beside, true, sms, &tiles);
  if (bag::is_quantized(fmt) && p.num_peers <= 0 && !(c.t.flags & kNoBag) && p.index_size <= 0x7fffff00LL) {
    FewBagsCall few{};
    few.bits = fmt;
    few.words = bag::few_by_words(c.t);
    few.units = bag::few_units(c.t, fmt);
    few.warp_chunks = kVariantInfo[v].cpl;
    few.mapped = c.t.flags & kPruned;
    few.tiles = (c.t.cols + bag::kFewColumns - 1) / bag::kFewColumns;
    few.bags = p.output_size;
    few.beside = p.bags_beside;
    few.rows = p.index_size;
    if (few_bags_pay(few, sms)) {
      return launch<bag::BagCall>(bag::few_bags(fmt), dim3((unsigned)p.output_size, (unsigned)few.tiles), c, stream, bag::kFewThreads);
    }
  }
  const int64_t blocks = blocks_of(p.output_size, v);
  if (blocks <= 0 || blocks > 0x7fffffffLL || tiles > 65535) {
    return cudaErrorInvalidValue;
  }
  // The deep form while what is on the chip fits it at once.  With a pruning map, one more trip to memory in every
  // stretch, up to two such launches' worth and whatever runs beside: 2-bit D = 128, 11000 bags 16.9 against 14.5 us,
  // 14000 20.0 / 18.5, 20000 27.6 / 25.5; quarter warps on 16 streams 9.5 / 7.1.  (Dense tables lose there: 8-bit D = 128,
  // 14000 bags 29.7 against 33.6; 10000 bags on 16 streams 7.0 against 8.3.  Narrower groups do once anything runs beside
  // them: 4-bit D = 64, 4096 bags on 16 streams 3.2 against 3.6.)
  const int form = form_of(c.t);
  const int64_t bags = kVariantInfo[v].g == 32 ? bags_at_a_time(p.output_size, p.bags_beside) : p.output_size + p.bags_beside;
  const int64_t fit = deep_fit(sms);
  const bool deep = form == bag::kMapped ? blocks * tiles <= 2 * fit : form != bag::kWide && blocks_of(bags, v) * tiles <= fit;
  return launch<bag::BagCall>(single_kernel(v, deep ? bag::kDeepForms + form : form), dim3((unsigned)blocks, (unsigned)tiles), c, stream);
}

// ---- several tables per launch --------------------------------------------------

struct UnitsLaunch {
  bag::BagUnits units;
  unsigned blocks;
  int form;
};

MultiPlan::MultiPlan() = default;
MultiPlan::~MultiPlan() = default;

// One launch takes up to kMaxTables tables of any row formats with kMaxUnits
// column tiles in all.
cudaError_t build_multi_plan(const SpmdmParams* tables, const int* bit_rates, size_t count, MultiPlan* plan) {
  int64_t bags = 0;
  for (size_t t = 0; t < count; ++t) {
    bags += tables[t].output_size;
  }
  struct Unit {
    size_t table;
    int variant, tile;
    int64_t blocks;
    int form;
    double work;
  };
  std::vector<Unit> order;
  std::vector<BagTable> bag_tables(count);
  const int64_t sms = sm_count();
  for (size_t t = 0; t < count; ++t) {
    if (tables[t].output_size <= 0) {
      continue;  // nothing to pool, nothing to store
    }
    int tiles = 0;
    bag_table_of(tables[t], &bag_tables[t]);
    const int v = pick_variant(bag_tables[t], format_of(tables[t], bit_rates[t]), bags, 0, false, sms, &tiles);
    const int64_t blocks = blocks_of(tables[t].output_size, v);
    if (blocks > 0x7fffffffLL || tiles > 65535) {
      return cudaErrorInvalidValue;
    }
    for (int i = 0; i < tiles; ++i) {
      order.push_back({t, v, i, blocks, form_of(bag_tables[t]),
                       (double)tables[t].index_size / std::max<int64_t>(1, blocks) * bag_tables[t].data_bytes});
    }
  }
  // Tables of one form go together, the longest-running blocks first: the short ones fill the last wave.
  std::stable_sort(order.begin(), order.end(), [](const Unit& a, const Unit& b) {
    return a.form != b.form ? a.form > b.form : a.work > b.work;
  });
  std::vector<int> place(count);  // of a table in the launch being filled
  for (size_t i = 0; i < order.size();) {
    plan->launches.emplace_back(new UnitsLaunch);
    UnitsLaunch& l = *plan->launches.back();
    bag::BagUnits& u = l.units;
    u.count = 0;
    l.form = order[i].form;
    int64_t blocks = 0;
    int tables_in = 0;
    std::fill(place.begin(), place.end(), -1);
    for (; i < order.size() && order[i].form == l.form && u.count < bag::kMaxUnits &&
         blocks + order[i].blocks <= 0x7fffffffLL; ++i) {
      int& at = place[order[i].table];
      if (at < 0) {
        if (tables_in == bag::kMaxTables) {
          break;
        }
        at = tables_in++;
        const SpmdmParams& p = tables[order[i].table];
        u.t[at] = bag_tables[order[i].table];
        std::copy(p.peer_out, p.peer_out + p.num_peers, u.peers[at]);
      }
      const int k = u.count++;
      u.first_block[k] = (int32_t)blocks;
      u.unit[k] = {(uint8_t)order[i].variant, (uint8_t)at, (uint16_t)order[i].tile};
      blocks += order[i].blocks;
    }
    u.first_block[u.count] = (int32_t)blocks;
    l.blocks = (unsigned)blocks;
  }
  return cudaSuccess;
}

cudaError_t launch_multi_plan(const MultiPlan& plan, cudaStream_t stream) {
  for (const auto& l : plan.launches) {
    const bag::BagUnitsFn fn = l->form == bag::kWide ? bag_units_wide()
        : l->form == bag::kMapped                    ? bag_units_mapped()
        : l->form == bag::kFull                      ? bag_units_full()
                                                     : bag_units_lean();
    const cudaError_t e = launch<bag::BagUnits>(fn, dim3(l->blocks), l->units, stream);
    if (e != cudaSuccess) {
      return e;
    }
  }
  return cudaSuccess;
}

cudaError_t launch_tables(const SpmdmParams* tables, const int* bit_rates, size_t count, cudaStream_t stream) {
  if (g_kernel_choice.load(std::memory_order_relaxed) == FBGEMM_B200_KERNEL_GENERIC) {
    for (size_t t = 0; t < count; ++t) {
      const cudaError_t e = tables[t].output_size > 0 ? launch_spmdm(tables[t], bit_rates[t], stream) : cudaSuccess;
      if (e != cudaSuccess) {
        return e;
      }
    }
    return cudaSuccess;
  }
  MultiPlan plan;
  const cudaError_t e = build_multi_plan(tables, bit_rates, count, &plan);
  return e == cudaSuccess ? launch_multi_plan(plan, stream) : e;
}

}  // namespace fbgemm_b200
