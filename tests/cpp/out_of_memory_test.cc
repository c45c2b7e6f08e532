// Host allocations that fail inside an entry point come back as a return code; nothing is thrown through the C ABI.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <new>
#include <vector>

#include "fbgemm_b200/embedding_c_api.h"

static int fail_in = -1;  // allocations until one fails

void* operator new(std::size_t bytes) {
  if (fail_in >= 0 && fail_in-- == 0) {
    throw std::bad_alloc();
  }
  if (void* p = std::malloc(bytes ? bytes : 1)) {
    return p;
  }
  throw std::bad_alloc();
}
void operator delete(void* p) noexcept {
  std::free(p);
}
void operator delete(void* p, std::size_t) noexcept {
  std::free(p);
}

int main() {
  // the entry points below only look at tables before they allocate: any non-null context will do
  std::vector<unsigned char> memory(1 << 20, 0);
  auto* ctx = reinterpret_cast<fbgemm_b200_ctx*>(memory.data());
  fbgemm_b200_table_call table;
  std::memset(&table, 0, sizeof(table));
  table.cfg.bit_rate = 8;
  table.cfg.index_bytes = table.cfg.offset_bytes = 8;
  table.cfg.block_size = 16;
  table.cfg.output_stride = table.cfg.input_stride = -1;
  table.cfg.use_offsets = table.cfg.absolute_offsets = 1;
  const int64_t column = 0;
  for (int at = 0; at < 3; ++at) {   // the set itself, its tables, their columns
    fbgemm_b200_table_set* set = reinterpret_cast<fbgemm_b200_table_set*>(1);
    fail_in = at;
    const int rc = fbgemm_b200_table_set_create(ctx, &table, &column, 1, &set);
    const bool failed = fail_in < 0;
    fail_in = -1;
    if (!failed || rc != FBGEMM_B200_ENOMEM || set != nullptr || !std::strstr(fbgemm_b200_last_error(), "memory")) {
      std::printf("table_set_create, allocation %d: rc %d, %s\n", at, rc, fbgemm_b200_last_error());
      return 1;
    }
  }
  fbgemm_b200_multi_plan* plan = reinterpret_cast<fbgemm_b200_multi_plan*>(1);
  fail_in = 0;
  if (fbgemm_b200_multi_plan_create(ctx, &table, 1, 0, 0, 0, &plan) != FBGEMM_B200_ENOMEM || plan != nullptr) {
    std::printf("multi_plan_create\n");
    return 1;
  }
  fail_in = -1;
  return 0;
}
