// The single-table lookup kernels for fp32, fp16, bf16 and FP8 rows (see bag_kernel.cuh).
#include "bag_kernel.cuh"

namespace fbgemm_b200 {

void bag_kernels_plain(bag::BagFn (*fn)[4]) {
  using namespace bag;
#define ENTRY(FMT, VB, CPL, G)                                                         \
  fn[id_##FMT##_##VB##_##CPL##_##G][0] = bag_kernel<FMT, VB, CPL, G, false>;          \
  fn[id_##FMT##_##VB##_##CPL##_##G][1] = bag_kernel<FMT, VB, CPL, G, true>;           \
  fn[id_##FMT##_##VB##_##CPL##_##G][2] = deep_kernel<FMT, VB, CPL, G, false>();       \
  fn[id_##FMT##_##VB##_##CPL##_##G][3] = deep_kernel<FMT, VB, CPL, G, true>();
  FBGEMM_B200_BAG_VARIANTS_PLAIN(ENTRY)
#undef ENTRY
}

}  // namespace fbgemm_b200
