// The single-table lookup kernels for 4-bit rows (see bag_kernel.cuh).
#include "bag_kernel.cuh"

namespace fbgemm_b200 {

void bag_kernels_4(bag::BagFn (*fn)[4]) {
  using namespace bag;
#define ENTRY(FMT, VB, CPL, G)                                                         \
  fn[id_##FMT##_##VB##_##CPL##_##G][0] = bag_kernel<FMT, VB, CPL, G, false>;          \
  fn[id_##FMT##_##VB##_##CPL##_##G][1] = bag_kernel<FMT, VB, CPL, G, true>;           \
  fn[id_##FMT##_##VB##_##CPL##_##G][2] = deep_kernel<FMT, VB, CPL, G, false>();       \
  fn[id_##FMT##_##VB##_##CPL##_##G][3] = deep_kernel<FMT, VB, CPL, G, true>();
  FBGEMM_B200_BAG_VARIANTS_4(ENTRY)
#undef ENTRY
}

}  // namespace fbgemm_b200
