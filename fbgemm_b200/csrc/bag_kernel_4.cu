// The single-table lookup kernels for 4-bit rows (see bag_kernel.cuh).
#include "bag_kernel.cuh"

namespace fbgemm_b200 {

void bag_kernels_4(bag::BagFn (*fn)[bag::kForms]) {
  using namespace bag;
#define ENTRY(FMT, VB, CPL, G)                                                        \
  fn[id_##FMT##_##VB##_##CPL##_##G][0] = bag_kernel<FMT, VB, CPL, G, kLean>;         \
  fn[id_##FMT##_##VB##_##CPL##_##G][1] = bag_kernel<FMT, VB, CPL, G, kMapped>;       \
  fn[id_##FMT##_##VB##_##CPL##_##G][2] = bag_kernel<FMT, VB, CPL, G, kWide>;         \
  fn[id_##FMT##_##VB##_##CPL##_##G][3] = bag_kernel_deep<FMT, VB, CPL, G, kLean>;    \
  fn[id_##FMT##_##VB##_##CPL##_##G][4] = bag_kernel_deep<FMT, VB, CPL, G, kMapped>;
  FBGEMM_B200_BAG_VARIANTS_4(ENTRY)
#undef ENTRY
}

}  // namespace fbgemm_b200
