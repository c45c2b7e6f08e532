// The single-table lookup kernels for 8-bit rows (see bag_kernel.cuh).
#include "bag_kernel.cuh"

namespace fbgemm_b200 {

void bag_kernels_8(bag::BagFn (*fn)[bag::kForms]) {
  using namespace bag;
#define ENTRY(FMT, VB, CPL, G)                                                                \
  fn[id_##FMT##_##VB##_##CPL##_##G][kLean] = bag_kernel<FMT, VB, CPL, G, kLean>;              \
  fn[id_##FMT##_##VB##_##CPL##_##G][kFull] = bag_kernel<FMT, VB, CPL, G, kFull>;              \
  fn[id_##FMT##_##VB##_##CPL##_##G][kWide] = bag_kernel<FMT, VB, CPL, G, kWide>;              \
  fn[id_##FMT##_##VB##_##CPL##_##G][kMapped] = bag_kernel<FMT, VB, CPL, G, kMapped>;          \
  fn[id_##FMT##_##VB##_##CPL##_##G][kDeepForms + kLean] = bag_kernel_deep<FMT, VB, CPL, G, kLean>; \
  fn[id_##FMT##_##VB##_##CPL##_##G][kDeepForms + kFull] = bag_kernel_deep<FMT, VB, CPL, G, kFull>; \
  fn[id_##FMT##_##VB##_##CPL##_##G][kDeepForms + kMapped] = bag_kernel_deep<FMT, VB, CPL, G, kMapped>;
  FBGEMM_B200_BAG_VARIANTS_8(ENTRY)
#undef ENTRY
}

}  // namespace fbgemm_b200
