// The single-table lookup kernels for fp32, fp16, bf16 and FP8 rows (see bag_kernel.cuh).
#include "bag_kernel.cuh"

namespace fbgemm_b200 {

void bag_kernels_plain(bag::BagFn (*fn)[bag::kForms]) {
  using namespace bag;
#define ENTRY(FMT, VB, CPL, G)                                                        \
  fn[id_##FMT##_##VB##_##CPL##_##G][0] = bag_kernel<FMT, VB, CPL, G, kLean>;         \
  fn[id_##FMT##_##VB##_##CPL##_##G][1] = bag_kernel<FMT, VB, CPL, G, kMapped>;       \
  fn[id_##FMT##_##VB##_##CPL##_##G][2] = bag_kernel<FMT, VB, CPL, G, kWide>;         \
  fn[id_##FMT##_##VB##_##CPL##_##G][3] = bag_kernel_deep<FMT, VB, CPL, G, kLean>;    \
  fn[id_##FMT##_##VB##_##CPL##_##G][4] = bag_kernel_deep<FMT, VB, CPL, G, kMapped>;
  FBGEMM_B200_BAG_VARIANTS_PLAIN(ENTRY)
#undef ENTRY
}

}  // namespace fbgemm_b200
