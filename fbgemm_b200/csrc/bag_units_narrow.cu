// The multi-table lookup kernel for tables whose rows all lie within 4 GB (see bag_kernel.cuh).
#include "bag_kernel.cuh"

namespace fbgemm_b200 {

bag::BagUnitsFn bag_units_narrow() {
  return bag::bag_units_kernel<false>;
}

}  // namespace fbgemm_b200
