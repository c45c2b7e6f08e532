// The multi-table lookup kernel for tables of any size (see bag_kernel.cuh).
#include "bag_kernel.cuh"

namespace fbgemm_b200 {

bag::BagUnitsFn bag_units_wide() {
  return bag::bag_units_kernel<true>;
}

}  // namespace fbgemm_b200
