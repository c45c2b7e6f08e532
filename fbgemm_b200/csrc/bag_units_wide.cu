// The multi-table lookup kernel with all options and 64-bit positions and rows (see bag_kernel.cuh).
#include "bag_kernel.cuh"

namespace fbgemm_b200 {

bag::BagUnitsFn bag_units_wide() {
  return bag::bag_units_kernel<bag::kWide>;
}

}  // namespace fbgemm_b200
