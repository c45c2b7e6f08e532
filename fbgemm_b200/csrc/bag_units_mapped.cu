// The multi-table lookup kernel with all options and pruning maps (see bag_kernel.cuh).
#include "bag_kernel.cuh"

namespace fbgemm_b200 {

bag::BagUnitsFn bag_units_mapped() {
  return bag::bag_units_kernel<bag::kMapped>;
}

}  // namespace fbgemm_b200
