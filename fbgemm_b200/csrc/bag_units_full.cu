// The multi-table lookup kernel with all options but pruning maps (see bag_kernel.cuh).
#include "bag_kernel.cuh"

namespace fbgemm_b200 {

bag::BagUnitsFn bag_units_full() {
  return bag::bag_units_kernel<bag::kFull>;
}

}  // namespace fbgemm_b200
