// The multi-table lookup kernel of tables whose indices all name rows (see bag_kernel.cuh).
#include "bag_kernel.cuh"

namespace fbgemm_b200 {

bag::BagUnitsFn bag_units_lean() {
  return bag::bag_units_kernel<bag::kLean>;
}

}  // namespace fbgemm_b200
