// Instantiations of the three-kernel iteration (fused.cuh): FP64, edges 96, 128.
#include "fused.cuh"

namespace rism3d {
namespace fused {

template <> Vtable<double> table_medium<double>(int N, int V) {
  switch (N) {
    case 96: return table_v<double, 96>(V);
    case 128: return table_v<double, 128>(V);
  }
  return {nullptr, nullptr};
}

}  // namespace fused
}  // namespace rism3d
