// Instantiations of the plane kernels (fused.cuh): FP64, cell edges 60, 64, 80.
#include "fused.cuh"

namespace rism3d {
namespace fused {

template <> Vtable<double> table_b<double>(int N, int V) {
  switch (N) {
    case 60: return table_v<double, 60>(V);
    case 64: return table_v<double, 64>(V);
    case 80: return table_v<double, 80>(V);
  }
  return {};
}

}  // namespace fused
}  // namespace rism3d
