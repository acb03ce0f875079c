// Instantiations of the plane kernels (fused.cuh): FP32, cell edges 60, 64, 72, 80.
#include "fused.cuh"

namespace rism3d {
namespace fused {

template <> Vtable<float> table_b<float>(int N, int V) {
  switch (N) {
    case 60: return table_v<float, 60>(V);
    case 64: return table_v<float, 64>(V);
    case 72: return table_v<float, 72>(V);
    case 80: return table_v<float, 80>(V);
  }
  return {};
}

}  // namespace fused
}  // namespace rism3d
