// Instantiations of the plane kernels (fused.cuh): FP64, cell edges 32, 36, 40, 48.
#include "fused.cuh"

namespace rism3d {
namespace fused {

template <> Vtable<double> table_a<double>(int N, int V) {
  switch (N) {
    case 32: return table_v<double, 32>(V);
    case 36: return table_v<double, 36>(V);
    case 40: return table_v<double, 40>(V);
    case 48: return table_v<double, 48>(V);
  }
  return {};
}

}  // namespace fused
}  // namespace rism3d
