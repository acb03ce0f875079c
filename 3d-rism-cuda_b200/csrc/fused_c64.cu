// Instantiations of the plane kernels (fused.cuh): FP64, cell edges 128, 160, 256.
#include "fused.cuh"

namespace rism3d {
namespace fused {

template <> Vtable<double> table_c<double>(int N, int V) {
  switch (N) {
    case 128: return table_v<double, 128>(V);
    case 160: return table_v<double, 160>(V);
    case 256: return table_v<double, 256>(V);
  }
  return {};
}

}  // namespace fused
}  // namespace rism3d
