// Instantiations of the plane kernels (fused.cuh): FP32, cell edges 96, 128, 256.
#include "fused.cuh"

namespace rism3d {
namespace fused {

template <> Vtable<float> table_c<float>(int N, int V) {
  switch (N) {
    case 96: return table_v<float, 96>(V);
    case 128: return table_v<float, 128>(V);
    case 256: return table_v<float, 256>(V);
  }
  return {};
}

}  // namespace fused
}  // namespace rism3d
