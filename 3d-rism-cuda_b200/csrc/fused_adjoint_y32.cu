// Instantiations of the adjoint's one-launch solve (fused_adjoint.cuh): FP32,
// cell edges 80, 96, 100, 108, 120, 128, 256.
#include "fused_adjoint.cuh"

namespace rism3d {
namespace fused {

template <> AdjointLaunch<float> adjoint_table_y<float>(int N, int V) {
  switch (N) {
    case 80: return adjoint_table_v<float, 80>(V);
    case 96: return adjoint_table_v<float, 96>(V);
    case 100: return adjoint_table_v<float, 100>(V);
    case 108: return adjoint_table_v<float, 108>(V);
    case 120: return adjoint_table_v<float, 120>(V);
    case 128: return adjoint_table_v<float, 128>(V);
    case 256: return adjoint_table_v<float, 256>(V);
  }
  return nullptr;
}

}  // namespace fused
}  // namespace rism3d
