// Instantiations of the adjoint's one-launch solve (fused_adjoint.cuh): FP64,
// cell edges 32, 36, 40, 48, 60, 64, 72.
#include "fused_adjoint.cuh"

namespace rism3d {
namespace fused {

template <> AdjointLaunch<double> adjoint_table_x<double>(int N, int V) {
  switch (N) {
    case 32: return adjoint_table_v<double, 32>(V);
    case 36: return adjoint_table_v<double, 36>(V);
    case 40: return adjoint_table_v<double, 40>(V);
    case 48: return adjoint_table_v<double, 48>(V);
    case 60: return adjoint_table_v<double, 60>(V);
    case 64: return adjoint_table_v<double, 64>(V);
    case 72: return adjoint_table_v<double, 72>(V);
  }
  return nullptr;
}

}  // namespace fused
}  // namespace rism3d
