// Instantiations of the adjoint's one-launch solve (fused_adjoint.cuh): FP64.
#include "fused_adjoint.cuh"

namespace rism3d {
namespace fused {

template <> AdjointLaunch<double> adjoint_table<double>(int N, int V) {
  switch (N) {
    case 32: return adjoint_table_v<double, 32>(V);
    case 48: return adjoint_table_v<double, 48>(V);
    case 64: return adjoint_table_v<double, 64>(V);
    case 96: return adjoint_table_v<double, 96>(V);
    case 128: return adjoint_table_v<double, 128>(V);
    case 256: return adjoint_table_v<double, 256>(V);
  }
  return nullptr;
}

}  // namespace fused
}  // namespace rism3d
