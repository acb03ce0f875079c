// Instantiations of the three-kernel iteration (fused.cuh): FP64, edges 32, 48, 64.
#include "fused.cuh"

namespace rism3d {
namespace fused {

template <> Vtable<double> table_small<double>(int N, int V) {
  switch (N) {
    case 32: return table_v<double, 32>(V);
    case 48: return table_v<double, 48>(V);
    case 64: return table_v<double, 64>(V);
  }
  return {nullptr, nullptr};
}

}  // namespace fused
}  // namespace rism3d
