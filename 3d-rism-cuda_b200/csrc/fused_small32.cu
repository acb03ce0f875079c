// Instantiations of the three-kernel iteration (fused.cuh): FP32, edges 32, 48, 64.
#include "fused.cuh"

namespace rism3d {
namespace fused {

template <> Vtable<float> table_small<float>(int N, int V) {
  switch (N) {
    case 32: return table_v<float, 32>(V);
    case 48: return table_v<float, 48>(V);
    case 64: return table_v<float, 64>(V);
  }
  return {nullptr, nullptr};
}

}  // namespace fused
}  // namespace rism3d
