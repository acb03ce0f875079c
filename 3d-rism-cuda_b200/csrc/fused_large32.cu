// Instantiations of the three-kernel iteration (fused.cuh): FP32, edges 256.
#include "fused.cuh"

namespace rism3d {
namespace fused {

template <> Vtable<float> table_large<float>(int N, int V) {
  switch (N) {
    case 256: return table_v<float, 256>(V);
  }
  return {nullptr, nullptr};
}

}  // namespace fused
}  // namespace rism3d
