// Instantiations of the three-kernel iteration (fused.cuh): FP32, edges 96, 128.
#include "fused.cuh"

namespace rism3d {
namespace fused {

template <> Vtable<float> table_medium<float>(int N, int V) {
  switch (N) {
    case 96: return table_v<float, 96>(V);
    case 128: return table_v<float, 128>(V);
  }
  return {nullptr, nullptr};
}

}  // namespace fused
}  // namespace rism3d
