// Instantiations of the three-kernel iteration (fused.cuh): FP64, edges 256.
#include "fused.cuh"

namespace rism3d {
namespace fused {

template <> Vtable<double> table_large<double>(int N, int V) {
  switch (N) {
    case 256: return table_v<double, 256>(V);
  }
  return {nullptr, nullptr};
}

}  // namespace fused
}  // namespace rism3d
