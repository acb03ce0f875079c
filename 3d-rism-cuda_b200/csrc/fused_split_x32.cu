// Instantiations of the split form of the folded iteration (fused_split.cuh):
// FP32, edges 32, 36, 40, 48, 60, 64, 72, 80, 96, 100, 108.
#include "fused_split.cuh"

namespace rism3d {
namespace fused {

template <> SplitRun<float> split_table_x<float>(int N, int V, int *lines) {
  switch (N) {
    case 32: return split_v<float, 32>(V, lines);
    case 36: return split_v<float, 36>(V, lines);
    case 40: return split_v<float, 40>(V, lines);
    case 48: return split_v<float, 48>(V, lines);
    case 60: return split_v<float, 60>(V, lines);
    case 64: return split_v<float, 64>(V, lines);
    case 72: return split_v<float, 72>(V, lines);
    case 80: return split_v<float, 80>(V, lines);
    case 96: return split_v<float, 96>(V, lines);
    case 100: return split_v<float, 100>(V, lines);
    case 108: return split_v<float, 108>(V, lines);
  }
  return nullptr;
}

}  // namespace fused
}  // namespace rism3d
