// Instantiations of the split form of the folded iteration (fused_split.cuh):
// FP32, edges 120, 128, 144, 160, 180, 192, 200, 216, 240, 256.
#include "fused_split.cuh"

namespace rism3d {
namespace fused {

template <> SplitRun<float> split_table_y<float>(int N, int V, int *lines) {
  switch (N) {
    case 120: return split_v<float, 120>(V, lines);
    case 128: return split_v<float, 128>(V, lines);
    case 144: return split_v<float, 144>(V, lines);
    case 160: return split_v<float, 160>(V, lines);
    case 180: return split_v<float, 180>(V, lines);
    case 192: return split_v<float, 192>(V, lines);
    case 200: return split_v<float, 200>(V, lines);
    case 216: return split_v<float, 216>(V, lines);
    case 240: return split_v<float, 240>(V, lines);
    case 256: return split_v<float, 256>(V, lines);
  }
  return nullptr;
}

}  // namespace fused
}  // namespace rism3d
