// The three-kernel iteration (fused.cuh) as the solver sees it.
#pragma once

#include "passes.cuh"

namespace rism3d {
namespace fused {

// The form that a cell's iteration takes.
enum Form { kLibrary, kPlanes, kSplit };

// Cubic cells, by what a step took on a B200 (us; V = 2, library passes /
// planes / split; one launch where that is the planes' form).  The plane
// kernels move fewer bytes and launch less; their cost is the exchange and
// barriers inside a plane, which grow where a row's threads do not fit a warp
// (R2 = 6, 10, 12) and with the registers of long FP64 lines.
//   FP64   64  45 / 23 / 36      72  58 / 49 / 46      80  66 / 41 / 51
//          96 103 / 73 / 68     100  96 / 110 / 104   108 125 / 169 / 155
//         120 165 / 179 / 161   128 179 / 132 / 152   144 233 / 327 / 231
//         160 339 / 320 / 336   180 584 / 658 / 551   192 590 / 603 / 555
//         200 819 / 844 / 724   216 830 / 1059 / 916  240 1317 / 1339 / 1169
//         256 1283 / 1107 / 1121
//   FP32   64  44 / 19 / 33      72  55 / 29 / 40      80  60 / 33 / 46
//          96  77 / 47 / 55     100  76 / 79 / 72     108  92 / 112 / 84
//         120 124 / 123 / 105   128 129 / 89 / 103    144 169 / 171 / 141
//         160 238 / 203 / 188   180 365 / 425 / 326   192 372 / 346 / 311
//         200 488 / 465 / 398   216 528 / 632 / 521   240 833 / 794 / 661
//         256 817 / 653 / 650
// Smaller edges, library passes / the planes' one launch:
//   FP64   32  32 / 15           36  31 / 16           40  34 / 22
//          48  37 / 21           60  43 / 30
//   FP32   32  29 / 12           36  32 / 13           40  34 / 16
//          48  36 / 16           60  39 / 19
// Four sites, library passes / the form chosen:
//   FP64   32  35 / 18   36  37 / 26   40  41 / 33   48  48 / 31   60  67 / 53
//          64  68 / 37   72  96 / 71   80 129 / 90   96 200 / 137 120 329 / 315
//         128 369 / 311 160 751 / 741 256 2819 / 2368
//   FP32   32  33 / 14   36  33 / 21   40  35 / 25   48  41 / 22   60  49 / 36
//          64  51 / 24   72  65 / 42   80  76 / 49   96 119 / 73  120 192 / 186
//         128 205 / 149 160 398 / 395 256 1493 / 1300
// Edges with another prime factor than 2, 3 and 5, above 256, and one, three or
// more than four sites run the library passes.
// Cells that are not cubic run the split form (72x60x48 50 / - / 41).
inline Form cubic_form(int N, bool fp64) {
  switch (N) {
    case 32: case 36: case 40: case 48: case 60: case 64: case 80: case 128: case 256:
      return kPlanes;
    case 72: case 96:
      return fp64 ? kSplit : kPlanes;
    case 160:
      return fp64 ? kPlanes : kSplit;
    case 120: case 144: case 180: case 192: case 200: case 240:
      return kSplit;
    case 100: case 108: case 216:
      return fp64 ? kLibrary : kSplit;
  }
  return kLibrary;
}

// set-up (attributes, cluster counts; false: not on this device) for nb solutes
// and, where not part of it, of the kernels of a cycle; launch of kernel 0 (plane A), 1 (z lines), 2 (plane R), 3 (the pass after the loop) or 4 (a
// whole phase) of one (T, edge, sites)
template <typename T>
struct Vtable {
  bool (*setup)(FusedPlan &, int nb, bool host_driven) = nullptr;
  bool (*planes)(FusedPlan &, int room) = nullptr;
  cudaError_t (*launch)(const FusedPlan &, int, bool, int, int, const IterArgs<T> &,
                        cudaStream_t) = nullptr;
};

// one translation unit per group of edges: up to 48, 60-80, above
template <typename T> Vtable<T> table_a(int N, int V);
template <typename T> Vtable<T> table_b(int N, int V);
template <typename T> Vtable<T> table_c(int N, int V);
template <typename T> Vtable<T> table(int N, int V) {
  return N <= 48 ? table_a<T>(N, V) : N <= 80 ? table_b<T>(N, V) : table_c<T>(N, V);
}

// The split form (fused_split.cuh): kernel `which` of the axis (0 x, 1 y, 2
// z) whose edge the table was asked for; lines: rows per block of the row
// kernels.
template <typename T>
using SplitRun = cudaError_t (*)(int which, int axis, bool ref, int hnc, int nb,
                                 const IterArgs<T> &, cudaStream_t);
template <typename T> SplitRun<T> split_table_x(int N, int V, int *lines);   // 32-108
template <typename T> SplitRun<T> split_table_y(int N, int V, int *lines);   // 120-256
template <typename T> SplitRun<T> split_table(int N, int V, int *lines) {
  return N <= 108 ? split_table_x<T>(N, V, lines) : split_table_y<T>(N, V, lines);
}

}  // namespace fused
}  // namespace rism3d
