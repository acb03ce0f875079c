// The three-kernel iteration (fused.cuh) as the solver sees it.
#pragma once

#include "passes.cuh"

namespace rism3d {
namespace fused {

// set-up (attributes, cluster counts; false: not on this device) and launch
// of kernel 0 (plane A), 1 (z lines), 2 (plane R), 3 (the pass after the loop) or 4 (a
// whole phase) of one (T, edge, sites)
template <typename T>
struct Vtable {
  bool (*setup)(FusedPlan &, int);
  cudaError_t (*launch)(const FusedPlan &, int, bool, int, int, const IterArgs<T> &, cudaStream_t);
};

// one translation unit per group of edges
template <typename T> Vtable<T> table_small(int N, int V);    // 32, 48, 64
template <typename T> Vtable<T> table_medium(int N, int V);   // 96, 128
template <typename T> Vtable<T> table_large(int N, int V);    // 256

}  // namespace fused
}  // namespace rism3d
