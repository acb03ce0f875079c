// Arguments and device state of the adjoint's one-launch solve
// (fused_adjoint.cuh), shared with its host side (adjoint.cu).
#pragma once

#include "fused_api.cuh"

namespace rism3d {
namespace fused {

constexpr int kAdjDepth = 6;   // Anderson history of the adjoint solve

struct AdjointState {
  int done;        // 0 running, 1 converged, 2 diverged, 3 step limit, 4 stalled
                   // at the FP32 floor, 5 launched without its clusters
  unsigned bar;    // arrival count of the barriers: zero again once every block
                   // has left, else a wait gave up
  int it, ns, slot, since_best;
  double best, bnorm;
  double gram[kAdjDepth * kAdjDepth];
  double coef[kAdjDepth];
};

template <typename T>
struct AdjointArgs {
  IterArgs<T> it;              // cell, transform buffer, tables, chi, barrier
  const T *G, *w;              // closure derivative and right-hand side [V][N]
  T *xi, *Lxi;                 // [V][N]
  T *ys, *rs;                  // histories [kAdjDepth][V][N]
  double *part;                // dots of every block
  int max_blocks;              // that it has room for
  AdjointState *st;
  double eta, tol;
  int maxit;
};

// launch (clusters null) or cluster count of a whole solve; false: not on
// this device
template <typename T>
using AdjointLaunch = bool (*)(const AdjointArgs<T> &, int *clusters, cudaStream_t);
template <typename T> AdjointLaunch<T> adjoint_table_x(int N, int V);   // 32-72
template <typename T> AdjointLaunch<T> adjoint_table_y(int N, int V);   // 80-128, 256
template <typename T> AdjointLaunch<T> adjoint_table(int N, int V) {    // null: no instantiation
  return N <= 72 ? adjoint_table_x<T>(N, V) : adjoint_table_y<T>(N, V);
}

}  // namespace fused
}  // namespace rism3d
