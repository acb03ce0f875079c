// The folded iteration for cells whose edges differ: the stages of fused.cuh
// as five kernels, each templated on one edge only, so that any combination
// of instantiated edges works:
//
//   rows A (nx), columns (ny), z lines (nz), inverse columns (ny), rows R (nx)
//
// The columns pass through memory on their own (64 B per point and cycle more
// than the plane kernels in FP64 with two sites, still 328 against 456 B and
// five launches against a dozen).  chi comes from an octant table (chi_octant)
// instead of a spline evaluation per point and cycle.
#pragma once

#include "fused.cuh"

namespace rism3d {
namespace fused {

// One batch of LB rows per block: row r of ny nz P is (p, z, y)
template <typename T, int N, int V, bool REF>
__global__ void __launch_bounds__(Lines<N>::TH, (Lines<N>::template minb<T>()))
    k_rows_a(IterArgs<T> a0, bool hnc) {
  typedef CxT<T> C;
  using L = Lines<N>;
  extern __shared__ __align__(16) unsigned char fused_sm[];
  const IterArgs<T> a = solute_view<T, V>(a0);
  if (a.st->done) return;
  const int row_l = threadIdx.x / L::R2, t = threadIdx.x % L::R2;
  const int rows = a.ny * a.nz, r = blockIdx.x * L::LB + row_l;
  const bool live = row_l < L::LB && r < rows * ((V + 1) / 2);
  const int p = live ? r / rows : 0, yz = live ? r - p * rows : 0, z = yz / a.ny, y = yz - z * a.ny;
  const size_t base = (size_t)yz * N;
  update_row<T, N, V, REF, false>(a, a.st, reinterpret_cast<C *>(fused_sm) + row_l * L::LS, t, live,
                                  (size_t)(2 * p) * a.n + base,
                                  cmul(a.tw[N + y], a.tw[N + a.ny + z]), (y + z) & 1,
                                  a.buf + (size_t)p * a.n + base, a.tw, a.roots, hnc);
}

template <typename T, int N, int V, bool REF>
__global__ void __launch_bounds__(Lines<N>::TH, (Lines<N>::template minb<T>()))
    k_rows_r(IterArgs<T> a0, bool hnc) {
  typedef CxT<T> C;
  using L = Lines<N>;
  extern __shared__ __align__(16) unsigned char fused_sm[];
  const IterArgs<T> a = solute_view<T, V>(a0);
  if (a.st->done) {                                // this solute has stopped
    if (blockIdx.x == 0 && threadIdx.x == 0) loop_test_all(a0);
    return;
  }
  const int row_l = threadIdx.x / L::R2, t = threadIdx.x % L::R2;
  const int rows = a.ny * a.nz, r = blockIdx.x * L::LB + row_l;
  const bool live = row_l < L::LB && r < rows * ((V + 1) / 2);
  const int p = live ? r / rows : 0, yz = live ? r - p * rows : 0, z = yz / a.ny, y = yz - z * a.ny;
  const size_t base = (size_t)yz * N;
  C *line = reinterpret_cast<C *>(fused_sm) + row_l * L::LS;
  double acc[6] = {0, 0, 0, 0, 0, 0};
  rows_inverse<T, N>(a.buf + (size_t)p * a.n + base, line, t, live, a.roots);
  if (live)
    residual_row<T, N, V, REF, false>(a, a.st, line, t, 2 * p,
                                      (size_t)(2 * p) * a.n + base,
                                      cmul(a.tw[N + y], a.tw[N + a.ny + z]), (y + z) & 1, a.tw,
                                      a.st->count <= 0, hnc, acc);
  block_sums<L::TH>(acc, a.part);
  finish_cycle(a0, a, V);
}

// After the loop (fused.cuh, k_plane_final): the last cycle's inverse columns
// are in the buffer already
template <typename T, int N, int V, bool REF>
__global__ void __launch_bounds__(Lines<N>::TH) k_rows_final(IterArgs<T> a0, bool hnc) {
  typedef CxT<T> C;
  using L = Lines<N>;
  extern __shared__ __align__(16) unsigned char fused_sm[];
  const IterArgs<T> a = solute_view<T, V>(a0);
  const bool snap = !REF && a.hout, update = a.st->done == 3 && a.st->mode != 0;
  if (!snap && !update) return;
  const int row_l = threadIdx.x / L::R2, t = threadIdx.x % L::R2;
  const int rows = a.ny * a.nz, r = blockIdx.x * L::LB + row_l;
  const bool live = row_l < L::LB && r < rows * ((V + 1) / 2);
  const int p = live ? r / rows : 0, yz = live ? r - p * rows : 0, z = yz / a.ny, y = yz - z * a.ny;
  C *line = reinterpret_cast<C *>(fused_sm) + row_l * L::LS;
  rows_inverse<T, N>(a.buf + (size_t)p * a.n + (size_t)yz * N, line, t, live, a.roots);
  if (live)
    final_row<T, N, V, REF>(a, line, t, p, (size_t)yz * N, cmul(a.tw[N + y], a.tw[N + a.ny + z]),
                            (y + z) & 1, snap, update, hnc);
}

// LB columns of one xy plane per block, in place
template <typename T, int N, int V, bool INV>
__global__ void __launch_bounds__(Lines<N>::TH, (Lines<N>::template minb<T>()))
    k_columns(IterArgs<T> a0) {
  typedef CxT<T> C;
  using L = Lines<N>;
  extern __shared__ __align__(16) unsigned char fused_sm[];
  const IterArgs<T> a = solute_view<T, V>(a0);
  if (a.st->done) return;
  const int tiles = (a.nx + L::LB - 1) / L::LB, plane = blockIdx.x / tiles,
            c0 = (blockIdx.x - plane * tiles) * L::LB;
  C *pc = a.buf + (size_t)plane * a.nx * N + c0;
  columns<T, N, INV, false>(pc, pc, a.nx, min(L::LB, a.nx - c0), reinterpret_cast<C *>(fused_sm),
                     a.roots + a.nx);
}

template <typename T, int N, int V>
__global__ void __launch_bounds__(ZShape<T, N, V>::TH, (ZShape<T, N, V>::MINB))
    k_zlines_any(IterArgs<T> a0) {
  extern __shared__ __align__(16) unsigned char fused_sm[];
  const IterArgs<T> a = solute_view<T, V>(a0);
  if (a.st->done) return;
  zline_tile<T, N, V, false, false>(a, reinterpret_cast<CxT<T> *>(fused_sm),
                                    a.roots + a.nx + a.ny, a.nx, a.ny, blockIdx.x);
}

// which: 0 rows A, 1 columns, 2 z lines, 3 inverse columns, 4 rows R, 5 the
// pass after the loop; which < 0: set-up (attributes).  rows_blocks: blocks of
// the row kernels.
template <typename T, int N, int V>
struct SplitKernels {
  static_assert(V % 2 == 0, "whole site pairs");
  using L = Lines<N>;
  using Z = ZShape<T, N, V>;
  template <typename K> static void attr(K k, size_t b, cudaError_t &e) {
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)b);
  }
  static int rows_blocks(int ny, int nz) {
    return (int)(((long long)ny * nz * ((V + 1) / 2) + L::LB - 1) / L::LB);
  }
  template <bool REF>
  static void rows(int which, int hnc, int nb, const IterArgs<T> &a, cudaStream_t st,
                   cudaError_t &e) {
    const size_t s = L::template smem<T>();
    const dim3 g(rows_blocks(a.ny, a.nz), nb);
    if (which < 0) {
      attr(k_rows_a<T, N, V, REF>, s, e);
      attr(k_rows_r<T, N, V, REF>, s, e);
      attr(k_rows_final<T, N, V, REF>, s, e);
    } else if (which == 0) {
      k_rows_a<T, N, V, REF><<<g, L::TH, s, st>>>(a, hnc != 0);
    } else if (which == 4) {
      k_rows_r<T, N, V, REF><<<g, L::TH, s, st>>>(a, hnc != 0);
    } else {
      k_rows_final<T, N, V, REF><<<g, L::TH, s, st>>>(a, hnc != 0);
    }
  }
  static cudaError_t run(int which, int axis, bool ref, int hnc, int nb, const IterArgs<T> &a,
                         cudaStream_t st) {
    cudaError_t e = cudaSuccess;
    if (axis == 0) {
      if constexpr (sizeof(T) == 4) {
        if (ref || which < 0) rows<true>(which, hnc, nb, a, st, e);
      }
      if (!ref || which < 0) rows<false>(which, hnc, nb, a, st, e);
    } else if (axis == 1) {
      const size_t s = sizeof(CxT<T>) * L::LB * (size_t)N;
      const dim3 g((a.nx + L::LB - 1) / L::LB * a.nz * ((V + 1) / 2), nb);
      if (which < 0) {
        attr(k_columns<T, N, V, false>, s, e);
        attr(k_columns<T, N, V, true>, s, e);
      } else if (which == 1) {
        k_columns<T, N, V, false><<<g, L::TH, s, st>>>(a);
      } else {
        k_columns<T, N, V, true><<<g, L::TH, s, st>>>(a);
      }
    } else {
      if (which < 0) attr(k_zlines_any<T, N, V>, Z::smem(), e);
      else
        k_zlines_any<T, N, V><<<dim3((a.nx + Z::CW - 1) / Z::CW * (a.ny / 2), nb), Z::TH, Z::smem(),
                                st>>>(a);
    }
    return e == cudaSuccess ? cudaGetLastError() : e;
  }
};

template <typename T, int N>
SplitRun<T> split_v(int V, int *lines) {
  if (lines) *lines = Lines<N>::LB;
  switch (V) {
    case 2: return SplitKernels<T, N, 2>::run;
    case 4: return SplitKernels<T, N, 4>::run;
  }
  return nullptr;
}

}  // namespace fused
}  // namespace rism3d
