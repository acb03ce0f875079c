// The Anderson-accelerated transposed-Jacobian solve of the adjoint as one
// launch (cells and sites of fused.cuh).  A step of the host-driven solve is
// a dozen launches, a copy of seven dots to the host and a wait: 88 us at
// 64^3, where the work is a few us.  Here a step is three stages with a
// barrier over the blocks between them:
//   planes  xi = sum_i c_i y_i of one xy plane, packed, x- and y-DFT
//   z lines z-DFT, OZ product, inverse z-DFT (zline_tile)
//   planes  inverse y- and x-DFT: L xi; r = (G - 1)(w + L xi) - G xi, the
//           history slots r and y = xi + eta r, and the Gram dots
// after which every block reduces all dots in the same order and solves the
// bordered normal equations for the next coefficients (one warp, a row per
// lane).  The steps, their order and the stopping tests are those of the
// host-driven solve in adjoint.cu.
#pragma once

#include "adjoint_state.h"
#include "fused.cuh"

namespace rism3d {
namespace fused {

// Coefficients of min |sum c_i r_i|, sum c_i = 1, over m <= kAdjDepth stored
// residuals (gram[a][b] = <r_a, r_b>): Gauss-Jordan elimination with partial
// pivoting of the bordered system, lane l < m + 1 holding row l.  All lanes of
// one warp call it.
__device__ __forceinline__ void anderson_warp(const double *gram, int m, double *coef) {
  constexpr int D = kAdjDepth + 1;
  const int lane = threadIdx.x & 31, dd = m + 1;
  double sc = 0.0;
  for (int a = 0; a < m; ++a) sc = fmax(sc, gram[a * kAdjDepth + a]);
  if (!(sc > 0.0)) sc = 1.0;
  double row[D + 1];
#pragma unroll
  for (int k = 0; k < D; ++k) {
    double v = 0.0;
    if (lane < m && k < m) v = gram[lane * kAdjDepth + k] / sc;
    else if ((lane < m && k == m) || (lane == m && k < m)) v = 1.0;
    row[k] = v;
  }
  row[D] = lane == m ? 1.0 : 0.0;
  int mine = -1;                                   // the column this lane's row solves for
#pragma unroll
  for (int col = 0; col < D; ++col) {
    if (col < dd) {
      double best = (lane < dd && mine < 0) ? fabs(row[col]) : -1.0;
      int who = lane;
      for (int o = 4; o > 0; o >>= 1) {
        const double b2 = __shfl_xor_sync(0xffffffffu, best, o);
        const int w2 = __shfl_xor_sync(0xffffffffu, who, o);
        if (b2 > best || (b2 == best && w2 < who)) { best = b2; who = w2; }
      }
      who = __shfl_sync(0xffffffffu, who, 0);
      if (lane == who) mine = col;
      const double piv = __shfl_sync(0xffffffffu, row[col], who);
      const bool ok = fabs(piv) >= 1e-300;
      const double f = ok ? row[col] / piv : 0.0;
#pragma unroll
      for (int k = 0; k <= D; ++k) {
        const double p = __shfl_sync(0xffffffffu, row[k], who);
        if (lane != who && lane < dd) row[k] -= f * p;
      }
    }
  }
  double d = 0.0;
#pragma unroll
  for (int k = 0; k < D; ++k)
    if (k == mine) d = row[k];
  if (mine >= 0 && mine < m) coef[mine] = fabs(d) < 1e-300 ? 0.0 : row[D] / d;
}

template <typename T, int N, int V>
__device__ __forceinline__ void adjoint_forward(const AdjointArgs<T> &g, const AdjointState *s,
                                                CxT<T> *sm, const CxT<T> *tw,
                                                const CxT<T> *roots) {
  typedef CxT<T> C;
  using L = Lines<N>;
  constexpr int R1 = L::R1, R2 = L::R2, LB = L::LB, ST = L::ST, LS = L::LS;
  using W = Vecs<T, R1, false>;
  constexpr int P = (V + 1) / 2, VW = W::VW;
  const IterArgs<T> &a = g.it;
  const size_t n = (size_t)a.n;
  const int rank = blockIdx.x % L::NC, ncl = gridDim.x / L::NC;
  const int row_l = threadIdx.x / R2, t = threadIdx.x % R2;
  C *line = sm + row_l * LS;
  double cf[kAdjDepth];
  const int ns = s->it > 0 ? s->ns : 0;
#pragma unroll
  for (int i = 0; i < kAdjDepth; ++i) cf[i] = i < ns ? s->coef[i] : 0.0;
  for (int plane = blockIdx.x / L::NC; plane < N * P; plane += ncl) {
    const int p = plane / N, z = plane % N;
    C *pb = a.buf + (size_t)plane * N * N;
    __syncthreads();                               // the columns' exchange is free
#pragma unroll 1
    for (int rb = 0; rb < L::SH; rb += LB) {
      const bool live = L::FULL || (row_l < LB && rb + row_l < L::SH);
      const int y = rank * L::SH + (live ? rb + row_l : 0);
      const size_t base = (size_t)(2 * p) * n + ((size_t)z * N + y) * N;
      const C tyz = cmul(tw[N + y], tw[2 * N + z]);
      const int dyz = (y + z) & 1;
      row_sync<R2>();                              // the exchange's last readers are done
#pragma unroll 1
      for (int q = 0; q < (live ? W::TOT : 0); ++q) {
        const int x0 = VW * (t + R2 * q);
        T xv[2][VW];
#pragma unroll
        for (int b = 0; b < 2; ++b) {
#pragma unroll
          for (int k = 0; k < VW; ++k) xv[b][k] = T(0);
          const size_t j = base + b * n + x0;
          if (ns == 0) {
            ldv(xv[b], g.xi + j);
          } else {
            T yv[kAdjDepth][VW];
#pragma unroll
            for (int i = 0; i < kAdjDepth; ++i)
              if (i < ns) ldv(yv[i], g.ys + (size_t)i * V * n + j);
#pragma unroll
            for (int k = 0; k < VW; ++k) {
              double v = 0.0;
#pragma unroll
              for (int i = 0; i < kAdjDepth; ++i)
                if (i < ns) v += cf[i] * (double)yv[i][k];
              xv[b][k] = (T)v;
            }
            stv(g.xi + j, xv[b]);
          }
        }
#pragma unroll
        for (int k = 0; k < VW; ++k) {
          const int x = x0 + k;
          C c, w;
          c.x = xv[0][k];
          c.y = xv[1][k];
          const C kf = cmul(tw[x], tyz);
          const T dir = ((x & 1) ^ dyz) ? T(-1) : T(1);
          w.x = kf.x * dir;
          w.y = kf.y * dir;
          line[(x / R2) * ST + x % R2] = cmul(c, w);
        }
      }
      row_sync<R2>();
      rows_forward<T, N>(line, pb + (size_t)y * N, t, live, roots);
    }
    plane_sync<L::NC>();                           // every row of the plane is in L2
    columns<T, N, false, L::FULL>(pb + rank * L::SH, pb + rank * L::SH, N, L::SH, sm, roots);
  }
}

template <typename T, int N, int V>
__device__ __forceinline__ void adjoint_residual(const AdjointArgs<T> &g, const AdjointState *s,
                                                 CxT<T> *sm, const CxT<T> *tw,
                                                 const CxT<T> *roots) {
  typedef CxT<T> C;
  using L = Lines<N>;
  constexpr int R1 = L::R1, R2 = L::R2, LB = L::LB, ST = L::ST, LS = L::LS, TH = L::TH;
  using W = Vecs<T, R1, false>;
  constexpr int P = (V + 1) / 2, VW = W::VW;
  __shared__ double red[(TH + 31) / 32][kAdjDepth + 1];
  const IterArgs<T> &a = g.it;
  const size_t n = (size_t)a.n, tot = (size_t)V * n;
  const int slot = s->slot, nd = s->ns < kAdjDepth ? s->ns + 1 : kAdjDepth;
  const int rank = blockIdx.x % L::NC, cl = blockIdx.x / L::NC, ncl = gridDim.x / L::NC;
  const int row_l = threadIdx.x / R2, t = threadIdx.x % R2;
  C *line = sm + row_l * LS;
  C *scr = a.scr + (size_t)cl * N * N;
  const T invvol = (T)a.invvol;
  double acc[kAdjDepth + 1];
#pragma unroll
  for (int i = 0; i <= kAdjDepth; ++i) acc[i] = 0.0;
  for (int plane = cl; plane < N * P; plane += ncl) {
    const int p = plane / N, z = plane % N;
    columns<T, N, true, L::FULL>(a.buf + (size_t)plane * N * N + rank * L::SH, scr + rank * L::SH, N, L::SH,
                        sm, roots);
    __syncthreads();                               // the columns' exchange is free
    plane_sync<L::NC>();                           // every column of the plane is in L2
#pragma unroll 1
    for (int rb = 0; rb < L::SH; rb += LB) {
      const bool live = L::FULL || (row_l < LB && rb + row_l < L::SH);
      const int y = rank * L::SH + (live ? rb + row_l : 0);
      rows_inverse<T, N>(scr + (size_t)y * N, line, t, live, roots);
      const size_t base = (size_t)(2 * p) * n + ((size_t)z * N + y) * N;
      const C tyz = cmul(tw[N + y], tw[2 * N + z]);
      const int dyz = (y + z) & 1;
#pragma unroll 1
      for (int q = 0; q < (live ? W::TOT : 0); ++q) {
        const int x0 = VW * (t + R2 * q);
        C h[VW];
#pragma unroll
        for (int k = 0; k < VW; ++k) {
          const int x = x0 + k;
          const C kf = cmul(tw[x], tyz);
          const T sc = invvol * (((x & 1) ^ dyz) ? T(-1) : T(1));
          C w;
          w.x = kf.x * sc;
          w.y = -kf.y * sc;
          h[k] = cmul(line[(x / R2) * ST + x % R2], w);
        }
#pragma unroll
        for (int b = 0; b < 2; ++b) {
          const size_t j = base + b * n + x0;
          T gv[VW], wv[VW], xv[VW], rv[kAdjDepth][VW], lw[VW], rw[VW], yw[VW];
          ldv(gv, g.G + j);
          ldv(wv, g.w + j);
          ldv(xv, g.xi + j);
#pragma unroll
          for (int i = 0; i < kAdjDepth; ++i)
            if (i < nd && i != slot) ldv(rv[i], g.rs + (size_t)i * tot + j);
#pragma unroll
          for (int k = 0; k < VW; ++k) {
            lw[k] = b ? h[k].y : h[k].x;
            const double G = gv[k], x = xv[k];
            rw[k] = (T)((G - 1.0) * ((double)wv[k] + (double)lw[k]) - G * x);
            const double r = (double)rw[k];        // the stored value enters the dots
#pragma unroll
            for (int i = 0; i < kAdjDepth; ++i)
              if (i < nd) acc[i] += r * (i == slot ? r : (double)rv[i][k]);
            acc[kAdjDepth] += r * r;
            yw[k] = (T)(x + g.eta * r);
          }
          stv(g.Lxi + j, lw);
          stv(g.rs + (size_t)slot * tot + j, rw);
          stv(g.ys + (size_t)slot * tot + j, yw);
        }
      }
    }
    if (plane + ncl < N * P) plane_sync<L::NC>();  // the scratch plane is free again
  }
#pragma unroll
  for (int i = 0; i <= kAdjDepth; ++i) {
    double v = acc[i];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    acc[i] = v;
  }
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0)
#pragma unroll
    for (int i = 0; i <= kAdjDepth; ++i) red[wid][i] = acc[i];
  __syncthreads();
  if (threadIdx.x <= kAdjDepth) {
    double v = 0.0;
    for (int w = 0; w < TH / 32; ++w) v += red[w][threadIdx.x];
    g.part[(size_t)threadIdx.x * gridDim.x + blockIdx.x] = v;
  }
}

// Reduction of the dots, stopping tests and the next coefficients, the same
// in every block (s: the block's own copy of the state).
__device__ __forceinline__ void adjoint_finalize(AdjointState *s, const double *part, int nblk,
                                                 double tol, int maxit, int fp32) {
  __shared__ double red[kAdjDepth + 1][32];
  double v[kAdjDepth + 1];
#pragma unroll
  for (int k = 0; k <= kAdjDepth; ++k) v[k] = 0.0;
  for (int b = threadIdx.x; b < nblk; b += blockDim.x)
#pragma unroll
    for (int k = 0; k <= kAdjDepth; ++k) v[k] += __ldcg(part + (size_t)k * nblk + b);
#pragma unroll
  for (int k = 0; k <= kAdjDepth; ++k)
    for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
  if ((threadIdx.x & 31) == 0)
#pragma unroll
    for (int k = 0; k <= kAdjDepth; ++k) red[k][threadIdx.x >> 5] = v[k];
  __syncthreads();
  if (threadIdx.x < 32) {
    if (threadIdx.x <= kAdjDepth) {
      double t = 0.0;
      for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[threadIdx.x][w];
      red[threadIdx.x][0] = t;
    }
    __syncwarp();
    if (threadIdx.x == 0) {
      const double rn = sqrt(red[kAdjDepth][0]);
      if (!isfinite(red[kAdjDepth][0])) {
        s->done = 2;
      } else {
        if (s->bnorm < 0.0) s->bnorm = rn;         // xi = 0: r = (G - 1) w
        if (rn <= tol * s->bnorm) s->done = 1;
        else if (rn < 0.99 * s->best) { s->best = rn; s->since_best = 0; }
        else if (fp32 && ++s->since_best > 200 && rn <= 10.0 * tol * s->bnorm) s->done = 4;
      }
      if (!s->done) {
        const int sl = s->slot;
        for (int i = 0; i < kAdjDepth; ++i)
          s->gram[sl * kAdjDepth + i] = s->gram[i * kAdjDepth + sl] = red[i][0];
        s->gram[sl * kAdjDepth + sl] = red[kAdjDepth][0];
        s->ns = s->ns < kAdjDepth ? s->ns + 1 : kAdjDepth;
        s->slot = (sl + 1) % kAdjDepth;
        s->it += 1;
        if (s->it >= maxit) s->done = 3;
      }
    }
    __syncwarp();
    if (!s->done) anderson_warp(s->gram, s->ns, s->coef);
  }
  __syncthreads();
}

template <typename T, int N, int V>
__global__ void __cluster_dims__(Lines<N>::NC, 1, 1)
    __launch_bounds__(Lines<N>::TH, (Lines<N>::template minp<T, V>())) k_adjoint_solve(AdjointArgs<T> g) {
  typedef CxT<T> C;
  extern __shared__ __align__(16) unsigned char fused_sm[];
  __shared__ AdjointState s;
  C *sm = reinterpret_cast<C *>(fused_sm);
  if (cluster_ctas() != Lines<N>::NC) {            // see the launches in fused.cuh
    if (blockIdx.x == 0 && threadIdx.x == 0) g.st->done = 5;
    return;
  }
  C *tw = reinterpret_cast<C *>(fused_sm + tables_at<T, N, V>()), *roots = tw + 3 * N;
  for (int i = threadIdx.x; i < 3 * N; i += blockDim.x) tw[i] = g.it.tw[i];
  for (int i = threadIdx.x; i < N; i += blockDim.x) roots[i] = g.it.roots[i];
  if (threadIdx.x == 0) s = *g.st;
  __syncthreads();
  __shared__ GridBarrier bar;
  const unsigned nblk = gridDim.x;
  if (threadIdx.x == 0) enter_barrier(bar, &g.st->bar, g.it.delay);
  __syncthreads();
  while (!s.done) {
    adjoint_forward<T, N, V>(g, &s, sm, tw, roots);
    if (!grid_barrier(bar)) break;
#pragma unroll 1
    for (int tile = blockIdx.x; tile < ZShape<T, N, V>::TILES; tile += nblk) {
      zline_tile<T, N, V, false, true>(g.it, sm, roots, N, N, tile);
      __syncthreads();
    }
    if (!grid_barrier(bar)) break;
    adjoint_residual<T, N, V>(g, &s, sm, tw, roots);
    if (!grid_barrier(bar)) break;
    adjoint_finalize(&s, g.part, (int)nblk, g.tol, g.maxit, sizeof(T) == 4);
  }
  if (threadIdx.x == 0) {
    if (blockIdx.x == 0) {
      g.st->done = s.done;
      g.st->it = s.it;
    }
    leave_barrier(bar);
  }
}

// Launch of the whole solve; false: this device cannot hold it at once
template <typename T, int N, int V>
bool adjoint_launch(const AdjointArgs<T> &g, int *clusters, cudaStream_t st) {
  using L = Lines<N>;
  const size_t s = tables_at<T, N, V>() + 4 * N * sizeof(CxT<T>);
  if (cudaFuncSetAttribute(k_adjoint_solve<T, N, V>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)s) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  const int planes = N * ((V + 1) / 2), room = g.max_blocks / L::NC;
  const int ncl = plane_clusters(k_adjoint_solve<T, N, V>, L::NC, L::TH, s,
                                 planes < room ? planes : room);
  if (ncl < 1) return false;
  if (clusters) {                                  // asked for the count only
    *clusters = ncl;
    return true;
  }
  return launch_plane(k_adjoint_solve<T, N, V>, ncl, L::NC, 1, L::TH, s, st, true, g) == cudaSuccess;
}

template <typename T, int N>
AdjointLaunch<T> adjoint_table_v(int V) {
  switch (V) {
    case 2: return adjoint_launch<T, N, 2>;
    case 4: return adjoint_launch<T, N, 4>;
  }
  return nullptr;
}

}  // namespace fused
}  // namespace rism3d
