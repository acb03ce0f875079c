// One iteration in three kernels, with the 3D transforms folded in (cubic
// cells whose edge N = R1 R2 has an instantiation, two or four solvent sites):
//
//   k_plane_a  update + closure + packing of one xy plane, x- and y-DFT
//   k_zline    z-DFT, OZ product of every mirror pair, inverse z-DFT
//   k_plane_r  inverse y- and x-DFT of one xy plane, residual, Gram sums,
//              and in the last block the stopping test and AN2's 2 x 2 solve
//
// What bounds the iteration is bytes: the passes and a library transform move
// 456 B per point and cycle in FP64 with two sites (passes A / K / R 264, two
// 3D transforms of three read-write passes each 192), and on small grids the
// dozen launches cost more than the work.  Folded, the cycle moves 264 B in
// three launches:
//   plane A  reads t, U, the new residual and two history grids, writes t and
//            one history grid (112) and the transform buffer (16);
//   z lines  read and write the buffer (32) and read half of fk (8);
//   plane R  reads the buffer, t, U and the two residual histories and writes
//            the new residual (96), so plane A needs no inverse transform.
// A plane is worked on by a cluster of CTAs: each transforms its share of the
// rows, the half-transformed plane is exchanged through L2, and after one
// cluster barrier each transforms its share of the columns.  (A plane of
// complex FP64 at N = 256 is 1 MB: more than the distributed shared memory of
// a portable cluster leaves room for at two CTAs per SM.)
//
// The residual goes to whichever of three slots holds no history
// (DevState.rp): if the update of this cycle is applied, finalize renames
// that slot, so the history is never copied and a stop leaves it untouched.
//
// A line of N = R1 R2 points is transformed in two register stages with one
// shared-memory exchange (n = t + R2 j, k = s + R1 k2):
//   A_t[s] = W_N^(t s) sum_j a[t + R2 j] W_R1^(j s),  X[s + R1 k2] = sum_t A_t[s] W_R2^(t k2)
// and backwards, starting from the groups of equal k mod R1 (so the z kernel
// goes forth and back with two exchanges in all).
#pragma once

#include "dft.cuh"
#include "fused_api.cuh"

namespace rism3d {
namespace fused {

template <typename T> using CxT = typename Cx<T>::t;

// ---- shapes: N = R1 R2, both even (z lines pair up registers of mirror
// points, rows move in pairs of points), R1 >= R2.  LB lines per batch of a
// block, NC CTAs per plane, CW owner columns of a z tile.  LB and NC are
// chosen so that the planes' CTAs fill the SMs in few, even rounds: a block is
// 96-256 threads, of which the SM holds 512 in FP64 (128 registers).
template <int N> struct Shape;
#define RISM3D_SHAPE(N, r1, r2, lb, nc, cw) \
  template <> struct Shape<N> { static constexpr int R1 = r1, R2 = r2, LB = lb, NC = nc, CW = cw; };
RISM3D_SHAPE(32, 8, 4, 16, 2, 8)
RISM3D_SHAPE(36, 6, 6, 12, 3, 6)
RISM3D_SHAPE(40, 10, 4, 20, 2, 10)
RISM3D_SHAPE(48, 8, 6, 16, 3, 8)
RISM3D_SHAPE(60, 10, 6, 30, 2, 15)
RISM3D_SHAPE(64, 8, 8, 32, 2, 16)
RISM3D_SHAPE(72, 12, 6, 36, 2, 18)
RISM3D_SHAPE(80, 10, 8, 16, 5, 8)
RISM3D_SHAPE(96, 12, 8, 16, 6, 8)
RISM3D_SHAPE(100, 10, 10, 10, 5, 5)
RISM3D_SHAPE(108, 18, 6, 18, 3, 9)
RISM3D_SHAPE(120, 12, 10, 10, 4, 5)
RISM3D_SHAPE(128, 16, 8, 16, 4, 8)
RISM3D_SHAPE(144, 12, 12, 12, 3, 6)
RISM3D_SHAPE(160, 16, 10, 16, 5, 8)
RISM3D_SHAPE(180, 18, 10, 15, 4, 6)
RISM3D_SHAPE(192, 16, 12, 16, 6, 8)
RISM3D_SHAPE(200, 20, 10, 20, 5, 10)
RISM3D_SHAPE(216, 18, 12, 18, 6, 9)
RISM3D_SHAPE(240, 20, 12, 15, 8, 6)
RISM3D_SHAPE(256, 16, 16, 16, 8, 8)
#undef RISM3D_SHAPE

template <int N> struct Lines {
  static constexpr int R1 = Shape<N>::R1, R2 = Shape<N>::R2, LB = Shape<N>::LB, NC = Shape<N>::NC,
                       CW = Shape<N>::CW;
  // threads: one stage-1 item each of a batch of lines or a z tile's columns,
  // in whole warps
  static constexpr int ITEMS = (LB > 2 * CW ? LB : 2 * CW) * R2, TH = (ITEMS + 31) / 32 * 32;
  static constexpr int ST = R2 | 1;                // row-exchange stride (no bank conflicts)
  static constexpr int LS = R1 * ST;               // shared points of one row
  static constexpr int SH = N / NC;                // lines per CTA
  // every thread has a line in every batch: no tests in the loops
  static constexpr bool FULL = LB * R2 == TH && SH % LB == 0, ZFULL = 2 * CW * R2 == TH;
  static_assert(R1 * R2 == N && R1 % 2 == 0 && R2 % 2 == 0 && R1 >= R2 && SH * NC == N, "line split");
  template <typename T> static constexpr size_t smem() { return sizeof(CxT<T>) * LB * (size_t)LS; }
  // a whole-phase launch of a small grid has one block per SM at most: all
  // registers, and all points of a thread in flight at once
  template <typename T, int V> __host__ __device__ static constexpr int minp() {
    return (N * NC * ((V + 1) / 2) <= 148) ? 1 : minb<T>();
  }
  // resident CTAs asked of the compiler: 128 registers in FP64, 80 in FP32
  template <typename T> __host__ __device__ static constexpr int minb() {
    return (sizeof(T) == 8 ? 512 : 768) / TH > 0 ? (sizeof(T) == 8 ? 512 : 768) / TH : 1;
  }
};

// Pointwise loops: a thread takes vectors of VW neighbouring points (16 bytes
// where its R1 points allow), NV of them at a time (WIDE: all) with every load before the
// first use.  FP64: 4 points x 10 streams = 320 B in flight per thread.
template <typename T, int R1, bool WIDE> struct Vecs {
  static constexpr int VW = sizeof(T) == 8 ? 2 : (R1 % 4 == 0 ? 4 : 2);
  static constexpr int TOT = R1 / VW;              // vectors per thread and row
  static constexpr int NV = WIDE ? TOT : (sizeof(T) == 8 && TOT % 2 == 0) ? 2 : 1;
  static constexpr int CH = TOT / NV;              // chunks
  static_assert(R1 % VW == 0, "points per thread");
};
template <int B> struct VecT;
template <> struct VecT<8> { typedef float2 t; };
template <> struct VecT<16> { typedef float4 t; };
// streams of the state: read or written once per kernel, first to leave L2
template <typename T, int W> __device__ __forceinline__ void ldv(T (&o)[W], const T *p) {
  typedef typename VecT<sizeof(T) * W>::t B;
  union { B b; T t[W]; } u;
  u.b = __ldcs(reinterpret_cast<const B *>(p));
#pragma unroll
  for (int k = 0; k < W; ++k) o[k] = u.t[k];
}
template <typename T, int W> __device__ __forceinline__ void stv(T *p, const T (&o)[W]) {
  typedef typename VecT<sizeof(T) * W>::t B;
  union { B b; T t[W]; } u;
#pragma unroll
  for (int k = 0; k < W; ++k) u.t[k] = o[k];
  __stcs(reinterpret_cast<B *>(p), u.b);
}

template <typename T> __device__ __forceinline__ void pf(const T *p) {
  asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;\n"
               ::: "memory");
}
__device__ __forceinline__ unsigned cluster_ctas() {
  unsigned n;
  asm("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(n));
  return n;
}
// Threads that share a row: the R2 consecutive threads of stage 1 also do its
// R1 stage-2 items (s = t, t + R2, ...), so that where R2 divides a warp the
// row exchange needs no block barrier.
template <int R2> __device__ __forceinline__ void row_sync() {
  if (32 % R2 == 0) __syncwarp();
  else __syncthreads();
}
template <int NC> __device__ __forceinline__ void plane_sync() {
  if (NC > 1) cluster_sync();
  else __syncthreads();
}

template <typename T> __device__ __forceinline__ T *rp_slot(const IterArgs<T> &a, int V, int i) {
  return i < 2 ? a.RP + (size_t)i * V * a.n : a.RPx;
}

// DFT along y of ncol columns of a plane: column x of src (row pitch `pitch`)
// -> column x of dst (dst may be src: a column is read whole before it is
// written)
template <typename T, int N, bool INV, bool FULL>
__device__ __forceinline__ void columns(const CxT<T> *src, CxT<T> *dst, int pitch, int ncol,
                                        CxT<T> *sm, const CxT<T> *roots) {
  typedef CxT<T> C;
  using L = Lines<N>;
  constexpr int R1 = L::R1, R2 = L::R2, LB = L::LB;
  const int col = threadIdx.x % LB, t = threadIdx.x / LB;
#pragma unroll 1
  for (int cb = 0; cb < ncol; cb += LB) {
    const bool live = FULL || (t < R2 && cb + col < ncol);
    C v[R1];
    if (live) {
      const C *s0 = src + cb + col;
#pragma unroll
      for (int j = 0; j < R1; ++j) v[j] = __ldcg(s0 + (size_t)(t + R2 * j) * pitch);
      dft::run<R1, INV>(v);
#pragma unroll
      for (int s = 1; s < R1; ++s) v[s] = dft::cmulw<INV>(v[s], roots[t * s]);
    }
    __syncthreads();                               // the exchange's last readers are done
    if (live)
#pragma unroll
      for (int s = 0; s < R1; ++s) sm[(s * R2 + t) * LB + col] = v[s];
    __syncthreads();
#pragma unroll 1
    for (int i = threadIdx.x; i < LB * R1; i += L::TH) {
      const int c = i % LB, s = i / LB;
      if (FULL || cb + c < ncol) {
        C w[R2];
#pragma unroll
        for (int k = 0; k < R2; ++k) w[k] = sm[(s * R2 + k) * LB + c];
        dft::run<R2, INV>(w);
        C *d0 = dst + cb + c;
#pragma unroll
        for (int k = 0; k < R2; ++k) __stcg(d0 + (size_t)(s + R1 * k) * pitch, w[k]);
      }
    }
  }
}

// Row batches: thread threadIdx.x < LB R2 works on row threadIdx.x / R2 of its
// batch where that row exists (live); the others only take part in the row
// barriers.
//
// x-DFT of a row in its exchange slots (line[(x / R2) ST + x % R2], complete)
// to dst; a thread's stage-1 inputs and outputs are its own slots.
template <typename T, int N>
__device__ __forceinline__ void rows_forward(CxT<T> *line, CxT<T> *dst, int t, bool live,
                                             const CxT<T> *roots) {
  typedef CxT<T> C;
  using L = Lines<N>;
  constexpr int R1 = L::R1, R2 = L::R2, ST = L::ST;
  if (live) {
    C v[R1];
#pragma unroll
    for (int j = 0; j < R1; ++j) v[j] = line[j * ST + t];
    dft::run<R1, false>(v);
#pragma unroll
    for (int s = 1; s < R1; ++s) v[s] = cmul(v[s], roots[t * s]);
#pragma unroll
    for (int s = 0; s < R1; ++s) line[s * ST + t] = v[s];
  }
  row_sync<R2>();
  if (live) {
#pragma unroll 1
    for (int s = t; s < R1; s += R2) {
      C w[R2];
#pragma unroll
      for (int k = 0; k < R2; ++k) w[k] = line[s * ST + k];
      dft::run<R2, false>(w);
#pragma unroll
      for (int k = 0; k < R2; ++k) __stcg(dst + s + R1 * k, w[k]);
    }
  }
}

// Inverse x-DFT of the row src into line[(x / R2) ST + x % R2], not yet
// twiddled; every thread of the row may read it on return.
template <typename T, int N>
__device__ __forceinline__ void rows_inverse(const CxT<T> *src, CxT<T> *line, int t, bool live,
                                             const CxT<T> *roots) {
  typedef CxT<T> C;
  using L = Lines<N>;
  constexpr int R1 = L::R1, R2 = L::R2, ST = L::ST, NI = (R1 + R2 - 1) / R2;
  {
    C v[R1];
    if (live) {
#pragma unroll
      for (int j = 0; j < R1; ++j) v[j] = __ldcg(src + t + R2 * j);
      dft::run<R1, true>(v);
#pragma unroll
      for (int s = 1; s < R1; ++s) v[s] = dft::cmulw<true>(v[s], roots[t * s]);
    }
    row_sync<R2>();                                // the exchange's last readers are done
    if (live)
#pragma unroll
      for (int s = 0; s < R1; ++s) line[s * ST + t] = v[s];
  }
  row_sync<R2>();
  C w[NI][R2];
#pragma unroll
  for (int i = 0; i < NI; ++i) {
    const int s = t + R2 * i;
    if (live && s < R1) {
#pragma unroll
      for (int k = 0; k < R2; ++k) w[i][k] = line[s * ST + k];
      dft::run<R2, true>(w[i]);
    }
  }
  row_sync<R2>();
#pragma unroll
  for (int i = 0; i < NI; ++i) {
    const int s = t + R2 * i;
    if (live && s < R1) {
#pragma unroll
      for (int k = 0; k < R2; ++k) {
        const int x = s + R1 * k;
        line[(x / R2) * ST + x % R2] = w[i][k];
      }
    }
  }
  row_sync<R2>();
}

// ---------------------------------------------------------------- plane A
// One row of a batch: the update of the last cycle, closure, packed and
// twiddled, then its x-DFT to dst.
template <typename T, int N, int V, bool REF, bool WIDE>
__device__ __forceinline__ void update_row(const IterArgs<T> &a, const DevState *st, CxT<T> *line,
                                           int t, bool live, size_t base, CxT<T> tyz,
                                           int dyz, CxT<T> *dst, const CxT<T> *tw,
                                           const CxT<T> *roots, bool hnc) {
  typedef CxT<T> C;
  using L = Lines<N>;
  constexpr int R1 = L::R1, R2 = L::R2, ST = L::ST;
  using W = Vecs<T, R1, WIDE>;
  constexpr int VW = W::VW, NV = W::NV;
  const int mode = st->mode, slot = st->upd_slot;
  const T s1 = (T)st->s1, s2 = (T)st->s2, m = (T)st->m;
  const size_t n = (size_t)a.n;
  row_sync<R2>();                                  // the exchange's last readers are done
  if (live) {
    T *pt = a.t + base, *py = a.Y + (size_t)slot * V * n + base;
    const T *pu = a.U + base, *pr = rp_slot(a, V, st->rp[slot]) + base,   // this cycle's residual
            *p0 = a.Y + base, *p1 = a.Y + (size_t)V * n + base;
#pragma unroll 1
    for (int c = 0; c < W::CH; ++c) {
      T tv[2][NV][VW], uv[2][NV][VW];
      int x0[NV];
#pragma unroll
      for (int q = 0; q < NV; ++q) {
        x0[q] = VW * (t + R2 * (q + NV * c));
        ldv(tv[0][q], pt + x0[q]);
        ldv(uv[0][q], pu + x0[q]);
        ldv(tv[1][q], pt + n + x0[q]);
        ldv(uv[1][q], pu + n + x0[q]);
      }
      if (mode != 0) {
        T rv[2][NV][VW], y0[2][NV][VW], y1[2][NV][VW];
#pragma unroll
        for (int q = 0; q < NV; ++q)
#pragma unroll
          for (int b = 0; b < 2; ++b) {
            ldv(rv[b][q], pr + b * n + x0[q]);
            ldv(y0[b][q], p0 + b * n + x0[q]);
            ldv(y1[b][q], p1 + b * n + x0[q]);
          }
#pragma unroll
        for (int q = 0; q < NV; ++q)
#pragma unroll
          for (int b = 0; b < 2; ++b) {
            T yw[VW];
#pragma unroll
            for (int k = 0; k < VW; ++k) {
              // newdt (AN2), anderson_cuda.cu:11-23, or newdt0 (Picard)
              const T tt = tv[b][q][k], r = rv[b][q][k], yy = tt + m * r;
              yw[k] = yy;
              tv[b][q][k] = mode == 2 ? yy + s1 * (y0[b][q][k] - yy) + s2 * (y1[b][q][k] - yy)
                                      : tt + r;
            }
            stv(py + b * n + x0[q], yw);
            stv(pt + b * n + x0[q], tv[b][q]);
          }
      }
      // closure + c_SR (calculate_cuda.cu:1-29) and the forward pre-twiddle
      // (timekf, fft3d.cu:41-49): dir * dkf * (c_a + i c_b)
#pragma unroll
      for (int q = 0; q < NV; ++q)
#pragma unroll
        for (int k = 0; k < VW; ++k) {
          const int x = x0[q] + k;
          C cc;
          cc.x = cfun_rt<REF>(tv[0][q][k], uv[0][q][k], hnc);
          cc.y = cfun_rt<REF>(tv[1][q][k], uv[1][q][k], hnc);
          const C kf = cmul(tw[x], tyz);
          const T dir = ((x & 1) ^ dyz) ? T(-1) : T(1);
          C w;
          w.x = kf.x * dir;
          w.y = kf.y * dir;
          line[(x / R2) * ST + x % R2] = cmul(cc, w);
        }
    }
  }
  row_sync<R2>();
  rows_forward<T, N>(line, dst, t, live, roots);
}

template <typename T, int N, int V, bool REF, bool WIDE>
__device__ __forceinline__ void planes_a(const IterArgs<T> &a, const DevState *st, CxT<T> *sm,
                                         const CxT<T> *tw, const CxT<T> *roots, bool hnc) {
  typedef CxT<T> C;
  using L = Lines<N>;
  constexpr int R2 = L::R2, LB = L::LB, P = (V + 1) / 2;
  const size_t n = (size_t)a.n;
  const int rank = blockIdx.x % L::NC, ncl = gridDim.x / L::NC;
  const int row_l = threadIdx.x / R2, t = threadIdx.x % R2;
  for (int plane = blockIdx.x / L::NC; plane < N * P; plane += ncl) {
    const int p = plane / N, z = plane % N;
    C *pb = a.buf + (size_t)plane * N * N;
    __syncthreads();                               // the columns' exchange is free
#pragma unroll 1
    for (int rb = 0; rb < L::SH; rb += LB) {
      const bool live = L::FULL || (row_l < LB && rb + row_l < L::SH);
      const int y = rank * L::SH + (live ? rb + row_l : 0);
      update_row<T, N, V, REF, WIDE>(a, st, sm + row_l * L::LS, t, live,
                                     (size_t)(2 * p) * n + ((size_t)z * N + y) * N,
                                     cmul(tw[N + y], tw[2 * N + z]), (y + z) & 1,
                                     pb + (size_t)y * N, tw, roots, hnc);
    }
    plane_sync<L::NC>();                           // every row of the plane is in L2
    C *pc = pb + rank * L::SH;
    columns<T, N, false, L::FULL>(pc, pc, N, L::SH, sm, roots);
  }
}

template <typename T, int N, int V, bool REF>
__global__ void __cluster_dims__(Lines<N>::NC, 1, 1)
    __launch_bounds__(Lines<N>::TH, (Lines<N>::template minb<T>())) k_plane_a(IterArgs<T> a0, bool hnc) {
  extern __shared__ __align__(16) unsigned char fused_sm[];
  const IterArgs<T> a = solute_view<T, V>(a0);
  if (a.st->done) return;
  planes_a<T, N, V, REF, false>(a, a.st, reinterpret_cast<CxT<T> *>(fused_sm), a.tw, a.roots, hnc);
}

// ---------------------------------------------------------------- plane R
// The points of one row after the inverse transform (line, not yet twiddled;
// sites v0 and v0 + 1): residuals, their sums, the new residual slot.
template <typename T, int N, int V, bool REF, bool WIDE>
__device__ __forceinline__ void residual_row(const IterArgs<T> &a, const DevState *st,
                                             const CxT<T> *line, int t, int v0,
                                             size_t base, CxT<T> tyz, int dyz, const CxT<T> *tw,
                                             bool gram, bool hnc, double (&acc)[6]) {
  typedef CxT<T> C;
  using L = Lines<N>;
  constexpr int R1 = L::R1, R2 = L::R2, ST = L::ST;
  using W = Vecs<T, R1, WIDE>;
  constexpr int VW = W::VW, NV = W::NV;
  const size_t n = (size_t)a.n;
  const T invvol = (T)a.invvol;
  const T *pt = a.t + base, *pu = a.U + base, *p0 = rp_slot(a, V, st->rp[0]) + base,
          *p1 = rp_slot(a, V, st->rp[1]) + base, *pq = REF ? a.R0 + base : nullptr;
  T *pr = rp_slot(a, V, st->rp[2]) + base;
#pragma unroll 1
  for (int c = 0; c < W::CH; ++c) {
    T tv[2][NV][VW], uv[2][NV][VW], r0[2][NV][VW], r1[2][NV][VW], qv[2][NV][VW];
    int x0[NV];
#pragma unroll
    for (int q = 0; q < NV; ++q) {
      x0[q] = VW * (t + R2 * (q + NV * c));
#pragma unroll
      for (int b = 0; b < 2; ++b) {
        ldv(tv[b][q], pt + b * n + x0[q]);
        ldv(uv[b][q], pu + b * n + x0[q]);
        ldv(r0[b][q], p0 + b * n + x0[q]);
        ldv(r1[b][q], p1 + b * n + x0[q]);
        if (REF) ldv(qv[b][q], pq + b * n + x0[q]);
      }
    }
#pragma unroll
    for (int q = 0; q < NV; ++q) {
      T rw[2][VW];
#pragma unroll
      for (int k = 0; k < VW; ++k) {
        const int x = x0[q] + k;
        // inverse post-twiddle (timekb, fft3d.cu:52-60): (1/V) dir conj(dkf)
        const C kf = cmul(tw[x], tyz);
        const T sc = invvol * (((x & 1) ^ dyz) ? T(-1) : T(1));
        C w;
        w.x = kf.x * sc;
        w.y = -kf.y * sc;
        const C h = cmul(line[(x / R2) * ST + x % R2], w);
#pragma unroll
        for (int b = 0; b < 2; ++b) {
          const T R = residual_rt<REF>(b ? h.y : h.x, tv[b][q][k], uv[b][q][k],
                                       REF ? qv[b][q][k] : T(0), hnc);
          rw[b][k] = R;
          const double r = (double)R;
          acc[0] += r * r;                     // cal_rms.cu:18
          if (gram) {                          // theta30, anderson_cuda.cu:33-39
            const double wt = a.sp->irho[v0 + b];
            const double d0 = r - (double)r0[b][q][k], d1 = r - (double)r1[b][q][k];
            acc[1] += wt * r * d0;
            acc[2] += wt * r * d1;
            acc[3] += wt * d0 * d0;
            acc[4] += wt * d0 * d1;
            acc[5] += wt * d1 * d1;
          }
        }
      }
#pragma unroll
      for (int b = 0; b < 2; ++b) {
        stv(pr + b * n + x0[q], rw[b]);
      }
    }
  }
}

// Block sums of R^2 and the Gram terms into this block's row of the partials
template <int TH>
__device__ __forceinline__ void block_sums(double (&acc)[6], double *part) {
  __shared__ double red[TH / 32][6];
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    double v = acc[k];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    acc[k] = v;
  }
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0)
    for (int k = 0; k < 6; ++k) red[wid][k] = acc[k];
  __syncthreads();
  if (threadIdx.x < 6) {
    double s = 0.0;
    for (int w = 0; w < TH / 32; ++w) s += red[w][threadIdx.x];
    part[(size_t)threadIdx.x * gridDim.x + blockIdx.x] = s;
  }
}

template <typename T, int N, int V, bool REF, bool WIDE>
__device__ __forceinline__ void planes_r(const IterArgs<T> &a, const DevState *st, CxT<T> *sm,
                                         const CxT<T> *tw, const CxT<T> *roots, bool hnc) {
  typedef CxT<T> C;
  using L = Lines<N>;
  constexpr int R2 = L::R2, LB = L::LB, P = (V + 1) / 2;
  const bool gram = st->count <= 0;
  const size_t n = (size_t)a.n;
  const int rank = blockIdx.x % L::NC, cl = blockIdx.x / L::NC, ncl = gridDim.x / L::NC;
  const int row_l = threadIdx.x / R2, t = threadIdx.x % R2;
  C *line = sm + row_l * L::LS;
  C *scr = a.scr + (size_t)cl * N * N;
  double acc[6] = {0, 0, 0, 0, 0, 0};
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
      if (live)
        residual_row<T, N, V, REF, WIDE>(a, st, line, t, 2 * p,
                                         (size_t)(2 * p) * n + ((size_t)z * N + y) * N,
                                         cmul(tw[N + y], tw[2 * N + z]), (y + z) & 1, tw, gram,
                                         hnc, acc);
    }
    if (plane + ncl < N * P) plane_sync<L::NC>();  // the scratch plane is free again
  }
  block_sums<L::TH>(acc, a.part);
}

// The last block of a solute to finish reduces all block sums and steers the
// loop.
template <typename T>
__device__ __forceinline__ void finish_cycle(const IterArgs<T> &a0, const IterArgs<T> &a, int V) {
  __shared__ bool last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(a.count, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  finalize_block(a.st, a.part, gridDim.x, (double)a.n * V, a.hist, a.hist_cap);
  if (threadIdx.x == 0) {
    *a.count = 0u;
    if (a.st->done) a.st->after_done = 1;          // nothing is left to do in the loop
    loop_test_all(a0);
  }
}

template <typename T, int N, int V, bool REF>
__global__ void __cluster_dims__(Lines<N>::NC, 1, 1)
    __launch_bounds__(Lines<N>::TH, (Lines<N>::template minb<T>())) k_plane_r(IterArgs<T> a0, bool hnc) {
  extern __shared__ __align__(16) unsigned char fused_sm[];
  const IterArgs<T> a = solute_view<T, V>(a0);
  DevState *st = a.st;
  if (st->done) {                                  // this solute has stopped
    if (blockIdx.x == 0 && threadIdx.x == 0) loop_test_all(a0);
    return;
  }
  planes_r<T, N, V, REF, false>(a, st, reinterpret_cast<CxT<T> *>(fused_sm), a.tw, a.roots, hnc);
  finish_cycle(a0, a, V);
}

// Once after the loop: snapshot of h (Re of the last OZ) and g (closure of
// the t used in that cycle), and when maxstep ended the loop the pending
// update (iterate.cu:61 runs before the step bound is tested).
template <typename T, int N, int V, bool REF>
__device__ __forceinline__ void final_row(const IterArgs<T> &a, const CxT<T> *line, int t, int p,
                                          size_t row, CxT<T> tyz, int dyz, bool snap, bool update,
                                          bool hnc) {
  typedef CxT<T> C;
  constexpr int R2 = Lines<N>::R2, ST = Lines<N>::ST;
  const DevState *st = a.st;
  const int mode = st->mode, slot = st->upd_slot;
  const T s1 = (T)st->s1, s2 = (T)st->s2, m = (T)st->m;
  const T *Rn = rp_slot(a, V, st->rp[slot]);       // renamed into the history already
  const size_t n = (size_t)a.n;
#pragma unroll 1
  for (int x = t; x < N; x += R2) {
    const C kf = cmul(a.tw[x], tyz);
    const T sc = (T)a.invvol * (((x & 1) ^ dyz) ? T(-1) : T(1));
    C w;
    w.x = kf.x * sc;
    w.y = -kf.y * sc;
    const C h = cmul(line[(x / R2) * ST + x % R2], w);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const size_t iv = (size_t)(2 * p + q) * n + row + x;
      const T tv = a.t[iv];
      if (snap) {
        a.hout[iv] = (double)(q ? h.y : h.x);
        a.gout[iv] = (double)closure_rt(tv - a.U[iv], hnc);
      }
      if (update) {
        const T R = Rn[iv], yv = tv + m * R;
        T tn = tv + R;
        if (mode == 2) tn = yv + s1 * (a.Y[iv] - yv) + s2 * (a.Y[(size_t)V * n + iv] - yv);
        a.Y[(size_t)slot * V * n + iv] = yv;
        a.t[iv] = tn;
      }
    }
  }
}

template <typename T, int N, int V, bool REF>
__global__ void __cluster_dims__(Lines<N>::NC, 1, 1) __launch_bounds__(Lines<N>::TH)
    k_plane_final(IterArgs<T> a0, bool hnc) {
  typedef CxT<T> C;
  using L = Lines<N>;
  constexpr int R2 = L::R2, LB = L::LB, P = (V + 1) / 2;
  extern __shared__ __align__(16) unsigned char fused_sm[];
  C *sm = reinterpret_cast<C *>(fused_sm);
  const IterArgs<T> a = solute_view<T, V>(a0);
  const bool snap = !REF && a.hout, update = a.st->done == 3 && a.st->mode != 0;
  if (!snap && !update) return;
  const int rank = blockIdx.x % L::NC, cl = blockIdx.x / L::NC, ncl = gridDim.x / L::NC;
  const int row_l = threadIdx.x / R2, t = threadIdx.x % R2;
  C *line = sm + row_l * L::LS;
  C *scr = a.scr + (size_t)cl * N * N;
  for (int plane = cl; plane < N * P; plane += ncl) {
    const int p = plane / N, z = plane % N;
    columns<T, N, true, L::FULL>(a.buf + (size_t)plane * N * N + rank * L::SH, scr + rank * L::SH, N, L::SH,
                        sm, a.roots);
    __syncthreads();
    plane_sync<L::NC>();
#pragma unroll 1
    for (int rb = 0; rb < L::SH; rb += LB) {
      const bool live = L::FULL || (row_l < LB && rb + row_l < L::SH);
      const int y = rank * L::SH + (live ? rb + row_l : 0);
      rows_inverse<T, N>(scr + (size_t)y * N, line, t, live, a.roots);
      if (live)
        final_row<T, N, V, REF>(a, line, t, p, ((size_t)z * N + y) * N,
                                cmul(a.tw[N + y], a.tw[2 * N + z]), (y + z) & 1, snap, update, hnc);
    }
    if (plane + ncl < N * P) plane_sync<L::NC>();
  }
}

// ---------------------------------------------------------------- z lines
// A block owns CW neighbouring kx columns at one ky < ny/2 and their mirrors
// (kx' = nx-1-kx, ky' = ny-1-ky), so every k and -k meet in it.  After the
// forward DFT the owner's points kz = s + R1 k of one thread mirror the
// points of the neighbouring lane's group R1-1-s, register R2-1-k: each lane
// takes half of the pairs with one shuffle each way.
template <typename T, int N, int V>
struct ZShape {
  static constexpr int CW = Lines<N>::CW, COLS = 2 * CW, TH = Lines<N>::TH;
  static constexpr int P = (V + 1) / 2;
  static constexpr int TILES = ((N + CW - 1) / CW) * (N / 2);      // of a cubic cell
  static constexpr int MINB = (sizeof(T) == 8 ? 512 : 1024) / TH > 0 ? (sizeof(T) == 8 ? 512 : 1024) / TH : 1;
  static constexpr size_t smem() { return sizeof(CxT<T>) * (size_t)P * COLS * N; }
};

template <typename C>
__device__ __forceinline__ C shfl_pair(unsigned mask, C v) {
  v.x = __shfl_xor_sync(mask, v.x, 1);
  v.y = __shfl_xor_sync(mask, v.y, 1);
  return v;
}

// N = nz; CUBIC: nx = ny = N and chi from the per-|k|^2 table, else the octant
// table; a tile past the last column repeats it for its spare columns' loads.
template <typename T, int N, int V, bool WIDE, bool CUBIC>
__device__ __forceinline__ void zline_tile(const IterArgs<T> &a, CxT<T> *sm, const CxT<T> *roots,
                                           int nx, int ny, int tile) {
  typedef CxT<T> C;
  using Z = ZShape<T, N, V>;
  constexpr int R1 = Shape<N>::R1, R2 = Shape<N>::R2, CW = Z::CW, COLS = Z::COLS, P = Z::P;
  static_assert(!CUBIC || N % CW == 0, "z tiles");
  const long long n = a.n, plane = (long long)nx * ny;
  const int tx = (nx + CW - 1) / CW, ky = tile / tx, x0 = (tile % tx) * CW;
  // fk and chi of an item's pairs: loaded ahead of the exchange where they fit
  // in registers, else asked into L2 now
  constexpr int H = R2 / 2;
  constexpr bool AHEAD = WIDE && H * (V * V + 2) * sizeof(T) <= 24 * 8;
  double2 fkv[H];
  T X[H][V * V];
  auto pair_kz = [&](int i, int k) {
    const int side = i & 1, s = (i >> 1) / CW;
    return side ? N - 1 - (R1 - 1 - s + R1 * k) : s + R1 * k;
  };
  auto load_pair = [&](int i, int k, double2 &fk, T (&x)[V * V]) {
    // beta fk is stored for kz < N/2, the conjugate of the mirror's beyond
    const int kx = CUBIC ? x0 + (i >> 1) % CW : min(x0 + (i >> 1) % CW, nx - 1), kz = pair_kz(i, k);
    fk = make_double2(0.0, 0.0);
    if (!a.nofk) {
      const bool lo = kz < N / 2;
      const long long j = kx + (long long)nx * ky + plane * kz;
      fk = __ldg(a.fkh + (lo ? j : n - 1 - j));
      if (!lo) fk.y = -fk.y;
    }
    if constexpr (CUBIC) chi_cubic<T, V>(a, kx, ky, kz, x);
    else chi_octant<T, V>(a, kx, ky, kz, x);
  };
  if constexpr (!AHEAD) {
    if (!a.nofk)                                   // rows of CW points and their mirrors
      for (int i = threadIdx.x; i < N; i += Z::TH) {
        const int kz = i % (N / 2);
        pf(a.fkh + plane * kz +
           (i < N / 2 ? x0 + (long long)nx * ky
                      : max(nx - x0 - CW, 0) + (long long)nx * (ny - 1 - ky)));
      }
  }
  const int col = threadIdx.x % COLS, t = threadIdx.x / COLS;
  const int cx = x0 + (col < CW ? col : COLS - 1 - col);           // its owner column
  const bool live = (Lines<N>::ZFULL || t < R2) && (CUBIC || cx < nx);
  C *g = a.buf + (col < CW ? (size_t)ky * nx + cx : (size_t)(ny - 1 - ky) * nx + nx - 1 - cx);
  if (live) {
#pragma unroll
    for (int p = 0; p < P; ++p) {
      C v[R1];
#pragma unroll
      for (int j = 0; j < R1; ++j) v[j] = __ldcg(g + (size_t)p * n + (size_t)(t + R2 * j) * plane);
      dft::run<R1, false>(v);
#pragma unroll
      for (int s = 1; s < R1; ++s) v[s] = cmul(v[s], roots[t * s]);
#pragma unroll
      for (int s = 0; s < R1; ++s) sm[(p * N + s * R2 + t) * COLS + col] = v[s];
    }
  }
  if constexpr (AHEAD)
    if (threadIdx.x < COLS * R1)
#pragma unroll
      for (int k = 0; k < H; ++k) load_pair(threadIdx.x, k, fkv[k], X[k]);
  __syncthreads();
#pragma unroll 1
  for (int i0 = 0; i0 < COLS * R1; i0 += Z::TH) {
    const int i = i0 + threadIdx.x;
    const bool act = i < COLS * R1;
    const unsigned mask = __ballot_sync(0xffffffffu, act);
    if (!act) continue;
    const int side = i & 1, o = (i >> 1) % CW, s = (i >> 1) / CW;
    const int grp = side ? R1 - 1 - s : s, cl = side ? COLS - 1 - o : o;
    C v[P][R2];
#pragma unroll
    for (int p = 0; p < P; ++p) {
#pragma unroll
      for (int k = 0; k < R2; ++k) v[p][k] = sm[(p * N + grp * R2 + k) * COLS + cl];
      dft::run<R2, false>(v[p]);
    }
    const int kx = x0 + o;
#pragma unroll
    for (int k = 0; k < H; ++k) {
      // the owner point of this lane's pair k
      const int kz = pair_kz(i, k);
      if constexpr (!AHEAD) load_pair(i, k, fkv[0], X[0]);
      const double2 fk = fkv[AHEAD ? k : 0];
      C y[P], ym[P], out[P], outm[P];
#pragma unroll
      for (int p = 0; p < P; ++p) {
        const C q = shfl_pair(mask, v[p][R2 - 1 - k]);
        y[p] = side ? q : v[p][k];
        ym[p] = side ? v[p][k] : q;
      }
      kspace_product_x<T, V>(a, fk, X[AHEAD ? k : 0], kx, ky, kz, y, ym, out, outm);
#pragma unroll
      for (int p = 0; p < P; ++p) {
        v[p][k] = side ? outm[p] : out[p];
        v[p][R2 - 1 - k] = shfl_pair(mask, side ? out[p] : outm[p]);
      }
    }
#pragma unroll
    for (int p = 0; p < P; ++p) {
      dft::run<R2, true>(v[p]);
#pragma unroll
      for (int k = 0; k < R2; ++k)
        sm[(p * N + grp * R2 + k) * COLS + cl] =
            k ? dft::cmulw<true>(v[p][k], roots[k * grp]) : v[p][k];
    }
    if constexpr (AHEAD && R1 > R2)
      if (i + Z::TH < COLS * R1)
#pragma unroll
        for (int k = 0; k < H; ++k) load_pair(i + Z::TH, k, fkv[k], X[k]);
  }
  __syncthreads();
  if (live) {
#pragma unroll
    for (int p = 0; p < P; ++p) {
      C v[R1];
#pragma unroll
      for (int s = 0; s < R1; ++s) v[s] = sm[(p * N + s * R2 + t) * COLS + col];
      dft::run<R1, true>(v);
#pragma unroll
      for (int j = 0; j < R1; ++j) __stcg(g + (size_t)p * n + (size_t)(t + R2 * j) * plane, v[j]);
    }
  }
}

template <typename T, int N, int V>
__global__ void __launch_bounds__(ZShape<T, N, V>::TH, (ZShape<T, N, V>::MINB)) k_zline(IterArgs<T> a0) {
  extern __shared__ __align__(16) unsigned char fused_sm[];
  const IterArgs<T> a = solute_view<T, V>(a0);
  if (a.st->done) return;
  zline_tile<T, N, V, false, true>(a, reinterpret_cast<CxT<T> *>(fused_sm), a.roots, N, N, blockIdx.x);
}

// ---------------------------------------------------------------- one launch
// A whole phase in one launch, for grids whose three kernels take about as
// long as their launches: the same three stages with a barrier over the
// solute's blocks between them (all resident: cooperative launch).  Every
// block keeps its own copy of the loop state and reduces all block sums
// itself, in the same order, so the stopping test and the 2 x 2 solve need no
// further exchange.  A block always works on the same planes, so the state
// arrays are only ever touched by the SM that wrote them; the transform
// buffer, the exchange planes and the sums go through L2.
//
// Debugging aid (RISM3D_STAGE_DELAY): a block sleeps up to `delay` ns before a
// stage, another time in each block and stage, so that results which depend on
// the blocks' relative speed show.
__device__ __forceinline__ void stage_delay(unsigned delay, unsigned salt) {
  const unsigned h = (blockIdx.x * 2654435761u) ^ (salt * 2246822519u) ^ (blockIdx.y * 40503u);
  __nanosleep((h >> 8) % delay);
}

// The arrival count of one solute's blocks is zero at every launch: the last
// block to leave the kernel (leave_barrier) clears it, and after a wait that
// gave up the host side does.  A launch on a count left over from another
// would run through every barrier without waiting.
//
// A block's side of it lies in shared memory and the barrier is a call: inline,
// its values took registers that the stages' loops need (k_phase spilled 204 B
// a thread instead of 32 at 128^3 in FP64, 19.2 instead of 17.5 ms a solve).
struct GridBarrier {
  unsigned *count;                                 // arrivals
  unsigned due, nblk;                              // of the last barrier; blocks
  unsigned delay;                                  // stage_delay, ns
  int ok;                                          // no wait gave up
};
// Arrival and wait, with a bound on the wait: false when the other blocks never
// came (the caller leaves, and is not counted out: so the host side learns).
constexpr unsigned kBarrierPolls = 1u << 24;
static __device__ __noinline__ bool grid_barrier(GridBarrier &b) {
  unsigned *count = nullptr;
  unsigned due = 0u, delay = 0u;
  if (threadIdx.x == 0) {                          // its own values: off the way
    count = b.count;
    due = b.due + b.nblk;
    delay = b.delay;
    b.due = due;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
    unsigned v, polls = 0;
    do {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(count) : "memory");
    } while ((int)(v - due) < 0 && ++polls < kBarrierPolls);      // the count may wrap
    if ((int)(v - due) < 0) b.ok = 0;
    if (delay) stage_delay(delay, due);
  }
  __syncthreads();
  return b.ok != 0;
}
// One thread, before the first barrier (a block barrier follows)
static __device__ __noinline__ void enter_barrier(GridBarrier &b, unsigned *count, unsigned delay) {
  b = GridBarrier{count, 0u, gridDim.x, delay, 1};
  if (delay) stage_delay(delay, 0u);
}
// One thread of each block, after its last barrier: the last of the blocks,
// which no other polls any more, clears the count.
static __device__ __noinline__ void leave_barrier(GridBarrier &b) {
  if (b.ok && atomicAdd(b.count, 1u) == b.due + b.nblk - 1u) atomicExch(b.count, 0u);
}

// A whole phase that runs without its clusters does nothing and says so
static __device__ __noinline__ void refuse_phase(DevState *st) {
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    st->fault = 2;
    st->done = 2;
    st->after_done = 1;
  }
}

// byte offset of the tables: after the largest of the stages' exchanges
template <typename T, int N, int V> __host__ __device__ constexpr size_t tables_at() {
  const size_t row = sizeof(CxT<T>) * Lines<N>::LB * Lines<N>::LS,
               z = sizeof(CxT<T>) * (size_t)((V + 1) / 2) * 2 * Lines<N>::CW * N;
  return row > z ? row : z;
}

template <typename T, int N, int V, bool REF>
__global__ void __cluster_dims__(Lines<N>::NC, 1, 1)
    __launch_bounds__(Lines<N>::TH, (Lines<N>::template minp<T, V>())) k_phase(IterArgs<T> a0, bool hnc) {
  typedef CxT<T> C;
  extern __shared__ __align__(16) unsigned char fused_sm[];
  constexpr bool WIDE = Lines<N>::template minp<T, V>() == 1 && Lines<N>::template minb<T>() > 1;
  __shared__ DevState ss;
  C *sm = reinterpret_cast<C *>(fused_sm);
  const IterArgs<T> a = solute_view<T, V>(a0);
  if (cluster_ctas() != Lines<N>::NC) {            // see the launches
    refuse_phase(a.st);
    return;
  }
  // the phase and root tables, read at every stage, stay in shared memory
  // (every barrier's acquire empties L1)
  C *tw = reinterpret_cast<C *>(fused_sm + tables_at<T, N, V>()), *roots = tw + 3 * N;
  for (int i = threadIdx.x; i < 3 * N; i += blockDim.x) tw[i] = a.tw[i];
  for (int i = threadIdx.x; i < N; i += blockDim.x) roots[i] = a.roots[i];
  if (threadIdx.x == 0) ss = *a.st;
  __syncthreads();
  __shared__ GridBarrier bar;
  const unsigned nblk = gridDim.x;
  if (threadIdx.x == 0) enter_barrier(bar, a.bar + blockIdx.y, a.delay);
  __syncthreads();
  while (!ss.done) {
    planes_a<T, N, V, REF, WIDE>(a, &ss, sm, tw, roots, hnc);
    if (!grid_barrier(bar)) break;
#pragma unroll 1
    for (int tile = blockIdx.x; tile < ZShape<T, N, V>::TILES; tile += nblk) {
      zline_tile<T, N, V, WIDE, true>(a, sm, roots, N, N, tile);
      __syncthreads();
    }
    if (!grid_barrier(bar)) break;
    planes_r<T, N, V, REF, WIDE>(a, &ss, sm, tw, roots, hnc);
    if (!grid_barrier(bar)) break;
    finalize_block(&ss, a.part, (int)nblk, (double)a.n * V, blockIdx.x == 0 ? a.hist : nullptr,
                   a.hist_cap);
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    if (blockIdx.x == 0) {
      if (!bar.ok) ss.done = 2;
      ss.after_done = 1;
      *a.st = ss;
    }
    leave_barrier(bar);
  }
}

// ---------------------------------------------------------------- launches
// The plane kernels carry their cluster size (__cluster_dims__), not the
// launch: ncu replays a cooperative launch without its attributes, and with
// clusters of one CTA plane_sync orders nothing -- a 32^3 solve then ran its
// 10000 steps without converging.  The two whole-phase kernels check it.
//
// Clusters of a plane kernel: one per plane, at most what is resident at once
// (a cluster then walks its planes with one scratch plane).
template <typename K>
int plane_clusters(K kernel, int nc, int threads, size_t smem, int planes) {
  int num = 0;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(nc);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  if (cudaOccupancyMaxActiveClusters(&num, kernel, &cfg) != cudaSuccess || num < 1) {
    cudaGetLastError();
    return 0;
  }
  return num < planes ? num : planes;
}

template <typename K, typename... A>
cudaError_t launch_plane(K kernel, int nclusters, int nc, int nb, int threads, size_t smem,
                         cudaStream_t st, bool cooperative, A... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(nclusters * nc, nb);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeCooperative;
  at.val.cooperative = 1;
  cfg.attrs = &at;
  cfg.numAttrs = cooperative ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

// The kernels of one (arithmetic, edge, sites) and their launch shapes
template <typename T, int N, int V>
struct Kernels {
  using L = Lines<N>;
  using Z = ZShape<T, N, V>;
  static constexpr int P = (V + 1) / 2;
  static_assert(V % 2 == 0, "whole site pairs");
  // A phase as one launch, by what a step took on a B200 (us, loop of three
  // launches / one launch; V = 2): FP64 N = 32 25 / 16, 64 31 / 23, 80 52 / 41,
  // 128 152 / 132, 160 336 / 320, 256 1022 / 1082; V = 4: 64 47 / 39, 80 109 /
  // 93, 128 316 / 354 (the one kernel's registers spill).  FP32 one launch is
  // never slower: 64 31 / 19, 128 101 / 89, 256 592 / 575.
  static constexpr bool ONE = sizeof(T) == 4 || N <= 80 || (N <= 160 && V <= 2);
  template <typename K> static cudaError_t allow(K k, size_t b) {
    return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)b);
  }
  static constexpr size_t phase_smem() {
    return tables_at<T, N, V>() + 4 * N * sizeof(CxT<T>);
  }
  // Attributes and cluster counts; false when the device cannot run them.  Only
  // the kernels that the cell will launch are touched: each costs 1-4 ms the
  // first time in a process, when the driver loads it.
  static bool setup(FusedPlan &f, int nb, bool host) {
    const size_t s = L::template smem<T>();
    f.nc = L::NC;
    cudaError_t e = allow(k_plane_final<T, N, V, false>, s);
    if constexpr (sizeof(T) == 4)
      if (e == cudaSuccess) e = allow(k_plane_final<T, N, V, true>, s);
    // clusters of one phase launch: resident ones shared by the nb solutes
    if constexpr (ONE) {
      if (!host) {
        if (e == cudaSuccess) e = allow(k_phase<T, N, V, false>, phase_smem());
        if (e == cudaSuccess)
          f.cp[0] = plane_clusters(k_phase<T, N, V, false>, L::NC, L::TH, phase_smem(), 1 << 30) / nb;
        f.cp[1] = f.cp[0];
        if constexpr (sizeof(T) == 4) {
          if (e == cudaSuccess) e = allow(k_phase<T, N, V, true>, phase_smem());
          if (e == cudaSuccess)
            f.cp[1] = plane_clusters(k_phase<T, N, V, true>, L::NC, L::TH, phase_smem(), 1 << 30) / nb;
        }
        for (int r = 0; r < 2; ++r) f.cp[r] = f.cp[r] < N * P ? f.cp[r] : N * P;
      }
    }
    if (e != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    if ((f.cp[0] == 0 || f.cp[1] == 0) && !setup_planes(f, N * P)) return false;
    for (int r = 0; r < 2; ++r) {
      f.cs = f.cs > f.cp[r] ? f.cs : f.cp[r];
      f.cs = f.cs > f.cr[r] ? f.cs : f.cr[r];
    }
    return true;
  }
  // the same of the kernels of a cycle; room: exchange planes
  static bool setup_planes(FusedPlan &f, int room) {
    const size_t s = L::template smem<T>();
    cudaError_t e = allow(k_plane_a<T, N, V, false>, s);
    if (e == cudaSuccess) e = allow(k_plane_r<T, N, V, false>, s);
    if (e == cudaSuccess) e = allow(k_zline<T, N, V>, Z::smem());
    if constexpr (sizeof(T) == 4) {
      if (e == cudaSuccess) e = allow(k_plane_a<T, N, V, true>, s);
      if (e == cudaSuccess) e = allow(k_plane_r<T, N, V, true>, s);
    }
    if (e != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    const int planes = N * P, rp = planes < room ? planes : room;
    f.ca[0] = plane_clusters(k_plane_a<T, N, V, false>, L::NC, L::TH, s, planes);
    f.cr[0] = plane_clusters(k_plane_r<T, N, V, false>, L::NC, L::TH, s, rp);
    f.ca[1] = f.ca[0];
    f.cr[1] = f.cr[0];
    if constexpr (sizeof(T) == 4) {
      f.ca[1] = plane_clusters(k_plane_a<T, N, V, true>, L::NC, L::TH, s, planes);
      f.cr[1] = plane_clusters(k_plane_r<T, N, V, true>, L::NC, L::TH, s, rp);
    }
    f.planes = f.ca[0] > 0 && f.cr[0] > 0 && f.ca[1] > 0 && f.cr[1] > 0;
    return f.planes;
  }
  // which: 0 plane A, 1 z lines, 2 plane R, 3 the pass after the loop, 4 a
  // whole phase
  static cudaError_t launch(const FusedPlan &f, int which, bool ref, int hnc, int nb,
                            const IterArgs<T> &a, cudaStream_t st) {
    if (which == 1) {
      k_zline<T, N, V><<<dim3(Z::TILES, nb), Z::TH, Z::smem(), st>>>(a);
      return cudaGetLastError();
    }
    if constexpr (sizeof(T) == 4) {
      if (ref) return launch_planes<true>(f, which, hnc != 0, nb, a, st);
    }
    return launch_planes<false>(f, which, hnc != 0, nb, a, st);
  }
  template <bool REF>
  static cudaError_t launch_planes(const FusedPlan &f, int which, bool hnc, int nb,
                                   const IterArgs<T> &a, cudaStream_t st) {
    const size_t s = L::template smem<T>();
    if constexpr (ONE)
      if (which == 4)
        return launch_plane(k_phase<T, N, V, REF>, f.cp[REF], L::NC, nb, L::TH, phase_smem(),
                            st, true, a, hnc);
    const int ncl = which == 0 ? f.ca[REF] : which == 2 ? f.cr[REF] : f.cs;
    return launch_plane(which == 0   ? k_plane_a<T, N, V, REF>
                        : which == 2 ? k_plane_r<T, N, V, REF>
                                     : k_plane_final<T, N, V, REF>,
                        ncl, L::NC, nb, L::TH, s, st, false, a, hnc);
  }
};

template <typename T, int N>
Vtable<T> table_v(int V) {
  switch (V) {
    case 2: return {Kernels<T, N, 2>::setup, Kernels<T, N, 2>::setup_planes, Kernels<T, N, 2>::launch};
    case 4: return {Kernels<T, N, 4>::setup, Kernels<T, N, 4>::setup_planes, Kernels<T, N, 4>::launch};
  }
  return {};
}

}  // namespace fused
}  // namespace rism3d
