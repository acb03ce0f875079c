// Device code shared by the iteration's kernels: the argument block, the
// closures and residuals, the k-space product of one mirror pair, and the
// reduction that steers the loop.
#pragma once

#include "rism3d_impl.h"

namespace rism3d {

template <typename T> struct Cx;
template <> struct Cx<double> { typedef double2 t; };
template <> struct Cx<float> { typedef float2 t; };

template <typename T>
struct IterArgs {
  long long n;
  int nx, ny, nz;
  FastDiv fdx, fdy;         // division by nx and ny
  const double *xs;         // chi table per odd-square sum (cubic cells) or null
  const float *xs32;        // the same table in FP32 (read by the FP32 passes)
  typename Cx<T>::t *buf;   // [P][N]
  T *t, *U, *Y, *RP;        // t, U: [V][N]; Y, RP: [2][V][N]
  const T *R0;              // refinement: base residual [V][N] (t = d, U = x0)
  double *hout, *gout;      // final snapshot, [V][N] (may be null)
  const typename Cx<T>::t *tw;  // px[nx] py[ny] pz[nz]
  double invvol, dv;
  const double2 *fkh;       // [N/2]
  const double *chi;        // [ntab][V*V][4]
  int ntab;
  double dk;
  double bx, by, bz;
  DevState *st;
  const StageParams *sp;
  double *part;
  int nblocks;
  unsigned *count;          // blocks of pass R done (reset by the last one)
  double *hist;             // per-iteration rms (single solves, verbose) or null
  int hist_cap;
  int nofk;                 // refinement: q cf fk cancels, fk is not read
  const float2 *xroots;     // fused-axis passes: W_nx^m, m < nx (nx == ny)
  const float2 *fkt;        // fused-axis pass K (nx = 256): beta fk as [nz/2][nx][ny]
  // three-kernel iteration (fused.cuh)
  T *RPx;                   // third residual slot [V][N]
  typename Cx<T>::t *scr;   // plane exchange, scr_n points per solute
  long long scr_n;
  const typename Cx<T>::t *roots;   // W_N^m, m < N (the cell edge); non-cubic: [nx] [ny] [nz]
  const T *xo;              // non-cubic: chi_ab [nz/2][ny/2][nx/2][V*V], by |2 i + 1| per axis
  cudaGraphConditionalHandle cond;  // loop body: the while node to steer
  int loop;                 // 1: plane R runs the loop test itself
  int body_kernels;         // kernels of one cycle in this form
  int nb;                   // solutes
  unsigned *gcount;         // solutes whose plane R is done (nb > 1)
  unsigned *bar;            // arrival counts of a whole-phase launch [nb]
  unsigned delay;           // longest sleep of a block before a stage (ns; debugging)
};

namespace {

constexpr int kThreads = 256;


// Batched solves: blockIdx.y selects the solute; every per-solute array is
// laid out solute-major ([B][...]) and this view offsets the pointers, so
// the kernel bodies below are the single-solute code unchanged.
template <typename T, int V>
__device__ __forceinline__ IterArgs<T> solute_view(const IterArgs<T> &a) {
  constexpr int P = (V + 1) / 2;
  IterArgs<T> s = a;
  const size_t b = blockIdx.y, n = (size_t)a.n;
  if (b == 0) return s;
  s.buf = a.buf + b * P * n;
  s.t = a.t + b * V * n;
  s.U = a.U + b * V * n;
  s.Y = a.Y + b * 2 * V * n;
  s.RP = a.RP + b * 2 * V * n;
  if (a.hout) { s.hout = a.hout + b * V * n; s.gout = a.gout + b * V * n; }
  if (a.R0) s.R0 = a.R0 + b * V * n;
  s.fkh = a.fkh + b * (n / 2);
  s.st = a.st + b;
  s.part = a.part + b * 6 * (size_t)a.nblocks;
  s.count = a.count + b;
  if (a.RPx) {
    s.RPx = a.RPx + b * V * n;
    s.scr = a.scr + b * (size_t)a.scr_n;
  }
  return s;
}

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
template <typename C> __device__ __forceinline__ C mk(double x, double y);
template <> __device__ __forceinline__ double2 mk<double2>(double x, double y) {
  return make_double2(x, y);
}
template <> __device__ __forceinline__ float2 mk<float2>(double x, double y) {
  return make_float2((float)x, (float)y);
}

// Vector access to PTS (1 or 2) consecutive points of a real or complex
// array; point pairs start at even indices, so 2-wide accesses are aligned.
template <typename T> struct V2;
template <> struct V2<float> { typedef float2 t; typedef float4 c; };
template <> struct V2<double> { typedef double2 t; typedef double4 c; };

template <int PTS, typename T>
__device__ __forceinline__ void ldr(const T *__restrict__ p, T (&o)[PTS]) {
  if (PTS == 1) {
    o[0] = p[0];
  } else {
    const typename V2<T>::t w = *reinterpret_cast<const typename V2<T>::t *>(p);
    o[0] = w.x;
    o[PTS - 1] = w.y;
  }
}
template <int PTS, typename T>
__device__ __forceinline__ void str(T *__restrict__ p, const T (&o)[PTS]) {
  if (PTS == 1) {
    p[0] = o[0];
  } else {
    typename V2<T>::t w;
    w.x = o[0];
    w.y = o[PTS - 1];
    *reinterpret_cast<typename V2<T>::t *>(p) = w;
  }
}
template <int PTS, typename C>
__device__ __forceinline__ void ldc(const C *__restrict__ p, C (&o)[PTS]) {
#pragma unroll
  for (int k = 0; k < PTS; ++k) o[k] = p[k];
}
template <int PTS, typename C>
__device__ __forceinline__ void stc(C *__restrict__ p, const C (&o)[PTS]) {
#pragma unroll
  for (int k = 0; k < PTS; ++k) p[k] = o[k];
}
// FP32 complex pairs move as one 16-byte access
template <>
__device__ __forceinline__ void ldc<2, float2>(const float2 *__restrict__ p, float2 (&o)[2]) {
  const float4 w = *reinterpret_cast<const float4 *>(p);
  o[0] = make_float2(w.x, w.y);
  o[1] = make_float2(w.z, w.w);
}
template <>
__device__ __forceinline__ void stc<2, float2>(float2 *__restrict__ p, const float2 (&o)[2]) {
  *reinterpret_cast<float4 *>(p) = make_float4(o[0].x, o[0].y, o[1].x, o[1].y);
}

__device__ __forceinline__ double fexp(double x) { return exp(x); }
__device__ __forceinline__ float fexp(float x) { return expf(x); }

// calculate_cuda.cu:1-20: KH g = 1 + x (x >= 0) or e^x; HNC g = e^x.
template <int CLOS, typename T>
__device__ __forceinline__ T closure(T x) {
  if (CLOS == 0) return x >= T(0) ? T(1) + x : fexp(x);
  return fexp(x);
}

__device__ __forceinline__ double fexpm1(double x) { return expm1(x); }
__device__ __forceinline__ float fexpm1(float x) { return expm1f(x); }

// C(x0 + d) - C(x0) to the relative precision of the difference itself
// (refinement form).  KH: C(x) - 1 = max(x, 0) + expm1(min(x, 0)), so with
// a = min(x0 + d, 0), b = min(x0, 0)
//   C(x0 + d) - C(x0) = [max(x0 + d, 0) - max(x0, 0)] + e^b expm1(a - b),
// where the linear bracket is d itself when both arguments are >= 0 and
// a - b is d itself when both are < 0: e^x0 expm1(d) on the exponential
// branch, d on the linear one, and in the two mixed cases (|x0| <= |d|)
// x - expm1(x0) and expm1(x) - x0.  One exp and one expm1 per call and no
// branches, so the lanes of a warp never split over the four cases.
template <int CLOS, typename T>
__device__ __forceinline__ T closure_diff(T x0, T d) {
  if (CLOS == 1) return fexp(x0) * fexpm1(d);
  const T x = x0 + d;
  const bool pos = x >= T(0), pos0 = x0 >= T(0);
  const T zero = T(0);
  const T lin = (pos && pos0) ? d : (fmax(x, zero) - fmax(x0, zero));
  const T b = fmin(x0, zero);
  const T da = (!pos && !pos0) ? d : (fmin(x, zero) - b);
  return lin + fexp(b) * fexpm1(da);
}

// Residual of the cycle at the current state: plain h + 1 - C(t - U);
// refinement R0 + h - [C(x0 + d) - C(x0)] (t = d, U = x0, h = L[dc]).
template <int CLOS, bool REF, typename T>
__device__ __forceinline__ T residual(T h, T t, T U, T r0) {
  if (REF) return r0 + h - closure_diff<CLOS>(U, t);
  return h + T(1) - closure<CLOS>(t - U);
}

// Packed FFT input: plain c_SR = C(t - U) - 1 - t; refinement dc = dg - d.
template <int CLOS, bool REF, typename T>
__device__ __forceinline__ T cfun(T t, T U) {
  if (REF) return closure_diff<CLOS>(U, t) - t;
  return closure<CLOS>(t - U) - T(1) - t;
}

// The same three with the closure chosen at run time (uniform): one exp (and
// expm1) for either closure.
template <typename T> __device__ __forceinline__ T closure_rt(T x, bool hnc) {
  const T e = fexp(x);
  return (!hnc && x >= T(0)) ? T(1) + x : e;
}
template <typename T> __device__ __forceinline__ T closure_diff_rt(T x0, T d, bool hnc) {
  const T x = x0 + d, zero = T(0);
  const bool pos = x >= zero && !hnc, pos0 = x0 >= zero && !hnc;
  const T b = hnc ? x0 : fmin(x0, zero);
  const T lin = hnc ? zero : (pos && pos0) ? d : (fmax(x, zero) - fmax(x0, zero));
  const T da = (!pos && !pos0) ? d : (fmin(x, zero) - b);
  return lin + fexp(b) * fexpm1(da);
}
template <bool REF, typename T>
__device__ __forceinline__ T residual_rt(T h, T t, T U, T r0, bool hnc) {
  if (REF) return r0 + h - closure_diff_rt(U, t, hnc);
  return h + T(1) - closure_rt(t - U, hnc);
}
template <bool REF, typename T> __device__ __forceinline__ T cfun_rt(T t, T U, bool hnc) {
  if (REF) return closure_diff_rt(U, t, hnc) - t;
  return closure_rt(t - U, hnc) - T(1) - t;
}

// Point index -> (ix, iy, iz), +-1 checkerboard dir = (-1)^(ix+iy+iz)
// (set_ir, fft3d.cu:86-94) and dkf = exp(-i pi sum x_d/n_d)
// (set_kf, fft3d.cu:71-83) as a product of three per-axis phases.
__device__ __forceinline__ void split_index(long long j, const FastDiv &fdx,
                                            const FastDiv &fdy, int &ix, int &iy,
                                            int &iz) {
  const unsigned u = (unsigned)j;                 // N < 2^31
  const unsigned r = fdx.div(u);
  ix = (int)(u - r * fdx.d);
  iz = (int)fdy.div(r);
  iy = (int)(r - (unsigned)iz * fdy.d);
}

template <typename C>
__device__ __forceinline__ void point_phase(long long j, const FastDiv &fdx,
                                            const FastDiv &fdy, const C *tw,
                                            int &ix, int &iy, int &iz, int &dir,
                                            C &dkf) {
  split_index(j, fdx, fdy, ix, iy, iz);
  dir = ((ix + iy + iz) & 1) ? -1 : 1;
  const int nx = (int)fdx.d, ny = (int)fdy.d;
  dkf = cmul(cmul(tw[ix], tw[nx + iy]), tw[nx + ny + iz]);
}

// chi_ab(|k|) of a cubic cell from its per-|k|^2 table: |k| = (pi/L) sqrt(s),
// s a sum of three odd squares (solvent_spline.cu:36-47).  Rows of an odd
// number of values are read one value at a time (they are not all aligned).
template <typename T, int V>
__device__ __forceinline__ void chi_cubic(const IterArgs<T> &a, int ix, int iy, int iz,
                                          T (&X)[V * V]) {
  const int ox = 2 * ix - a.nx + 1, oy = 2 * iy - a.ny + 1, oz = 2 * iz - a.nz + 1;
  const unsigned sq = (unsigned)(ox * ox + oy * oy + oz * oz);
  const size_t row = (size_t)((sq - 3u) >> 3) * V * V;
  if constexpr (sizeof(T) == 4 && V * V % 4 == 0) {
    const float4 *xr = reinterpret_cast<const float4 *>(a.xs32 + row);   // 16-byte rows
#pragma unroll
    for (int ab = 0; ab < V * V / 4; ++ab) {
      const float4 q = xr[ab];
      X[4 * ab] = q.x;
      X[4 * ab + 1] = q.y;
      X[4 * ab + 2] = q.z;
      X[4 * ab + 3] = q.w;
    }
  } else if constexpr (sizeof(T) == 4) {
#pragma unroll
    for (int ab = 0; ab < V * V; ++ab) X[ab] = a.xs32[row + ab];
  } else if constexpr (V * V % 2 == 0) {
    const double2 *xr = reinterpret_cast<const double2 *>(a.xs + row);
#pragma unroll
    for (int ab = 0; ab < V * V / 2; ++ab) {
      const double2 q = xr[ab];
      X[2 * ab] = (T)q.x;
      X[2 * ab + 1] = (T)q.y;
    }
  } else {
#pragma unroll
    for (int ab = 0; ab < V * V; ++ab) X[ab] = (T)a.xs[row + ab];
  }
}

// chi_ab(|k|) of a non-cubic cell from its octant table: |k| depends on the
// distance of each index from the middle alone.
template <typename T, int V>
__device__ __forceinline__ void chi_octant(const IterArgs<T> &a, int ix, int iy, int iz,
                                           T (&X)[V * V]) {
  const int hx = a.nx / 2, hy = a.ny / 2, hz = a.nz / 2;
  const int mx = ix < hx ? hx - 1 - ix : ix - hx, my = iy < hy ? hy - 1 - iy : iy - hy,
            mz = iz < hz ? hz - 1 - iz : iz - hz;
  const T *row = a.xo + ((size_t)mx + (size_t)hx * (my + (size_t)hy * mz)) * V * V;
  if constexpr (V * V * sizeof(T) % 16 == 0) {
#pragma unroll
    for (int ab = 0; ab < V * V; ab += 16 / (int)sizeof(T)) {
      union { float4 b; T t[16 / sizeof(T)]; } u;
      u.b = *reinterpret_cast<const float4 *>(row + ab);
#pragma unroll
      for (int e = 0; e < 16 / (int)sizeof(T); ++e) X[ab + e] = u.t[e];
    }
  } else {
#pragma unroll
    for (int ab = 0; ab < V * V; ++ab) X[ab] = row[ab];
  }
}

// chi_ab(|k|) of any cell: natural spline on knots k_i = dk (i+1) with the
// bisection semantics of splint.cc:9-16 on uniform knots
template <typename T, int V>
__device__ __forceinline__ void chi_spline(const IterArgs<T> &a, int ix, int iy, int iz,
                                           T (&X)[V * V]) {
  const double kx = 2.0 * kPi * (ix - a.nx / 2.0 + 0.5) / a.bx;   // set_g
  const double ky = 2.0 * kPi * (iy - a.ny / 2.0 + 0.5) / a.by;
  const double kz = 2.0 * kPi * (iz - a.nz / 2.0 + 0.5) / a.bz;
  const double kk = sqrt(kx * kx + ky * ky + kz * kz);
  int k0 = (int)(kk / a.dk) - 1;
  k0 = k0 < 0 ? 0 : (k0 > a.ntab - 2 ? a.ntab - 2 : k0);
  while (k0 < a.ntab - 2 && a.dk * (k0 + 2) <= kk) ++k0;
  while (k0 > 0 && a.dk * (k0 + 1) > kk) --k0;
  const double tt = kk - a.dk * (k0 + 1);
  const double2 *cf = reinterpret_cast<const double2 *>(a.chi + (size_t)k0 * V * V * 4);
#pragma unroll
  for (int ab = 0; ab < V * V; ++ab) {
    const double2 lo = cf[2 * ab], hi2 = cf[2 * ab + 1];
    X[ab] = (T)(((hi2.y * tt + hi2.x) * tt + lo.y) * tt + lo.x);
  }
}

// One mirror pair of k points: j (the owner, j < N/2, grid indices ix iy iz)
// and jm = N-1-j with k(jm) = -k(j).  y/ym are the forward-transformed
// packed site pairs at j and jm; out/outm receive the OZ result repacked
// for the inverse transform.
// fk is beta fk at the owner point (zero when a.nofk).
// X: chi_ab there, in T.
template <typename T, int V>
__device__ __forceinline__ void kspace_product_x(const IterArgs<T> &a, double2 fk,
                                                 const T (&X)[V * V], int ix, int iy, int iz,
                                                 const typename Cx<T>::t *y,
                                                 const typename Cx<T>::t *ym,
                                                 typename Cx<T>::t *out,
                                                 typename Cx<T>::t *outm) {
  typedef typename Cx<T>::t C;
  constexpr int P = (V + 1) / 2;
  const StageParams *sp = a.sp;
  const int dir = ((ix + iy + iz) & 1) ? -1 : 1;
  // unpack the site pairs and finish the forward transform
  // (timeirvol * dv, fft3d.cu:32) and subtract q cf fk (mqvfk)
  // (in the working precision T: the FP32 passes round F to FP32 anyway)
  C F[V];
  const T sc = (T)(a.dv * 0.5 * dir);
  const T fx = (T)fk.x, fy = (T)fk.y;
#pragma unroll
  for (int p = 0; p < P; ++p) {
    const T qa = (T)sp->qcf[2 * p];
    F[2 * p] = mk<C>(sc * (y[p].x - ym[p].x) - qa * fx, sc * (y[p].y + ym[p].y) - qa * fy);
    if (2 * p + 1 < V) {
      const T qb = (T)sp->qcf[2 * p + 1];
      F[2 * p + 1] = mk<C>(sc * (y[p].y - ym[p].y) - qb * fx, -sc * (y[p].x + ym[p].x) - qb * fy);
    }
  }
  C H[V];
#pragma unroll
  for (int va = 0; va < V; ++va) {
    T hr = 0, hi = 0;
#pragma unroll
    for (int vb = 0; vb < V; ++vb) {
      const T x = X[va * V + vb];
      hr += F[vb].x * x;                       // oz, calculate_cuda.cu:44-58
      hi += F[vb].y * x;
    }
    H[va] = mk<C>(hr, hi);
  }
  // repack for the inverse: dir (h_a + i h_b) at k and its mirror
  // (timeirvol before the inverse, fft3d.cu:34)
  const T d = (T)dir;
#pragma unroll
  for (int p = 0; p < P; ++p) {
    const C ha = H[2 * p];
    const C hb = (2 * p + 1 < V) ? H[2 * p + 1] : mk<C>(0.0, 0.0);
    out[p] = mk<C>(d * (ha.x - hb.y), d * (ha.y + hb.x));
    outm[p] = mk<C>(-d * (ha.x + hb.y), -d * (hb.x - ha.y));
  }
}

template <typename T, int V>
__device__ __forceinline__ void kspace_pair_fk(const IterArgs<T> &a, double2 fk, int ix, int iy,
                                               int iz, const typename Cx<T>::t *y,
                                               const typename Cx<T>::t *ym,
                                               typename Cx<T>::t *out, typename Cx<T>::t *outm) {
  T X[V * V];
  if (a.xs) chi_cubic<T, V>(a, ix, iy, iz, X);
  else chi_spline<T, V>(a, ix, iy, iz, X);
  kspace_product_x<T, V>(a, fk, X, ix, iy, iz, y, ym, out, outm);
}

template <typename T, int V>
__device__ __forceinline__ void kspace_pair(const IterArgs<T> &a, long long j, int ix, int iy,
                                            int iz, const typename Cx<T>::t *y,
                                            const typename Cx<T>::t *ym,
                                            typename Cx<T>::t *out, typename Cx<T>::t *outm) {
  const double2 fk = a.nofk ? make_double2(0.0, 0.0) : a.fkh[j];
  kspace_pair_fk<T, V>(a, fk, ix, iy, iz, y, ym, out, outm);
}

// ------------------------------------------------------------- finalize
// Run by the last block of pass R to finish: fixed-order reduction of the
// block sums, then the host logic of iterate.cu:52-62 and AN2::calculate
// (anderson.cu:35-63) on one thread -- no separate launch, no host sync.
__device__ void finalize_block(DevState *st, const double *part, int nblocks,
                               double nv_points, double *hist, int hist_cap) {
  // whole warps of any number: a butterfly in each warp, then one thread per
  // sum over the warps
  __shared__ double red[6][32];
  double s[6] = {0, 0, 0, 0, 0, 0};
  for (int b = threadIdx.x; b < nblocks; b += blockDim.x)
#pragma unroll
    for (int k = 0; k < 6; ++k) s[k] += __ldcg(part + (size_t)k * nblocks + b);
#pragma unroll
  for (int k = 0; k < 6; ++k)
    for (int o = 16; o > 0; o >>= 1) s[k] += __shfl_xor_sync(0xffffffffu, s[k], o);
  if ((threadIdx.x & 31) == 0)
#pragma unroll
    for (int k = 0; k < 6; ++k) red[k][threadIdx.x >> 5] = s[k];
  __syncthreads();
  if (threadIdx.x < 6) {
    double v = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) v += red[threadIdx.x][w];
    red[threadIdx.x][0] = v;
  }
  __syncthreads();
  if (threadIdx.x != 0) return;
  for (int k = 0; k < 6; ++k) st->sums[k] = red[k][0];
  const double rms = sqrt(red[0][0] / nv_points);
  st->rms = rms;
  if (st->measure) return;
  st->iter += 1;
  if (hist && st->iter <= hist_cap) hist[st->iter - 1] = rms;  // iterate.cu:63 output
  if (!isfinite(rms)) { st->done = 2; st->mode = 0; return; }  // iterate.cu:54-57
  if (rms <= st->conv) { st->done = 1; st->mode = 0; return; } // :58-59
  if (st->watch) {                       // a phase that may hand over early
    if (rms < 0.9 * st->best) { st->best = rms; st->since = 0; }
    else if (++st->since > 30) { st->done = 4; st->mode = 0; return; }
  }
  if (st->count > 0) {                                         // anderson.cu:43-49
    st->count -= 1;
    st->mode = 1;
  } else {                                                     // anderson.cu:50-61
    // [[a00 a01][a01 a11]] x = [c0 c1], eliminated as leg() does (:87-112)
    double a00 = red[3][0], a01 = red[4][0], a11 = red[5][0];
    double c0 = red[1][0], c1 = red[2][0];
    double p = a00;
    double a01n = a01 / p;
    double r = c0 / p;
    double a11n = a11 - a01 * a01n;
    double c1n = c1 - a01 * r;
    double x1 = c1n / a11n;
    double x0 = r - a01n * x1;
    st->s1 = x0 + st->mp * ((st->binary == 0) ? 0.0 : 1.0);
    st->s2 = x1 + st->mp * ((st->binary == 0) ? 1.0 : 0.0);
    st->mode = 2;
  }
  st->upd_slot = st->binary;
  st->binary = (st->binary == 0) ? 1 : 0;
  if (st->rotate) {                    // the new residual becomes this history entry
    const int f = st->rp[2];
    st->rp[2] = st->rp[st->upd_slot];
    st->rp[st->upd_slot] = f;
  }
  if (st->iter >= st->maxstep) st->done = 3;   // iterate.cu:51 loop bound
}

// End of one device-side loop body: keep looping while any solute is still
// running or has not yet had the idle pass after its stop (the snapshot);
// the body count is bounded by the phase's step limit plus a margin.
__device__ __forceinline__ void loop_test(cudaGraphConditionalHandle h, DevState *st, int nb,
                                          int body_kernels) {
  bool more = false;
  int cap = 1;                 // the largest step budget left to any solute
  for (int b = 0; b < nb; ++b) {
    if (!(__ldcg(&st[b].done) && __ldcg(&st[b].after_done) >= 1)) more = true;
    cap = max(cap, __ldcg(&st[b].maxstep));
  }
  const int loops = ++st[0].loops;
  st[0].launched += body_kernels;
  cap = cap < 1000000 ? cap : 1000000;
  if (loops >= cap + 4) more = false;
  cudaGraphSetConditional(h, more ? 1u : 0u);
}

// The loop test at the end of plane R: called once per solute and body, by
// one thread; the last solute's call runs the test.
template <typename T>
__device__ __forceinline__ void loop_test_all(const IterArgs<T> &a0) {
  if (!a0.loop) return;
  __threadfence();
  if (a0.nb > 1) {
    if (atomicAdd(a0.gcount, 1u) != (unsigned)a0.nb - 1u) return;
    *a0.gcount = 0u;
    __threadfence();
  }
  loop_test(a0.cond, a0.st, a0.nb, a0.body_kernels);
}

}  // namespace

}  // namespace rism3d
