// Cubic B-spline shift family (reference: src/holotomocupy/shift.py:15-221,
// kernels src/holotomocupy/cuda_kernels.py:131-290, 377-843).
//
// coeff: the periodic B-spline prefilter ifft2(fft2(psi) / B3) of shift.py:74-82.
//   The symbol B3[ky,kx] = (4 + 2 cos 2pi ky/nzpsi)(4 + 2 cos 2pi kx/npsi) is a
//   product, and along one axis 1 / (4 + 2 cos w) is a two-pole recursion
//   (k_bspline2d, k_bspline_cols).  Other symbols (ht_shift_filter) run as one
//   row pass and one column pass, each an FFT, a multiply by the symbol and an
//   inverse FFT.
// S / dS / d2S: 4x4-tap stencils at the sample position
//   x = mag (tx - n/2) - r_x + (mag-1)/2 + npsi/2 (same for y with r_y, nz,
//   nzpsi), zero outside the coefficient grid (cuda_kernels.py:177-222).
// S^T and the object part of dS^T: the reference scatters with atomics; here
//   every coefficient gathers from the output pixels whose 4x4 footprint
//   contains it (found from the inverse of the monotone sample map and
//   re-checked with the forward formula), so results are deterministic.
// Position part of dS^T: per-angle sums Re<g, dS/dr_y c>, Re<g, dS/dr_x c>
//   reduced in double precision inside the kernel (no dt1/dt2 images).
// Element type T is float2 (complex64 objects) or float (float32 objects).
#include "lines.cuh"
#include "holotomo_b200_internal.h"

#include <algorithm>
#include <cmath>
#include <vector>

namespace ht {

// ----------------------------------------------------------- the basis
// x6-scaled cubic B-spline and its derivatives (cuda_kernels.py:131-159)
__device__ __forceinline__ float bs0(float t) {
  if (-2.0f < t && t <= -1.0f) return (t + 2.0f) * (t + 2.0f) * (t + 2.0f);
  if (-1.0f < t && t <= 1.0f) return 4.0f - 6.0f * t * t + 3.0f * fabsf(t) * t * t;
  if (1.0f < t && t <= 2.0f) return (2.0f - t) * (2.0f - t) * (2.0f - t);
  return 0.0f;
}
__device__ __forceinline__ float bs1(float t) {
  if (-2.0f < t && t <= -1.0f) return 3.0f * (t + 2.0f) * (t + 2.0f);
  if (-1.0f < t && t <= 1.0f) return -12.0f * t + 9.0f * fabsf(t) * t;
  if (1.0f < t && t <= 2.0f) return -3.0f * (2.0f - t) * (2.0f - t);
  return 0.0f;
}
__device__ __forceinline__ float bs2(float t) {
  if (-2.0f < t && t <= -1.0f) return 6.0f * (t + 2.0f);
  if (-1.0f < t && t <= 1.0f) return -12.0f + 18.0f * fabsf(t);
  if (1.0f < t && t <= 2.0f) return 6.0f * (2.0f - t);
  return 0.0f;
}

// sample coordinate along one axis for output index t (cuda_kernels.py:179-184)
__device__ __forceinline__ float spline_x(float mag, int t, int nhalf, float shift, int npsihalf) {
  const float half = (mag - 1.0f) / 2.0f;
  return (mag * (float)(t - nhalf) - shift + half) + (float)npsihalf;
}

template <class T>
struct Ops;
template <>
struct Ops<float2> {
  static __device__ __forceinline__ float2 zero() { return make_float2(0.f, 0.f); }
  static __device__ __forceinline__ void fma(float2& a, float w, float2 v) {
    a.x += w * v.x;
    a.y += w * v.y;
  }
  static __device__ __forceinline__ float redot(float2 a, float2 b) { return a.x * b.x + a.y * b.y; }
};
template <>
struct Ops<float> {
  static __device__ __forceinline__ float zero() { return 0.f; }
  static __device__ __forceinline__ void fma(float& a, float w, float v) { a += w * v; }
  static __device__ __forceinline__ float redot(float a, float b) { return a * b; }
};

struct ShiftDims {
  int n, npsi, nz, nzpsi;
};

// ------------------------------------------------------- separable tiles
// The stencils are separable, so a CTA takes kTileX x kTileY outputs of one image
// in two steps: every input row its outputs reach is reduced along x at the
// tile's kTileX columns (a lane per column, its weights in registers) into
// shared memory, then each output sums its rows -- about 4 + 4 taps an output
// instead of 4 x 4, and the weights of a column and of a row are formed once.
// The tile is taken in parts where its rows exceed the buffer: the part halves
// until they fit.
constexpr int kTileX = 32, kTileY = 64, kTileThreads = 256, kTileWarps = kTileThreads / 32;
// reduced rows a buffer holds: those of a whole tile up to m = 1 (64 m + 4), half a tile for three sets
constexpr int tile_rows(int sets) { return sets == 3 ? 40 : 72; }

// Rows [lo, hi) that the outputs c0 .. c0 + part - 1 reach, halving part until
// they number at most max_rows; range(i, &first, &count) gives output i's rows.
template <class F>
__device__ __forceinline__ void tile_part(int c0, int max_rows, int& part, int& lo, int& hi, F range) {
  const int lane = threadIdx.x % 32;
  for (;;) {
    lo = 0x7fffffff;
    hi = 0;
    for (int i = lane; i < part; i += 32) {
      int p, c;
      range(c0 + i, p, c);
      if (c > 0) {
        lo = min(lo, p);
        hi = max(hi, p + c);
      }
    }
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    if (hi == 0) lo = 0;
    if (hi - lo <= max_rows || part == 1) return;
    part /= 2;
  }
}

// --------------------------------------------------- forward stencils
// MODE 0: S;  MODE 1: dS;  MODE 2: d2S;  MODE 3: the position part of dS^T.
//   dS  (cuda_kernels.py:600-609): phi phi c1 - (phi'_x phi_y dr_x + phi_x phi'_y dr_y) c
//   d2S (cuda_kernels.py:437-450, c1 paired with d1, c2 with d2, as in the reference)
//   MODE 3: acc[b, 0] += sum Re<g, dt1>, acc[b, 1] += sum Re<g, dt2> with
//     dt1 = sum -phi'_y phi_x c, dt2 = sum -phi'_x phi_y c (cuda_kernels.py:744-751)
// Along y the terms gather into one sum per derivative order of phi_y; set q
// of a reduced row is what phi_y's q-th derivative multiplies.
constexpr int stencil_sets(int mode) { return mode == 0 ? 1 : (mode == 2 ? 3 : 2); }
constexpr int stencil_orders(int mode) { return mode == 0 ? 0 : (mode == 2 ? 2 : 1); }

struct StencilRow {
  int i0, first, count;  // floor of the position - 1; the rows inside the grid
  float w[3][4];         // phi_y and its derivatives at the taps
};

template <class T, int MODE>
__global__ void __launch_bounds__(kTileThreads)
k_shift_stencil(T* __restrict__ out, const T* __restrict__ c, const T* __restrict__ c1, const T* __restrict__ c2,
                const float* __restrict__ r, const float* __restrict__ mag, const float* __restrict__ d1,
                const float* __restrict__ d2, const T* __restrict__ g, double* __restrict__ acc, ShiftDims D) {
  constexpr int NS = stencil_sets(MODE), ORD = stencil_orders(MODE);
  constexpr int ROWS = tile_rows(NS);
  __shared__ T rows[ROWS][NS][kTileX];
  __shared__ StencilRow yr[kTileY];
  const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
  const int tx = blockIdx.x * kTileX + lane, ty0 = blockIdx.y * kTileY;
  const long b = blockIdx.z;
  const float m0 = mag[b];
  if (threadIdx.x < kTileY) {
    StencilRow& R = yr[threadIdx.x];
    const float y = spline_x(m0, ty0 + threadIdx.x, D.nz / 2, r[2 * b + 0], D.nzpsi / 2);
    const int iy = (int)fminf(fmaxf(floorf(y), -4.f), (float)D.nzpsi + 4.f);  // beyond the grid: no rows either way
    const float dy = y - floorf(y);
    R.i0 = iy - 1;
    R.first = max(iy - 1, 0);
    R.count = ty0 + (int)threadIdx.x < D.nz ? max(min(iy + 3, D.nzpsi) - R.first, 0) : 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float u = dy - (float)(j - 1);
      R.w[0][j] = bs0(u);
      if (ORD >= 1) R.w[1][j] = bs1(u);
      if (ORD >= 2) R.w[2][j] = bs2(u);
    }
  }
  const float x = spline_x(m0, tx, D.n / 2, r[2 * b + 1], D.npsi / 2);
  const int ix = (int)fminf(fmaxf(floorf(x), -4.f), (float)D.npsi + 4.f);
  const float dx = x - floorf(x);
  float px[3][4];
  bool ok[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float u = dx - (float)(j - 1);
    ok[j] = ix + j - 1 >= 0 && ix + j - 1 < D.npsi && tx < D.n;
    px[0][j] = bs0(u);
    if (ORD >= 1) px[1][j] = bs1(u);
    if (ORD >= 2) px[2][j] = bs2(u);
  }
  float d1x = 0.f, d1y = 0.f, d2x = 0.f, d2y = 0.f;
  if (MODE == 1 || MODE == 2) {
    d1x = d1[2 * b + 1];
    d1y = d1[2 * b + 0];
  }
  if (MODE == 2) {
    d2x = d2[2 * b + 1];
    d2y = d2[2 * b + 0];
  }
  const long off = b * D.npsi * D.nzpsi + ix - 1;
  __syncthreads();
  double s1 = 0.0, s2 = 0.0;
  int part = kTileY;
  for (int y0 = 0; y0 < kTileY && ty0 + y0 < D.nz; y0 += part) {
    int lo, hi;
    tile_part(y0, ROWS, part, lo, hi, [&](int i, int& p, int& n) {
      p = yr[i].first;
      n = yr[i].count;
    });
    // along x: sums of one array with phi_x's derivative of order o
    for (int q = warp; q < hi - lo; q += kTileWarps) {
      const long row = off + (long)(lo + q) * D.npsi;
      auto taps = [&](const T* a, T(&v)[4]) {
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = ok[j] ? __ldg(&a[row + j]) : Ops<T>::zero();
      };
      auto sum = [&](const T(&v)[4], int o) {
        T t = Ops<T>::zero();
#pragma unroll
        for (int j = 0; j < 4; ++j) Ops<T>::fma(t, px[o][j], v[j]);
        return t;
      };
      T v[4];
      taps(c, v);
      T set[3];
      if (MODE == 0) {
        set[0] = sum(v, 0);
      } else if (MODE == 3) {
        set[0] = sum(v, 1);
        set[1] = sum(v, 0);
      } else if (MODE == 1) {
        T v1[4];
        taps(c1, v1);
        set[0] = sum(v1, 0);
        Ops<T>::fma(set[0], -d1x, sum(v, 1));
        set[1] = Ops<T>::zero();
        Ops<T>::fma(set[1], -d1y, sum(v, 0));
      } else {
        T v1[4], v2[4];
        taps(c1, v1);
        taps(c2, v2);
        set[0] = set[1] = set[2] = Ops<T>::zero();
        Ops<T>::fma(set[0], d1x * d2x, sum(v, 2));
        Ops<T>::fma(set[0], -d1x, sum(v1, 1));
        Ops<T>::fma(set[0], -d2x, sum(v2, 1));
        Ops<T>::fma(set[1], d1x * d2y + d1y * d2x, sum(v, 1));
        Ops<T>::fma(set[1], -d1y, sum(v1, 0));
        Ops<T>::fma(set[1], -d2y, sum(v2, 0));
        Ops<T>::fma(set[2], d1y * d2y, sum(v, 0));
      }
#pragma unroll
      for (int k = 0; k < NS; ++k) rows[q][k][lane] = set[k];
    }
    __syncthreads();
    for (int i = y0 + warp; i < y0 + part; i += kTileWarps) {
      const int ty = ty0 + i, q0 = yr[i].i0 - lo, f = yr[i].first - lo, n = yr[i].count;
      T t[NS];
#pragma unroll
      for (int k = 0; k < NS; ++k) t[k] = Ops<T>::zero();
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (q0 + j >= f && q0 + j < f + n)
#pragma unroll
          for (int k = 0; k < NS; ++k) Ops<T>::fma(t[MODE == 3 ? k : 0], yr[i].w[k][j], rows[q0 + j][k][lane]);
      if (tx < D.n && ty < D.nz) {
        const long o = (b * D.nz + ty) * D.n + tx;
        if (MODE == 3) {
          const T gv = g[o];
          s1 -= (double)Ops<T>::redot(gv, t[NS - 1]);
          s2 -= (double)Ops<T>::redot(gv, t[0]);
        } else {
          out[o] = t[0];
        }
      }
    }
    __syncthreads();
  }
  if (MODE != 3) return;
  // block reduction in double
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    s1 += __shfl_down_sync(0xffffffffu, s1, o);
    s2 += __shfl_down_sync(0xffffffffu, s2, o);
  }
  __shared__ double red[2][kTileWarps];
  if (lane == 0) {
    red[0][warp] = s1;
    red[1][warp] = s2;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double t1 = 0, t2 = 0;
    for (int i = 0; i < kTileWarps; ++i) {
      t1 += red[0][i];
      t2 += red[1][i];
    }
    atomicAdd(&acc[2 * b + 0], t1);
    atomicAdd(&acc[2 * b + 1], t2);
  }
}

// ------------------------------------------------ adjoint (gather form)
// out[b, iy, ix] = sum over output pixels (ty, tx) whose footprint holds
// (iy, ix) of phi(dy - (iy - iy(ty))) phi(dx - (ix - ix(tx))) g[b, ty, tx].
__device__ __forceinline__ void cand_range(float m0, float C0, int i, int nhalf, int nmax, int& lo, int& hi) {
  // x(t) = m0 (t - nhalf) + C0 lies in [i-2, i+2).  A (near) zero
  // magnification maps every t to one point: all t are candidates.
  if (!(fabsf(m0) > 1e-3f)) {
    lo = 0;
    hi = nmax - 1;
    return;
  }
  float a = ((float)(i - 2) - C0) / m0 + (float)nhalf;
  float b = ((float)(i + 2) - C0) / m0 + (float)nhalf;
  const float l = fminf(fmaxf(fminf(a, b), -1e7f), 1e7f);
  const float h = fminf(fmaxf(fmaxf(a, b), -1e7f), 1e7f);
  lo = max(0, (int)floorf(l) - 1);
  hi = min(nmax - 1, (int)ceilf(h) + 1);
}

// The pixels whose footprint holds a cell are neighbours, 4 / |m| + 1 at most: up
// to kAdjTaps of them for |m| >= kAdjMag, where the separable tile is used; a
// smaller magnification sums them pixel by pixel.
constexpr int kAdjTaps = 8;
constexpr float kAdjMag = 0.6f;
struct AdjTaps {
  int p0, cnt;
  float w[kAdjTaps];
};
__device__ __forceinline__ AdjTaps adj_taps(int cell, int npix, int ncell, float shift, float m0) {
  AdjTaps t;
  t.p0 = t.cnt = 0;
#pragma unroll
  for (int k = 0; k < kAdjTaps; ++k) t.w[k] = 0.f;
  const float C = -shift + (m0 - 1.0f) / 2.0f + (float)(ncell / 2);
  int p, p1;
  cand_range(m0, C, cell, npix / 2, npix, p, p1);
  for (; p <= p1; ++p) {
    const float x = spline_x(m0, p, npix / 2, shift, ncell / 2);
    const int j = cell - (int)floorf(x);
    if (j < -1 || j > 2) continue;
    if (t.cnt == 0) t.p0 = p;
    const float w = bs0(x - floorf(x) - (float)j);
#pragma unroll
    for (int k = 0; k < kAdjTaps; ++k)
      if (k == p - t.p0) t.w[k] = w;
    t.cnt = min(p - t.p0 + 1, kAdjTaps);
  }
  return t;
}

template <class T>
__global__ void __launch_bounds__(kTileThreads)
k_shift_adj(T* __restrict__ out, const T* __restrict__ g, const float* __restrict__ r, const float* __restrict__ mag,
            ShiftDims D) {
  constexpr int ROWS = 96;
  __shared__ T rows[ROWS][kTileX];
  __shared__ AdjTaps xt[kTileX], yt[kTileY];
  const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
  const int ix = blockIdx.x * kTileX + lane, iy0 = blockIdx.y * kTileY;
  const long b = blockIdx.z;
  const float m0 = mag[b];
  const float rx = r[2 * b + 1], ry = r[2 * b + 0];
  const T* gb = g + b * D.nz * D.n;
  T* ob = out + b * D.nzpsi * D.npsi + ix;
  if (!(fabsf(m0) >= kAdjMag)) {
    if (ix >= D.npsi) return;
    const float half = (m0 - 1.0f) / 2.0f;
    int tx0, tx1, ty0, ty1;
    cand_range(m0, -rx + half + (float)(D.npsi / 2), ix, D.n / 2, D.n, tx0, tx1);
    for (int iy = iy0 + warp; iy < min(iy0 + kTileY, D.nzpsi); iy += kTileWarps) {
      cand_range(m0, -ry + half + (float)(D.nzpsi / 2), iy, D.nz / 2, D.nz, ty0, ty1);
      T acc = Ops<T>::zero();
      for (int ty = ty0; ty <= ty1; ++ty) {
        const float y = spline_x(m0, ty, D.nz / 2, ry, D.nzpsi / 2);
        const int jy = iy - (int)floorf(y);
        if (jy < -1 || jy > 2) continue;
        const float wy = bs0(y - floorf(y) - (float)jy);
        T racc = Ops<T>::zero();
        for (int tx = tx0; tx <= tx1; ++tx) {
          const float x = spline_x(m0, tx, D.n / 2, rx, D.npsi / 2);
          const int jx = ix - (int)floorf(x);
          if (jx < -1 || jx > 2) continue;
          Ops<T>::fma(racc, bs0(x - floorf(x) - (float)jx), __ldg(&gb[(long)ty * D.n + tx]));
        }
        Ops<T>::fma(acc, wy, racc);
      }
      ob[(long)iy * D.npsi] = acc;
    }
    return;
  }
  AdjTaps none;
  none.p0 = none.cnt = 0;
  if (threadIdx.x < kTileX)
    xt[lane] = ix < D.npsi ? adj_taps(ix, D.n, D.npsi, rx, m0) : none;
  else if (threadIdx.x < kTileX + kTileY) {
    const int i = threadIdx.x - kTileX;
    yt[i] = iy0 + i < D.nzpsi ? adj_taps(iy0 + i, D.nz, D.nzpsi, ry, m0) : none;
  }
  __syncthreads();
  const AdjTaps t = xt[lane];
  int part = kTileY;
  for (int c0 = 0; c0 < kTileY && iy0 + c0 < D.nzpsi; c0 += part) {
    int lo, hi;
    tile_part(c0, ROWS, part, lo, hi, [&](int i, int& p, int& n) {
      p = yt[i].p0;
      n = yt[i].cnt;
    });
    for (int q = warp; q < hi - lo; q += kTileWarps) {
      const T* grow = gb + (long)(lo + q) * D.n + t.p0;
      T sum = Ops<T>::zero();
#pragma unroll
      for (int k = 0; k < kAdjTaps; ++k)
        if (k < t.cnt) Ops<T>::fma(sum, t.w[k], __ldg(&grow[k]));
      rows[q][lane] = sum;
    }
    __syncthreads();
    for (int i = c0 + warp; i < c0 + part; i += kTileWarps) {
      const int p = yt[i].p0 - lo, n = yt[i].cnt;
      T acc = Ops<T>::zero();
#pragma unroll
      for (int k = 0; k < kAdjTaps; ++k)
        if (k < n) Ops<T>::fma(acc, yt[i].w[k], rows[p + k][lane]);
      if (ix < D.npsi && iy0 + i < D.nzpsi) ob[(long)(iy0 + i) * D.npsi] = acc;
    }
    __syncthreads();
  }
}

// ------------------------------------------- back-projection shift
// Sback (shift.py:138-148; cuda_kernels.py:294-370, dir = 1): the detector
// image g is spread onto the coefficient grid with the B-spline stretched by
// the image's magnification m.  Pixel (tx, ty) sits at
// x = (m (tx - n/2) - r_x + (m - 1)/2) + npsi/2 (y likewise), ix = floor(x),
// dx = x - ix, and reaches the cells ix + jx for jx in [ceil(dx - 2m),
// (int)(dx + 2m)) with weight phi((dx - jx) / m) (and the same in y; the upper
// bound drops the last tap of non-zero weight when dx + 2m is not an integer,
// as the reference has it).
//
// Here the transpose is a gather: every coefficient cell sums the pixels whose tap
// windows contain it, found around the cell's preimage and tested with the exact
// membership rule above, in a fixed order (rows, then pixels within a row), so the
// result does not depend on scheduling and every cell is written once (no clearing
// pass, no atomics).
__device__ __forceinline__ float sback_phi(float t, float m) {
  t /= m;
  const float a = fabsf(t);
  if (t > -2.f && t <= -1.f) return (t + 2.f) * (t + 2.f) * (t + 2.f);
  if (t > -1.f && t <= 1.f) return 4.f - 6.f * t * t + 3.f * a * t * t;
  if (t > 1.f && t <= 2.f) return (2.f - t) * (2.f - t) * (2.f - t);
  return 0.f;
}

// Pixel p's position on the coefficient axis (the reference's float
// arithmetic) and whether its window reaches cell `cell`; *w is the tap weight.
__device__ __forceinline__ bool sback_tap(int p, int npix, int ncell, float shift, float m0, int cell, float* w) {
  const float half = (m0 - 1.0f) / 2.0f;
  const float x = (m0 * (float)(p - npix / 2) - shift + half) + (float)(ncell / 2);
  const int ix = (int)floorf(x);
  const float dx = x - (float)ix;
  const float span = 2.0f * m0;
  const int j = cell - ix;
  if (j < (int)ceilf(dx - span) || j >= (int)(dx + span)) return false;
  *w = sback_phi(dx - (float)j, m0);
  return true;
}

// The pixels whose windows can reach `cell`: sback_tap admits pixel p only
// when its position x(p) lies in (cell - 2m, cell + 2m], so p lies within
// (cell -+ 2m - c) / m + npix / 2; the range is widened by 0.01 cell units
// (far above the float rounding of x) and one pixel on each side, and
// membership is still decided by sback_tap.
__device__ __forceinline__ void sback_range(int cell, int npix, int ncell, float shift, float m0, int* p0, int* p1) {
  const float c = -shift + (m0 - 1.0f) / 2.0f + (float)(ncell / 2);
  const float lo = ((float)cell - 2.0f * m0 - 0.01f - c) / m0 + (float)(npix / 2);
  const float hi = ((float)cell + 2.0f * m0 + 0.01f - c) / m0 + (float)(npix / 2);
  *p0 = max(0, (int)floorf(fmaxf(lo, -1.0f)) - 1);
  *p1 = min(npix - 1, (int)ceilf(fminf(hi, (float)npix)) + 1);
}

// A cell line's taps.  sback_tap admits the pixels at x in [cell + 1 - 2m,
// cell + 2m], m apart: at most four neighbours (six leaves room for rounding).
constexpr int kSbackTaps = 6;
struct SbackTaps {
  int p0, cnt;  // first pixel, number of pixels
  float w[kSbackTaps];
};
__device__ __forceinline__ SbackTaps sback_taps(int cell, int npix, int ncell, float shift, float m0) {
  SbackTaps t;
  t.p0 = t.cnt = 0;
#pragma unroll
  for (int k = 0; k < kSbackTaps; ++k) t.w[k] = 0.f;
  int p, p1;
  sback_range(cell, npix, ncell, shift, m0, &p, &p1);
  for (; p <= p1; ++p) {
    float w;
    if (!sback_tap(p, npix, ncell, shift, m0, cell, &w)) continue;
    if (t.cnt == 0) t.p0 = p;
#pragma unroll
    for (int k = 0; k < kSbackTaps; ++k)
      if (k == p - t.p0) t.w[k] = w;
    t.cnt = min(p - t.p0 + 1, kSbackTaps);
  }
  return t;
}

// A CTA covers kSbackCX x kSbackCY cells of one image.  The taps are separable:
// the CTA first sums each pixel row its cells reach along x (a lane per cell
// column, its x taps in registers) into shared memory, then each cell sums its
// y taps over those rows -- about 5 + 4 taps a cell at m = 0.8 instead of 4 x 4,
// in the order of the double sum (rows, then pixels within a row).  The rows
// of the tile's cells fit the buffer down to m = 0.75; a smaller m takes the
// tile in parts.  128 images of 512^2 at m = 0.8: 0.85 ms when every cell
// tested a 16 x 16 candidate mask.
constexpr int kSbackCX = 32, kSbackCY = 64, kSbackThreads = 256;
constexpr int kSbackRows = 96;

__global__ void __launch_bounds__(kSbackThreads)
k_sback(const float2* __restrict__ g, float2* __restrict__ f, const float* __restrict__ r,
        const float* __restrict__ mag, int nmag, ShiftDims S) {
  __shared__ float2 rows[kSbackRows][kSbackCX];
  __shared__ SbackTaps xt[kSbackCX], yt[kSbackCY];
  const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
  constexpr int WARPS = kSbackThreads / 32;
  const int xx = blockIdx.x * kSbackCX + lane, y0 = blockIdx.y * kSbackCY;
  const long b = blockIdx.z;
  const float m0 = mag[nmag == 1 ? 0 : b];
  const float ry = r[2 * b + 0], rx = r[2 * b + 1];
  // m <= 0: the reference's tap ranges are empty
  SbackTaps none;
  none.p0 = none.cnt = 0;
  if (threadIdx.x < kSbackCX)
    xt[lane] = (m0 > 0.f && xx < S.npsi) ? sback_taps(xx, S.n, S.npsi, rx, m0) : none;
  else if (threadIdx.x < kSbackCX + kSbackCY) {
    const int i = threadIdx.x - kSbackCX;
    yt[i] = (m0 > 0.f && y0 + i < S.nzpsi) ? sback_taps(y0 + i, S.nz, S.nzpsi, ry, m0) : none;
  }
  __syncthreads();
  const SbackTaps tx = xt[lane];
  const float2* gb = g + b * (long)S.nz * S.n + tx.p0;
  float2* fb = f + b * (long)S.nzpsi * S.npsi + xx;
  int part = kSbackCY;
  for (int c0 = 0; c0 < kSbackCY && y0 + c0 < S.nzpsi; c0 += part) {
    int lo, hi;
    tile_part(c0, kSbackRows, part, lo, hi, [&](int i, int& p, int& n) {
      p = yt[i].p0;
      n = yt[i].cnt;
    });
    for (int q = warp; q < hi - lo; q += WARPS) {
      const float2* grow = gb + (long)(lo + q) * S.n;
      float2 sum = make_float2(0.f, 0.f);
#pragma unroll
      for (int k = 0; k < kSbackTaps; ++k)
        if (k < tx.cnt) {
          const float2 v = __ldg(&grow[k]);
          sum.x += tx.w[k] * v.x;
          sum.y += tx.w[k] * v.y;
        }
      rows[q][lane] = sum;
    }
    __syncthreads();
    for (int i = warp; i < part; i += WARPS) {
      const int yy = y0 + c0 + i;
      const int p = yt[c0 + i].p0 - lo, c = yt[c0 + i].cnt;
      float2 acc = make_float2(0.f, 0.f);
#pragma unroll
      for (int k = 0; k < kSbackTaps; ++k)
        if (k < c) {
          const float w = yt[c0 + i].w[k];
          const float2 v = rows[p + k][lane];
          acc.x += w * v.x;
          acc.y += w * v.y;
        }
      if (xx < S.npsi && yy < S.nzpsi) fb[(long)yy * S.npsi] = acc;
    }
    __syncthreads();
  }
}

// ------------------------------------------------- cubic B-spline prefilter
// Along one axis the filter solves b c[k-1] + 4 c[k] + b c[k+1] = s[k] on the
// periodic line (b = 1; smaller for the spline of a magnification below 1).
// With q = 1 / (2 + sqrt(4 - b^2)) and the pole p = -b q, 1 / (b z + 4 + b/z) =
// q / ((1 - p/z)(1 - p z)): a causal recursion u[k] = s[k] + p u[k-1] and an
// anticausal one c[k] = q u[k] + p c[k+1] (Unser, Aldroubi and Eden 1993).  A
// recursion forgets its start as p^k (|p| <= 2 - sqrt(3)), so a strip of the line
// started kBsWarm samples early (p^16 = 7e-10, far below half an ulp) is the
// periodic filter: the strips run in parallel, with 3.5 multiply-adds a sample
// instead of two FFTs, and the pass is bound by memory.
struct BsPole {
  float p, q;
};
static BsPole bs_pole(double b) {
  const double q = 1.0 / (2.0 + std::sqrt(4.0 - b * b));
  return {(float)(-b * q), (float)q};
}
constexpr int kBsWarm = 16, kBsStrip = 32;
template <class T>
constexpr int bs2d_strip() { return sizeof(T) == 8 ? 16 : 32; }  // see k_bspline2d

// a + w v
__device__ __forceinline__ float2 bs_fma(float w, float2 v, float2 a) {
  return make_float2(fmaf(w, v.x, a.x), fmaf(w, v.y, a.y));
}
__device__ __forceinline__ float bs_fma(float w, float v, float a) { return fmaf(w, v, a); }
__device__ __forceinline__ float2 bs_mul(float w, float2 v) { return make_float2(w * v.x, w * v.y); }
__device__ __forceinline__ float bs_mul(float w, float v) { return w * v; }

// One strip of L: samples ld(0 .. L + 2 kBsWarm - 1) from kBsWarm before its first
// one; the coefficients are left in u[0 .. L - 1].
template <int L, class T, class LD>
__device__ __forceinline__ void bspline_strip(T (&u)[L + kBsWarm], const BsPole P, LD ld) {
  T c = Ops<T>::zero();
#pragma unroll
  for (int i = 0; i < kBsWarm; ++i) c = bs_fma(P.p, c, ld(i));
#pragma unroll
  for (int i = 0; i < L + kBsWarm; ++i) u[i] = c = bs_fma(P.p, c, ld(i + kBsWarm));
  c = Ops<T>::zero();
#pragma unroll
  for (int i = L + kBsWarm - 1; i >= 0; --i) {
    c = bs_fma(P.p, c, bs_mul(P.q, u[i]));
    u[i] = c;
  }
}

__device__ __forceinline__ int wrap_index(int i, int n) {
  i %= n;
  return i < 0 ? i + n : i;
}

// Both axes in one pass, psi != out: a CTA filters a kBsTile x kBsTile tile with
// its warm-up margin in shared memory, first along x (a thread per row and
// strip), then along y (a thread per column and strip) into global memory.  The
// margins of neighbouring tiles come from L2.  Strips of 16 for complex images
// (384 threads, three CTAs an SM: 90 images of 512^2 in 0.15 ms against 0.18 with
// strips of 32, 0.3 with the FFT passes), of 32 for real ones (0.07 ms; 0.43 with
// the FFT passes on complex copies).
constexpr int kBsTile = 64, kBsSpan = kBsTile + 2 * kBsWarm;
template <class T>
constexpr int bs2d_threads() { return kBsSpan * (kBsTile / bs2d_strip<T>()); }

template <class T>
__global__ void __launch_bounds__(bs2d_threads<T>(), 3)
k_bspline2d(const T* __restrict__ in, T* __restrict__ out, int ny, int nx, int tx, int ty, BsPole P) {
  constexpr int L = bs2d_strip<T>(), THREADS = bs2d_threads<T>();
  extern __shared__ float2 smem[];
  T(*tile)[kBsSpan + 1] = reinterpret_cast<T(*)[kBsSpan + 1]>(smem);
  const long img = blockIdx.x / (tx * ty);
  const int bt = (int)(blockIdx.x % (tx * ty));
  const int x0 = (bt % tx) * kBsTile, y0 = (bt / tx) * kBsTile;
  const T* src = in + img * ny * nx;
  {
    constexpr int WARPS = THREADS / 32, CPL = kBsSpan / 32;
    const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
    int col[CPL];
#pragma unroll
    for (int j = 0; j < CPL; ++j) col[j] = wrap_index(x0 - kBsWarm + lane + 32 * j, nx);
#pragma unroll 4
    for (int i = warp; i < kBsSpan; i += WARPS) {
      const T* row = src + (long)wrap_index(y0 - kBsWarm + i, ny) * nx;
#pragma unroll
      for (int j = 0; j < CPL; ++j) tile[i][lane + 32 * j] = __ldg(&row[col[j]]);
    }
  }
  __syncthreads();
  T u[L + kBsWarm];
  {
    const int i = threadIdx.x % kBsSpan, c0 = (threadIdx.x / kBsSpan) * L;
    bspline_strip<L, T>(u, P, [&](int k) { return tile[i][c0 + k]; });
    __syncthreads();
#pragma unroll
    for (int k = 0; k < L; ++k) tile[i][kBsWarm + c0 + k] = u[k];
  }
  __syncthreads();
  if (threadIdx.x >= kBsTile * (kBsTile / L)) return;
  const int j = threadIdx.x % kBsTile, r0 = (threadIdx.x / kBsTile) * L;
  bspline_strip<L, T>(u, P, [&](int k) { return tile[r0 + k][kBsWarm + j]; });
  if (x0 + j >= nx) return;
  T* dst = out + (img * ny + y0 + r0) * nx + x0 + j;
#pragma unroll
  for (int k = 0; k < L; ++k)
    if (y0 + r0 + k < ny) dst[(long)k * nx] = u[k];
}

// Along the rows' axis only, [n, ncols], in place or not: a CTA holds whole
// columns (threads of one strip across blockDim.x columns, blockDim.y strips),
// every load before the first store.  The neighbouring strips' margins come
// from L1.
template <class T>
__global__ void __launch_bounds__(512)
k_bspline_cols(const T* in, T* out, int n, long ncols, BsPole P) {
  const long col = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const bool valid = col < ncols;
  const int k0 = threadIdx.y * kBsStrip;
  const T* src = in + (valid ? col : 0);
  int r = wrap_index(k0 - kBsWarm, n);
  T u[kBsStrip + kBsWarm];
  bspline_strip<kBsStrip, T>(u, P, [&](int) {
    const T v = src[(long)r * ncols];
    r = r + 1 == n ? 0 : r + 1;
    return v;
  });
  __syncthreads();
  if (!valid) return;
#pragma unroll
  for (int k = 0; k < kBsStrip; ++k)
    if (k0 + k < n) out[(long)(k0 + k) * ncols + col] = u[k];
}

// The spline at the grid points, out = B c with B = (1, 4, 1) along both axes,
// periodic: the prefilter's inverse.  A warp takes 32 columns of kSplineRows rows,
// each row's sum along x formed once.
constexpr int kSplineRows = 16, kSplineWarps = 8;
__global__ void __launch_bounds__(32 * kSplineWarps)
k_bspline_grid(const float2* __restrict__ c, float2* __restrict__ out, int ny, int nx) {
  const int x = blockIdx.x * 32 + threadIdx.x, y0 = (blockIdx.y * kSplineWarps + threadIdx.y) * kSplineRows;
  if (x >= nx || y0 >= ny) return;
  const float2* src = c + (long)blockIdx.z * ny * nx;
  float2* dst = out + (long)blockIdx.z * ny * nx + x;
  const int xm = x == 0 ? nx - 1 : x - 1, xp = x + 1 == nx ? 0 : x + 1;
  auto row = [&](int y) {
    const float2* r = src + (long)y * nx;
    const float2 a = __ldg(&r[xm]), b = __ldg(&r[x]), d = __ldg(&r[xp]);
    return make_float2((a.x + d.x) + 4.f * b.x, (a.y + d.y) + 4.f * b.y);
  };
  float2 p = row(y0 == 0 ? ny - 1 : y0 - 1), q = row(y0);
#pragma unroll 4
  for (int y = y0; y < min(y0 + kSplineRows, ny); ++y) {
    const float2 n = row(y + 1 == ny ? 0 : y + 1);
    dst[(long)y * nx] = make_float2((p.x + n.x) + 4.f * q.x, (p.y + n.y) + 4.f * q.y);
    p = q;
    q = n;
  }
}

template <class T>
static cudaError_t bspline2d(const T* in, T* out, long batch, int ny, int nx, double b, cudaStream_t st) {
  constexpr int smem = kBsSpan * (kBsSpan + 1) * (int)sizeof(T);
  const cudaError_t e = allow_smem(k_bspline2d<T>, smem);
  if (e != cudaSuccess) return e;
  const int tx = (nx + kBsTile - 1) / kBsTile, ty = (ny + kBsTile - 1) / kBsTile;
  k_bspline2d<T><<<(unsigned)(batch * tx * ty), bs2d_threads<T>(), smem, st>>>(in, out, ny, nx, tx, ty, bs_pole(b));
  count_launch();
  return cudaGetLastError();
}

template <class T>
static cudaError_t bspline_cols(const T* in, T* out, int n, long ncols, cudaStream_t st) {
  // strips of 32 rows up to 4096 rows; columns a block: 32 (whole 256-byte lines) up to 256 rows, then as
  // many as 256 threads take (16 at 512 rows, 8 at 1024), at least 4 (32-byte sectors; 512 threads at 4096)
  const int strips = (n + kBsStrip - 1) / kBsStrip;
  const int cw = strips <= 8 ? 32 : (strips <= 16 ? 16 : (strips <= 32 ? 8 : 4));
  k_bspline_cols<T><<<(unsigned)((ncols + cw - 1) / cw), dim3(cw, strips), 0, st>>>(in, out, n, ncols, bs_pole(1.0));
  count_launch();
  return cudaGetLastError();
}

// -------------------------------------------------- prefilter passes
// data [nrows, N] in place: FFT, * sym[k], IFFT (sym carries 1/N)
template <int N>
__global__ void __launch_bounds__(RowCfg<N>::THREADS)
k_symbol_rows(const float2* in, float2* out, long nrows, const float* __restrict__ sym,
              const float2* __restrict__ tw4) {
  constexpr int T = RowCfg<N>::T;
  extern __shared__ float2 smem[];
  const int line = threadIdx.x / T, t = threadIdx.x % T;
  const long row = (long)blockIdx.x * RowCfg<N>::LINES + line;
  const bool valid = row < nrows;
  SmRow sm{smem + line * SmRow::padded(N)};
  for (int k = t; k < N; k += T) sm.st(k, valid ? in[row * N + k] : make_float2(0.f, 0.f));
  __syncthreads();
  fft_line<N, false>(sm, t, tw4, line_sync<T>());
  for (int k = t; k < N; k += T) sm.st(k, cscale(sm.ld(k), __ldg(&sym[k])));
  __syncthreads();
  fft_line<N, true>(sm, t, tw4, line_sync<T>());
  if (!valid) return;
  for (int k = t; k < N; k += T) out[row * N + k] = sm.ld(k);
}

// data [nimg, N, ncols] in place along the column axis.  The forward FFT's
// first stage loads the block's C columns from global memory and the inverse
// FFT's last stage stores them back (a warp covers 32 / C rows of C adjacent
// columns per access); the tile passes shared memory only between stages.
template <int N>
__global__ void __launch_bounds__(ColCfg<N>::THREADS, ColCfg<N>::MIN_BLOCKS)
k_symbol_cols(const float2* in, float2* out, int ncols, const float* __restrict__ sym,
              const float2* __restrict__ tw4) {
  constexpr int C = ColCfg<N>::C;
  constexpr int T = ColCfg<N>::T;
  extern __shared__ float2 tile[];
  const int c = threadIdx.x % C, t = threadIdx.x / C;
  const bool valid = blockIdx.x * C + c < ncols;
  const int col = min((int)blockIdx.x * C + c, ncols - 1);
  const long off = (long)blockIdx.y * N * ncols + col;
  SmCol<C> sm{tile + c};
  fft_line_from<N, false, typename ColCfg<N>::PL>(GColIn{in + off, ncols, valid}, sm, t, tw4);
  for (int k = t; k < N; k += T) sm.st(k, cscale(sm.ld(k), __ldg(&sym[k])));
  __syncthreads();
  fft_line_to<N, true, typename ColCfg<N>::PL>(sm, GColOut{out + off, ncols, valid}, t, tw4);
}

// The column pass at 512 rows: one 32-thread group per column, 16 samples a
// thread, radices 8-8-8.  Thread t holds butterflies t and t + 32 of the
// forward FFT's last stage (P = 64), i.e. samples b + 64 j, which are also
// the samples of the inverse FFT's first stage (P = 1) on the same
// butterflies: the symbol multiplies them in registers and the spectrum makes
// no round trip through shared memory between the two transforms.  The same
// butterflies as k_symbol_cols; the results agree to an ulp (the compiler
// may fuse a complex product's multiply-adds differently in the two).  For the
// prefilter in place and for magnifications above 1: 128 images of 512^2 take 432 us,
// 471 with k_symbol_cols.
constexpr int kSym512C = 8, kSym512Threads = 32 * kSym512C;

__global__ void __launch_bounds__(kSym512Threads)
k_symbol_cols512(const float2* in, float2* out, int ncols, const float* __restrict__ sym,
                 const float2* __restrict__ tw4) {
  constexpr int N = 512, E = 16, C = kSym512C;
  extern __shared__ float2 tile[];
  const int c = threadIdx.x % C, t = threadIdx.x / C;
  const bool valid = blockIdx.x * C + c < ncols;
  const int col = min((int)blockIdx.x * C + c, ncols - 1);
  const long off = (long)blockIdx.y * N * ncols + col;
  SmCol<C> sm{tile + c};
  const CtaSync sync{};
  float2 v[E];
  // forward FFT: stage 1 (from global memory) and stage 2
  fft_stage<N, E, 8, 1, false, false, true>(v, SplitView<GColIn, SmCol<C>>{GColIn{in + off, ncols, valid}, sm}, t,
                                            tw4, sync);
  fft_stage<N, E, 8, 8, false, true, true>(v, sm, t, tw4, sync);
  // stage 3 (P = 64) kept in registers: v[8 s + j] = X[b_s + 64 j], b_s = t + 32 s; times the symbol
#pragma unroll
  for (int s2 = 0; s2 < 2; ++s2) {
    const int b = t + 32 * s2;
#pragma unroll
    for (int j = 0; j < 8; ++j) v[8 * s2 + j] = sm.ld(b + 64 * j);
    float2 w[8];
    twiddles<8, false>(tw4, b, N, w);
#pragma unroll
    for (int j = 1; j < 8; ++j) v[8 * s2 + j] = cmul(v[8 * s2 + j], w[j]);
    Dft<8, false>::run(&v[8 * s2]);
#pragma unroll
    for (int j = 0; j < 8; ++j) v[8 * s2 + j] = cscale(v[8 * s2 + j], __ldg(&sym[b + 64 * j]));
  }
  sync();  // every stage-3 load is done before the stores below
  // inverse FFT: stage 1 (P = 1) on the same butterflies, then stages 2 and 3 (to global memory)
#pragma unroll
  for (int s2 = 0; s2 < 2; ++s2) {
    const int b = t + 32 * s2;
    Dft<8, true>::run(&v[8 * s2]);
#pragma unroll
    for (int j = 0; j < 8; ++j) sm.st(b * 8 + j, v[8 * s2 + j]);
  }
  sync();
  fft_stage<N, E, 8, 8, true, true, true>(v, sm, t, tw4, sync);
  fft_stage<N, E, 8, 64, true, false, false>(v, SplitView<SmCol<C>, GColOut>{sm, GColOut{out + off, ncols, valid}},
                                             t, tw4, sync);
}

template <int N>
static cudaError_t l_symbol_rows(const float2* in, float2* out, long nrows, const float* sym, const float2* tw,
                                 cudaStream_t st) {
  using CF = RowCfg<N>;
  cudaError_t e = allow_smem(k_symbol_rows<N>, CF::SMEM);
  if (e != cudaSuccess) return e;
  k_symbol_rows<N><<<(unsigned)((nrows + CF::LINES - 1) / CF::LINES), CF::THREADS, CF::SMEM, st>>>(in, out, nrows,
                                                                                                 sym, tw); ::ht::count_launch();
  return cudaGetLastError();
}

template <int N>
static cudaError_t l_symbol_cols(const float2* in, float2* out, long nimg, int ncols, const float* sym,
                                 const float2* tw, cudaStream_t st) {
  if constexpr (N == 512) {
    constexpr int smem = N * kSym512C * (int)sizeof(float2);
    k_symbol_cols512<<<dim3((ncols + kSym512C - 1) / kSym512C, (unsigned)nimg), kSym512Threads, smem, st>>>(
        in, out, ncols, sym, tw);
    ::ht::count_launch();
    return cudaGetLastError();
  }
  using CF = ColCfg<N>;
  cudaError_t e = allow_smem(k_symbol_cols<N>, CF::SMEM);
  if (e != cudaSuccess) return e;
  k_symbol_cols<N><<<dim3((ncols + CF::C - 1) / CF::C, (unsigned)nimg), CF::THREADS, CF::SMEM, st>>>(in, out, ncols,
                                                                                                   sym, tw);
  ::ht::count_launch();
  return cudaGetLastError();
}

cudaError_t symbol_rows(int N, const float2* in, float2* out, long nrows, const float* sym, const float2* tw,
                        cudaStream_t st) {
  switch (N) {
#define X(S) \
  case S:    \
    return l_symbol_rows<S>(in, out, nrows, sym, tw, st);
    HT_SIZE_CASES(X)
#undef X
    default:
      return cudaErrorInvalidValue;
  }
}

cudaError_t symbol_cols(int N, const float2* in, float2* out, long nimg, int ncols, const float* sym,
                        const float2* tw, cudaStream_t st) {
  switch (N) {
#define X(S) \
  case S:    \
    return l_symbol_cols<S>(in, out, nimg, ncols, sym, tw, st);
    HT_SIZE_CASES(X)
#undef X
    default:
      return cudaErrorInvalidValue;
  }
}

}  // namespace ht

// ================================================================= C ABI
struct ht_shift_s {
  int n, npsi, nz, nzpsi, is_complex, device;
  float* symx;  // [npsi]  1 / (npsi (4 + 2 cos 2 pi k / npsi))
  float* symy;  // [nzpsi]
  const float2* tw_x;
  const float2* tw_y;
};

extern "C" int ht_shift_create(int n, int npsi, int nz, int nzpsi, int is_complex, ht_shift_s** out) {
  using namespace ht;
  HT_REQUIRE(out != nullptr, "ht_shift_create: null pointer");
  HT_REQUIRE(n > 0 && npsi > 0 && nz > 0 && nzpsi > 0, "ht_shift_create: sizes must be positive");
  ht_shift_s* s = new ht_shift_s{n, npsi, nz, nzpsi, is_complex ? 1 : 0, 0, nullptr, nullptr, nullptr, nullptr};
  cudaGetDevice(&s->device);
  const bool fft_ok = fft_size_supported(npsi) && fft_size_supported(nzpsi);
  if (fft_ok) {
    s->tw_x = twiddle_table(npsi, s->device);
    s->tw_y = twiddle_table(nzpsi, s->device);
  }
  std::vector<float> hx(npsi), hy(nzpsi);
  for (int k = 0; k < npsi; ++k) hx[k] = (float)(1.0 / (npsi * (4.0 + 2.0 * std::cos(2.0 * M_PI * k / npsi))));
  for (int k = 0; k < nzpsi; ++k) hy[k] = (float)(1.0 / (nzpsi * (4.0 + 2.0 * std::cos(2.0 * M_PI * k / nzpsi))));
  cudaError_t e = cudaMalloc(&s->symx, sizeof(float) * npsi);
  if (e == cudaSuccess) e = cudaMalloc(&s->symy, sizeof(float) * nzpsi);
  if (e == cudaSuccess) e = cudaMemcpy(s->symx, hx.data(), sizeof(float) * npsi, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(s->symy, hy.data(), sizeof(float) * nzpsi, cudaMemcpyHostToDevice);
  if (e != cudaSuccess || (fft_ok && (!s->tw_x || !s->tw_y))) {
    if (e != cudaSuccess) set_error(std::string("ht_shift_create: ") + cudaGetErrorString(e));
    cudaFree(s->symx);
    cudaFree(s->symy);
    delete s;
    return kCudaError;
  }
  *out = s;
  return kOk;
}

extern "C" int ht_shift_destroy(ht_shift_s* s) {
  if (!s) return ht::kOk;
  cudaFree(s->symx);
  cudaFree(s->symy);
  delete s;
  return ht::kOk;
}

namespace {
ht::ShiftDims dims(const ht_shift_s* s) { return ht::ShiftDims{s->n, s->npsi, s->nz, s->nzpsi}; }
dim3 out_grid(const ht_shift_s* s, long batch) {
  return dim3((s->n + ht::kTileX - 1) / ht::kTileX, (s->nz + ht::kTileY - 1) / ht::kTileY, (unsigned)batch);
}
dim3 coef_grid(const ht_shift_s* s, long batch) {
  return dim3((s->npsi + ht::kTileX - 1) / ht::kTileX, (s->nzpsi + ht::kTileY - 1) / ht::kTileY, (unsigned)batch);
}
const int kBlock = ht::kTileThreads;
}  // namespace

namespace {
bool prefilter_sizes_ok(const ht_shift_s* s, const char* name) {
  if (ht::fft_size_supported(s->npsi) && ht::fft_size_supported(s->nzpsi)) return true;
  ht::set_error(std::string(name) + ": npsi and nzpsi must be supported FFT lengths");
  return false;
}
}  // namespace

extern "C" int ht_shift_coeff(ht_shift_s* s, const void* psi, void* out, long batch, void* stream) {
  using namespace ht;
  HT_REQUIRE(s && psi && out, "ht_shift_coeff: null pointer");
  HT_REQUIRE(s->is_complex, "ht_shift_coeff: works on complex64 data (pass real data as complex)");
  if (!prefilter_sizes_ok(s, "ht_shift_coeff")) return kUnsupported;
  if (batch == 0) return kOk;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const float2* src = static_cast<const float2*>(psi);
  float2* dst = static_cast<float2*>(out);
  const long total = batch * s->nzpsi * s->npsi;
  if (src + total <= dst || dst + total <= src) {
    HT_CHECK_CUDA(bspline2d<float2>(src, dst, batch, s->nzpsi, s->npsi, 1.0, st));
    return kOk;
  }
  // in place: line by line (the tiles of the one-pass kernel read their neighbours)
  HT_CHECK_CUDA(symbol_rows(s->npsi, src, dst, batch * s->nzpsi, s->symx, s->tw_x, st));
  HT_CHECK_CUDA(symbol_cols(s->nzpsi, dst, dst, batch, s->npsi, s->symy, s->tw_y, st));
  return kOk;
}

extern "C" int ht_shift_coeff_real(ht_shift_s* s, const float* psi, float* out, long batch, void* stream) {
  using namespace ht;
  HT_REQUIRE(s && psi && out, "ht_shift_coeff_real: null pointer");
  HT_REQUIRE(batch >= 0, "ht_shift_coeff_real: batch must be non-negative");
  if (!prefilter_sizes_ok(s, "ht_shift_coeff_real")) return kUnsupported;
  if (batch == 0) return kOk;
  const long total = batch * s->nzpsi * s->npsi;
  HT_REQUIRE(psi + total <= out || out + total <= psi, "ht_shift_coeff_real: psi and out must not overlap");
  HT_CHECK_CUDA(bspline2d<float>(psi, out, batch, s->nzpsi, s->npsi, 1.0, static_cast<cudaStream_t>(stream)));
  return kOk;
}

extern "C" int ht_shift_coeffback(ht_shift_s* s, const void* psi, void* out, long batch, float b, void* stream) {
  using namespace ht;
  HT_REQUIRE(s && psi && out, "ht_shift_coeffback: null pointer");
  HT_REQUIRE(batch >= 0, "ht_shift_coeffback: batch must be non-negative");
  HT_REQUIRE(b >= 0.f && b <= 1.f, "ht_shift_coeffback: b must be in [0, 1]");
  if (!prefilter_sizes_ok(s, "ht_shift_coeffback")) return kUnsupported;
  if (batch == 0) return kOk;
  const float2* src = static_cast<const float2*>(psi);
  float2* dst = static_cast<float2*>(out);
  const long total = batch * s->nzpsi * s->npsi;
  HT_REQUIRE(src + total <= dst || dst + total <= src, "ht_shift_coeffback: psi and out must not overlap");
  HT_CHECK_CUDA(bspline2d<float2>(src, dst, batch, s->nzpsi, s->npsi, b, static_cast<cudaStream_t>(stream)));
  return kOk;
}

extern "C" int ht_shift_coeff_z(ht_shift_s* s, const void* in, void* out, long ncols, void* stream) {
  using namespace ht;
  HT_REQUIRE(s && in && out, "ht_shift_coeff_z: null pointer");
  HT_REQUIRE(ncols >= 0, "ht_shift_coeff_z: ncols must be non-negative");
  if (!fft_size_supported(s->nzpsi)) {
    set_error("ht_shift_coeff_z: nzpsi must be a supported FFT length");
    return kUnsupported;
  }
  if (ncols == 0) return kOk;
  HT_REQUIRE(ncols <= 0x7fffffffL, "ht_shift_coeff_z: ncols too large");
  HT_CHECK_CUDA(bspline_cols<float2>(static_cast<const float2*>(in), static_cast<float2*>(out), s->nzpsi, ncols,
                                     static_cast<cudaStream_t>(stream)));
  return kOk;
}

extern "C" int ht_shift_spline(ht_shift_s* s, const void* c, void* out, long batch, void* stream) {
  using namespace ht;
  HT_REQUIRE(s && c && out, "ht_shift_spline: null pointer");
  HT_REQUIRE(batch >= 0, "ht_shift_spline: batch must be non-negative");
  const long img = (long)s->nzpsi * s->npsi;
  const float2* src = static_cast<const float2*>(c);
  float2* dst = static_cast<float2*>(out);
  HT_REQUIRE(src + batch * img <= dst || dst + batch * img <= src, "ht_shift_spline: c and out must not overlap");
  const int rows = kSplineRows * kSplineWarps;
  for (long b = 0; b < batch; b += 65535) {
    const dim3 grid((s->npsi + 31) / 32, (s->nzpsi + rows - 1) / rows, (unsigned)std::min(65535L, batch - b));
    k_bspline_grid<<<grid, dim3(32, kSplineWarps), 0, static_cast<cudaStream_t>(stream)>>>(src + b * img, dst + b * img,
                                                                                           s->nzpsi, s->npsi);
    count_launch();
    HT_CHECK_CUDA(cudaGetLastError());
  }
  return kOk;
}

extern "C" int ht_shift_filter(ht_shift_s* s, const void* psi, void* out, long batch, const float* symx,
                               const float* symy, void* stream) {
  using namespace ht;
  HT_REQUIRE(s && psi && out && symx && symy, "ht_shift_filter: null pointer");
  if (!fft_size_supported(s->npsi) || !fft_size_supported(s->nzpsi)) {
    set_error("ht_shift_filter: npsi and nzpsi must be supported FFT lengths");
    return kUnsupported;
  }
  HT_REQUIRE(batch >= 0, "ht_shift_filter: batch must be non-negative");
  if (batch == 0) return kOk;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  HT_CHECK_CUDA(symbol_rows(s->npsi, static_cast<const float2*>(psi), static_cast<float2*>(out), batch * s->nzpsi,
                            symx, s->tw_x, st));
  HT_CHECK_CUDA(symbol_cols(s->nzpsi, static_cast<float2*>(out), static_cast<float2*>(out), batch, s->npsi, symy,
                            s->tw_y, st));
  return kOk;
}

extern "C" int ht_shift_Sback(ht_shift_s* s, const void* g, const float* r, const float* mag, int nmag, void* out,
                              long batch, void* stream) {
  using namespace ht;
  HT_REQUIRE(s && g && r && mag && out, "ht_shift_Sback: null pointer");
  HT_REQUIRE(nmag == 1 || nmag == batch, "ht_shift_Sback: nmag must be 1 or batch");
  HT_REQUIRE(batch >= 0 && batch <= 65535, "ht_shift_Sback: batch must be in [0, 65535]");
  if (batch == 0) return kOk;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const dim3 sgrid((s->npsi + kSbackCX - 1) / kSbackCX, (s->nzpsi + kSbackCY - 1) / kSbackCY, (unsigned)batch);
  k_sback<<<sgrid, kSbackThreads, 0, st>>>(static_cast<const float2*>(g), static_cast<float2*>(out), r, mag, nmag,
                                           dims(s));
  count_launch();
  HT_CHECK_CUDA(cudaGetLastError());
  return kOk;
}

template <int MODE>
static int shift_stencil(ht_shift_s* s, void* out, const void* c, const void* c1, const void* c2, const float* r,
                         const float* mag, const float* d1, const float* d2, long batch, void* stream) {
  using namespace ht;
  HT_REQUIRE(s && out && c && r && mag, "shift: null pointer");
  HT_REQUIRE(MODE < 1 || (c1 && d1), "shift: null first-derivative operand");
  HT_REQUIRE(MODE < 2 || (c2 && d2), "shift: null second-derivative operand");
  if (batch == 0) return kOk;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (s->is_complex) {
    k_shift_stencil<float2, MODE><<<out_grid(s, batch), kBlock, 0, st>>>(
        (float2*)out, (const float2*)c, (const float2*)c1, (const float2*)c2, r, mag, d1, d2, nullptr, nullptr, dims(s));
    ::ht::count_launch();
  }
  else {
    k_shift_stencil<float, MODE><<<out_grid(s, batch), kBlock, 0, st>>>(
        (float*)out, (const float*)c, (const float*)c1, (const float*)c2, r, mag, d1, d2, nullptr, nullptr, dims(s));
    ::ht::count_launch();
  }
  HT_CHECK_CUDA(cudaGetLastError());
  return kOk;
}

extern "C" int ht_shift_S(ht_shift_s* s, const void* c, const float* r, const float* mag, void* out, long batch,
                          void* stream) {
  return shift_stencil<0>(s, out, c, nullptr, nullptr, r, mag, nullptr, nullptr, batch, stream);
}

extern "C" int ht_shift_dS(ht_shift_s* s, const void* c, const float* r, const float* mag, const void* c1,
                           const float* dr, void* out, long batch, void* stream) {
  return shift_stencil<1>(s, out, c, c1, nullptr, r, mag, dr, nullptr, batch, stream);
}

extern "C" int ht_shift_d2S(ht_shift_s* s, const void* c, const float* r, const float* mag, const void* c1,
                            const float* dr1, const void* c2, const float* dr2, void* out, long batch,
                            void* stream) {
  return shift_stencil<2>(s, out, c, c1, c2, r, mag, dr1, dr2, batch, stream);
}

extern "C" int ht_shift_Sadj(ht_shift_s* s, const void* g, const float* r, const float* mag, void* out, long batch,
                             void* stream) {
  using namespace ht;
  HT_REQUIRE(s && g && r && mag && out, "ht_shift_Sadj: null pointer");
  if (batch == 0) return kOk;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (s->is_complex) {
    k_shift_adj<float2><<<coef_grid(s, batch), kBlock, 0, st>>>((float2*)out, (const float2*)g, r, mag,
                                                                       dims(s));
    ::ht::count_launch();
  }
  else {
    k_shift_adj<float><<<coef_grid(s, batch), kBlock, 0, st>>>((float*)out, (const float*)g, r, mag, dims(s));
    ::ht::count_launch();
  }
  HT_CHECK_CUDA(cudaGetLastError());
  return kOk;
}

extern "C" int ht_shift_dSadj(ht_shift_s* s, const void* c, const float* r, const float* mag, const void* g,
                              void* out1, double* out2, long batch, void* stream) {
  using namespace ht;
  HT_REQUIRE(s && c && r && mag && g && out1 && out2, "ht_shift_dSadj: null pointer");
  if (batch == 0) return kOk;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  HT_CHECK_CUDA(cudaMemsetAsync(out2, 0, sizeof(double) * 2 * batch, st));
  if (s->is_complex) {
    k_shift_adj<float2><<<coef_grid(s, batch), kBlock, 0, st>>>((float2*)out1, (const float2*)g, r, mag,
                                                                       dims(s)); ::ht::count_launch();
    k_shift_stencil<float2, 3><<<out_grid(s, batch), kBlock, 0, st>>>(
        nullptr, (const float2*)c, nullptr, nullptr, r, mag, nullptr, nullptr, (const float2*)g, out2, dims(s));
    ::ht::count_launch();
  } else {
    k_shift_adj<float><<<coef_grid(s, batch), kBlock, 0, st>>>((float*)out1, (const float*)g, r, mag, dims(s)); ::ht::count_launch();
    k_shift_stencil<float, 3><<<out_grid(s, batch), kBlock, 0, st>>>(
        nullptr, (const float*)c, nullptr, nullptr, r, mag, nullptr, nullptr, (const float*)g, out2, dims(s));
    ::ht::count_launch();
  }
  HT_CHECK_CUDA(cudaGetLastError());
  return kOk;
}

extern "C" int ht_filter_rows(int N, const void* in, void* out, long nrows, const float* sym, void* stream) {
  using namespace ht;
  HT_REQUIRE(in && out && sym, "ht_filter_rows: null pointer");
  if (!fft_size_supported(N)) {
    set_error("ht_filter_rows: unsupported row length");
    return kUnsupported;
  }
  if (nrows == 0) return kOk;
  int dev = 0;
  cudaGetDevice(&dev);
  const float2* tw = twiddle_table(N, dev);
  if (!tw) return kCudaError;
  HT_CHECK_CUDA(symbol_rows(N, static_cast<const float2*>(in), static_cast<float2*>(out), nrows, sym, tw,
                            static_cast<cudaStream_t>(stream)));
  return kOk;
}
