// USFFT Radon transform R / RT (reference: src/holotomocupy/tomo.py:12-116,
// gather kernel src/holotomocupy/cuda_kernels.py:3-76).
//
// R(obj)[theta, z, :] = crop . IFFT_n . gather_theta . FFT2_2n . embed(obj * phi)
// with the reference's fftshift-by-sign multiplications folded into the
// passes.  ZI consecutive slices are interleaved (their samples stored
// together): a spectral cell or a polar sample is one vector of ZI * 8 bytes,
// 128 bytes for more than eight slices, and each Gaussian window serves ZI
// slices:
//   1. row pass (length 2n) over the n non-zero rows of the padded slice:
//      embed obj*phi, pre-sign (-1)^(row+col), FFT, post column sign (-1)^kx
//      -> fa  [zb][n][2n][ZI];
//   2. column pass (length 2n, rows outside n/2..3n/2 are zero): FFT, post
//      row sign (-1)^ky -> the centred spectrum fde [zb][2n][2n][ZI];
//   3. gather: each polar sample is an 81-tap Gaussian-weighted sum of fde
//      (m = 4 at every supported size) -> gs [zb][ntheta][n][ZI];
//   4. detector IFFT of the polar samples: sign, IFFT_n, sign, /4.
// RT runs the exact adjoint: detector FFT with signs -> gs; a gather per
// spectral cell replaces the reference's atomic scatter (lists of the samples
// whose window holds a cell of each 2 x 2 tile, made once per handle); then
// column IFFT keeping the central rows, row IFFT, crop, * phi.  The pairs and
// weights come from the forward's own formulas, so R^T is the exact transpose
// of R and deterministic.
//
// The FFT passes take ZC <= ZI slices a block (shared memory holds ZC lines)
// with the slice index fastest over the threads: the first stage loads from
// global memory and the last one stores there, in vectors of ZC samples on the
// interleaved side and runs of 32 / ZC samples on the other.
//
// The samples lie in the disc of radius n cells about the centre, so the
// cells further out than any window reaches are neither stored nor read.
//
// Angle cosines and sines come from a table computed in double precision on
// the host (the reference's __cosf/__sinf error of ~5e-7 moves R by up to
// ~1e-4 relative at n >= 512, so the exact values are used).
#include "lines.cuh"
#include "holotomo_b200_internal.h"

#include <algorithm>
#include <cmath>
#include <numeric>
#include <vector>

namespace ht {

struct GatherGeom {
  int n, ntheta, m;
  float coeff0, coeff1;   // pi/mu, -pi^2/mu
  const float2* cs;       // [ntheta] (cos theta, sin theta)
  const float* th_sorted; // [ntheta] theta mod pi, ascending
  const int* th_index;    // [ntheta] original index of th_sorted[i]
};

// Interleave for a call of nz slices: 16 fills a 128-byte line per cell or
// sample, so that the gathers move whole lines (64-byte vectors took the same
// number of L1 cycles each: one per line touched); fewer slices take the
// smallest vector that holds them.
static int interleave(int nz) { return nz > 8 ? 16 : (nz > 4 ? 8 : 4); }

// Slices of a call's first run.  At 1024^2 and above, where a slice's workspace is
// 50 MB and more, up to four slices past a multiple of 16 take a run of their own at
// their own interleave, in the first run's workspace, instead of 16 slices' room:
// 20 slices of 2048^2 at 2048 angles hold 5.6 GB instead of 9.1 and take 5.10 + 5.88 ms
// (R, R^T) instead of 6.49 + 6.03.  A longer remainder is faster with the others (28
// slices: R 7.28 ms against 7.33, R^T, whose lists would be read twice, 7.10 against 8.48).
static int first_run(int n, int nz) {
  const int rest = nz % 16;
  return n >= 1024 && nz > 16 && rest <= 4 ? nz - rest : nz;
}

// Slices a block of an FFT pass takes: 8 lines up to 1024 samples (64 KB), 4
// beyond (a 32-byte sector of the interleaved layout).
template <int N2, int ZI>
constexpr int zc_of() {
  return (N2 <= 1024 && ZI >= 8) ? 8 : 4;
}

// Plan of the Radon transform's lines of N samples: the row plan, except that
// 24 samples a thread are faster for the lines of 384 and 768 samples (BH
// iteration at 384^3 x 672 x 4: 67.5 against 69.0 ms).
template <int N>
struct RadonPlan : Plan<N> {};
template <>
struct RadonPlan<384> : PlanOf<384, 24, 8, 8, 3, 2> {};
template <>
struct RadonPlan<768> : PlanOf<768, 24, 8, 8, 4, 3> {};

// ZC lines of length N per block, slice index fastest.
template <int N, int ZC>
struct ZCfg {
  using PL = RadonPlan<N>;
  static constexpr int THREADS = ZC * PL::T;
  static constexpr int SMEM = ZC * N * (int)sizeof(float2);
};

// Cells of the centred grid (index i: frequency i - n) that a pass stores and
// reads: the windows of the samples, which lie within n of the centre, and the
// boxes the gather joins two of them in reach less than 13 cells further.
__device__ __forceinline__ bool in_disc(int n, int ky, int kx) {
  const int y = ky - n, x = kx - n, r = n + 16;
  return y * y + x * x <= r * r;
}

// Block index -> (line index, slices z0 .. z0 + ZC - 1 of batch zb): the blocks
// of one line's slices are neighbours.
template <int ZI, int ZC>
struct LineBlock {
  int line, zb, l0;
  __device__ __forceinline__ LineBlock(int bx, int by) {
    constexpr int PARTS = ZI / ZC;
    line = bx / PARTS;
    l0 = (bx % PARTS) * ZC;
    zb = by;
  }
};

// ---------------------------------------------- the 9x9 Gaussian window
// For sample tx of angle th: base indices and separable weights
// (cuda_kernels.py:22-45).  x0 = (tx - n/2)/n cos(th), y0 = -(tx - n/2)/n sin(th).
struct Window {
  int bx, by;
  float x0, y0;
};

__device__ __forceinline__ void window_base(const GatherGeom& G, int tx, float2 cs, Window& w) {
  const int n = G.n;
  const float twon = (float)(2 * n);
  const float rho = (float)(tx - n / 2) / (float)n;
  w.x0 = rho * cs.x;
  w.y0 = -rho * cs.y;
  w.bx = (int)floorf(twon * w.x0) - G.m;
  w.by = (int)floorf(twon * w.y0) - G.m;
}
__device__ __forceinline__ float wx_tap(const GatherGeom& G, const Window& w, int i) {
  const float inv_twon = 1.0f / (float)(2 * G.n);
  const float w0 = (float)(w.bx + i) * inv_twon - w.x0;
  return __expf(G.coeff1 * w0 * w0);
}
__device__ __forceinline__ float wy_tap(const GatherGeom& G, const Window& w, int i) {
  const float inv_twon = 1.0f / (float)(2 * G.n);
  const float w1 = (float)(w.by + i) * inv_twon - w.y0;
  return G.coeff0 * __expf(G.coeff1 * w1 * w1);
}

// A sample of the caller's arrays, complex or real (imaginary part 0 in, dropped out).
__device__ __forceinline__ float2 ld_c(const float2* p) { return *p; }
__device__ __forceinline__ float2 ld_c(const float* p) { return make_float2(*p, 0.f); }
__device__ __forceinline__ void st_c(float2* p, float2 v) { *p = v; }
__device__ __forceinline__ void st_c(float* p, float2 v) { *p = v.x; }

// ------------------------------------------------------ 1: rows (R)
// obj [nz, n, n] -> fa [zb][n][2n][ZI];  grid (n ZI / ZC, nzb)
template <class T>
struct TRowFwdIn {
  const T* p;        // obj row of this slice
  const float* phi;  // phi row
  int n, pr;         // pr: padded row (sign)
  static constexpr bool kCentralHalf = true;
  __device__ __forceinline__ float2 ld(int q) const {
    float s = __ldg(&phi[q - n / 2]);
    if ((pr + q) & 1) s = -s;
    return cscale(ld_c(p + (q - n / 2)), s);   // past the last slice: slice 0's line, not stored
  }
};
// Interleaved line: sample k at k * stride, the odd ones negated.
struct TSignOut {
  float2* p;
  long stride;
  bool valid;
  __device__ __forceinline__ void st(int k, float2 v) const {
    if (valid) p[k * stride] = (k & 1) ? make_float2(-v.x, -v.y) : v;
  }
};

template <int N2, int ZI, class T>
__global__ void __launch_bounds__(ZCfg<N2, zc_of<N2, ZI>()>::THREADS)
k_trow_fwd(const T* __restrict__ obj, const float* __restrict__ phi, float2* __restrict__ fa, int nz,
           const float2* __restrict__ tw4) {
  constexpr int ZC = zc_of<N2, ZI>();
  constexpr int n = N2 / 2;
  extern __shared__ float2 smem[];
  const LineBlock<ZI, ZC> B(blockIdx.x, blockIdx.y);
  const int l = threadIdx.x % ZC, t = threadIdx.x / ZC, r = B.line;
  if (B.zb * ZI + B.l0 >= nz) return;
  const int z = B.zb * ZI + B.l0 + l;
  const bool valid = z < nz;
  const TRowFwdIn<T> in{obj + ((long)(valid ? z : 0) * n + r) * n, phi + r * n, n, r + n / 2};
  const TSignOut out{fa + ((long)B.zb * n + r) * N2 * ZI + B.l0 + l, ZI, valid};
  fft_line_io<N2, false, RadonPlan<N2>>(in, SmCol<ZC>{smem + l}, out, t, tw4);
}

// --------------------------------------------------- 2: columns (R)
// fa [zb][n][2n][ZI] -> fde [zb][2n][2n][ZI];  grid (2n ZI / ZC, nzb).  The
// rows outside the central n are zero and not read; the cells outside the
// disc are not stored (21 % of the grid).
// (The slices past the last one of a ragged batch are read too, whatever the
// workspace holds there: no slice's line meets another's, and theirs are not
// stored.)
struct TColFwdIn {
  const float2* p;  // fa at row 0 of this column and slice
  int n;
  long rowstride;
  static constexpr bool kCentralHalf = true;
  __device__ __forceinline__ float2 ld(int k) const { return p[(k - n / 2) * rowstride]; }
};
struct TColFwdOut {
  float2* p;  // fde at row 0 of this column and slice
  int n, kx;
  long rowstride;
  bool valid;
  __device__ __forceinline__ void st(int k, float2 v) const {
    if (valid && in_disc(n, k, kx)) p[k * rowstride] = (k & 1) ? make_float2(-v.x, -v.y) : v;
  }
};

template <int N2, int ZI>
__global__ void __launch_bounds__(ZCfg<N2, zc_of<N2, ZI>()>::THREADS)
k_tcol_fwd(const float2* __restrict__ fa, float2* __restrict__ fde, int nz, const float2* __restrict__ tw4) {
  constexpr int ZC = zc_of<N2, ZI>();
  constexpr int n = N2 / 2;
  extern __shared__ float2 smem[];
  const LineBlock<ZI, ZC> B(blockIdx.x, blockIdx.y);
  const int l = threadIdx.x % ZC, t = threadIdx.x / ZC, kx = B.line;
  if (B.zb * ZI + B.l0 >= nz) return;
  const bool valid = B.zb * ZI + B.l0 + l < nz;
  const TColFwdIn in{fa + (long)B.zb * n * N2 * ZI + (long)kx * ZI + B.l0 + l, n, (long)N2 * ZI};
  const TColFwdOut out{fde + (long)B.zb * N2 * N2 * ZI + (long)kx * ZI + B.l0 + l, n, kx, (long)N2 * ZI, valid};
  fft_line_io<N2, false, RadonPlan<N2>>(in, SmCol<ZC>{smem + l}, out, t, tw4);
}

// ------------------------------------------------- 3: polar gather (R)
// fde [zb][2n][2n][ZI] -> gs [zb][ntheta][n][ZI].  ZI/2 consecutive lanes share
// the samples of NA angles (neighbours in the sorted order) at one radius, each
// lane reading one float4 (two slices) of a cell's vector.  The windows of two
// neighbouring angles overlap where their lines lie within a few cells, so the
// pair walks the box that holds both and each cell loaded serves both samples:
// about 105 loads instead of 162.  Sparse angles go one by one (NA = 1), as does
// a pair whose box is wider than kBoxW.  L1 moves 128 bytes a cycle, a request
// of four cells' vectors takes four: 64 slices of 512^2 at 900 angles take 0.78 ms
// in pairs and 0.84 one by one (62 % of L1's rate, half of the issue slots), at
// 225 angles 0.30 and 0.24; boxes of 2 x 2 samples save half of the loads again
// but take 0.87 and 0.35: their zero weights cost more multiply-adds than that
// and their 128 registers leave half the warps.
constexpr int kBoxW = 12;
constexpr int kGatherThreads = 256;

template <int ZI, int S, int WM, bool WRAP>
__device__ __forceinline__ void gather_box(const float4* __restrict__ f, const GatherGeom& G, const Window (&w)[S],
                                           int minx, int miny, int W, int H, float4 (&acc)[S]) {
  constexpr int Q = ZI / 2, CH = S == 1 ? WM : 4;  // CH: loads in flight
  const int n = G.n, twon = 2 * n;
  const float inv_twon = 1.0f / (float)twon;
  float wx[S][WM];
#pragma unroll
  for (int s = 0; s < S; ++s)
#pragma unroll
    for (int j = 0; j < WM; ++j) {
      const float w0 = (float)(minx + j) * inv_twon - w[s].x0;
      wx[s][j] = (unsigned)(minx + j - w[s].bx) < 9u ? __expf(G.coeff1 * w0 * w0) : 0.f;
    }
#pragma unroll
  for (int s = 0; s < S; ++s) acc[s] = make_float4(0.f, 0.f, 0.f, 0.f);
  const int c0 = n + minx;
#pragma unroll 1
  for (int i = 0; i < H; ++i) {
    int row = n + miny + i;
    row += (row < 0) ? twon : 0;
    row -= (row >= twon) ? twon : 0;
    const float4* frow = f + ((long)row * twon + (WRAP ? 0 : c0)) * Q;
    float2 a[S], b[S];
#pragma unroll
    for (int s = 0; s < S; ++s) a[s] = b[s] = make_float2(0.f, 0.f);
#pragma unroll
    for (int j0 = 0; j0 < WM; j0 += CH) {
      float4 v[CH];
#pragma unroll
      for (int jj = 0; jj < CH; ++jj) {
        const int j = j0 + jj;
        if (j >= WM) break;
        v[jj] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (j < 9 || j < W) {
          int c = j;
          if (WRAP) {
            c += c0;
            c += (c < 0) ? twon : 0;
            c -= (c >= twon) ? twon : 0;
          }
          v[jj] = __ldg(&frow[c * Q]);
        }
      }
#pragma unroll
      for (int jj = 0; jj < CH; ++jj) {
        if (j0 + jj >= WM) break;
#pragma unroll
        for (int s = 0; s < S; ++s) {
          const float2 k = make_float2(wx[s][j0 + jj], wx[s][j0 + jj]);
          a[s] = p2_fma(k, make_float2(v[jj].x, v[jj].y), a[s]);
          b[s] = p2_fma(k, make_float2(v[jj].z, v[jj].w), b[s]);
        }
      }
    }
#pragma unroll
    for (int s = 0; s < S; ++s) {
      const float w1 = (float)(miny + i) * inv_twon - w[s].y0;
      const float ey = (unsigned)(miny + i - w[s].by) < 9u ? G.coeff0 * __expf(G.coeff1 * w1 * w1) : 0.f;
      acc[s] = make_float4(fmaf(ey, a[s].x, acc[s].x), fmaf(ey, a[s].y, acc[s].y), fmaf(ey, b[s].x, acc[s].z),
                           fmaf(ey, b[s].y, acc[s].w));
    }
  }
}

template <int ZI, int S, int WM>
__device__ __forceinline__ void gather_group(const float4* __restrict__ f, const GatherGeom& G, const Window (&w)[S],
                                             int minx, int miny, int W, int H, float4 (&acc)[S]) {
  if (G.n + minx >= 0 && G.n + minx + W <= 2 * G.n)
    gather_box<ZI, S, WM, false>(f, G, w, minx, miny, W, H, acc);
  else
    gather_box<ZI, S, WM, true>(f, G, w, minx, miny, W, H, acc);
}

// Block of kGatherThreads / (ZI/2) groups: GR radii x GA groups of angles, whose
// cells stay in L1.  grid (radial tiles x angle tiles, nzb)
template <int ZI, int NA>
struct GatherTile {
  static constexpr int GR = 8, GA = kGatherThreads / (ZI / 2) / GR;
};

template <int ZI, int NA>
__global__ void __launch_bounds__(kGatherThreads, NA == 2 ? 3 : 4)
k_tgather(const float2* __restrict__ fde, float2* __restrict__ gs, GatherGeom G, int nz, int rtiles) {
  using TL = GatherTile<ZI, NA>;
  constexpr int Q = ZI / 2;
  const int n = G.n, twon = 2 * n;
  const int q = threadIdx.x % Q, grp = threadIdx.x / Q;
  const int zb = blockIdx.y;
  const int tx = (int)(blockIdx.x % rtiles) * TL::GR + grp % TL::GR;
  const int ia0 = ((int)(blockIdx.x / rtiles) * TL::GA + grp / TL::GR) * NA;
  if (zb * ZI + 2 * q >= nz || tx >= n || ia0 >= G.ntheta) return;
  const float4* f = reinterpret_cast<const float4*>(fde + (long)zb * twon * twon * ZI) + q;
  float4* out = reinterpret_cast<float4*>(gs + (long)zb * G.ntheta * n * ZI) + q;
  Window w[NA];
  int th[NA];
  int minx = 1 << 30, miny = 1 << 30, maxx = -(1 << 30), maxy = -(1 << 30);
#pragma unroll
  for (int a = 0; a < NA; ++a) {
    th[a] = G.th_index[min(ia0 + a, G.ntheta - 1)];
    window_base(G, tx, G.cs[th[a]], w[a]);
    minx = min(minx, w[a].bx);
    maxx = max(maxx, w[a].bx);
    miny = min(miny, w[a].by);
    maxy = max(maxy, w[a].by);
  }
  float4 acc[NA];
  const int W = maxx - minx + 9, H = maxy - miny + 9;
  if (NA == 1) {
    gather_group<ZI, NA, 9>(f, G, w, minx, miny, 9, 9, acc);
  } else if (W <= kBoxW && H <= kBoxW) {
    gather_group<ZI, NA, kBoxW>(f, G, w, minx, miny, W, H, acc);
  } else {
#pragma unroll
    for (int s = 0; s < NA; ++s) {
      const Window one[1] = {w[s]};
      float4 v[1];
      gather_group<ZI, 1, 9>(f, G, one, w[s].bx, w[s].by, 9, 9, v);
      acc[s] = v[0];
    }
  }
#pragma unroll
  for (int a = 0; a < NA; ++a)
    if (ia0 + a < G.ntheta) out[((long)th[a] * n + tx) * Q] = acc[a];
}

// --------------------------------------- 4: detector IFFT (R), detector FFT (RT)
// gs [zb][ntheta][n][ZI] <-> sino [ntheta, ldz rows, n];  grid (ntheta ZI / ZC, nzb).
// symx: the detector-axis filter, whose frequency kx sits at sample kx - n/2 (mod n).
struct TSinoScale {
  const float* symx;
  int n;
  float s;
  __device__ __forceinline__ float2 at(int tx, float2 v) const {
    float k = (tx & 1) ? -s : s;
    if (symx) {
      const int h = tx + n / 2;
      k *= __ldg(&symx[h >= n ? h - n : h]);
    }
    return cscale(v, k);
  }
};
struct TSinoIfftIn {
  const float2* p;
  int stride;
  TSinoScale sc;  // 1/n of the gather, (-1)^tx before the IFFT, the filter
  __device__ __forceinline__ float2 ld(int tx) const { return sc.at(tx, p[(long)tx * stride]); }
};
template <class T>
struct TSinoIfftOut {
  T* p;
  float s;  // ifft 1/n and /4; (-1)^k
  bool valid;
  __device__ __forceinline__ void st(int k, float2 v) const {
    if (valid) st_c(p + k, cscale(v, (k & 1) ? -s : s));
  }
};
template <int N, int ZI, class T>
__global__ void __launch_bounds__(ZCfg<N, zc_of<2 * N, ZI>()>::THREADS)
k_tsino_ifft(const float2* __restrict__ gs, T* __restrict__ sino, int ntheta, int nz, int ldz,
             const float2* __restrict__ tw4, const float* __restrict__ symx) {
  constexpr int ZC = zc_of<2 * N, ZI>();
  extern __shared__ float2 smem[];
  const LineBlock<ZI, ZC> B(blockIdx.x, blockIdx.y);
  const int l = threadIdx.x % ZC, t = threadIdx.x / ZC, th = B.line;
  if (B.zb * ZI + B.l0 >= nz) return;
  const int z = B.zb * ZI + B.l0 + l;
  const bool valid = z < nz;
  const TSinoIfftIn in{gs + ((long)B.zb * ntheta + th) * N * ZI + B.l0 + l, ZI,
                       TSinoScale{symx, N, 1.0f / (float)N}};
  const TSinoIfftOut<T> out{sino + ((long)th * ldz + (valid ? z : 0)) * N, 1.0f / (4.f * (float)N), valid};
  fft_line_io<N, true, RadonPlan<N>>(in, SmCol<ZC>{smem + l}, out, t, tw4);
}

template <class T>
struct TSinoFftIn {
  const T* p;
  __device__ __forceinline__ float2 ld(int k) const {
    const float2 v = ld_c(p + k);
    return (k & 1) ? make_float2(-v.x, -v.y) : v;
  }
};
struct TSinoFftOut {
  float2* p;
  int stride;
  TSinoScale sc;  // the caller's scale, (-1)^tx, the filter
  bool valid;
  __device__ __forceinline__ void st(int tx, float2 v) const {
    if (valid) p[(long)tx * stride] = sc.at(tx, v);
  }
};
template <int N, int ZI, class T>
__global__ void __launch_bounds__(ZCfg<N, zc_of<2 * N, ZI>()>::THREADS)
k_tsino_fft(const T* __restrict__ sino, float2* __restrict__ gs, int ntheta, int nz, int ldz,
            const float2* __restrict__ tw4, const float* __restrict__ symx, float scale) {
  constexpr int ZC = zc_of<2 * N, ZI>();
  extern __shared__ float2 smem[];
  const LineBlock<ZI, ZC> B(blockIdx.x, blockIdx.y);
  const int l = threadIdx.x % ZC, t = threadIdx.x / ZC, th = B.line;
  if (B.zb * ZI + B.l0 >= nz) return;
  const int z = B.zb * ZI + B.l0 + l;
  const bool valid = z < nz;
  const TSinoFftIn<T> in{sino + ((long)th * ldz + (valid ? z : 0)) * N};
  const TSinoFftOut out{gs + ((long)B.zb * ntheta + th) * N * ZI + B.l0 + l, ZI, TSinoScale{symx, N, scale}, valid};
  fft_line_io<N, false, RadonPlan<N>>(in, SmCol<ZC>{smem + l}, out, t, tw4);
}

// -------------------------------------------- RT 2: sparse cell gather
// The pairs (sample, spectral cell) of R's gridding and their weights depend
// only on the angles, so ht_tomo_create lists them once: for every tile of 2 x 2
// cells the samples whose window holds any of its cells -- found by a search
// (the angles whose line passes within kTileReach, by binary search in the
// sorted angles; the radial samples near the tile) with window membership and
// weights from the forward's own formulas -- and the four cells' weights (0
// where the window misses the cell).  Each list is padded to a multiple of
// four entries with weight 0.  A sample's vector is loaded once for the four
// cells (1.23 times the samples of one cell, so 3.2 times fewer vector loads
// than cell by cell), by ZI/2 lanes, for ZG slice batches a pass.  Bound by L1:
// 4 cycles a vector request, 4 for a request of weights.  The exact transpose
// of R, deterministic, no atomics.
constexpr float kTileReach = 8.3f;  // window cells lie within 5 sqrt(2) of the sample centre, a tile's within sqrt(1/2) of its own

__device__ __forceinline__ int lower_bound_f(const float* a, int n, float v) {
  int lo = 0, hi = n;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (a[mid] < v)
      lo = mid + 1;
    else
      hi = mid;
  }
  return lo;
}

__device__ __forceinline__ int upper_bound_f(const float* a, int n, float v) {
  int lo = 0, hi = n;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (a[mid] <= v)
      lo = mid + 1;
    else
      hi = mid;
  }
  return lo;
}

// (X - n - b) mod 2n for the window base b: b lies in [-n - m, n - m] and X - n
// in [-n, n), so one correction either way reduces it
__device__ __forceinline__ int window_index(int X, int n, int b) {
  int i = X - n - b;
  i += (i < 0) ? 2 * n : 0;
  i -= (i >= 2 * n) ? 2 * n : 0;
  return i;
}

// Visit (sample index j*n + t, weights of the cells (X, Y), (X+1, Y), (X, Y+1),
// (X+1, Y+1)) for every sample of angle j whose window holds one of them.
template <class F>
__device__ __forceinline__ void tile_angle_pairs(const GatherGeom& G, int j, float px, float py, int X, int Y, F& f) {
  const int n = G.n, twon = 2 * n;
  const float2 cs = G.cs[j];
  const float s = px * cs.x - py * cs.y;  // projection onto (cos, -sin)
  const int t0 = max(0, (int)ceilf((s - kTileReach) * 0.5f) + n / 2);
  const int t1 = min(n - 1, (int)floorf((s + kTileReach) * 0.5f) + n / 2);
  for (int tx = t0; tx <= t1; ++tx) {
    Window w;
    window_base(G, tx, cs, w);
    const int i0 = window_index(X, n, w.bx), i1 = window_index(Y, n, w.by);
    const bool x0 = i0 <= 8, x1 = i0 <= 7 || i0 == twon - 1;
    const bool y0 = i1 <= 8, y1 = i1 <= 7 || i1 == twon - 1;
    if (!((x0 || x1) && (y0 || y1))) continue;
    if (!f.wants_weights) {
      f(j * n + tx, make_float4(0.f, 0.f, 0.f, 0.f));
      continue;
    }
    const float wx0 = x0 ? wx_tap(G, w, i0) : 0.f, wx1 = x1 ? wx_tap(G, w, i0 == twon - 1 ? 0 : i0 + 1) : 0.f;
    const float wy0 = y0 ? wy_tap(G, w, i1) : 0.f, wy1 = y1 ? wy_tap(G, w, i1 == twon - 1 ? 0 : i1 + 1) : 0.f;
    f(j * n + tx, make_float4(wx0 * wy0, wx1 * wy0, wx0 * wy1, wx1 * wy1));
  }
}

// The angles whose line passes near a tile, in a fixed order: all of them, or one or
// two ranges of the sorted ones.
struct AngleSpan {
  int first[2], len[2];
  bool sorted;
  __device__ __forceinline__ int count() const { return len[0] + len[1]; }
  __device__ __forceinline__ int at(const GatherGeom& G, int k) const {
    if (!sorted) return k;
    return G.th_index[k < len[0] ? first[0] + k : first[1] + k - len[0]];
  }
};

// visit(px, py, span) for the centre of the tile at cell (X, Y) and its periodic
// images within reach of the sample disc.
template <class V>
__device__ __forceinline__ void tile_images(const GatherGeom& G, int X, int Y, V visit) {
  const int n = G.n, twon = 2 * n;
  const float PI = 3.14159265358979f;
  const float lim = (float)n + 10.0f;
  for (int oy = -1; oy <= 1; ++oy) {
    for (int ox = -1; ox <= 1; ++ox) {
      const float px = (float)(X - n + ox * twon) + 0.5f, py = (float)(Y - n + oy * twon) + 0.5f;
      if (fabsf(px) > lim || fabsf(py) > lim) continue;
      AngleSpan span{{0, 0}, {G.ntheta, 0}, false};
      const float R = sqrtf(px * px + py * py);
      if (R > kTileReach) {
        // angles with R |sin(theta + phi)| <= reach, theta taken mod pi
        const float dlt = asinf(fminf(1.0f, kTileReach / R)) + 1e-4f;
        float c = -atan2f(py, px);
        c = c - PI * floorf(c / PI);
        const float a = c - dlt, b = c + dlt;
        float ia[2] = {a, 0.f}, ib[2] = {b, -1.f};
        if (a < 0.f) {
          ia[0] = 0.f;
          ia[1] = a + PI;
          ib[1] = PI;
        } else if (b >= PI) {
          ib[0] = PI;
          ib[1] = b - PI;
        }
        span.sorted = true;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          span.first[q] = lower_bound_f(G.th_sorted, G.ntheta, ia[q]);
          span.len[q] = max(upper_bound_f(G.th_sorted, G.ntheta, ib[q]) - span.first[q], 0);
        }
      }
      visit(px, py, span);
    }
  }
}

struct PairCount {
  static constexpr bool wants_weights = false;
  int n = 0;
  __device__ void operator()(int, float4) { ++n; }
};

struct PairFill {
  static constexpr bool wants_weights = true;
  int* idx;
  float4* w;
  int p = 0;
  __device__ void operator()(int i, float4 v) {
    idx[p] = i;
    w[p] = v;
    ++p;
  }
};

// Tiles within kNearTiles of the centre, where many lines pass: a warp each, its
// lanes taking consecutive stretches of the angles (the lists' order is that of one
// thread), against a thread each for the others.  One thread a centre tile outlasts
// the rest of the launch: ht_tomo_create took 10.6 ms at 512^2 x 900 angles, 5.3 with
// 16 tiles either way, 4.2 with 32; at 64^2 x 90 angles 1.9 ms, 1.0, 0.9.
constexpr int kNearTiles = 32;
__host__ __device__ inline int near_first(int n) { return n / 2 > kNearTiles ? n / 2 - kNearTiles : 0; }
__host__ __device__ inline int near_side(int n) {
  return (n < n / 2 + kNearTiles ? n : n / 2 + kNearTiles) - near_first(n);
}
__device__ __forceinline__ bool near_tile(int n, int tx, int ty) {
  return (unsigned)(tx - near_first(n)) < (unsigned)near_side(n) &&
         (unsigned)(ty - near_first(n)) < (unsigned)near_side(n);
}

// Tiles in row-major order over the n x n tiles of the 2n x 2n cells.
__global__ void k_cell_count(GatherGeom G, int* __restrict__ cnt) {
  const long c = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const int tx = (int)(c % G.n), ty = (int)(c / G.n);
  if (c >= (long)G.n * G.n || near_tile(G.n, tx, ty)) return;
  PairCount f;
  tile_images(G, 2 * tx, 2 * ty, [&](float px, float py, const AngleSpan& span) {
    for (int k = 0; k < span.count(); ++k) tile_angle_pairs(G, span.at(G, k), px, py, 2 * tx, 2 * ty, f);
  });
  cnt[c] = (f.n + 3) / 4 * 4;
}

__global__ void k_cell_fill(GatherGeom G, const long* __restrict__ off, int* __restrict__ idx,
                            float4* __restrict__ wgt) {
  const long c = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const int tx = (int)(c % G.n), ty = (int)(c / G.n);
  if (c >= (long)G.n * G.n || near_tile(G.n, tx, ty)) return;
  PairFill f{idx + off[c], wgt + off[c]};
  tile_images(G, 2 * tx, 2 * ty, [&](float px, float py, const AngleSpan& span) {
    for (int k = 0; k < span.count(); ++k) tile_angle_pairs(G, span.at(G, k), px, py, 2 * tx, 2 * ty, f);
  });
  const int last = f.p > 0 ? f.idx[f.p - 1] : 0;
  while (f.p < (int)(off[c + 1] - off[c])) f(last, make_float4(0.f, 0.f, 0.f, 0.f));
}

// The same for the near tiles; grid: a warp per tile.  FILL: the lists, else the counts.
template <bool FILL>
__global__ void k_cell_near(GatherGeom G, int* __restrict__ cnt, const long* __restrict__ off, int* __restrict__ idx,
                            float4* __restrict__ wgt) {
  const int lane = threadIdx.x % 32, side = near_side(G.n);
  const int tile = (int)((blockIdx.x * blockDim.x + threadIdx.x) / 32);
  if (tile >= side * side) return;
  const int tx = near_first(G.n) + tile % side, ty = near_first(G.n) + tile / side;
  const long c = (long)ty * G.n + tx;
  int total = 0;
  tile_images(G, 2 * tx, 2 * ty, [&](float px, float py, const AngleSpan& span) {
    const int per = (span.count() + 31) / 32, k0 = min(lane * per, span.count()), k1 = min(k0 + per, span.count());
    PairCount n;
    for (int k = k0; k < k1; ++k) tile_angle_pairs(G, span.at(G, k), px, py, 2 * tx, 2 * ty, n);
    int before = n.n;  // inclusive sum over the lanes
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, before, o);
      if (lane >= o) before += v;
    }
    const int all = __shfl_sync(0xffffffffu, before, 31);
    if constexpr (FILL) {
      const long at = off[c] + total + before - n.n;
      PairFill f{idx + at, wgt + at};
      for (int k = k0; k < k1; ++k) tile_angle_pairs(G, span.at(G, k), px, py, 2 * tx, 2 * ty, f);
    }
    total += all;
  });
  if constexpr (FILL) {
    __syncwarp();
    if (lane != 0) return;
    const int last = total > 0 ? idx[off[c] + total - 1] : 0;
    PairFill f{idx + off[c], wgt + off[c], total};
    while (f.p < (int)(off[c + 1] - off[c])) f(last, make_float4(0.f, 0.f, 0.f, 0.f));
  } else if (lane == 0) {
    cnt[c] = (total + 3) / 4 * 4;
  }
}

// A list's entries p0, p0 + step, ... (groups of four) summed into acc[batch][cell].
template <int ZI, int ZG>
__device__ __forceinline__ void tile_sum(const int* __restrict__ idx, const float4* __restrict__ wgt, int nl, int p0,
                                         int step, const float4* __restrict__ gb, long bstride, int nb,
                                         float4 (&acc)[ZG][4]) {
  constexpr int Q = ZI / 2;
#pragma unroll
  for (int g = 0; g < ZG; ++g)
#pragma unroll
    for (int k = 0; k < 4; ++k) acc[g][k] = make_float4(0.f, 0.f, 0.f, 0.f);
  int4 next = p0 < nl ? __ldg(reinterpret_cast<const int4*>(idx + p0)) : make_int4(0, 0, 0, 0);
  for (int p = p0; p < nl; p += step) {
    const int ii[4] = {next.x, next.y, next.z, next.w};
    // the next four samples' indices are on their way while these four's vectors
    // load (250 slices of 256^2 at 361 angles: 521 us to 480)
    if (p + step < nl) next = __ldg(reinterpret_cast<const int4*>(idx + p + step));
    float4 u[4][ZG];
#pragma unroll
    for (int e = 0; e < 4; ++e)
#pragma unroll
      for (int g = 0; g < ZG; ++g)
        u[e][g] = g < nb ? __ldg(&gb[g * bstride + (long)ii[e] * Q]) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float4 w4 = __ldg(&wgt[p + e]);
      const float ww[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float2 w2 = make_float2(ww[k], ww[k]);
#pragma unroll
        for (int g = 0; g < ZG; ++g) {
          float4& a = acc[g][k];
          const float2 lo = p2_fma(w2, make_float2(u[e][g].x, u[e][g].y), make_float2(a.x, a.y));
          const float2 hi = p2_fma(w2, make_float2(u[e][g].z, u[e][g].w), make_float2(a.z, a.w));
          a = make_float4(lo.x, lo.y, hi.x, hi.y);
        }
      }
    }
  }
}

// Lists longer than this are summed by a whole block: near the centre, where
// all the lines cross, a list is tens of times the average, and one group of
// lanes walking it would outlast the rest of the launch.
constexpr int kHeavyList = 512;
constexpr int kCellThreads = 256;

// gs [zb][ntheta][n][ZI] -> fde [zb][2n][2n][ZI].  ZG slice batches a pass,
// ngroups passes; block b takes pass b % ngroups (the passes over one stretch
// of the lists run together, so the lists come from DRAM once) of tile block
// b / ngroups: the first nheavy of them one long list each, the others
// TX x TY tiles, a list per group of ZI/2 lanes.
template <int ZI>
struct CellTile {
  static constexpr int GROUPS = kCellThreads / (ZI / 2);
  static constexpr int TX = ZI == 4 ? 16 : 8;
  static constexpr int TY = GROUPS / TX;
};

template <int ZI, int ZG>
__global__ void __launch_bounds__(kCellThreads, 2)
k_tcell(const float2* __restrict__ gs, float2* __restrict__ fde, const long* __restrict__ off,
        const int* __restrict__ idx, const float4* __restrict__ wgt, const int* __restrict__ heavy, int nheavy, int n,
        long nsamp, int nz, int ngroups) {
  constexpr int Q = ZI / 2;
  using TL = CellTile<ZI>;
  __shared__ float4 red[kCellThreads / 32][ZG][4][Q];
  const int grp = (int)(blockIdx.x % ngroups);
  const int blk = (int)(blockIdx.x / ngroups);
  const int q = threadIdx.x % Q, lg = threadIdx.x / Q;
  const int zb0 = grp * ZG;
  // batches of this pass that hold this lane's slices
  int nb = 0;
#pragma unroll
  for (int g = 0; g < ZG; ++g) nb += ((zb0 + g) * ZI + 2 * q < nz) ? 1 : 0;
  const float4* gb = reinterpret_cast<const float4*>(gs + (long)zb0 * nsamp * ZI) + q;
  const long bstride = nsamp * Q;
  float4 acc[ZG][4];
  const int twon = 2 * n;
  int X, Y;
  if (blk < nheavy) {
    const int tile = heavy[blk];
    X = 2 * (tile % n);
    Y = 2 * (tile / n);
    const long o = off[tile];
    tile_sum<ZI, ZG>(idx + o, wgt + o, (int)(off[tile + 1] - o), 4 * lg, 4 * TL::GROUPS, gb, bstride, nb, acc);
    // the groups of a warp, then the warps, in a fixed order
#pragma unroll
    for (int g = 0; g < ZG; ++g)
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        float4& a = acc[g][k];
#pragma unroll
        for (int o2 = 16; o2 >= Q; o2 >>= 1) {
          a.x += __shfl_down_sync(0xffffffffu, a.x, o2);
          a.y += __shfl_down_sync(0xffffffffu, a.y, o2);
          a.z += __shfl_down_sync(0xffffffffu, a.z, o2);
          a.w += __shfl_down_sync(0xffffffffu, a.w, o2);
        }
        if (threadIdx.x % 32 < Q) red[threadIdx.x / 32][g][k][q] = a;
      }
    __syncthreads();
    if (lg != 0) return;
#pragma unroll
    for (int g = 0; g < ZG; ++g)
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        float4 a = red[0][g][k][q];
        for (int w = 1; w < kCellThreads / 32; ++w) {
          const float4 b = red[w][g][k][q];
          a = make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
        }
        acc[g][k] = a;
      }
  } else {
    const int tb = blk - nheavy, bx = (n + TL::TX - 1) / TL::TX;
    const int tx = (tb % bx) * TL::TX + lg % TL::TX, ty = (tb / bx) * TL::TY + lg / TL::TX;
    if (tx >= n || ty >= n) return;
    X = 2 * tx;
    Y = 2 * ty;
    const long o = off[ty * n + tx];
    const int nl = (int)(off[ty * n + tx + 1] - o);
    if (nl > kHeavyList) return;
    tile_sum<ZI, ZG>(idx + o, wgt + o, nl, 0, 4, gb, bstride, nb, acc);
  }
  float4* dst = reinterpret_cast<float4*>(fde) + q;
#pragma unroll
  for (int g = 0; g < ZG; ++g) {
    if (g >= nb) break;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int y = Y + k / 2, x = X + k % 2;
      if (in_disc(n, y, x)) dst[(((long)(zb0 + g) * twon + y) * twon + x) * Q] = acc[g][k];
    }
  }
}

// ------------------------------------------- RT 3: column IFFT
// fde [zb][2n][2n][ZI] -> fb [zb][n][2n][ZI] (central rows);  grid (2n ZI / ZC, nzb).
struct TColAdjIn {
  const float2* p;  // fde at row 0 of this column and slice
  int n, kx;
  long rowstride;
  __device__ __forceinline__ float2 ld(int k) const {
    // outside the disc: the centre row's cell, dropped (a load without a branch)
    const bool in = in_disc(n, k, kx);
    const float2 v = p[(in ? k : n) * rowstride];
    const float s = ((k + kx) & 1) ? -1.f : 1.f;  // pre-sign (-1)^(ky+kx)
    return in ? cscale(v, s) : make_float2(0.f, 0.f);
  }
};
struct TColAdjOut {
  float2* p;  // fb at row 0 of this column and slice
  int n;
  long rowstride;
  float s;    // 1 / 2n
  bool valid;
  static constexpr bool kCentralHalf = true;
  __device__ __forceinline__ void st(int k, float2 v) const {
    if (valid && k >= n / 2 && k < 3 * n / 2) p[(k - n / 2) * rowstride] = cscale(v, (k & 1) ? -s : s);  // post sign
  }
};

template <int N2, int ZI>
__global__ void __launch_bounds__(ZCfg<N2, zc_of<N2, ZI>()>::THREADS)
k_tcol_adj(const float2* __restrict__ fde, float2* __restrict__ fb, int nz, const float2* __restrict__ tw4) {
  constexpr int ZC = zc_of<N2, ZI>();
  constexpr int n = N2 / 2;
  extern __shared__ float2 smem[];
  const LineBlock<ZI, ZC> B(blockIdx.x, blockIdx.y);
  const int l = threadIdx.x % ZC, t = threadIdx.x / ZC, kx = B.line;
  if (B.zb * ZI + B.l0 >= nz) return;
  const bool valid = B.zb * ZI + B.l0 + l < nz;
  const TColAdjIn in{fde + (long)B.zb * N2 * N2 * ZI + (long)kx * ZI + B.l0 + l, n, kx, (long)N2 * ZI};
  const TColAdjOut out{fb + (long)B.zb * n * N2 * ZI + (long)kx * ZI + B.l0 + l, n, (long)N2 * ZI, 1.0f / (float)N2,
                       valid};
  fft_line_io<N2, true, RadonPlan<N2>>(in, SmCol<ZC>{smem + l}, out, t, tw4);
}

// ---------------------------------------------- RT 4: row IFFT
// fb [zb][n][2n][ZI] -> out [nz, n, n] = crop(IFFT) * (-1)^q * phi;  grid (n ZI / ZC, nzb)
struct TLineIn {
  const float2* p;
  int stride;
  __device__ __forceinline__ float2 ld(int k) const { return p[(long)k * stride]; }
};
template <class T>
struct TRowAdjOut {
  T* p;              // out row of this slice
  const float* phi;  // phi row
  int n;
  float s;           // 1 / 2n
  bool valid;
  static constexpr bool kCentralHalf = true;
  __device__ __forceinline__ void st(int q, float2 v) const {
    if (!valid || q < n / 2 || q >= 3 * n / 2) return;
    float ph = __ldg(&phi[q - n / 2]) * s;
    if (q & 1) ph = -ph;
    st_c(p + (q - n / 2), cscale(v, ph));
  }
};

template <int N2, int ZI, class T>
__global__ void __launch_bounds__(ZCfg<N2, zc_of<N2, ZI>()>::THREADS)
k_trow_adj(const float2* __restrict__ fb, const float* __restrict__ phi, T* __restrict__ out, int nz,
           const float2* __restrict__ tw4) {
  constexpr int ZC = zc_of<N2, ZI>();
  constexpr int n = N2 / 2;
  extern __shared__ float2 smem[];
  const LineBlock<ZI, ZC> B(blockIdx.x, blockIdx.y);
  const int l = threadIdx.x % ZC, t = threadIdx.x / ZC, r = B.line;
  if (B.zb * ZI + B.l0 >= nz) return;
  const int z = B.zb * ZI + B.l0 + l;
  const bool valid = z < nz;
  const TLineIn in{fb + ((long)B.zb * n + r) * N2 * ZI + B.l0 + l, ZI};
  const TRowAdjOut<T> dst{out + ((long)(valid ? z : 0) * n + r) * n, phi + r * n, n, 1.0f / (float)N2, valid};
  fft_line_io<N2, true, RadonPlan<N2>>(in, SmCol<ZC>{smem + l}, dst, t, tw4);
}

// ================================================================ launch
template <int N2, int ZI, class T>
static cudaError_t tomo_R_sized(const T* obj, T* sino, const float* phi, float2* fa, float2* fde,
                                float2* gs, const GatherGeom& G, bool pairs, int nz, int ldz, const float2* tw_n,
                                const float2* tw_2n, const float* symx, cudaStream_t st) {
  constexpr int n = N2 / 2;
  constexpr int ZC = zc_of<N2, ZI>(), PARTS = ZI / ZC;
  using C2 = ZCfg<N2, ZC>;
  using C1 = ZCfg<n, ZC>;
  const int nzb = (nz + ZI - 1) / ZI;
  cudaError_t e;
  if ((e = allow_smem(k_trow_fwd<N2, ZI, T>, C2::SMEM)) != cudaSuccess) return e;
  if ((e = allow_smem(k_tcol_fwd<N2, ZI>, C2::SMEM)) != cudaSuccess) return e;
  if ((e = allow_smem(k_tsino_ifft<n, ZI, T>, C1::SMEM)) != cudaSuccess) return e;
  k_trow_fwd<N2, ZI, T><<<dim3(n * PARTS, nzb), C2::THREADS, C2::SMEM, st>>>(obj, phi, fa, nz, tw_2n);
  count_launch();
  k_tcol_fwd<N2, ZI><<<dim3(N2 * PARTS, nzb), C2::THREADS, C2::SMEM, st>>>(fa, fde, nz, tw_2n);
  count_launch();
  {
    KTimer kt("k_tgather", st, (double)nz);
    auto go = [&](auto kern, int na, int ga, int gr) {
      const int rt = (n + gr - 1) / gr, at = (G.ntheta + na * ga - 1) / (na * ga);
      kern<<<dim3(rt * at, nzb), kGatherThreads, 0, st>>>(fde, gs, G, nz, rt);
    };
    using T2 = GatherTile<ZI, 2>;
    using T1 = GatherTile<ZI, 1>;
    if (pairs)
      go(k_tgather<ZI, 2>, 2, T2::GA, T2::GR);
    else
      go(k_tgather<ZI, 1>, 1, T1::GA, T1::GR);
  }
  count_launch();
  k_tsino_ifft<n, ZI, T><<<dim3(G.ntheta * PARTS, nzb), C1::THREADS, C1::SMEM, st>>>(gs, sino, G.ntheta, nz, ldz, tw_n,
                                                                                symx);
  count_launch();
  return cudaGetLastError();
}

struct CellLists {
  const long* off;    // [n*n + 1] first entry of each tile's list
  const int* idx;     // sample indices
  const float4* wgt;  // weights of the tile's four cells
  const int* heavy;   // tiles with more than kHeavyList entries, longest first
  int nheavy;
};

template <int N2, int ZI, class T>
static cudaError_t tomo_RT_sized(const T* sino, T* obj, const float* phi, float2* fab, float2* fde,
                                 float2* gs, const GatherGeom& G, const CellLists& L, int nz, int ldz,
                                 const float2* tw_n,
                                 const float2* tw_2n, const float* symx, float scale, cudaStream_t st) {
  constexpr int n = N2 / 2;
  constexpr int ZC = zc_of<N2, ZI>(), PARTS = ZI / ZC;
  using C2 = ZCfg<N2, ZC>;
  using C1 = ZCfg<n, ZC>;
  const int nzb = (nz + ZI - 1) / ZI;
  cudaError_t e;
  if ((e = allow_smem(k_tsino_fft<n, ZI, T>, C1::SMEM)) != cudaSuccess) return e;
  if ((e = allow_smem(k_tcol_adj<N2, ZI>, C2::SMEM)) != cudaSuccess) return e;
  if ((e = allow_smem(k_trow_adj<N2, ZI, T>, C2::SMEM)) != cudaSuccess) return e;
  k_tsino_fft<n, ZI, T><<<dim3(G.ntheta * PARTS, nzb), C1::THREADS, C1::SMEM, st>>>(sino, gs, G.ntheta, nz, ldz, tw_n,
                                                                               symx, scale);
  count_launch();
  {
    KTimer kt("k_tcell", st, (double)nz);
    using TL = CellTile<ZI>;
    const int blocks = L.nheavy + ((n + TL::TX - 1) / TL::TX) * ((n + TL::TY - 1) / TL::TY);
    auto go = [&](auto kern, int zg) {
      const int ngroups = (nzb + zg - 1) / zg;
      kern<<<(unsigned)blocks * ngroups, kCellThreads, 0, st>>>(gs, fde, L.off, L.idx, L.wgt, L.heavy, L.nheavy, n,
                                                                (long)G.ntheta * n, nz, ngroups);
    };
    if (nzb > 1)
      go(k_tcell<ZI, 2>, 2);
    else
      go(k_tcell<ZI, 1>, 1);
  }
  count_launch();
  k_tcol_adj<N2, ZI><<<dim3(N2 * PARTS, nzb), C2::THREADS, C2::SMEM, st>>>(fde, fab, nz, tw_2n);
  count_launch();
  k_trow_adj<N2, ZI, T><<<dim3(n * PARTS, nzb), C2::THREADS, C2::SMEM, st>>>(fab, phi, obj, nz, tw_2n);
  count_launch();
  return cudaGetLastError();
}

#define HT_TOMO_SIZES(X) X(18, 36) X(24, 48) X(32, 64) X(48, 96) X(64, 128) X(96, 192) X(128, 256) \
  X(192, 384) X(256, 512) X(384, 768) X(512, 1024) X(768, 1536) X(1024, 2048) X(1536, 3072) X(2048, 4096)

}  // namespace ht

// ================================================================= C ABI
struct ht_tomo_s {
  int n, nz, ntheta, m, device;
  float mu;
  float* phi;          // [n, n] deapodisation * mask * norm (the reference's phi)
  float2* cs;          // [ntheta] (cos, sin) of the angles
  float* th_sorted;    // [ntheta] angles mod pi, ascending
  int* th_index;       // [ntheta]
  float2* fde;         // workspace [nzb][2n][2n][ZI]
  float2* fab;         // workspace [nzb][n][2n][ZI]
  float2* gs;          // workspace [nzb][ntheta][n][ZI]
  const float2* tw_n;
  const float2* tw_2n;
  long* cl_off;        // R^T lists: [n*n + 1] first entry of each 2 x 2 tile of cells
  int* cl_idx;         // [entries] sample index
  float4* cl_wgt;      // [entries] weights of the tile's four cells
  int* cl_heavy;       // [nheavy] tiles with long lists
  int nheavy;
  bool pairs;          // R gathers two angles at once (their lines lie within a few cells)
  float* symx;         // [n] 1 / (4 + 2 cos 2 pi k / n): the B-spline prefilter along the detector axis
};

namespace ht {
static cudaError_t build_cell_lists(ht_tomo_s* t);
}

static bool tomo_size_ok(int n) {
  switch (n) {
#define X(A, B) case A:
    HT_TOMO_SIZES(X)
#undef X
    return true;
    default:
      return false;
  }
}

static void tomo_free(ht_tomo_s* t) {
  cudaFree(t->phi);
  cudaFree(t->cs);
  cudaFree(t->th_sorted);
  cudaFree(t->th_index);
  cudaFree(t->fde);
  cudaFree(t->fab);
  cudaFree(t->gs);
  cudaFree(t->cl_off);
  cudaFree(t->cl_idx);
  cudaFree(t->cl_wgt);
  cudaFree(t->cl_heavy);
  cudaFree(t->symx);
}

extern "C" int ht_tomo_create(int n, int nz, int ntheta, const float* theta_host, const float* phi_host,
                              ht_tomo_s** out) {
  using namespace ht;
  HT_REQUIRE(out && theta_host && phi_host, "ht_tomo_create: null pointer");
  HT_REQUIRE(n > 0 && nz > 0 && ntheta > 0, "ht_tomo_create: sizes must be positive");
  if (!tomo_size_ok(n)) {
    set_error("ht_tomo_create: n must be one of 18,24,32,48,64,96,128,192,256,384,512,768,1024,1536,2048");
    return kUnsupported;
  }
  // USFFT parameters (tomo.py:14-16)
  const double eps = 1e-3;
  const double mu = -std::log(eps) / (2.0 * n * n);
  const int m = (int)std::ceil(2.0 * n / M_PI * std::sqrt(-mu * std::log(eps) + (mu * n) * (mu * n) / 4.0));
  if (m != 4) {
    set_error("ht_tomo_create: the gridding half-width m must be 4 (it is for every n >= 8)");
    return kUnsupported;
  }
  ht_tomo_s* t = new ht_tomo_s{};
  t->n = n;
  t->nz = nz;
  t->ntheta = ntheta;
  t->m = m;
  t->mu = (float)mu;
  cudaGetDevice(&t->device);
  std::vector<float2> cs(ntheta);
  std::vector<float> thm(ntheta);
  for (int i = 0; i < ntheta; ++i) {
    const double th = (double)theta_host[i];
    cs[i] = make_float2((float)std::cos(th), (float)std::sin(th));
    double r = std::fmod(th, M_PI);
    if (r < 0) r += M_PI;
    thm[i] = (float)r;
    if (thm[i] >= (float)M_PI) thm[i] = 0.f;
  }
  std::vector<int> idx(ntheta);
  std::iota(idx.begin(), idx.end(), 0);
  std::stable_sort(idx.begin(), idx.end(), [&](int a, int b) { return thm[a] < thm[b]; });
  std::vector<float> ths(ntheta);
  for (int i = 0; i < ntheta; ++i) ths[i] = thm[idx[i]];
  t->tw_n = twiddle_table(n, t->device);
  t->tw_2n = twiddle_table(2 * n, t->device);
  // two neighbouring angles' lines are at most n times their gap apart; up to
  // three cells their windows share most of a box (see k_tgather; 20 slices of 2048^2
  // at 1800 angles, 3.6 cells apart at the rim: 3.3 ms one by one, 3.6 in pairs)
  // Angles mod pi: over a full turn theta and theta + pi are neighbours, whose samples
  // of one radius lie on opposite sides.  They go one after the other, but in one
  // thread and over one line's cells: 64 slices of 512^2 at 900 angles over 2 pi take
  // 1.22 ms so and 1.25 in the order mod 2 pi one by one, at 1800 angles 2.08 and 2.06.
  int close = 0;
  for (int i = 0; i + 1 < ntheta; i += 2) close += (double)(ths[i + 1] - ths[i]) * n <= 3.0;
  t->pairs = 2 * close > ntheta / 2;
  const int run = first_run(n, nz), ZI = interleave(run);
  const size_t nzp = (size_t)((run + ZI - 1) / ZI) * ZI;
  cudaError_t e = cudaSuccess;
  auto alloc = [&](void** p, size_t b) {
    if (e == cudaSuccess) e = cudaMalloc(p, b);
  };
  alloc((void**)&t->phi, sizeof(float) * n * n);
  alloc((void**)&t->cs, sizeof(float2) * ntheta);
  alloc((void**)&t->th_sorted, sizeof(float) * ntheta);
  alloc((void**)&t->th_index, sizeof(int) * ntheta);
  alloc((void**)&t->fde, sizeof(float2) * nzp * 4 * n * n);
  alloc((void**)&t->fab, sizeof(float2) * nzp * 2 * n * n);
  alloc((void**)&t->gs, sizeof(float2) * nzp * ntheta * n);
  alloc((void**)&t->symx, sizeof(float) * n);
  std::vector<float> sx(n);
  for (int k = 0; k < n; ++k) sx[k] = (float)(1.0 / (4.0 + 2.0 * std::cos(2.0 * M_PI * k / n)));
  if (e == cudaSuccess) e = cudaMemcpy(t->phi, phi_host, sizeof(float) * n * n, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(t->cs, cs.data(), sizeof(float2) * ntheta, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(t->th_sorted, ths.data(), sizeof(float) * ntheta, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(t->th_index, idx.data(), sizeof(int) * ntheta, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(t->symx, sx.data(), sizeof(float) * n, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = build_cell_lists(t);
  if (e != cudaSuccess || !t->tw_n || !t->tw_2n) {
    if (e != cudaSuccess) set_error(std::string("ht_tomo_create: ") + cudaGetErrorString(e));
    cudaGetLastError();  // the next launch's check must not find this call's failure
    tomo_free(t);
    delete t;
    return kCudaError;
  }
  *out = t;
  return kOk;
}

extern "C" int ht_tomo_destroy(ht_tomo_s* t) {
  if (!t) return ht::kOk;
  tomo_free(t);
  delete t;
  return ht::kOk;
}

namespace ht {
static GatherGeom geom(const ht_tomo_s* t) {
  GatherGeom G;
  G.n = t->n;
  G.ntheta = t->ntheta;
  G.m = t->m;
  const float PI = 3.141592653589793238f;
  G.coeff0 = PI / t->mu;
  G.coeff1 = -PI * PI / t->mu;
  G.cs = t->cs;
  G.th_sorted = t->th_sorted;
  G.th_index = t->th_index;
  return G;
}

// The R^T lists (k_cell_count, k_cell_fill) on a private stream; the per-tile
// counts use the Fourier-grid workspace as scratch.
static cudaError_t build_cell_lists(ht_tomo_s* t) {
  const GatherGeom G = geom(t);
  const long ntiles = (long)t->n * t->n;
  int* cnt = reinterpret_cast<int*>(t->fde);
  cudaStream_t st = nullptr;
  cudaError_t e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
  if (e != cudaSuccess) return e;
  std::vector<int> len(ntiles), heavy;
  std::vector<long> off(ntiles + 1);
  const unsigned near_blocks = (unsigned)(near_side(t->n) * near_side(t->n) + 7) / 8;
  k_cell_near<false><<<near_blocks, 256, 0, st>>>(G, cnt, nullptr, nullptr, nullptr);
  count_launch();
  k_cell_count<<<(unsigned)((ntiles + 255) / 256), 256, 0, st>>>(G, cnt);
  count_launch();
  e = cudaMemcpyAsync(len.data(), cnt, sizeof(int) * ntiles, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e == cudaSuccess) {
    off[0] = 0;
    for (long i = 0; i < ntiles; ++i) {
      off[i + 1] = off[i] + len[i];
      if (len[i] > kHeavyList) heavy.push_back((int)i);
    }
    std::stable_sort(heavy.begin(), heavy.end(), [&](int a, int b) { return len[a] > len[b]; });
    t->nheavy = (int)heavy.size();
    const size_t tot = (size_t)std::max(off[ntiles], 4L);
    e = cudaMalloc(&t->cl_off, sizeof(long) * (ntiles + 1));
    if (e == cudaSuccess) e = cudaMalloc(&t->cl_heavy, sizeof(int) * std::max(t->nheavy, 1));
    if (e == cudaSuccess) e = cudaMalloc(&t->cl_idx, sizeof(int) * tot);
    if (e == cudaSuccess) e = cudaMalloc(&t->cl_wgt, sizeof(float4) * tot);
  }
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(t->cl_off, off.data(), sizeof(long) * (ntiles + 1), cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess && t->nheavy)
    e = cudaMemcpyAsync(t->cl_heavy, heavy.data(), sizeof(int) * t->nheavy, cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess) {
    k_cell_near<true><<<near_blocks, 256, 0, st>>>(G, nullptr, t->cl_off, t->cl_idx, t->cl_wgt);
    count_launch();
    k_cell_fill<<<(unsigned)((ntiles + 255) / 256), 256, 0, st>>>(G, t->cl_off, t->cl_idx, t->cl_wgt);
    count_launch();
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  cudaStreamDestroy(st);
  return e;
}
}  // namespace ht

namespace ht {
static CellLists lists(const ht_tomo_s* t) { return {t->cl_off, t->cl_idx, t->cl_wgt, t->cl_heavy, t->nheavy}; }

template <class F>
static cudaError_t by_interleave(int nz, F go) {
  switch (interleave(nz)) {
    case 16:
      return go(std::integral_constant<int, 16>{});
    case 8:
      return go(std::integral_constant<int, 8>{});
    default:
      return go(std::integral_constant<int, 4>{});
  }
}

template <class T>
static cudaError_t run_R(ht_tomo_s* t, const T* obj, T* sino, int nz, int ldz, const float* sym, cudaStream_t st) {
  const GatherGeom G = geom(t);
  switch (t->n) {
#define X(A, B)                                                                                                    \
  case A:                                                                                                          \
    return by_interleave(nz, [&](auto zi) {                                                                        \
      return tomo_R_sized<B, decltype(zi)::value, T>(obj, sino, t->phi, t->fab, t->fde, t->gs, G, t->pairs, nz,    \
                                                     ldz, t->tw_n, t->tw_2n, sym, st);                             \
    });
    HT_TOMO_SIZES(X)
#undef X
    default:
      return cudaErrorInvalidValue;
  }
}

template <class T>
static cudaError_t run_RT(ht_tomo_s* t, const T* sino, T* obj, int nz, int ldz, const float* sym, float scale,
                          cudaStream_t st) {
  const GatherGeom G = geom(t);
  switch (t->n) {
#define X(A, B)                                                                                                    \
  case A:                                                                                                          \
    return by_interleave(nz, [&](auto zi) {                                                                        \
      return tomo_RT_sized<B, decltype(zi)::value, T>(sino, obj, t->phi, t->fab, t->fde, t->gs, G, lists(t), nz,   \
                                                      ldz, t->tw_n, t->tw_2n, sym, scale, st);                     \
    });
    HT_TOMO_SIZES(X)
#undef X
    default:
      return cudaErrorInvalidValue;
  }
}

template <class T>
static int tomo_R(ht_tomo_s* t, const T* obj, T* sino, int nz, int ldz, const float* sym, void* stream) {
  HT_REQUIRE(t && obj && sino, "ht_tomo_R: null pointer");
  HT_REQUIRE(nz >= 0 && nz <= t->nz, "ht_tomo_R: nz exceeds the handle's slice capacity");
  HT_REQUIRE(ldz >= nz, "ht_tomo_R: ldz must be at least nz");
  if (nz == 0) return kOk;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int run = first_run(t->n, nz);
  const long n = t->n;
  HT_CHECK_CUDA(run_R(t, obj, sino, run, ldz, sym, st));
  if (run < nz) HT_CHECK_CUDA(run_R(t, obj + run * n * n, sino + run * n, nz - run, ldz, sym, st));
  return kOk;
}

template <class T>
static int tomo_RT(ht_tomo_s* t, const T* sino, T* obj, int nz, int ldz, const float* sym, float scale,
                   void* stream) {
  HT_REQUIRE(t && obj && sino, "ht_tomo_RT: null pointer");
  HT_REQUIRE(nz >= 0 && nz <= t->nz, "ht_tomo_RT: nz exceeds the handle's slice capacity");
  HT_REQUIRE(ldz >= nz, "ht_tomo_RT: ldz must be at least nz");
  if (nz == 0) return kOk;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int run = first_run(t->n, nz);
  const long n = t->n;
  HT_CHECK_CUDA(run_RT(t, sino, obj, run, ldz, sym, scale, st));
  if (run < nz) HT_CHECK_CUDA(run_RT(t, sino + run * n, obj + run * n * n, nz - run, ldz, sym, scale, st));
  return kOk;
}

static int tomo_R_c(ht_tomo_s* t, const void* obj, void* sino, int nz, int ldz, bool coeffx, void* stream) {
  HT_REQUIRE(t, "ht_tomo_R: null pointer");
  return tomo_R(t, static_cast<const float2*>(obj), static_cast<float2*>(sino), nz, ldz, coeffx ? t->symx : nullptr,
                stream);
}
static int tomo_RT_c(ht_tomo_s* t, const void* sino, void* obj, int nz, int ldz, bool coeffx, float scale,
                     void* stream) {
  HT_REQUIRE(t, "ht_tomo_RT: null pointer");
  return tomo_RT(t, static_cast<const float2*>(sino), static_cast<float2*>(obj), nz, ldz, coeffx ? t->symx : nullptr,
                 scale, stream);
}
}  // namespace ht

extern "C" int ht_tomo_R(ht_tomo_s* t, const void* obj, void* sino, int nz, void* stream) {
  return ht::tomo_R_c(t, obj, sino, nz, nz, false, stream);
}

extern "C" int ht_tomo_RT(ht_tomo_s* t, const void* sino, void* obj, int nz, void* stream) {
  return ht::tomo_RT_c(t, sino, obj, nz, nz, false, 1.0f, stream);
}

extern "C" int ht_tomo_R_coeffx(ht_tomo_s* t, const void* obj, void* sino, int nz, void* stream) {
  return ht::tomo_R_c(t, obj, sino, nz, nz, true, stream);
}

extern "C" int ht_tomo_RT_coeffx(ht_tomo_s* t, const void* sino, void* obj, int nz, float scale, void* stream) {
  return ht::tomo_RT_c(t, sino, obj, nz, nz, true, scale, stream);
}

extern "C" int ht_tomo_R_slab(ht_tomo_s* t, const void* obj, void* sino, int nz, int ldz, int coeffx, void* stream) {
  return ht::tomo_R_c(t, obj, sino, nz, ldz, coeffx != 0, stream);
}

extern "C" int ht_tomo_RT_slab(ht_tomo_s* t, const void* sino, void* obj, int nz, int ldz, int coeffx, float scale,
                               void* stream) {
  return ht::tomo_RT_c(t, sino, obj, nz, ldz, coeffx != 0, scale, stream);
}

extern "C" int ht_tomo_R_real(ht_tomo_s* t, const float* obj, float* sino, int nz, int ldz, void* stream) {
  return ht::tomo_R<float>(t, obj, sino, nz, ldz, nullptr, stream);
}

extern "C" int ht_tomo_RT_filter(ht_tomo_s* t, const void* sino, void* obj, int nz, int ldz, int is_real,
                                 const float* sym, float scale, void* stream) {
  if (is_real)
    return ht::tomo_RT(t, static_cast<const float*>(sino), static_cast<float*>(obj), nz, ldz, sym, scale, stream);
  return ht::tomo_RT(t, static_cast<const float2*>(sino), static_cast<float2*>(obj), nz, ldz, sym, scale, stream);
}
