// The 7-point operator over the whole mesh as a short march in z.
//
// A CTA owns a run of 256 places along the rows of the x-y plane and walks zc
// planes: the value and the z coupling of the plane above become those of the plane
// below, so each is loaded once per march instead of at three planes, and the x and
// y neighbours come from L1 and L2.  Runs along the rows leave no thread idle on any
// mesh; tiles of 32 x 8 places, which keep the y neighbours of wide meshes in L1,
// measured the same there (operator at 256^3 146 us either way) and slower where they
// do not fit: 59 us against 50 at 161 x 163 x 157, 99 against 50 at 8 x 512 x 1024,
// the CG step 212 against 58 at 2048 x 1 x 2048.  Bound by HBM.  The loop is unrolled twice, which puts the next plane's loads
// in flight before this plane's arithmetic (the CG step at 256^3: unrolled once
// 289 us, twice 183, four times 252; one plane per CTA 238) provided the output
// pointers are __restrict__.  Sixteen planes,
// which spread the CTA's first loads (the CG scalars) over the march, where
// that leaves sixteen CTAs per SM, else the power of two that does.
#pragma once

#include "pmf_kernels.h"

namespace pmf {

constexpr int kStX = 32, kStY = 8;

struct StencilShape {
  dim3 grid;
  int zc;
  int blocks() const { return (int)(grid.x * grid.y); }
};
inline StencilShape stencil_shape(const Grid& g) {
  StencilShape s;
  const long long runs = (g.MN + kStX * kStY - 1) / (kStX * kStY);
  s.zc = 16;
  while (s.zc > 1 && runs * ((g.P + s.zc - 1) / s.zc) < 16 * 148) s.zc /= 2;
  while ((g.P + s.zc - 1) / s.zc > 65535) s.zc *= 2;
  s.grid = dim3((unsigned)runs, (g.P + s.zc - 1) / s.zc);  // y: stretches of planes
  return s;
}

// this thread's (x, y) in the blockIdx.x-th run of 256 places along the rows
__device__ __forceinline__ int2 stencil_xy(const Grid& g) {
  const unsigned c = (blockIdx.x * kStY + threadIdx.y) * kStX + threadIdx.x, y = c / (unsigned)g.M;
  return make_int2((int)(c - y * g.M), (int)y);
}

// out(c, v, a) with v = val(c) and a = (A v)(c), evaluated in the order diagonal, x-, x+, y-, y+, z-, z+, for the
// cells of this thread's column with z0 <= ez < z1
template <typename T, class V, class O>
__device__ __forceinline__ void stencil_march(const Grid& g, const T* __restrict__ tx, const T* __restrict__ ty,
                                              const T* __restrict__ tz, const T* __restrict__ diag, int z0, int z1,
                                              V val, O out) {
  const int2 xy = stencil_xy(g);
  const int ex = xy.x, ey = xy.y;
  if (ex >= g.M || ey >= g.N) return;
  const bool xm = ex > 0, xp = ex < g.M - 1, ym = ey > 0, yp = ey < g.N - 1;
  long long c = (long long)z0 * g.MN + (long long)ey * g.M + ex;
  T vm = z0 > 0 ? val(c - g.MN) : (T)0, vc = val(c), tzc = tz[c];
#pragma unroll 2
  for (int ez = z0; ez < z1; ++ez) {
    const bool zp = ez < g.P - 1;
    const T vp = zp ? val(c + g.MN) : (T)0, tzp = zp ? tz[c + g.MN] : (T)0;
    T a = diag[c] * vc;
    if (xm) a -= tx[c] * val(c - 1);
    if (xp) a -= tx[c + 1] * val(c + 1);
    if (ym) a -= ty[c] * val(c - g.M);
    if (yp) a -= ty[c + g.M] * val(c + g.M);
    if (ez > 0) a -= tzc * vm;
    if (zp) a -= tzp * vp;
    out(c, vc, a);
    vm = vc;
    vc = vp;
    tzc = tzp;
    c += g.MN;
  }
}

// sum over a CTA of 32 x 8 threads in a fixed order, valid in thread (0, 0)
__device__ __forceinline__ double stencil_sum(double v) {
  __shared__ double red[kStY];
  v = warp_sum(v);
  if (threadIdx.x == 0) red[threadIdx.y] = v;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x == 0 && threadIdx.y == 0) {
#pragma unroll
    for (int i = 0; i < kStY; ++i) t += red[i];
  }
  return t;
}

}  // namespace pmf
