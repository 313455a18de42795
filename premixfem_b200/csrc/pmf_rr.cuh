// Small dense Rayleigh-Ritz problems, one warp each: the lowest m eigenpairs of
// the pencil (GA, GM) of order n <= NX <= 32.
//
// These problems (the projected problems of the local eigensolves, 16..30
// unknowns, and of the level-3 eigensolves, 4..16) are chains of short
// dependent steps, so they are bound by latency.  One warp per problem, lane l
// holding row l of the current matrix in registers, replaces CTA barriers by
// warp-synchronous steps and lets a dozen problems share an SM.  Against one CTA
// of 256 threads per problem: 64 problems of 18 unknowns 52 us a launch instead
// of 95, the 38 iterations of 512 problems of 24 unknowns 3.5 ms instead of
// 10.0, the 86 of 1 728 problems in FP64 storage 8.6 ms instead of 31.1.  Every
// loop over pivots is rolled: the registers shift by one column per step (the
// shift is the destination of the update's multiply-add), so all register indices
// are compile-time constants and the code stays small enough for the instruction
// cache.
#pragma once

#include "pmf_dense.cuh"

namespace pmf {

template <int NX, int MX>
struct __align__(16) WarpRR {
  double Lc[NX * NX];       // Lc[c*NX + j] = L[c+j][c] (columns of the factor, shifted), later free
  double B[NX * (NX + 1)];  // transposes; the reflectors
  double lu[4 * NX * MX];   // tridiagonal factors of the inverse iteration, [i*MX + vector]
  double z[NX * MX];        // eigenvectors of the tridiagonal matrix, [i*MX + vector]
  double dsc[NX], inv[NX], dg[NX], of[NX], beta[NX], ws[NX], lam[MX], ds[36], es[36];
};

// Lowest m eigenpairs (m <= MX) of the symmetric q x q matrix whose row l lane l
// holds in a[] (zero past q): eigenvalues to s.lam (ascending), eigenvectors to
// s.z.  Hv: NX*NX doubles for the reflectors.
//   1. Householder tridiagonalisation (Golub & Van Loan, Alg. 8.3.1);
//   2. eigenvalues by multisection: 32/m lanes per eigenvalue, two points each;
//      the Sturm count is the number of sign changes of the leading principal
//      minors (Givens' recurrence, one dependent multiply-add per row instead
//      of a division; rescaled every four rows);
//   3. eigenvectors by inverse iteration, one lane per vector, then Gram-Schmidt
//      in ascending order and back-transformation.
template <int NX, int MX>
__device__ __forceinline__ void warp_sym_lowest(WarpRR<NX, MX>& s, double (&a)[NX], int q, int m, double* Hv) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  // ---- 1. tridiagonalisation: at step k, a[j] = A[lane][k + j]
  for (int k = 0; k + 2 < q; ++k) {
    const double dk = __shfl_sync(full, a[0], k);
    const double x = (lane > k && lane < q) ? a[0] : 0.0;
    const double nrm2 = warp_sum(x * x);
    const double x0 = __shfl_sync(full, x, k + 1);
    double b = 0.0, alpha = x0, v = 0.0;
    if (nrm2 > 1e-300) {
      const double nrm = nrm2 * rsqrt(nrm2);
      alpha = x0 >= 0.0 ? -nrm : nrm;
      b = __drcp_rn(nrm2 + fabs(x0) * nrm);  // 2 / v^T v
      v = lane == k + 1 ? x0 - alpha : x;
    }
    if (lane == 0) {
      s.dg[k] = dk;
      s.of[k] = alpha;
      s.beta[k] = b;
    }
    const double vsh = __shfl_sync(full, v, (k + lane) & 31);
    if (lane < NX) Hv[k * NX + lane] = k + lane < q ? vsh : 0.0;  // Hv[k*NX + j] = v[k + j]
    __syncwarp();
    const double* vk = Hv + k * NX;
    double p0 = 0.0, p1 = 0.0, p2 = 0.0, p3 = 0.0;
#pragma unroll
    for (int j = 1; j < NX; ++j) {
      const double t = vk[j];
      if (j % 4 == 0) p0 += a[j] * t;
      else if (j % 4 == 1) p1 += a[j] * t;
      else if (j % 4 == 2) p2 += a[j] * t;
      else p3 += a[j] * t;
    }
    const double p = lane > k ? b * ((p0 + p1) + (p2 + p3)) : 0.0;
    const double K = 0.5 * b * warp_sum(p * v);
    const double w = p - K * v;
    const double wsh = __shfl_sync(full, w, (k + lane) & 31);
    if (lane < NX) s.ws[lane] = k + lane < q ? wsh : 0.0;
    __syncwarp();
#pragma unroll
    for (int j = 1; j < NX; ++j) a[j - 1] = a[j] - v * s.ws[j] - w * vk[j];
    a[NX - 1] = 0.0;
    __syncwarp();
  }
  {
    // the trailing 2 x 2 block (or the 1 x 1 matrix)
    const int k = max(0, q - 2);
    const double d0 = __shfl_sync(full, a[0], k);
    const double d1 = __shfl_sync(full, a[1], min(k + 1, 31));
    const double o = __shfl_sync(full, a[0], min(k + 1, 31));
    if (lane == 0) {
      s.dg[k] = d0;
      s.of[k] = 0.0;
      if (q > 1) {
        s.of[k] = o;
        s.dg[k + 1] = d1;
        s.of[k + 1] = 0.0;
      }
    }
  }
  __syncwarp();
  // ---- 2. eigenvalues; T is scaled by its Gershgorin radius for the counts
  double gl = 1e300, gh = -1e300, gm = 0.0;
  if (lane < q) {
    const double r = (lane > 0 ? fabs(s.of[lane - 1]) : 0.0) + fabs(s.of[lane]);
    gl = s.dg[lane] - r;
    gh = s.dg[lane] + r;
    gm = fabs(s.dg[lane]) + r;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    gl = fmin(gl, __shfl_xor_sync(full, gl, o));
    gh = fmax(gh, __shfl_xor_sync(full, gh, o));
    gm = fmax(gm, __shfl_xor_sync(full, gm, o));
  }
  // a matrix of zeros (a floating rank of one unknown) has its scale set to one: the inverse
  // iteration's growth, up to 1e19 / emax, is squared below
  const double emax = gm > 1e-100 ? gm : 1.0, isc = 1.0 / emax;
  // scaled diagonal, and squared couplings to the row before: at least 1e-36, a
  // coupling of 1e-18, which is below the rounding of T
  double *ds = s.ds, *es = s.es;
  {
    const double e = (lane > 0 && lane < q) ? s.of[lane - 1] * isc : 0.0;
    ds[lane] = lane < q ? s.dg[lane] * isc : 4.0;
    es[lane] = lane < q ? fmax(e * e, 1e-36) : 0.0;
    if (lane < 4) {
      ds[32 + lane] = 4.0;
      es[32 + lane] = 0.0;
    }
  }
  __syncwarp();
  {
    const int P = 32 / m;  // lanes per eigenvalue
    const int ge = min(lane / P, m - 1), part = lane % P;
    const bool live = lane < P * m;
    const unsigned gmask = (P >= 32 ? full : ((1u << P) - 1u));
    const double pad = 1e-14;
    double lo = gl * isc - pad, hi = gh * isc + pad;
    const double rs = 1.0 / (2 * P + 1);
    for (int round = 0; round < 48; ++round) {
      const bool open = hi - lo > 1e-14 * fmax(fabs(lo), fabs(hi)) + 1e-17;
      if (!__any_sync(full, open && live)) break;
      const double x0 = lo + (hi - lo) * ((2 * part + 1) * rs), x1 = lo + (hi - lo) * ((2 * part + 2) * rs);
      int c0 = 0, c1 = 0;
      double pa = 1.0, pb = ds[0] - x0, ra = 1.0, rb = ds[0] - x1;
      c0 += pb < 0.0;
      c1 += rb < 0.0;
      for (int i0 = 1; i0 < q; i0 += 4) {  // past q: a positive diagonal, no coupling, no sign change
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const double d = ds[i0 + u], e = es[i0 + u];
          const double pn = (d - x0) * pb - e * pa;
          const double rn = (d - x1) * rb - e * ra;
          c0 += (pn < 0.0) != (pb < 0.0);
          c1 += (rn < 0.0) != (rb < 0.0);
          pa = pb;
          pb = pn;
          ra = rb;
          rb = rn;
        }
        if (fabs(pa) + fabs(pb) < 1e-120) {
          pa *= 1e120;
          pb *= 1e120;
        }
        if (fabs(ra) + fabs(rb) < 1e-120) {
          ra *= 1e120;
          rb *= 1e120;
        }
      }
      const unsigned b0 = (__ballot_sync(full, live && c0 > ge) >> (ge * P)) & gmask;
      const unsigned b1 = (__ballot_sync(full, live && c1 > ge) >> (ge * P)) & gmask;
      // first point whose count exceeds the eigenvalue's index
      int f = 2 * P;
      if (b0) f = min(f, 2 * (__ffs(b0) - 1));
      if (b1) f = min(f, 2 * (__ffs(b1) - 1) + 1);
      const double w = hi - lo, nlo = f == 0 ? lo : lo + w * (f * rs), nhi = f == 2 * P ? hi : lo + w * ((f + 1) * rs);
      if (open) {
        lo = nlo;
        hi = nhi;
      }
    }
    if (live && part == 0) s.lam[ge] = 0.5 * (lo + hi) * emax;
  }
  __syncwarp();
  // ---- 3. inverse iteration, one lane per eigenvector (tridiagonal LU with partial pivoting)
  if (lane < m) {
    double* __restrict__ dl = s.lu + lane;
    double* __restrict__ rd = s.lu + NX * MX + lane;  // reciprocal pivots
    double* __restrict__ du = s.lu + 2 * NX * MX + lane;
    double* __restrict__ du2 = s.lu + 3 * NX * MX + lane;
    double* __restrict__ z = s.z + lane;
    const double lam = s.lam[lane] - 4e-15 * emax * (1 + lane);
    const double tiny = 1e-300 + 1e-16 * emax * 1e-3;
    unsigned piv = 0;
    double dcur = s.dg[0] - lam, ucur = q > 1 ? s.of[0] : 0.0;
    for (int i = 0; i < q; ++i) {
      const bool more = i + 1 < q;
      const double sub = more ? s.of[i] : 0.0;  // below the pivot
      const double dnext = more ? s.dg[i + 1] - lam : 0.0, unext = i + 2 < q ? s.of[i + 1] : 0.0;
      double dd = dcur, uu = ucur, u2 = 0.0, f = 0.0;
      if (more && !(fabs(dcur) >= fabs(sub))) {  // exchange rows i and i+1
        piv |= 1u << i;
        f = dcur * __drcp_rn(sub);
        dd = sub;
        uu = dnext;
        u2 = unext;
        const double t = ucur - f * dnext;
        ucur = -f * unext;
        dcur = t;
      } else if (more) {
        f = dcur != 0.0 ? sub * __drcp_rn(dcur) : 0.0;
        dcur = dnext - f * ucur;
        ucur = unext;
      }
      if (fabs(dd) < tiny) dd = dd < 0.0 ? -tiny : tiny;
      dl[i * MX] = f;
      rd[i * MX] = __drcp_rn(dd);
      du[i * MX] = uu;
      du2[i * MX] = u2;
      z[i * MX] = hash_uniform(0x5bd1e995ull * (lane + 1) + i);
    }
    for (int itr = 0; itr < 3; ++itr) {
      double zc = z[0];
#pragma unroll 4
      for (int i = 0; i + 1 < q; ++i) {
        const double zn = z[(i + 1) * MX], f = dl[i * MX];
        const bool ex = (piv >> i) & 1;
        const double top = ex ? zn : zc, bot = ex ? zc : zn;
        z[i * MX] = top;
        zc = bot - f * top;
      }
      double z1 = 0.0, z2 = 0.0, nrm = 0.0;
#pragma unroll 4
      for (int i = q - 1; i >= 0; --i) {
        double t = i == q - 1 ? zc : z[i * MX];
        t -= du2[i * MX] * z2;
        t = (t - du[i * MX] * z1) * rd[i * MX];
        z[i * MX] = t;
        nrm += t * t;
        z2 = z1;
        z1 = t;
      }
      nrm = rsqrt(fmax(nrm, 1e-300));
#pragma unroll 4
      for (int i = 0; i < q; ++i) z[i * MX] *= nrm;
    }
  }
  __syncwarp();
  // Gram-Schmidt in ascending order, each vector against all before it at once, twice
  {
    double zv[MX];
#pragma unroll
    for (int j = 0; j < MX; ++j) zv[j] = (j < m && lane < q) ? s.z[lane * MX + j] : 0.0;
#pragma unroll
    for (int j = 0; j < MX; ++j) {
      if (j < m) {
#pragma unroll 1
        for (int rep = 0; rep < (j > 0 ? 2 : 0); ++rep) {
          double d[MX];
#pragma unroll
          for (int i = 0; i < MX; ++i)
            if (i < j) d[i] = zv[i] * zv[j];
#pragma unroll
          for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int i = 0; i < MX; ++i)
              if (i < j) d[i] += __shfl_xor_sync(full, d[i], o);
#pragma unroll
          for (int i = 0; i < MX; ++i)
            if (i < j) zv[j] -= d[i] * zv[i];
        }
        zv[j] *= rsqrt(fmax(warp_sum(zv[j] * zv[j]), 1e-300));
      }
    }
    if (lane < q) {
#pragma unroll
      for (int j = 0; j < MX; ++j)
        if (j < m) s.z[lane * MX + j] = zv[j];
    }
  }
  __syncwarp();
  // back-transformation y = P_0 P_1 ... P_{q-3} z: PB lanes per vector, rows part, part + PB, ...
  constexpr int PB = MX <= 8 ? 4 : 2;
  constexpr int RB = (NX + PB - 1) / PB;
  {
    const int vec = min(lane / PB, m - 1), part = lane % PB;
    double zr[RB];
#pragma unroll
    for (int t = 0; t < RB; ++t) {
      const int i = part + PB * t;
      zr[t] = i < q ? s.z[i * MX + vec] : 0.0;
    }
    for (int k = q - 3; k >= 0; --k) {
      const double b = s.beta[k];
      const double* vk = Hv + k * NX - k;  // vk[i] = v_k[i], i > k
      double v[RB], d = 0.0;
#pragma unroll
      for (int t = 0; t < RB; ++t) {
        const int i = part + PB * t;
        v[t] = (i > k && i < q) ? vk[i] : 0.0;
        d += v[t] * zr[t];
      }
#pragma unroll
      for (int o = 1; o < PB; o <<= 1) d += __shfl_xor_sync(full, d, o);
      d *= b;
#pragma unroll
      for (int t = 0; t < RB; ++t) zr[t] -= d * v[t];
    }
    __syncwarp();
    if (lane < PB * m) {
#pragma unroll
      for (int t = 0; t < RB; ++t) {
        const int i = part + PB * t;
        if (i < q) s.z[i * MX + vec] = zr[t];
      }
    }
  }
  __syncwarp();
}

// Rayleigh-Ritz on a basis of n vectors with Gram matrices GM (in M) and GA (in
// A): load(0, a) and load(1, a) fill a[j] with GM[j][lane] and GA[j][lane] (zero
// where j or lane is not below n).  Y (n x min(m, rank), leading dimension
// ldy) gets the M-orthonormal coefficients of the lowest Ritz vectors, s.lam
// their Ritz values.  Returns the kept rank.
//
// The basis is scaled to unit M-norm, D = diag(GM)^-1/2; Cholesky D GM D = L L^T
// and H = L^-1 (D GA D) L^-T by two substitutions.  A vector whose pivot is at or
// below `drop` depends on the ones before it and leaves the basis (its row of H is
// decoupled above the spectrum), so a nearly dependent basis costs little more than
// another one.  A pivot d is known to eps / d, and one of that size enters the later
// ones as eps / sqrt(d): below eps^(2/3) it can lift a dependent vector's pivot over
// `drop`, and its Ritz value is noise.  So as soon as one vector is dropped the
// factorisation is repeated with the pivots held above 1e-9.
template <int NX, int MX, class F>
__device__ __forceinline__ int warp_rayleigh_ritz(WarpRR<NX, MX>& s, int n, int m, double drop, F load, double* Y,
                                                  int ldy) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  constexpr int LB = NX + 1;
  double a[NX];
  load(0, a);
  double dl = 0.0;
#pragma unroll
  for (int j = 0; j < NX; ++j)
    if (j == lane) dl = a[j];
  double mx = dl;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(full, mx, o));
  const double dsc = (lane < n && dl > 1e-28 * mx) ? 1.0 / sqrt(dl) : 0.0;
  if (lane < NX) s.dsc[lane] = dsc;
  __syncwarp();
  // Cholesky, right-looking: at step c, a[j] = (trailing matrix)[lane][c + j]
  unsigned kept = 0;
#pragma unroll 1
  for (double least = drop;; least = 1e-9) {
    if (kept) load(0, a);
    __syncwarp();
#pragma unroll
    for (int j = 0; j < NX; ++j) a[j] *= dsc * s.dsc[j];
    kept = 0;
    for (int c = 0; c < n; ++c) {
      const double d = __shfl_sync(full, a[0], c);
      const bool keep = d > least && s.dsc[c] != 0.0;
      const double r = keep ? rsqrt(d) : 0.0;
      const double lc = lane > c ? a[0] * r : (lane == c && keep ? d * r : 0.0);
      const double lsh = __shfl_sync(full, lc, (c + lane) & 31);
      if (lane < NX) s.Lc[c * NX + lane] = c + lane < n ? lsh : 0.0;
      if (lane == 0) s.inv[c] = r;
      kept |= (keep ? 1u : 0u) << c;
      __syncwarp();
#pragma unroll
      for (int j = 1; j < NX; ++j) a[j - 1] = a[j] - lc * s.Lc[c * NX + j];
      a[NX - 1] = 0.0;
    }
    if (kept == 0 || __popc(kept) == n || least >= 1e-9) break;
  }
  const int q = __popc(kept);
  // B = D GA D, symmetrised
  load(1, a);
#pragma unroll
  for (int j = 0; j < NX; ++j) {
    a[j] *= dsc * s.dsc[j];
    if (lane < NX) s.B[j * LB + lane] = a[j];
  }
  __syncwarp();
  if (lane < NX) {
#pragma unroll
    for (int j = 0; j < NX; ++j) a[j] = 0.5 * (a[j] + s.B[lane * LB + j]);
  }
  __syncwarp();
#pragma unroll 1
  for (int pass = 0; pass < 2; ++pass) {  // W = L^-1 B by columns (lane = column), then L^-1 W^T
    for (int i = 0; i < n; ++i) {
      const double x = a[0] * s.inv[i];
      if (lane < NX) s.B[i * LB + lane] = x;
#pragma unroll
      for (int j = 1; j < NX; ++j) a[j - 1] = a[j] - s.Lc[i * NX + j] * x;
      a[NX - 1] = 0.0;
    }
    __syncwarp();
#pragma unroll
    for (int j = 0; j < NX; ++j) {
      a[j] = (j < n && lane < n) ? s.B[lane * LB + j] : 0.0;
      if (pass == 1 && j < n && lane < n) a[j] = 0.5 * (a[j] + s.B[j * LB + lane]);
    }
    __syncwarp();
  }
  if (q < n) {
    double rsum = 0.0;
#pragma unroll
    for (int j = 0; j < NX; ++j) rsum += fabs(a[j]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) rsum = fmax(rsum, __shfl_xor_sync(full, rsum, o));
#pragma unroll
    for (int j = 0; j < NX; ++j)
      if (j == lane && j < n && !((kept >> j) & 1u)) a[j] = 1.0001 * rsum + 1e-300;
  }
  const int mm = min(m, q);
  if (mm == 0) return 0;
  warp_sym_lowest<NX, MX>(s, a, n, mm, s.B);
  // Y = D L^-T z, one lane per vector: at step i, a[j] = (remaining right-hand side)[i - j]
  if (lane < mm) {
#pragma unroll
    for (int j = 0; j < NX; ++j) a[j] = j < n ? s.z[(n - 1 - j) * MX + lane] : 0.0;
    for (int i = n - 1; i >= 0; --i) {
      const double y = a[0] * s.inv[i];
      Y[i * ldy + lane] = s.dsc[i] * y;
#pragma unroll
      for (int j = 1; j < NX; ++j) a[j - 1] = j <= i ? a[j] - s.Lc[(i - j) * NX + j] * y : 0.0;
    }
  }
  __syncwarp();
  return q;
}

}  // namespace pmf
