// Coarse-space kernels (FP64): level-2 Galerkin assembly, batched dense SPD
// inverses, the level-3 eigenproblem and the small coarse products used by the
// cycle executor.
#include <algorithm>
#include <cstdio>

#include "pmf_dense.cuh"
#include "pmf_kernels.h"
#include "pmf_rr.cuh"

namespace pmf {

// ---- coarse products over ranks of different sizes (RankLayout) -------------
__device__ __forceinline__ int rank_nr(const RankLayout& L, int r) { return (L.first[r + 1] - L.first[r]) * L.kmax; }
__device__ __forceinline__ long long rank_dof0(const RankLayout& L, int r) { return (long long)L.first[r] * L.kmax; }
// the rank whose range [off[r], off[r+1]) holds e (binary search)
__device__ __forceinline__ int rank_of(const long long* off, int nrank, long long e) {
  int lo = 0, hi = nrank - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (off[mid] <= e)
      lo = mid;
    else
      hi = mid - 1;
  }
  return lo;
}

// The cycle's coarse visits are short and follow one another, so they are bound
// by launches and the latency of a few dependent loads: one launch for the
// level-2 product with its accumulation into Z, one for the coarse residual's
// update with the level-3 restriction, and one for the level-3 solve with its
// prolongation and accumulation; five launches a V-cycle instead of ten.
// Coarse part of an iteration: 33 us instead of 53 (one rank of 256 unknowns),
// 40 instead of 72 (eight of 384), 100 instead of 153 (four of 2 244, whose two
// products with the inverses stream 161 MB each).

// Rows go in chunks of kCoarseRows within one rank, one CTA each; a chunk's table entry holds all a CTA
// needs to start loading, so that no chain of index loads precedes the data.

// out[g] = sum_j inv_r[i][j] in[dof0_r + j] for coarse dof g = dof0_r + i, four rows per warp at a time;
// Z = out (first) or Z += out
__global__ void __launch_bounds__(256) k_block_gemv_r(const CoarseChunk* chunks, const double* inv, const double* in,
                                                      double* out, double* Z, int first, const int* done) {
  if (done && *done) return;
  const CoarseChunk ch = chunks[blockIdx.x];
  const int lane = threadIdx.x & 31, i0 = (threadIdx.x >> 5) * 4;
  if (i0 >= ch.rows) return;
  const double* x = in + ch.dof0;
  const double* A = inv + ch.a_off + (long long)i0 * ch.nr;
  const int n1 = min(1, ch.rows - 1 - i0), n2 = min(2, ch.rows - 1 - i0), n3 = min(3, ch.rows - 1 - i0);
  double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;  // rows past the chunk repeat its last one
#pragma unroll 4
  for (int j = lane; j < ch.nr; j += 32) {
    const double v = x[j];
    a0 += A[j] * v;
    a1 += A[(long long)n1 * ch.nr + j] * v;
    a2 += A[(long long)n2 * ch.nr + j] * v;
    a3 += A[(long long)n3 * ch.nr + j] * v;
  }
  a0 = warp_sum(a0);
  a1 = warp_sum(a1);
  a2 = warp_sum(a2);
  a3 = warp_sum(a3);
  if (lane < 4 && i0 + lane < ch.rows) {
    const double v = lane == 0 ? a0 : lane == 1 ? a1 : lane == 2 ? a2 : a3;
    const long long g = ch.g0 + i0 + lane;
    out[g] = v;
    Z[g] = first ? v : Z[g] + v;
  }
}
void launch_block_gemv_r(const RankLayout& L, const double* inv, const double* in, double* out, double* Z, int first,
                         const int* done, cudaStream_t st) {
  { note_launch(); k_block_gemv_r<<<L.nchunk, 256, 0, st>>>(L.chunks, inv, in, out, Z, first, done); }
}

// c -= A2 dz (when dz is given) with A2 = Phi^T A Phi stored as 7 kmax x kmax
// blocks per subdomain row (diagonal + six face neighbours), then, when V is
// given, this chunk of rows' part of the level-3 restriction
// part[chunk][j] = sum_i V[i][j] c[i].  Eight lanes per row, a block each.
__global__ void __launch_bounds__(256) k_coarse_resid(const CoarseChunk* chunks, const SubInfo* subs, int kmax,
                                                      const double* blk, const double* dz, double* c, int en2,
                                                      const double* V, double* part, const int* done) {
  if (done && *done) return;
  __shared__ double cs[kCoarseRows];
  const CoarseChunk ch = chunks[blockIdx.x];
  const int b = threadIdx.x & 7, q = threadIdx.x >> 3;
  const long long g = ch.g0 + q;
  double acc = 0.0;
  if (q < ch.rows && dz) {
    const int s = (int)(g / kmax), i = (int)(g - (long long)s * kmax);
    const int nb = b == 0 ? s : (b < 7 ? subs[s].nb[b - 1] : -1);
    if (nb >= 0) {
      const double* B = blk + (((long long)s * 7 + b) * kmax + i) * kmax;
      const double* v = dz + (long long)nb * kmax;
#pragma unroll 8
      for (int j = 0; j < kmax; ++j) acc += B[j] * v[j];
    }
  }
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (b == 0 && q < ch.rows) {
    const double v = c[g] - acc;
    if (dz) c[g] = v;
    cs[q] = v;
  }
  if (!V) return;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  static_assert(kCoarseRows == 32, "a lane per row");
  for (int j = threadIdx.x >> 5; j < en2; j += 8) {
    const double v = warp_sum(lane < ch.rows ? V[ch.v_off + (long long)lane * en2 + j] * cs[lane] : 0.0);
    if (lane == 0) part[(long long)blockIdx.x * en2 + j] = v;
  }
}
void launch_coarse_resid(const RankLayout& L, const SubInfo* subs, const double* blk, const double* dz, double* c,
                         int en2, const double* V, double* part, const int* done, cudaStream_t st) {
  { note_launch(); k_coarse_resid<<<L.nchunk, 256, 0, st>>>(L.chunks, subs, L.kmax, blk, dz, c, en2, V, part, done); }
}

// Level-3 solve and prolongation for this chunk of rows: d = the ranks' sums of
// part, w = the rank's rows of A3^-1 d, dz = V w, Z = dz (first) or Z += dz.
// Every CTA adds up d (gs lanes per entry) and forms its rank's en2 entries of w itself.
__global__ void __launch_bounds__(256) k_lv3_solve(const CoarseChunk* chunks, const int* chunk_first, int n3, int en2,
                                                   int gs, const double* part, const double* A3inv, const double* V,
                                                   double* dz, double* Z, int first, const int* done) {
  if (done && *done) return;
  extern __shared__ double l3s[];
  double* d = l3s;       // n3
  double* w = l3s + n3;  // en2
  const CoarseChunk ch = chunks[blockIdx.x];
  const int lane = threadIdx.x & 31, gl = threadIdx.x % gs;
  for (int e0 = 0; e0 < n3; e0 += 256 / gs) {
    const int e = e0 + threadIdx.x / gs;
    double v = 0.0;
    if (e < n3) {
      const int rr = e / en2, j = e - rr * en2, c1 = chunk_first[rr + 1];
#pragma unroll 4
      for (int k = chunk_first[rr] + gl; k < c1; k += gs) v += part[(long long)k * en2 + j];
    }
    for (int o = gs >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (e < n3 && gl == 0) d[e] = v;
  }
  __syncthreads();
  for (int j = threadIdx.x >> 5; j < en2; j += 8) {
    const double* row = A3inv + (long long)(ch.rank * en2 + j) * n3;
    double acc = 0.0;
#pragma unroll 4
    for (int e = lane; e < n3; e += 32) acc += row[e] * d[e];
    acc = warp_sum(acc);
    if (lane == 0) w[j] = acc;
  }
  __syncthreads();
  const int q = threadIdx.x;
  if (q < ch.rows) {
    const double* Vi = V + ch.v_off + (long long)q * en2;
    double acc = 0.0;
#pragma unroll 4
    for (int j = 0; j < en2; ++j) acc += Vi[j] * w[j];
    dz[ch.g0 + q] = acc;
    Z[ch.g0 + q] = first ? acc : Z[ch.g0 + q] + acc;
  }
}
// The same in three launches for many ranks, where every CTA's own sums and products cost more than two
// launches: d by a warp per entry, w = A3^-1 d by a warp per row, then the prolongation.
__global__ void __launch_bounds__(256) k_lv3_sum(const int* chunk_first, int n3, int en2, const double* part, double* d,
                                                 const int* done) {
  if (done && *done) return;
  const int e = (int)((blockIdx.x * 256u + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (e >= n3) return;
  const int rr = e / en2, j = e - rr * en2, c1 = chunk_first[rr + 1];
  double v = 0.0;
  for (int k = chunk_first[rr] + lane; k < c1; k += 32) v += part[(long long)k * en2 + j];
  v = warp_sum(v);
  if (lane == 0) d[e] = v;
}
__global__ void __launch_bounds__(256) k_lv3_gemv(int n3, const double* A3inv, const double* d, double* w,
                                                  const int* done) {
  if (done && *done) return;
  const int i = (int)((blockIdx.x * 256u + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (i >= n3) return;
  const double* row = A3inv + (long long)i * n3;
  double acc = 0.0;
#pragma unroll 8
  for (int e = lane; e < n3; e += 32) acc += row[e] * d[e];
  acc = warp_sum(acc);
  if (lane == 0) w[i] = acc;
}
__global__ void __launch_bounds__(256) k_lv3_prolong(const CoarseChunk* chunks, int nchunk, int en2, const double* w,
                                                     const double* V, double* dz, double* Z, int first,
                                                     const int* done) {
  if (done && *done) return;
  const int c = blockIdx.x * 8 + (threadIdx.x >> 5), q = threadIdx.x & 31;  // a warp per chunk, a lane per row
  static_assert(kCoarseRows == 32, "a lane per row");
  if (c >= nchunk) return;
  const CoarseChunk ch = chunks[c];
  if (q >= ch.rows) return;
  const double* Vi = V + ch.v_off + (long long)q * en2;
  const double* wr = w + (long long)ch.rank * en2;
  double acc = 0.0;
#pragma unroll 4
  for (int j = 0; j < en2; ++j) acc += Vi[j] * wr[j];
  dz[ch.g0 + q] = acc;
  Z[ch.g0 + q] = first ? acc : Z[ch.g0 + q] + acc;
}

// Every CTA of the one launch reads en2 (nchunk + n3) values.  Coarse part of an iteration in one launch and in
// three, by that number: 3 072 (64 ranks of 256 unknowns, four vectors each) 50 us and 55, 4 096 52 and 50 (128
// ranks of 128) and 67 and 68 (64 of 384), 13 312 458 and 423 (64 of 1 536), 20 480 227 and 128 (512 of 192);
// 4 096 ranks of four unknowns 1 428 and 152.
bool lv3_split(const RankLayout& L, int n3, int en2) { return (long long)en2 * (L.nchunk + n3) > 4096; }
void launch_lv3_solve(const RankLayout& L, int n3, int en2, const double* part, double* dw, const double* A3inv,
                      const double* V, double* dz, double* Z, int first, const int* done, cudaStream_t st) {
  if (lv3_split(L, n3, en2)) {
    const int g = (n3 + 7) / 8;
    { note_launch(); k_lv3_sum<<<g, 256, 0, st>>>(L.chunk_first, n3, en2, part, dw, done); }
    { note_launch(); k_lv3_gemv<<<g, 256, 0, st>>>(n3, A3inv, dw, dw + n3, done); }
    { note_launch(); k_lv3_prolong<<<(L.nchunk + 7) / 8, 256, 0, st>>>(L.chunks, L.nchunk, en2, dw + n3, V, dz, Z, first, done); }
    return;
  }
  const int smem = (n3 + en2) * (int)sizeof(double);
  int gs = 1;  // lanes per entry of d: as many as leave no second pass
  while (gs < 32 && n3 * gs * 2 <= 256) gs *= 2;
  if (smem > 48 * 1024) cudaFuncSetAttribute(k_lv3_solve, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  { note_launch(); k_lv3_solve<<<L.nchunk, 256, smem, st>>>(L.chunks, L.chunk_first, n3, en2, gs, part, A3inv, V, dz, Z, first, done); }
}

// nv[s] = 1 / (value of subdomain s's first basis vector, a constant): the constant in the coarse space
template <typename T>
__global__ void k_null_coef(Grid g, const SubInfo* subs, int nsub, int kmax, const T* phi, double* nv) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= nsub) return;
  const SubInfo& S = subs[s];
  nv[s] = 1.0 / (double)phi[(((long long)S.z0 * g.N + S.y0) * g.M + S.x0) * kmax];
}
template <typename T>
void launch_null_coef(const Grid& g, const SubInfo* subs, int nsub, int kmax, const T* phi, double* nv,
                      cudaStream_t st) {
  { note_launch(); k_null_coef<T><<<(nsub + 255) / 256, 256, 0, st>>>(g, subs, nsub, kmax, phi, nv); }
}
template void launch_null_coef<float>(const Grid&, const SubInfo*, int, int, const float*, double*, cudaStream_t);
template void launch_null_coef<double>(const Grid&, const SubInfo*, int, int, const double*, double*, cudaStream_t);

// c <- c - nv (nv.c) / (nv.nv).  nv.c is the sum of the residual, zero up to the rounding of the restriction, and
// what is left of it the coarse solves multiply by up to 1e12 (the shift of the singular level-3 matrix).  One CTA:
// a load or two per thread and pass, bound by its own latency (3 us for 2 244 subdomains).  A batch has one CTA
// per problem, whose subdomains are a rank's; problems with a Dirichlet face are left alone.
__global__ void __launch_bounds__(1024) k_coarse_project(int nsub, int kmax, const int* first, const ProbInfo* probs,
                                                         const double* nv, double* c, const int* done) {
  if (done && *done) return;
  if (probs && probs[blockIdx.x].dmask) return;
  const int s0 = probs ? first[blockIdx.x] : 0, s1 = probs ? first[blockIdx.x + 1] : nsub;
  __shared__ double red[32];
  double t = 0.0, nn = 0.0;
  for (int s = s0 + threadIdx.x; s < s1; s += 1024) {
    const double v = nv[s];
    t += v * c[(long long)s * kmax];
    nn += v * v;
  }
  t = block_sum(t, red);
  __syncthreads();
  nn = block_sum(nn, red);
  __shared__ double q;
  if (threadIdx.x == 0) q = t / nn;
  __syncthreads();
  for (int s = s0 + threadIdx.x; s < s1; s += 1024) c[(long long)s * kmax] -= q * nv[s];
}
void launch_coarse_project(int nsub, int kmax, const RankLayout& L, const ProbInfo* probs, int nprob, const double* nv,
                           double* c, const int* done, cudaStream_t st) {
  { note_launch(); k_coarse_project<<<probs ? nprob : 1, 1024, 0, st>>>(nsub, kmax, L.first, probs, nv, c, done); }
}

// The block of a rank that holds a whole singular problem has its null pivot at the last unknown of the null vector, the
// last subdomain's constant.  Its rounding would be kept or dropped as it falls (1e-14 of the diagonal): of 48 boxes
// without a Dirichlet face in one rank, 1e-8 took one 17 instead of 12 iterations in FP64 and five of them 38 to 100 in
// mixed precision.  With row and column set to zero the inverse's rule drops it always.  One CTA per rank.
__global__ void __launch_bounds__(256) k_pin_null(RankLayout L, const ProbInfo* probs, double* dense) {
  if (probs && probs[blockIdx.x].dmask) return;
  const int r = blockIdx.x, n = rank_nr(L, r), e = n - L.kmax;
  double* A = dense + L.off2[r];
  for (int i = threadIdx.x; i < n; i += 256) A[(long long)e * n + i] = A[(long long)i * n + e] = 0.0;
}
void launch_pin_null(int nrank, const RankLayout& L, const ProbInfo* probs, double* dense, cudaStream_t st) {
  { note_launch(); k_pin_null<<<nrank, 256, 0, st>>>(L, probs, dense); }
}

__global__ void k_axpy(long long n, double a, const double* x, double* y, const int* done) {
  if (done && *done) return;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    y[i] += a * x[i];
}
__global__ void k_copy(long long n, const double* x, double* y, const int* done) {
  if (done && *done) return;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    y[i] = x[i];
}
void launch_axpy(long long n, double a, const double* x, double* y, const int* done, cudaStream_t st) {
  { note_launch(); k_axpy<<<(int)std::min<long long>((n + 255) / 256, 4096), 256, 0, st>>>(n, a, x, y, done); }
}
void launch_copy(long long n, const double* x, double* y, const int* done, cudaStream_t st) {
  { note_launch(); k_copy<<<(int)std::min<long long>((n + 255) / 256, 4096), 256, 0, st>>>(n, x, y, done); }
}

// ---------------------------------------------------------------------------
// Galerkin blocks of Phi^T A Phi (_PC_setup_lv2_J, src/PreMixFEM_3D.c:756-890).
// Warp i of the CTA for subdomain s computes row i of:
//   blk[s][0]   = Phi_s^T A_s Phi_s, A_s the principal submatrix of A on s
//                 (interior faces in difference form, globally interior
//                 boundary faces and Dirichlet terms on the diagonal);
//   blk[s][1+f] = -sum_{face f} t phi_s,i(c) phi_nb,j(c')  (neighbour coupling);
//   gface[s][f] =  sum_{face f} t phi_s,i(c) phi_s,j(c)    (boundary-face part of
//                 the diagonal block, removed again for rank-Neumann matrices).
template <typename T, int KM>
__global__ void k_galerkin(Grid g, const SubInfo* subs, int kmax, const double* tx, const double* ty,
                           const double* tz, const double* diag, const T* phi, double* blk, double* gface) {
  const int s = blockIdx.x;
  const SubInfo S = subs[s];
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (wid >= kmax) return;
  const int i = wid;
  const int nx = S.nx, ny = S.ny, nz = S.nz, ncells = nx * ny * nz;
  double acc[KM];
#pragma unroll
  for (int j = 0; j < KM; ++j) acc[j] = 0.0;
  for (int cl = lane; cl < ncells; cl += 32) {
    const int ii = cl % nx, tt = cl / nx, jj = tt % ny, kk = tt / ny;
    const long long cg = ((long long)(S.z0 + kk) * g.N + (S.y0 + jj)) * g.M + (S.x0 + ii);
    const double pi = (double)phi[cg * kmax + i];
    if (pi == 0.0) continue;
    const double dg = diag[cg];
    const double t_xm = ii > 0 ? tx[cg] : 0.0, t_xp = ii < nx - 1 ? tx[cg + 1] : 0.0;
    const double t_ym = jj > 0 ? ty[cg] : 0.0, t_yp = jj < ny - 1 ? ty[cg + g.M] : 0.0;
    const double t_zm = kk > 0 ? tz[cg] : 0.0, t_zp = kk < nz - 1 ? tz[cg + g.MN] : 0.0;
#pragma unroll
    for (int j = 0; j < KM; ++j) {
      if (j >= kmax) break;
      double a = dg * (double)phi[cg * kmax + j];
      if (ii > 0) a -= t_xm * (double)phi[(cg - 1) * kmax + j];
      if (ii < nx - 1) a -= t_xp * (double)phi[(cg + 1) * kmax + j];
      if (jj > 0) a -= t_ym * (double)phi[(cg - g.M) * kmax + j];
      if (jj < ny - 1) a -= t_yp * (double)phi[(cg + g.M) * kmax + j];
      if (kk > 0) a -= t_zm * (double)phi[(cg - g.MN) * kmax + j];
      if (kk < nz - 1) a -= t_zp * (double)phi[(cg + g.MN) * kmax + j];
      acc[j] += pi * a;
    }
  }
#pragma unroll
  for (int j = 0; j < KM; ++j) {
    if (j >= kmax) break;
    const double v = warp_sum(acc[j]);
    if (lane == 0) blk[(((long long)s * 7 + 0) * kmax + i) * kmax + j] = v;
  }
  // faces x-, x+, y-, y+, z-, z+
  for (int f = 0; f < 6; ++f) {
    const int axis = f >> 1, hi = f & 1;
    bool exists;
    int na, nb;  // face extents
    if (axis == 0) {
      exists = hi ? (S.x0 + nx < g.M) : (S.x0 > 0);
      na = ny;
      nb = nz;
    } else if (axis == 1) {
      exists = hi ? (S.y0 + ny < g.N) : (S.y0 > 0);
      na = nx;
      nb = nz;
    } else {
      exists = hi ? (S.z0 + nz < g.P) : (S.z0 > 0);
      na = nx;
      nb = ny;
    }
    double ag[KM], ac[KM];
#pragma unroll
    for (int j = 0; j < KM; ++j) ag[j] = ac[j] = 0.0;
    if (exists) {
      for (int idx = lane; idx < na * nb; idx += 32) {
        const int a = idx % na, b = idx / na;
        int ii, jj, kk;
        if (axis == 0) {
          ii = hi ? nx - 1 : 0;
          jj = a;
          kk = b;
        } else if (axis == 1) {
          ii = a;
          jj = hi ? ny - 1 : 0;
          kk = b;
        } else {
          ii = a;
          jj = b;
          kk = hi ? nz - 1 : 0;
        }
        const long long cg = ((long long)(S.z0 + kk) * g.N + (S.y0 + jj)) * g.M + (S.x0 + ii);
        const long long off = axis == 0 ? 1 : (axis == 1 ? g.M : g.MN);
        const long long cn = hi ? cg + off : cg - off;
        const double* tt = axis == 0 ? tx : (axis == 1 ? ty : tz);
        const double t = hi ? tt[cn] : tt[cg];
        const double pi = (double)phi[cg * kmax + i];
#pragma unroll
        for (int j = 0; j < KM; ++j) {
          if (j >= kmax) break;
          ag[j] += t * pi * (double)phi[cg * kmax + j];
          ac[j] -= t * pi * (double)phi[cn * kmax + j];
        }
      }
    }
#pragma unroll
    for (int j = 0; j < KM; ++j) {
      if (j >= kmax) break;
      const double vg = warp_sum(ag[j]);
      const double vc = warp_sum(ac[j]);
      if (lane == 0) {
        gface[(((long long)s * 6 + f) * kmax + i) * kmax + j] = vg;
        blk[(((long long)s * 7 + 1 + f) * kmax + i) * kmax + j] = vc;
      }
    }
  }
}

template <typename T>
void launch_galerkin(const Grid& g, const SubInfo* subs, int nsub, int kmax, const double* tx, const double* ty,
                     const double* tz, const double* diag, const T* phi, double* blk, double* gface,
                     cudaStream_t st) {
  const int threads = 32 * kmax;
  if (kmax <= 4)
    { note_launch(); k_galerkin<T, 4><<<nsub, threads, 0, st>>>(g, subs, kmax, tx, ty, tz, diag, phi, blk, gface); }
  else if (kmax <= 8)
    { note_launch(); k_galerkin<T, 8><<<nsub, threads, 0, st>>>(g, subs, kmax, tx, ty, tz, diag, phi, blk, gface); }
  else
    { note_launch(); k_galerkin<T, 16><<<nsub, threads, 0, st>>>(g, subs, kmax, tx, ty, tz, diag, phi, blk, gface); }
}
template void launch_galerkin<float>(const Grid&, const SubInfo*, int, int, const double*, const double*,
                                     const double*, const double*, const float*, double*, double*, cudaStream_t);
template void launch_galerkin<double>(const Grid&, const SubInfo*, int, int, const double*, const double*,
                                      const double*, const double*, const double*, double*, double*, cudaStream_t);

// Dense per-rank coarse matrices.  mode 0: the rank's principal block of
// Phi^T A Phi (level-2 matrix of _PC_setup_lv2_J); mode 1: the rank-Neumann
// matrix of _PC_setup_lv3_eigen (:938-1076), i.e. without the boundary-face
// terms of faces that leave the rank.  Padded dofs (j >= k_s) are identity.
__global__ void k_assemble_dense_r(const SubInfo* subs, int nrank, RankLayout L, long long total, const double* blk,
                                   const double* gface, int mode, double* dense) {
  const int kmax = L.kmax;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    const int r = rank_of(L.off2, nrank, e);
    const long long nr = rank_nr(L, r);
    const long long rem = e - L.off2[r];
    const int row = (int)(rem / nr), col = (int)(rem % nr);
    const int a = row / kmax, i = row % kmax, b = col / kmax, j = col % kmax;
    const int s = L.first[r] + a, s2 = L.first[r] + b;
    const SubInfo& S = subs[s];
    double v = 0.0;
    if (i >= S.k || j >= subs[s2].k) {
      v = (row == col) ? 1.0 : 0.0;
    } else if (a == b) {
      v = blk[(((long long)s * 7) * kmax + i) * kmax + j];
      if (mode == 1)
        for (int f = 0; f < 6; ++f)
          if (S.nb[f] >= 0 && subs[S.nb[f]].rank != r) v -= gface[(((long long)s * 6 + f) * kmax + i) * kmax + j];
    } else {
      for (int f = 0; f < 6; ++f)
        if (S.nb[f] == s2) v = blk[(((long long)s * 7 + 1 + f) * kmax + i) * kmax + j];
    }
    dense[e] = v;
  }
}
void launch_assemble_dense_r(const SubInfo* subs, int nrank, const RankLayout& L, long long total, const double* blk,
                             const double* gface, int mode, double* dense, cudaStream_t st) {
  const int nb = (int)std::min<long long>((total + 255) / 256, 148 * 32);
  { note_launch(); k_assemble_dense_r<<<nb, 256, 0, st>>>(subs, nrank, L, total, blk, gface, mode, dense); }
}
__global__ void k_add_diag_r(RankLayout L, double* dense, double mu, int relative) {
  const int r = blockIdx.x;
  const int n = rank_nr(L, r);
  double* A = dense + L.off2[r];
  __shared__ double mx;
  if (threadIdx.x == 0) {
    double m = 0.0;
    for (int i = 0; i < n; ++i) m = fmax(m, fabs(A[(long long)i * n + i]));
    mx = relative ? m * mu : mu;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += blockDim.x) A[(long long)i * n + i] += mx;
}
void launch_add_diag_r(const RankLayout& L, int nrank, double* dense, double mu, int relative, cudaStream_t st) {
  { note_launch(); k_add_diag_r<<<nrank, 256, 0, st>>>(L, dense, mu, relative); }
}

// In-place Gauss-Jordan inverse of SPD matrices (one CTA per matrix).
// Pivots <= tol * max diag are null directions: that row/column is dropped
// (zero in the result), which equals inverting the matrix with the index
// removed -- the same treatment as the semidefinite Cholesky of the oracle.
__global__ void k_spd_inverse(int n, double* a_all, double tol, int* nnull) {
  double* a = a_all + (long long)blockIdx.x * n * n;
  extern __shared__ double sh[];
  double* colk = sh;
  double* rowk = sh + n;
  __shared__ double red[32];
  __shared__ int nul;
  double mx = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) mx = fmax(mx, fabs(a[(long long)i * n + i]));
  // block max via shared reduction
  {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (lane == 0) red[wid] = mx;
    __syncthreads();
    if (threadIdx.x == 0) {
      double m = 0.0;
      for (int w = 0; w < (int)((blockDim.x + 31) >> 5); ++w) m = fmax(m, red[w]);
      red[0] = m;
      nul = 0;
    }
    __syncthreads();
  }
  const double scale = red[0] > 0 ? red[0] : 1.0;
  for (int k = 0; k < n; ++k) {
    const double piv = a[(long long)k * n + k];
    const bool isnull = !(piv > tol * scale);
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      colk[i] = a[(long long)i * n + k];
      rowk[i] = isnull ? 0.0 : (i == k ? 1.0 : a[(long long)k * n + i]) / piv;
    }
    __syncthreads();
    if (isnull) {
      for (int i = threadIdx.x; i < n; i += blockDim.x) {
        a[(long long)k * n + i] = 0.0;
        a[(long long)i * n + k] = 0.0;
      }
      if (threadIdx.x == 0) nul += 1;
    } else {
      // rank-1 update, one warp per row (no index division in the inner loop)
      const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
      for (int i = threadIdx.x >> 5; i < n; i += nw) {
        double* row = a + (long long)i * n;
        if (i == k) {
          for (int j = lane; j < n; j += 32) row[j] = rowk[j];
        } else {
          const double ci = colk[i];
          for (int j = lane; j < n; j += 32) row[j] = (j == k ? 0.0 : row[j]) - ci * rowk[j];
        }
      }
    }
    __syncthreads();
  }
  {
    const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    for (int i = threadIdx.x >> 5; i < n; i += nw)
      for (int j = i + 1 + lane; j < n; j += 32) {
        const double v = 0.5 * (a[(long long)i * n + j] + a[(long long)j * n + i]);
        a[(long long)i * n + j] = v;
        a[(long long)j * n + i] = v;
      }
  }
  if (threadIdx.x == 0 && nnull) atomicAdd(nnull, nul);
}
// D += A B for one 8 x 8 tile, k = 4, on the FP64 tensor cores.
__device__ __forceinline__ void dmma_8x8x4(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

// The same Gauss-Jordan inverse spread over the whole GPU, in panels of kGjPB
// pivots.  Eliminating the pivots P of a panel turns [A_PP A_PR; A_RP A_RR] into
//   A_PP <- Z = A_PP^-1,  A_PR <- Z A_PR,  A_RP <- -A_RP Z,  A_RR <- A_RR - A_RP Z A_PR,
// which is what the pivots one at a time give in exact arithmetic; Z comes
// from the pivot-by-pivot Gauss-Jordan of the diagonal block with the
// null-pivot rule above (a pivot at or below tol x max|diag| drops its row and
// column), so a null pivot zeroes its row and column of the result as before.
//
// The matrix stays symmetric up to sign: with s_i = -1 for the pivots already
// eliminated and +1 for the others, A_ij = s_i s_j A_ji.  So A_RP is s A_PR^T,
// its new value -s (Z A_PR)^T, and only the tiles on and below the diagonal
// are updated, each writing its mirror image as well: half the operations of
// the full update, and one kernel (k_gj_rows: R = Z A_PR) before it instead of
// three around it.  The products run on the FP64 tensor cores (m8n8k4) from
// shared memory whose pitch keeps fragment loads at their two wavefronts.  The
// CTA that updates the next panel's diagonal block also inverts it, so a panel
// costs two launches; the inversion, the longest chain, runs next to the other
// tiles' updates.  Matrix b has order ord(b) and starts at at(b); panels past a
// matrix's order leave it alone.
//
// Bound by FP64 arithmetic for many or large matrices and by the chain of
// panels for few small ones.  The two inverses of a set-up with four matrices of
// 2 244: 10.7 ms instead of 36.5 by the full update on the CUDA cores in five
// launches a panel; one of 256: 0.18 ms instead of 0.58 by a cluster of 8 CTAs
// with the rows in registers.
struct GjShape {
  const int* first;      // per-matrix orders (first[b+1] - first[b]) kmax, or null (all n)
  const long long* off;  // per-matrix offsets, or null (b n^2)
  int n, kmax;
  __device__ int ord(int b) const { return first ? (first[b + 1] - first[b]) * kmax : n; }
  __device__ long long at(int b) const { return off ? off[b] : (long long)b * n * n; }
};
constexpr int kGjPB = 64;   // pivots per panel and tile edge
constexpr int kGjLd = 72;   // pitch of operands stored [k][row or column]: 8 mod 16 doubles
constexpr int kGjLdZ = 68;  // pitch of an operand stored [row][k]: 4 mod 16 doubles
constexpr int kGjLdT = 65;  // pitch of a tile read by rows and by columns

// Inverse of the pb x pb matrix t (pitch kGjLdT) in place, pivot by pivot, by 256 threads holding 4 x 4
// entries each (rows ty + 16 a, columns tx + 16 b); a pivot at or below thr drops its row and column.
// buf: 4 x kGjPB doubles.  Returns the number of dropped pivots.
__device__ __forceinline__ int gj_invert_tile(double* t, int pb, double thr, double* buf) {
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  double v[4][4];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int i = ty + 16 * a, j = tx + 16 * b;
      v[a][b] = (i < pb && j < pb) ? t[i * kGjLdT + j] : 0.0;
    }
  int nul = 0;
#pragma unroll
  for (int ka = 0; ka < 4; ++ka) {
#pragma unroll 1
    for (int kl = 0; kl < 16; ++kl) {
      const int kk = 16 * ka + kl;
      if (kk >= pb) break;
      double* row = buf + (kk & 1) * 2 * kGjPB;
      double* col = row + kGjPB;
      if (ty == kl) {
#pragma unroll
        for (int b = 0; b < 4; ++b) row[tx + 16 * b] = v[ka][b];
      }
      if (tx == kl) {
#pragma unroll
        for (int a = 0; a < 4; ++a) col[ty + 16 * a] = v[a][ka];
      }
      __syncthreads();
      const double piv = row[kk];
      const bool isnull = !(piv > thr);
      const double rp = isnull ? 0.0 : 1.0 / piv;
      nul += isnull ? 1 : 0;
      double rk[4], ck[4];
#pragma unroll
      for (int b = 0; b < 4; ++b) rk[b] = (tx + 16 * b == kk ? 1.0 : row[tx + 16 * b]) * rp;
#pragma unroll
      for (int a = 0; a < 4; ++a) ck[a] = isnull ? 0.0 : col[ty + 16 * a];
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          const bool pr = a == ka && ty == kl, pc = b == ka && tx == kl;
          v[a][b] = pr ? rk[b] : (pc ? 0.0 : v[a][b]) - ck[a] * rk[b];
        }
    }
  }
  __syncthreads();
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int i = ty + 16 * a, j = tx + 16 * b;
      if (i < pb && j < pb) t[i * kGjLdT + j] = v[a][b];
    }
  __syncthreads();
  return nul;
}

// scale = max |a_ii| and Z of the first panel
__global__ void __launch_bounds__(256) k_gj_first(GjShape sh, const double* a_all, double tol, double* scale,
                                                  double* zbuf, int* nnull) {
  const int b = blockIdx.x;
  const int n = sh.ord(b);
  const double* a = a_all + sh.at(b);
  __shared__ double t[kGjPB * kGjLdT], buf[4 * kGjPB], red[8];
  const int tid = threadIdx.x, pb = min(kGjPB, n);
  double mx = 0.0;
  for (int i = tid; i < n; i += 256) mx = fmax(mx, fabs(a[(long long)i * n + i]));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if ((tid & 31) == 0) red[tid >> 5] = mx;
  for (int e = tid; e < pb * kGjPB; e += 256) {
    const int i = e / kGjPB, j = e % kGjPB;
    if (j < pb) t[i * kGjLdT + j] = a[(long long)i * n + j];
  }
  __syncthreads();
  double m = 0.0;
#pragma unroll
  for (int w = 0; w < 8; ++w) m = fmax(m, red[w]);
  m = m > 0 ? m : 1.0;
  if (tid == 0) scale[b] = m;
  const int nul = gj_invert_tile(t, pb, tol * m, buf);
  double* zb = zbuf + (long long)b * kGjPB * kGjPB;
  for (int e = tid; e < kGjPB * kGjPB; e += 256) {
    const int i = e / kGjPB, j = e % kGjPB;
    zb[e] = (i < pb && j < pb) ? t[i * kGjLdT + j] : 0.0;
  }
  if (tid == 0 && nnull && nul) atomicAdd(nnull, nul);
}

// acc += X^T Y over kGjPB k-values, X and Y stored [k][.] at pitch kGjLd: the warp's 16 x 32 part at
// (wi, wj) of a 64 x 64 tile.
template <bool XZ>
__device__ __forceinline__ void gj_mma_tile(const double* X, const double* Y, int wi, int wj, double (&acc)[2][4][2]) {
  const int lane = threadIdx.x & 31, r = lane >> 2, q = lane & 3;
#pragma unroll 4
  for (int k = 0; k < kGjPB; k += 4) {
    double x[2], y[4];
#pragma unroll
    for (int a = 0; a < 2; ++a)
      x[a] = XZ ? X[(wi + 8 * a + r) * kGjLdZ + k + q] : X[(k + q) * kGjLd + wi + 8 * a + r];
#pragma unroll
    for (int b = 0; b < 4; ++b) y[b] = Y[(k + q) * kGjLd + wj + 8 * b + r];
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) dmma_8x8x4(acc[a][b][0], acc[a][b][1], x[a], y[b]);
  }
}

// R = Z A_PR and a copy of A_PR, 64 columns per CTA (none for the panel's own columns)
__global__ void __launch_bounds__(256) k_gj_rows(GjShape sh, const double* a_all, int k0, const double* zbuf,
                                                 double* rbuf, double* lbuf) {
  const int b = blockIdx.y;
  const int n = sh.ord(b);
  const int j0 = blockIdx.x * kGjPB;
  if (k0 >= n || j0 >= n || j0 == k0) return;
  const int pb = min(kGjPB, n - k0);
  const double* a = a_all + sh.at(b);
  extern __shared__ __align__(16) double gj_sm[];
  double* zs = gj_sm;                   // [c][c'] at kGjLdZ
  double* as = gj_sm + kGjPB * kGjLdZ;  // [c'][j] at kGjLd
  const double* zb = zbuf + (long long)b * kGjPB * kGjPB;
  double* rb = rbuf + (long long)b * kGjPB * sh.n;
  double* lb = lbuf + (long long)b * kGjPB * sh.n;
  const int tid = threadIdx.x;
  for (int e = tid; e < kGjPB * kGjPB; e += 256) {
    const int c = e / kGjPB, j = e % kGjPB;
    zs[c * kGjLdZ + j] = zb[e];
    const double v = (c < pb && j0 + j < n) ? a[(long long)(k0 + c) * n + j0 + j] : 0.0;
    as[c * kGjLd + j] = v;
    if (j0 + j < n) lb[(long long)c * sh.n + j0 + j] = v;
  }
  __syncthreads();
  const int w = tid >> 5, wi = (w >> 1) * 16, wj = (w & 1) * 32, r = (tid & 31) >> 2, q = tid & 3;
  double acc[2][4][2] = {};
  gj_mma_tile<true>(zs, as, wi, wj, acc);
#pragma unroll
  for (int x = 0; x < 2; ++x)
#pragma unroll
    for (int y = 0; y < 4; ++y)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int c = wi + 8 * x + r, j = j0 + wj + 8 * y + 2 * q + h;
        if (j < n) rb[(long long)c * sh.n + j] = acc[x][y][h];
      }
}

// One tile (ti >= tj) of the panel's update and its mirror image: the rank-64
// update outside the panel, R and -s R^T in its row and column, Z on its
// diagonal.  CTA 0 takes the next panel's diagonal tile and inverts it.
__global__ void __launch_bounds__(256) k_gj_update(GjShape sh, double* a_all, int k0, const double* zbuf, double* znext,
                                                   const double* rbuf, const double* lbuf, int ntile, double tol,
                                                   const double* scale, int* nnull) {
  const int b = blockIdx.y;
  const int n = sh.ord(b);
  if (k0 >= n) return;
  const int tp = k0 / kGjPB, tn = min(tp + 1, ntile - 1);
  // tile list in row order, with the next panel's diagonal tile first
  int id = blockIdx.x;
  const int dn = tn * (tn + 1) / 2 + tn;
  id = id == 0 ? dn : (id <= dn ? id - 1 : id);
  int ti = (int)((sqrtf(8.0f * (float)id + 1.0f) - 1.0f) * 0.5f);
  while ((ti + 1) * (ti + 2) / 2 <= id) ++ti;
  while (ti * (ti + 1) / 2 > id) --ti;
  const int tj = id - ti * (ti + 1) / 2;
  const int i0 = ti * kGjPB, j0 = tj * kGjPB;
  if (i0 >= n) return;
  double* a = a_all + sh.at(b);
  const double* rb = rbuf + (long long)b * kGjPB * sh.n;
  const double* lb = lbuf + (long long)b * kGjPB * sh.n;
  extern __shared__ __align__(16) double gj_sm[];
  double* xs = gj_sm;                   // [c][i], old A_PR at the rows' columns; then the new tile
  double* ys = gj_sm + kGjPB * kGjLd;   // [c][j], R
  const int tid = threadIdx.x, c64 = tid & 63, r64 = tid >> 6;
  if (ti == tp && tj == tp) {
    const double* zb = zbuf + (long long)b * kGjPB * kGjPB;
    for (int c = r64; c < kGjPB; c += 4)
      if (k0 + c < n && k0 + c64 < n) a[(long long)(k0 + c) * n + k0 + c64] = zb[c * kGjPB + c64];
    return;
  }
  if (ti == tp || tj == tp) {
    const int o0 = ti == tp ? j0 : i0;  // the tile's rows and columns outside the panel
    const double s = o0 < k0 ? 1.0 : -1.0;
    for (int c = r64; c < kGjPB; c += 4) {
      const double v = o0 + c64 < n ? rb[(long long)c * sh.n + o0 + c64] : 0.0;
      if (k0 + c < n && o0 + c64 < n) a[(long long)(k0 + c) * n + o0 + c64] = v;
      xs[c * kGjLdT + c64] = v;
    }
    __syncthreads();
    for (int i = r64; i < kGjPB; i += 4)
      if (o0 + i < n && k0 + c64 < n) a[(long long)(o0 + i) * n + k0 + c64] = s * xs[c64 * kGjLdT + i];
    return;
  }
  double old[16];
#pragma unroll
  for (int u = 0; u < 16; ++u) {
    const int i = i0 + r64 + 4 * u, j = j0 + c64;
    old[u] = (i < n && j < n) ? a[(long long)i * n + j] : 0.0;
  }
  for (int c = r64; c < kGjPB; c += 4) {
    xs[c * kGjLd + c64] = i0 + c64 < n ? lb[(long long)c * sh.n + i0 + c64] : 0.0;
    ys[c * kGjLd + c64] = j0 + c64 < n ? rb[(long long)c * sh.n + j0 + c64] : 0.0;
  }
  __syncthreads();
  const int w = tid >> 5, wi = (w >> 1) * 16, wj = (w & 1) * 32, r = (tid & 31) >> 2, q = tid & 3;
  double acc[2][4][2] = {};
  gj_mma_tile<false>(xs, ys, wi, wj, acc);
  __syncthreads();
  double* t = xs;
#pragma unroll
  for (int x = 0; x < 2; ++x)
#pragma unroll
    for (int y = 0; y < 4; ++y)
#pragma unroll
      for (int h = 0; h < 2; ++h) t[(wi + 8 * x + r) * kGjLdT + wj + 8 * y + 2 * q + h] = acc[x][y][h];
  __syncthreads();
  const double si = i0 < k0 ? -1.0 : 1.0, sj = j0 < k0 ? -1.0 : 1.0;
#pragma unroll
  for (int u = 0; u < 16; ++u) {
    const int il = r64 + 4 * u, i = i0 + il, j = j0 + c64;
    const double v = old[u] - si * t[il * kGjLdT + c64];
    t[il * kGjLdT + c64] = v;
    if (i < n && j < n) a[(long long)i * n + j] = v;
  }
  __syncthreads();
  if (ti != tj) {
    const double sg = si * sj;
    for (int jl = r64; jl < kGjPB; jl += 4)
      if (j0 + jl < n && i0 + c64 < n) a[(long long)(j0 + jl) * n + i0 + c64] = sg * t[c64 * kGjLdT + jl];
  } else if (ti == tp + 1) {
    const int pb = min(kGjPB, n - i0);
    const int nul = gj_invert_tile(t, pb, tol * scale[b], ys);
    double* zb = znext + (long long)b * kGjPB * kGjPB;
    for (int i = r64; i < kGjPB; i += 4)
      zb[i * kGjPB + c64] = (i < pb && c64 < pb) ? t[i * kGjLdT + c64] : 0.0;
    if (tid == 0 && nnull && nul) atomicAdd(nnull, nul);
  }
}

// the diagonal tiles, the only ones whose two halves are computed separately
__global__ void __launch_bounds__(256) k_gj_sym(GjShape sh, double* a_all) {
  const int b = blockIdx.y;
  const int n = sh.ord(b), i0 = blockIdx.x * kGjPB;
  double* a = a_all + sh.at(b);
  for (int e = threadIdx.x; e < kGjPB * kGjPB; e += 256) {
    const int i = i0 + e / kGjPB, j = i0 + e % kGjPB;
    if (i < n && j < n && j > i) {
      const double v = 0.5 * (a[(long long)i * n + j] + a[(long long)j * n + i]);
      a[(long long)i * n + j] = v;
      a[(long long)j * n + i] = v;
    }
  }
}
// nb matrices of orders <= sh.n; returns false when the scratch could not be allocated
static bool gj_inverse(int nb, GjShape sh, double* a, double tol, int* nnull, cudaStream_t st) {
  const int n = sh.n;
  double* scr = nullptr;
  const size_t zsz = (size_t)nb * kGjPB * kGjPB, psz = (size_t)nb * kGjPB * n;
  if (cudaMallocAsync((void**)&scr, sizeof(double) * (nb + 2 * zsz + 2 * psz), st) != cudaSuccess) {
    (void)cudaGetLastError();
    return false;
  }
  double* zbuf = scr;
  double* rbuf = scr + 2 * zsz;
  double* lbuf = rbuf + psz;
  double* scale = lbuf + psz;
  const int sm_rows = (int)(sizeof(double) * kGjPB * (kGjLdZ + kGjLd));
  const int sm_upd = (int)(sizeof(double) * kGjPB * 2 * kGjLd);
  cudaFuncSetAttribute(k_gj_rows, cudaFuncAttributeMaxDynamicSharedMemorySize, sm_rows);
  cudaFuncSetAttribute(k_gj_update, cudaFuncAttributeMaxDynamicSharedMemorySize, sm_upd);
  { note_launch(); k_gj_first<<<nb, 256, 0, st>>>(sh, a, tol, scale, zbuf, nnull); }
  const int nt = (n + kGjPB - 1) / kGjPB;
  for (int k0 = 0, p = 0; k0 < n; k0 += kGjPB, p ^= 1) {
    double *z = zbuf + p * zsz, *zn = zbuf + (p ^ 1) * zsz;
    if (nt > 1) { note_launch(); k_gj_rows<<<dim3(nt, nb), 256, sm_rows, st>>>(sh, a, k0, z, rbuf, lbuf); }
    { note_launch(); k_gj_update<<<dim3(nt * (nt + 1) / 2, nb), 256, sm_upd, st>>>(sh, a, k0, z, zn, rbuf, lbuf, nt, tol, scale, nnull); }
  }
  { note_launch(); k_gj_sym<<<dim3(nt, nb), 256, 0, st>>>(sh, a); }
  cudaFreeAsync(scr, st);
  return true;
}

bool launch_spd_inverse_r(const RankLayout& L, int nrank, int nr_max, double* dense, double tol, int* nnull,
                          cudaStream_t st) {
  return gj_inverse(nrank, GjShape{L.first, L.off2, nr_max, L.kmax}, dense, tol, nnull, st);
}

void launch_spd_inverse(int nb, int n, double* a, double tol, int* nnull, cudaStream_t st) {
  if (gj_inverse(nb, GjShape{nullptr, nullptr, n, 0}, a, tol, nnull, st)) return;
  const int smem = 2 * n * sizeof(double);  // no room for the scratch: one CTA per matrix, in place
  if (smem > 48 * 1024) cudaFuncSetAttribute(k_spd_inverse, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  { note_launch(); k_spd_inverse<<<nb, 1024, smem, st>>>(n, a, tol, nnull); }
}

// ---------------------------------------------------------------------------
// Level-3 HEP (_PC_setup_lv3_eigen, :1086-1115): smallest en2 eigenpairs of
// each rank's dense rank-Neumann matrix.  SLEPc's shift-and-invert Krylov-
// Schur is replaced by block inverse subspace iteration with the precomputed
// (A + mu I)^-1, SVQB orthonormalisation and a Rayleigh-Ritz step on A; the
// eigenvectors come out orthonormal in the 2-norm as SLEPc returns them.
// work: 3 * nr * p doubles per rank.
#define PMF_L3_MAXP 32

// Out[i * p + c] = sum_l M[i][l] Xs[l * ldx + c] (- shift[c] Xs[i * ldx + c]) for c < q, with the
// block Xs staged in shared memory: one warp per row, lanes along l (coalesced
// row reads), eight column accumulators per pass, warp reductions.
__device__ void cta_rows_mm(const double* __restrict__ M, int nr, const double* Xs, int ldx, int q, double* Out,
                            int p, const double* shift) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int i = wid; i < nr; i += nw) {
    const double* row = M + (long long)i * nr;
    for (int c0 = 0; c0 < q; c0 += 8) {
      double acc[8];
#pragma unroll
      for (int c = 0; c < 8; ++c) acc[c] = 0.0;
      for (int l = lane; l < nr; l += 32) {
        const double mv = row[l];
        const double* xr = Xs + l * ldx + c0;
#pragma unroll
        for (int c = 0; c < 8; ++c)
          if (c0 + c < q) acc[c] += mv * xr[c];
      }
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const double v = warp_sum(acc[c]);
        if (lane == 0 && c0 + c < q)
          Out[(long long)i * p + c0 + c] = shift ? v - shift[c0 + c] * Xs[i * ldx + c0 + c] : v;
      }
    }
  }
}

// Xs[l * ldx + c] = X[l * p + c], c < q
__device__ __forceinline__ void cta_stage_block(const double* X, int nr, int p, int q, double* Xs, int ldx) {
  for (int e = threadIdx.x; e < nr * q; e += blockDim.x) {
    const int l = e / q, c = e - l * q;
    Xs[l * ldx + c] = X[(long long)l * p + c];
  }
  __syncthreads();
}

__global__ void __launch_bounds__(512) k_dense_smallest_eig(RankLayout L, int en2, int p, const double* A_all,
                                                             const double* inv_all, double* V_all, double* evals_all,
                                                             int* iters, double tol, int max_it, double* work_all,
                                                             int ldx) {
  extern __shared__ double xs[];  // nr x ldx staging block when ldx > 0
  const int r = blockIdx.x;
  const int nr = rank_nr(L, r);
  const double* A = A_all + L.off2[r];
  const double* inv = inv_all + L.off2[r];
  double* X = work_all + L.offw[r];
  double* Y = X + (long long)nr * p;
  double* AY = Y + (long long)nr * p;
  __shared__ double G[PMF_L3_MAXP * PMF_L3_MAXP], U[PMF_L3_MAXP * PMF_L3_MAXP], w[PMF_L3_MAXP],
      C[PMF_L3_MAXP * PMF_L3_MAXP], dsc[PMF_L3_MAXP], jac[64];
  __shared__ int ijac[32];
  __shared__ int keep, conv;
  __shared__ double anorm;
  const int tid = threadIdx.x, nt = blockDim.x;
  // scale of A: max |diag|
  if (tid == 0) {
    double m = 0.0;
    for (int i = 0; i < nr; ++i) m = fmax(m, fabs(A[(long long)i * nr + i]));
    anorm = m > 0 ? m : 1.0;
  }
  __syncthreads();
  for (long long e = tid; e < (long long)nr * p; e += nt) {
    const double v = hash_uniform(((unsigned long long)r << 40) ^ (unsigned long long)e);
    X[e] = v / anorm;
    AY[e] = -v;
  }
  __syncthreads();
  int it = 0;
  for (; it < max_it; ++it) {
    // Y = X - inv R with the residuals R in AY, as k_l3_mm and k_l3_init explain
    if (ldx > 0) {
      cta_stage_block(AY, nr, p, p, xs, ldx);
      cta_rows_mm(inv, nr, xs, ldx, p, Y, p, nullptr);
      __syncthreads();
      for (long long e = tid; e < (long long)nr * p; e += nt) Y[e] = X[e] - Y[e];
    } else {
      for (long long e = tid; e < (long long)nr * p; e += nt) {
        const int i = (int)(e / p), j = (int)(e % p);
        const double* row = inv + (long long)i * nr;
        double acc = 0.0;
        for (int l = 0; l < nr; ++l) acc += row[l] * AY[(long long)l * p + j];
        Y[e] = X[e] - acc;
      }
    }
    __syncthreads();
    // SVQB: G = Y^T Y, D^-1/2 G D^-1/2 = U w U^T, X = Y D^-1/2 U w^-1/2 (kept columns)
    for (int e = tid; e < p * p; e += nt) {
      const int a = e / p, b = e % p;
      double acc = 0.0;
      for (int l = 0; l < nr; ++l) acc += Y[(long long)l * p + a] * Y[(long long)l * p + b];
      G[a * PMF_L3_MAXP + b] = acc;
    }
    __syncthreads();
    if (tid < p) dsc[tid] = 1.0 / sqrt(fmax(G[tid * PMF_L3_MAXP + tid], 1e-300));
    __syncthreads();
    for (int e = tid; e < p * p; e += nt) {
      const int a = e / p, b = e % p;
      G[a * PMF_L3_MAXP + b] *= dsc[a] * dsc[b];
    }
    __syncthreads();
    cta_jacobi_eigh(G, U, w, p, PMF_L3_MAXP, ijac, jac);
    if (tid == 0) {
      int kk = 0;
      const double wmax = w[p - 1];
      for (int c = p - 1; c >= 0; --c)
        if (w[c] > 1e-12 * wmax) ++kk;
      keep = kk;
    }
    __syncthreads();
    const int q = keep;  // kept columns are the last q (largest w)
    for (int e = tid; e < p * q; e += nt) {
      const int a = e / q, c = e % q;
      const int cc = p - q + c;
      C[a * PMF_L3_MAXP + c] = dsc[a] * U[a * PMF_L3_MAXP + cc] / sqrt(w[cc]);
    }
    __syncthreads();
    for (long long e = tid; e < (long long)nr * q; e += nt) {
      const int i = (int)(e / q), c = (int)(e % q);
      double acc = 0.0;
      for (int a = 0; a < p; ++a) acc += Y[(long long)i * p + a] * C[a * PMF_L3_MAXP + c];
      X[(long long)i * p + c] = acc;
    }
    __syncthreads();
    // AY = A X (q columns), H = X^T A X
    if (ldx > 0) {
      cta_stage_block(X, nr, p, q, xs, ldx);
      cta_rows_mm(A, nr, xs, ldx, q, AY, p, nullptr);
    } else {
      for (long long e = tid; e < (long long)nr * q; e += nt) {
        const int i = (int)(e / q), c = (int)(e % q);
        const double* row = A + (long long)i * nr;
        double acc = 0.0;
        for (int l = 0; l < nr; ++l) acc += row[l] * X[(long long)l * p + c];
        AY[(long long)i * p + c] = acc;
      }
    }
    __syncthreads();
    for (int e = tid; e < q * q; e += nt) {
      const int a = e / q, b = e % q;
      double acc = 0.0;
      for (int l = 0; l < nr; ++l) acc += X[(long long)l * p + a] * AY[(long long)l * p + b];
      G[a * PMF_L3_MAXP + b] = acc;
    }
    __syncthreads();
    for (int e = tid; e < q * q; e += nt) {  // symmetrise
      const int a = e / q, b = e % q;
      if (a < b) {
        const double v = 0.5 * (G[a * PMF_L3_MAXP + b] + G[b * PMF_L3_MAXP + a]);
        G[a * PMF_L3_MAXP + b] = v;
        G[b * PMF_L3_MAXP + a] = v;
      }
    }
    __syncthreads();
    cta_jacobi_eigh(G, U, w, q, PMF_L3_MAXP, ijac, jac);
    // X <- X U (through Y as scratch)
    for (long long e = tid; e < (long long)nr * q; e += nt) {
      const int i = (int)(e / q), c = (int)(e % q);
      double ax = 0.0;
      for (int a = 0; a < q; ++a) ax += X[(long long)i * p + a] * U[a * PMF_L3_MAXP + c];
      Y[(long long)i * p + c] = ax;
    }
    __syncthreads();
    for (long long e = tid; e < (long long)nr * q; e += nt) {
      const int i = (int)(e / q), c = (int)(e % q);
      X[(long long)i * p + c] = Y[(long long)i * p + c];
    }
    __syncthreads();
    // recompute AY for the Ritz vectors and the residuals of the wanted ones
    if (ldx > 0) {
      cta_stage_block(X, nr, p, q, xs, ldx);
      cta_rows_mm(A, nr, xs, ldx, q, AY, p, w);
    } else {
      for (long long e = tid; e < (long long)nr * q; e += nt) {
        const int i = (int)(e / q), c = (int)(e % q);
        const double* row = A + (long long)i * nr;
        double acc = 0.0;
        for (int l = 0; l < nr; ++l) acc += row[l] * X[(long long)l * p + c];
        AY[(long long)i * p + c] = acc - w[c] * X[(long long)i * p + c];
      }
    }
    __syncthreads();
    if (tid == 0) conv = 1;
    __syncthreads();
    for (int c = tid; c < min(en2, q); c += nt) {
      double rr = 0.0;
      for (int l = 0; l < nr; ++l) rr += AY[(long long)l * p + c] * AY[(long long)l * p + c];
      if (sqrt(rr) > tol * anorm) conv = 0;
    }
    if (q < en2 && tid == 0) conv = 0;
    __syncthreads();
    if (conv) break;
    // fresh random directions in place of dropped columns, orthogonal to the kept ones: the inverse of a floating
    // rank, whose constant it takes 1e8 times, would turn others back into copies of the kept ones
    for (long long e = tid; e < (long long)nr * (p - q); e += nt) {
      const int i = (int)(e / (p - q)), c = q + (int)(e % (p - q));
      X[(long long)i * p + c] = hash_uniform(((unsigned long long)(r + 7) << 44) ^ ((unsigned long long)it << 32) ^
                                             (unsigned long long)e);
    }
    __syncthreads();
    for (int e = tid; e < (p - q) * q; e += nt) {
      const int c = q + e / q, k = e % q;
      double acc = 0.0;
      for (int l = 0; l < nr; ++l) acc += X[(long long)l * p + c] * X[(long long)l * p + k];
      G[c * PMF_L3_MAXP + k] = acc;
    }
    __syncthreads();
    for (long long e = tid; e < (long long)nr * (p - q); e += nt) {
      const long long i = e / (p - q);
      const int c = q + (int)(e % (p - q));
      double v = X[i * p + c];
      for (int k = 0; k < q; ++k) v -= G[c * PMF_L3_MAXP + k] * X[i * p + k];
      X[i * p + c] = v / anorm;
      AY[i * p + c] = -v;
    }
    __syncthreads();
  }
  double* V = V_all + L.offv[r];
  for (long long e = tid; e < (long long)nr * en2; e += nt) {
    const int i = (int)(e / en2), j = (int)(e % en2);
    V[e] = X[(long long)i * p + j];
  }
  if (tid < en2) evals_all[(long long)r * en2 + tid] = w[tid];
  if (tid == 0) iters[r] = it + 1;
}

// The same iteration in three launches over all ranks for p <= kL3Cols columns:
// Y and A Y on the FP64 tensor cores, then one CTA per rank for the projected
// problem.  Y = X - inv R with the residuals R = A X - X w is (A + mu I)^-1 X up to
// a factor per column, formed so that the inverse's rounding errors are multiplied
// by the residual: from Y = inv X a rank whose matrix is singular up to mu can stall
// above the tolerance and run to the iteration limit.  Y is not orthonormalised first: the Rayleigh-Ritz step
// takes the pencil (Y^T A Y, Y^T Y) on one warp (pmf_rr.cuh), whose Cholesky
// drops dependent columns; in exact arithmetic the Ritz pairs are the same, and
// from the second iteration on Y's columns are nearly orthogonal.  The Ritz
// vectors' images are A Y C, so an iteration streams each rank's two matrices
// once.  Dropped columns restart from random directions orthogonal to the kept
// ones: without that the shift-inverse would turn them back into copies of the
// lowest vector and they would be dropped again.  A converged rank's kernels
// return at once; the host checks every 4 iterations whether all have converged.
//
// Bound by latency for few small ranks (one rank of 256 unknowns: 1.4 ms a
// set-up, 4.6 ms with one CTA per rank for the whole iteration and CTA-wide
// Jacobi for the projected problems) and by streaming the matrices for large
// ones (four ranks of 2 244: 3.0 ms instead of 23).
struct L3Rank {
  double anorm;
  double w[PMF_L3_MAXP];
  int q, conv, it;
};
constexpr int kL3Cols = 16;    // most columns of the block
constexpr int kL3Rows = 32;    // rows per CTA of the products: 4 warps of 8
constexpr int kL3Tile = 128;   // rows of the block staged in shared memory at a time
constexpr int kL3Ld = 18;      // its pitch: 4 kL3Ld is 8 mod 16 doubles, so fragment loads take two wavefronts
constexpr int kL3Thr = 512;    // threads of the projected problem

__global__ void k_l3_init(RankLayout L, int p, const double* A_all, double* work_all, L3Rank* st) {
  const int r = blockIdx.x;
  const int nr = rank_nr(L, r);
  const double* A = A_all + L.off2[r];
  double* X = work_all + L.offw[r];
  __shared__ double red[32];
  double m = 0.0;
  for (int i = threadIdx.x; i < nr; i += blockDim.x) m = fmax(m, fabs(A[(long long)i * nr + i]));
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (lane == 0) red[wid] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    double v = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) v = fmax(v, red[w]);
    st[r].anorm = v > 0 ? v : 1.0;
    for (int c = 0; c < PMF_L3_MAXP; ++c) st[r].w[c] = 0.0;
    st[r].q = p;
    st[r].conv = 0;
    st[r].it = 0;
  }
  __syncthreads();
  // Random columns V as X = V / anorm and R = -V, which makes Y = inv V and a little of V: a direction that the inverse
  // dropped as null (the only one of a floating rank of one unknown, whose matrix is rounding) stays in the block.
  double* R = X + 2 * (long long)nr * p;
  const double an = st[r].anorm;
  for (long long e = threadIdx.x; e < (long long)nr * p; e += blockDim.x) {
    const double v = hash_uniform(((unsigned long long)r << 40) ^ (unsigned long long)e);
    X[e] = v / an;
    R[e] = -v;
  }
}

// Out = M In (REFINE: X - M In), blocks src / dst of the rank's workspace (0 X,
// 1 Y, 2 R or A Y).  Lane (r, q) of a warp holds of row r the entries k0 + 4 q + t,
// t < 4, of each 16: whole 128-byte row segments per load, used as the A fragments
// of four k-steps (the order of k within a dot product is free as long as B follows
// it).  m16n8k4 products, here and in the inverses, measured the same: neither
// kernel is bound by the tensor cores.
template <bool REFINE>
__global__ void __launch_bounds__(128) k_l3_mm(RankLayout L, int p, const double* M_all, double* work_all, int src,
                                               int dst, const L3Rank* st) {
  const int rk = blockIdx.y;
  if (st[rk].conv) return;
  const int nr = rank_nr(L, rk);
  const int lane = threadIdx.x & 31, r = lane >> 2, q = lane & 3;
  const int i0 = blockIdx.x * kL3Rows;
  if (i0 >= nr) return;
  const int i = i0 + (threadIdx.x >> 5) * 8 + r;
  const double* M = M_all + L.off2[rk];
  const double* In = work_all + L.offw[rk] + (long long)src * nr * p;
  double* Out = work_all + L.offw[rk] + (long long)dst * nr * p;
  __shared__ double xs[kL3Tile * kL3Ld];
  const bool vec = (nr & 1) == 0 && (reinterpret_cast<unsigned long long>(M) & 15) == 0;  // 16-byte aligned rows
  const double* row = M + (long long)min(i, nr - 1) * nr;
  double acc[2][2][2] = {};  // two independent chains per 8-column tile
  for (int l0 = 0; l0 < nr; l0 += kL3Tile) {
    const int lend = min(kL3Tile, nr - l0);
    for (int e = threadIdx.x; e < kL3Tile * kL3Cols; e += blockDim.x) {
      const int l = e / kL3Cols, c = e % kL3Cols;
      xs[l * kL3Ld + c] = (l < lend && c < p) ? In[(long long)(l0 + l) * p + c] : 0.0;
    }
    __syncthreads();
    for (int k0 = 0; k0 < lend; k0 += 32) {
      double m[2][4];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int k = k0 + 16 * u + 4 * q;
        if (vec && k + 3 < lend) {
          const double2 lo = *reinterpret_cast<const double2*>(row + l0 + k);
          const double2 hi = *reinterpret_cast<const double2*>(row + l0 + k + 2);
          m[u][0] = lo.x;
          m[u][1] = lo.y;
          m[u][2] = hi.x;
          m[u][3] = hi.y;
        } else {
#pragma unroll
          for (int t = 0; t < 4; ++t) m[u][t] = k + t < lend ? row[l0 + k + t] : 0.0;
        }
      }
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const double* xk = xs + (k0 + 16 * u + 4 * q + t) * kL3Ld + r;
          dmma_8x8x4(acc[u][0][0], acc[u][0][1], m[u][t], xk[0]);
          dmma_8x8x4(acc[u][1][0], acc[u][1][1], m[u][t], xk[8]);
        }
    }
    __syncthreads();
  }
  if (i < nr) {
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int c = 8 * n + 2 * q + h;
        const long long o = (long long)i * p + c;
        const double v = acc[0][n][h] + acc[1][n][h];
        if (c < p) Out[o] = REFINE ? work_all[L.offw[rk] + o] - v : v;
      }
  }
}

struct L3Smem {
  WarpRR<kL3Cols, kL3Cols> rr;
  double C[kL3Cols * kL3Cols];
  double G[2 * kL3Cols * kL3Cols];
  double part[kL3Thr / 32][kL3Cols * kL3Cols];  // per-warp partial Grams, then the pads' coefficients
  double red[32];
};

// Rayleigh-Ritz on (Y^T A Y, Y^T Y), X <- Y C, R = A X - X w from A Y C in the place of A Y, the residual norms
// of the wanted pairs, and fresh directions in place of dropped columns.
__global__ void __launch_bounds__(kL3Thr) k_l3_rr(RankLayout L, int en2, int p, double* work_all, L3Rank* st,
                                                  double tol, int it) {
  const int rk = blockIdx.x;
  if (st[rk].conv) return;
  extern __shared__ __align__(16) unsigned char l3_raw[];
  L3Smem& sm = *reinterpret_cast<L3Smem*>(l3_raw);
  const int nr = rank_nr(L, rk);
  double* X = work_all + L.offw[rk];
  const double* Y = X + (long long)nr * p;
  double* AY = X + 2 * (long long)nr * p;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nw = kL3Thr / 32;
  {
    // Grams: rows l of four per step, tiles (0,0), (0,1), (1,1) of the 16 x 16 result
    const int r = lane >> 2, q = lane & 3;
    double g[2][3][2] = {};
    const bool c0 = r < p, c1 = r + 8 < p;
#pragma unroll 4
    for (int l0 = 4 * wid; l0 < nr; l0 += 4 * nw) {
      const int l = l0 + q;
      const double* y = Y + (long long)l * p + r;
      const double* ay = AY + (long long)l * p + r;
      const bool in = l < nr;
      const double y0 = in && c0 ? y[0] : 0.0, y1 = in && c1 ? y[8] : 0.0;
      const double a0 = in && c0 ? ay[0] : 0.0, a1 = in && c1 ? ay[8] : 0.0;
      dmma_8x8x4(g[0][0][0], g[0][0][1], y0, y0);
      dmma_8x8x4(g[0][1][0], g[0][1][1], y0, y1);
      dmma_8x8x4(g[0][2][0], g[0][2][1], y1, y1);
      dmma_8x8x4(g[1][0][0], g[1][0][1], y0, a0);
      dmma_8x8x4(g[1][1][0], g[1][1][1], y0, a1);
      dmma_8x8x4(g[1][2][0], g[1][2][1], y1, a1);
    }
#pragma unroll
    for (int which = 0; which < 2; ++which) {
      double* o = sm.part[wid];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int c = 2 * q + h;
        o[r * 16 + c] = g[which][0][h];
        o[r * 16 + 8 + c] = g[which][1][h];
        o[(8 + r) * 16 + 8 + c] = g[which][2][h];
      }
      __syncthreads();
      if (tid < 256) {
        int a = tid >> 4, b = tid & 15;
        if (a >= 8 && b < 8) {  // the block below the diagonal is the mirror
          const int x = a;
          a = b;
          b = x;
        }
        double v = 0.0;
        for (int w = 0; w < nw; ++w) v += sm.part[w][a * 16 + b];
        sm.G[which * 256 + tid] = v;
      }
      __syncthreads();
    }
  }
  if (wid == 0) {
    auto load = [&](int which, double(&g)[kL3Cols]) {
#pragma unroll
      for (int j = 0; j < kL3Cols; ++j) g[j] = (j < p && lane < p) ? sm.G[which * 256 + j * 16 + lane] : 0.0;
    };
    const int q = warp_rayleigh_ritz<kL3Cols, kL3Cols>(sm.rr, p, p, 1e-12, load, sm.C, kL3Cols);
    if (lane == 0) st[rk].q = q;
    if (lane < min(p, q)) st[rk].w[lane] = sm.rr.lam[lane];
    sm.red[0] = q;
  }
  __syncthreads();
  const int q = (int)sm.red[0];
  __syncthreads();
  const int nw2 = min(en2, q);
  double res[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) res[c] = 0.0;
  for (int l = tid; l < nr; l += kL3Thr) {
    double y[kL3Cols], ay[kL3Cols];
#pragma unroll
    for (int a = 0; a < kL3Cols; ++a) {
      y[a] = a < p ? Y[(long long)l * p + a] : 0.0;
      ay[a] = a < p ? AY[(long long)l * p + a] : 0.0;
    }
#pragma unroll
    for (int c = 0; c < kL3Cols; ++c)
      if (c < q) {
        double x = 0.0;
#pragma unroll
        for (int a = 0; a < kL3Cols; ++a)
          if (a < p) x += y[a] * sm.C[a * kL3Cols + c];
        double ax = 0.0;
#pragma unroll
        for (int a = 0; a < kL3Cols; ++a)
          if (a < p) ax += ay[a] * sm.C[a * kL3Cols + c];
        const double d = ax - sm.rr.lam[c] * x;
        X[(long long)l * p + c] = x;
        AY[(long long)l * p + c] = d;
        if (c < 8 && c < nw2) res[c] += d * d;
      }
  }
  bool conv = q >= en2;
  const double thr = tol * st[rk].anorm;
#pragma unroll
  for (int c = 0; c < 8; ++c)
    if (c < nw2) {
      const double rr = block_sum(res[c], sm.red);
      __syncthreads();
      if (tid == 0) sm.G[c] = rr;
    }
  for (int c = 8; c < nw2; ++c) {  // rarely wanted: from the residuals this thread has just stored
    double v = 0.0;
    for (int l = tid; l < nr; l += kL3Thr) {
      const double d = AY[(long long)l * p + c];
      v += d * d;
    }
    const double rr = block_sum(v, sm.red);
    __syncthreads();
    if (tid == 0) sm.G[c] = rr;
  }
  __syncthreads();
  for (int c = 0; c < nw2; ++c) conv = conv && sqrt(sm.G[c]) <= thr;
  if (tid == 0) {
    st[rk].it = it + 1;
    st[rk].conv = conv ? 1 : 0;
  }
  if (conv || q == p) return;
  // fresh directions for the dropped columns, orthogonal to the kept ones (X, complete after the barriers above)
  auto rnd = [&](int l, int c) {
    return hash_uniform(((unsigned long long)(rk + 7) << 44) ^ ((unsigned long long)it << 32) ^
                        ((unsigned long long)l * (p - q) + (c - q)));
  };
  double* d = &sm.part[0][0];  // d[c * 16 + k] = <random column c, kept column k>
  for (int e = wid; e < (p - q) * q; e += nw) {
    const int c = q + e / q, k = e % q;
    double v = 0.0, xx = 0.0;
    for (int l = lane; l < nr; l += 32) {
      const double x = X[(long long)l * p + k];
      v += rnd(l, c) * x;
      xx += x * x;
    }
    v = warp_sum(v);
    xx = warp_sum(xx);
    if (lane == 0) d[c * 16 + k] = xx > 0.0 ? v / xx : 0.0;
  }
  __syncthreads();
  for (int l = tid; l < nr; l += kL3Thr)
    for (int c = q; c < p; ++c) {
      double v = rnd(l, c);
      for (int k = 0; k < q; ++k) v -= d[c * 16 + k] * X[(long long)l * p + k];
      X[(long long)l * p + c] = v / st[rk].anorm;
      AY[(long long)l * p + c] = -v;
    }
}

__global__ void k_l3_count(const L3Rank* st, int nrank, int* left) {
  __shared__ int n;
  if (threadIdx.x == 0) n = 0;
  __syncthreads();
  for (int r = threadIdx.x; r < nrank; r += blockDim.x)
    if (!st[r].conv) atomicAdd(&n, 1);
  __syncthreads();
  if (threadIdx.x == 0) *left = n;
}

__global__ void k_l3_out(RankLayout L, int en2, int p, const double* work_all, const L3Rank* st, double* V_all,
                         double* evals_all, int* iters) {
  const int r = blockIdx.x;
  const int nr = rank_nr(L, r);
  const double* X = work_all + L.offw[r];
  double* V = V_all + L.offv[r];
  for (long long e = threadIdx.x; e < (long long)nr * en2; e += blockDim.x) {
    const int i = (int)(e / en2), j = (int)(e % en2);
    V[e] = j < st[r].q ? X[(long long)i * p + j] : -X[((long long)2 * nr + i) * p + j];
  }
  if (threadIdx.x < en2) evals_all[(long long)r * en2 + threadIdx.x] = st[r].w[threadIdx.x];
  if (threadIdx.x == 0) iters[r] = st[r].it;
}

void launch_dense_smallest_eig(const RankLayout& L, int nrank, int nr, int en2, int p, const double* A,
                               const double* inv, double* V, double* evals, int* iters, double tol, int max_it,
                               double* work, cudaStream_t st) {
  L3Rank* rs = nullptr;
  int* left = nullptr;
  if (p <= kL3Cols && cudaMallocAsync((void**)&rs, sizeof(L3Rank) * nrank + 16, st) == cudaSuccess) {
    left = reinterpret_cast<int*>(rs + nrank);
    const int gx = (nr + kL3Rows - 1) / kL3Rows;
    cudaFuncSetAttribute(k_l3_rr, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(L3Smem));
    { note_launch(); k_l3_init<<<nrank, 256, 0, st>>>(L, p, A, work, rs); }
    for (int it = 0; it < max_it; ++it) {
      { note_launch(); k_l3_mm<true><<<dim3(gx, nrank), 128, 0, st>>>(L, p, inv, work, 2, 1, rs); }
      { note_launch(); k_l3_mm<false><<<dim3(gx, nrank), 128, 0, st>>>(L, p, A, work, 1, 2, rs); }
      { note_launch(); k_l3_rr<<<nrank, kL3Thr, sizeof(L3Smem), st>>>(L, en2, p, work, rs, tol, it); }
      if ((it + 1) % 4 == 0 || it + 1 == max_it) {
        int h = 1;
        { note_launch(); k_l3_count<<<1, 256, 0, st>>>(rs, nrank, left); }
        if (cudaMemcpyAsync(&h, left, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
            cudaStreamSynchronize(st) != cudaSuccess)
          break;  // the caller's stream check reports the error
        if (h == 0) break;
      }
    }
    { note_launch(); k_l3_out<<<nrank, 256, 0, st>>>(L, en2, p, work, rs, V, evals, iters); }
    cudaFreeAsync(rs, st);
    return;
  }
  (void)cudaGetLastError();
  // wider blocks: one CTA per rank, the iteration block staged in shared memory (odd leading dimension: no
  // bank conflicts) when it fits
  int ld = p | 1;
  size_t sm = (size_t)nr * ld * sizeof(double);
  if (sm > 160 * 1024) {
    ld = 0;
    sm = 0;
  } else {  // the kernel also holds ~26 KB of static shared memory
    cudaFuncSetAttribute(k_dense_smallest_eig, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  }
  { note_launch(); k_dense_smallest_eig<<<nrank, 512, sm, st>>>(L, en2, p, A, inv, V, evals, iters, tol, max_it, work, ld); }
}

}  // namespace pmf
