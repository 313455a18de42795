// Preconditioned CG over a batch of independent problems (the reference's
// KSPCG, src/Expe_scal.c:100-119, run once per problem) in one set of launches:
// every problem keeps its own CG scalars (PcgState), and every CG kernel is a
// two-dimensional grid whose blockIdx.y is the problem, so the dot products
// are reduced per problem in a fixed order.  The preconditioner application
// in between is the shared three-level cycle of the whole batch (its
// operators are block diagonal over the problems); it runs while any problem
// is still iterating, and the CG kernels of a finished problem do nothing.
#include <algorithm>

#include "pmf_kernels.h"
#include "pmf_stencil.cuh"

namespace pmf {

namespace {
constexpr int kBT = 256;  // threads of the CG kernels

// the cells of problem q handled by thread t of block b: c0 + b*kBT + t + k*nblk*kBT
struct ProbCells {
  long long c0, c1, stride;
};
__device__ __forceinline__ ProbCells prob_cells(const ProbInfo& p, int nblk) {
  return ProbCells{p.c0 + (long long)blockIdx.x * kBT + threadIdx.x, p.c1, (long long)nblk * kBT};
}
__device__ __forceinline__ double bfixed_sum(const double* part, int n, double* red) {
  double v = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) v += part[i];
  return block_sum(v, red);
}
}  // namespace

// r = b, x = 0, partial r.r per (problem, block)
__global__ void k_bpcg_start(const ProbInfo* probs, const double* b, double* x, double* r, float* r32, double* part,
                             int nblk) {
  __shared__ double red[32];
  const int q = blockIdx.y;
  const ProbCells pc = prob_cells(probs[q], nblk);
  double v = 0.0;
  for (long long c = pc.c0; c < pc.c1; c += pc.stride) {
    const double bc = b[c];
    x[c] = 0.0;
    r[c] = bc;
    if (r32) r32[c] = (float)bc;
    v += bc * bc;
  }
  v = block_sum(v, red);
  if (threadIdx.x == 0) part[(long long)q * nblk + blockIdx.x] = v;
}
__global__ void k_bpcg_start_fin(const double* part, int nblk, PcgState* st, double* x, double rtol, double atol,
                                 int max_it) {
  __shared__ double red[32];
  const int q = blockIdx.x;
  const double v = bfixed_sum(part + (long long)q * nblk, nblk, red);
  if (threadIdx.x == 0) {
    PcgState& s = st[q];
    const double dp = sqrt(v);
    s.x = x;
    s.dp = dp;
    s.rnorm0 = dp;
    s.ttol = fmax(rtol * dp, atol);  // KSPConvergedDefault
    s.its = 0;
    s.max_it = max_it;
    s.first = 1;
    s.beta = s.betaold = s.dpi = s.dpiold = s.alpha = 0.0;
    s.done = (!(dp == dp) || isinf(dp)) ? 4 : (dp <= s.ttol) ? 1 : 0;
  }
}

// beta = z.r of each problem from the per-subdomain partials of the final level-1 visit
__global__ void k_bpcg_beta_fin(const ProbInfo* probs, const double* part, PcgState* st) {
  __shared__ double red[32];
  const int q = blockIdx.x;
  PcgState& s = st[q];
  if (s.done) return;
  const double v = bfixed_sum(part + probs[q].s0, probs[q].s1 - probs[q].s0, red);
  if (threadIdx.x == 0) {
    s.beta = v;
    if (v == 0.0) {
      s.its += 1;
      s.done = 5;  // KSP_CONVERGED_ATOL
    }
  }
}

// p <- z (first) or z + (beta/betaold) p; w <- A p: a CTA covers 256 places along the
// rows of one layer of the shared mesh, whose problem is layer_prob[z] (separator
// layers: none); layers past the grid's y limit are taken in turn.  Places past
// the problem's own extent (the shared mesh is the largest of all problems in x
// and y) add nothing; everything there is zero and stays so.  A partial of p.w per
// run and layer, so problem q's partials are the contiguous range of its layers.
// (A solve of 16 problems of 24..80 cells per axis takes 18.4 ms;
// with this step and the next over the whole shared mesh 25.)
__global__ void __launch_bounds__(kStX * kStY) k_bpcg_iter_a(Grid g, const ProbInfo* probs, const int* layer_prob,
                                                             const double* tx, const double* ty, const double* tz,
                                                             const double* diag, const double* __restrict__ z,
                                                             const double* __restrict__ pin,
                                                             double* __restrict__ pout, double* __restrict__ w,
                                                             double* __restrict__ part, const PcgState* st) {
  const int2 xy = stencil_xy(g);
  for (int ez = blockIdx.y; ez < g.P; ez += gridDim.y) {
    const int q = layer_prob[ez];
    if (q < 0) continue;
    const PcgState& s = st[q];
    if (s.done) continue;
    const double b = s.first ? 0.0 : s.beta / s.betaold;  // the first step: pin is zero
    double v = 0.0;
    if (xy.x < probs[q].M && xy.y < probs[q].N)
      stencil_march(g, tx, ty, tz, diag, ez, ez + 1, [&](long long c) { return z[c] + b * pin[c]; },
                    [&](long long c, double pc, double a) {
                      pout[c] = pc;
                      w[c] = a;
                      v = pc * a;
                    });
    v = stencil_sum(v);
    if (threadIdx.x == 0 && threadIdx.y == 0) part[(long long)ez * gridDim.x + blockIdx.x] = v;
    __syncthreads();  // the sum's scratch is reused
  }
}
__global__ void __launch_bounds__(1024) k_bpcg_iter_a_fin(const ProbInfo* probs, const double* part, int per_layer,
                                                           PcgState* st) {
  __shared__ double red[32];
  const int q = blockIdx.x;
  PcgState& s = st[q];
  if (s.done) return;
  const ProbInfo pq = probs[q];
  const double* pp = part + (long long)pq.z0 * per_layer;
  const int n = pq.P * per_layer;
  double a8[8];
#pragma unroll
  for (int u = 0; u < 8; ++u) a8[u] = 0.0;
  for (int i0 = threadIdx.x; i0 < n; i0 += 8 * blockDim.x) {
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int i = i0 + u * blockDim.x;
      if (i < n) a8[u] += pp[i];
    }
  }
  const double dpi = block_sum(((a8[0] + a8[1]) + (a8[2] + a8[3])) + ((a8[4] + a8[5]) + (a8[6] + a8[7])), red);
  if (threadIdx.x == 0) {
    s.dpiold = s.dpi;
    s.dpi = dpi;
    s.betaold = s.beta;
    const bool flip = !s.first && ((dpi > 0) != (s.dpiold > 0));
    s.first = 0;
    if (dpi == 0.0 || flip) {
      s.its += 1;
      s.done = 3;  // KSP_DIVERGED_INDEFINITE_MAT
    } else {
      s.alpha = s.beta / dpi;
    }
  }
}

// x += alpha p, r -= alpha w, partial r.r over the problem's own cells: gridDim.x CTAs per layer
__global__ void __launch_bounds__(kBT) k_bpcg_iter_b(Grid g, const ProbInfo* probs, const int* layer_prob, double* r,
                                                     float* r32, const double* p, const double* w,
                                                     double* part, const PcgState* st) {
  __shared__ double red[32];
  for (int ez = blockIdx.y; ez < g.P; ez += gridDim.y) {
    const int q = layer_prob[ez];
    if (q < 0) continue;
    const PcgState& s = st[q];
    if (s.done) continue;
    const double a = s.alpha;
    double* x = s.x;
    const int M = probs[q].M, n = M * probs[q].N;
    const long long c0 = (long long)ez * g.MN;
    double v = 0.0;
#pragma unroll 4
    for (int i = blockIdx.x * kBT + threadIdx.x; i < n; i += gridDim.x * kBT) {
      const int ey = i / M;
      const long long c = c0 + (long long)ey * g.M + (i - ey * M);
      x[c] += a * p[c];
      const double rc = r[c] - a * w[c];
      r[c] = rc;
      if (r32) r32[c] = (float)rc;
      v += rc * rc;
    }
    v = block_sum(v, red);
    if (threadIdx.x == 0) part[(long long)ez * gridDim.x + blockIdx.x] = v;
  }
}
// the residual norms, iteration counts and stop codes (a warp per problem, its partials in order), then
// all_done = 1 when every problem has stopped (the shared preconditioner kernels test it)
__global__ void __launch_bounds__(1024) k_bpcg_iter_b_fin(const ProbInfo* probs, int nprob, const double* part,
                                                          int per_layer, PcgState* st, int* all_done, LoopCond loop) {
  __shared__ int any;
  if (threadIdx.x == 0) any = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  for (int q = threadIdx.x >> 5; q < nprob; q += 32) {
    PcgState& s = st[q];
    int d = s.done;
    if (!d) {
      const double* pp = part + (long long)probs[q].z0 * per_layer;
      const int n = probs[q].P * per_layer;
      double v = 0.0;
#pragma unroll 4
      for (int i = lane; i < n; i += 32) v += pp[i];
      v = warp_sum(v);
      if (lane == 0) {
        const double dp = sqrt(v);
        s.dp = dp;
        s.its += 1;
        if (!(dp == dp) || isinf(dp))
          d = 4;
        else if (dp <= s.ttol)
          d = 1;
        else if (s.its >= s.max_it)
          d = 2;
        s.done = d;
      }
    }
    if (lane == 0 && !d) any = 1;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    *all_done = any ? 0 : 1;
    loop_while(loop, any);
  }
}
__global__ void k_bpcg_all_done(const PcgState* st, int nprob, int* all_done) {
  __shared__ int any;
  if (threadIdx.x == 0) any = 0;
  __syncthreads();
  for (int q = threadIdx.x; q < nprob; q += blockDim.x)
    if (!st[q].done) any = 1;
  __syncthreads();
  if (threadIdx.x == 0) *all_done = any ? 0 : 1;
}

void launch_bpcg_start(const ProbInfo* probs, int nprob, const double* b, double* x, double* r, float* r32,
                       double* part, PcgState* st, double rtol, double atol, int max_it, int* all_done, int nblk, cudaStream_t s) {
  { note_launch(); k_bpcg_start<<<dim3(nblk, nprob), kBT, 0, s>>>(probs, b, x, r, r32, part, nblk); }
  { note_launch(); k_bpcg_start_fin<<<nprob, 256, 0, s>>>(part, nblk, st, x, rtol, atol, max_it); }
  { note_launch(); k_bpcg_all_done<<<1, 256, 0, s>>>(st, nprob, all_done); }
}
void launch_bpcg_beta(const ProbInfo* probs, int nprob, const double* part, PcgState* st, cudaStream_t s) {
  { note_launch(); k_bpcg_beta_fin<<<nprob, 256, 0, s>>>(probs, part, st); }
}
void launch_bpcg_iter_a(const Grid& g, const ProbInfo* probs, const int* layer_prob, int nprob, const double* tx,
                        const double* ty, const double* tz, const double* diag, const double* z, const double* pin,
                        double* pout, double* w, double* part, PcgState* st, cudaStream_t s) {
  // a partial per run and layer: pcg_part_capacity(g) of them
  const dim3 grid(stencil_shape(g).grid.x, std::min(g.P, 65535));
  { note_launch(); k_bpcg_iter_a<<<grid, dim3(kStX, kStY), 0, s>>>(g, probs, layer_prob, tx, ty, tz, diag, z, pin, pout, w, part, st); }
  { note_launch(); k_bpcg_iter_a_fin<<<nprob, 1024, 0, s>>>(probs, part, (int)grid.x, st); }
}
void launch_bpcg_iter_b(const Grid& g, const ProbInfo* probs, const int* layer_prob, int nprob, double* r, float* r32,
                        const double* p, const double* w, double* part, PcgState* st, int* all_done, LoopCond loop,
                        cudaStream_t s) {
  const int sub = std::max(1, std::min(32, (int)(g.MN / 2048)));  // CTAs per layer, fewer than its runs
  { note_launch(); k_bpcg_iter_b<<<dim3(sub, std::min(g.P, 65535)), kBT, 0, s>>>(g, probs, layer_prob, r, r32, p, w, part, st); }
  { note_launch(); k_bpcg_iter_b_fin<<<1, 1024, 0, s>>>(probs, nprob, part, sub, st, all_done, loop); }
}

}  // namespace pmf
