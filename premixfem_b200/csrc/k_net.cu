// Kernels of the learned-initialisation network (layer table in pmf_net.h).
//
// Forward: every layer is one implicit GEMM, out[row][cout] = sum over
// (tap, cin) of in[gather(row, tap)][cin] * W[tap][cin][cout], computed on
// the BF16 tensor cores (mma.sync m16n8k16, FP32 accumulation) with the bias,
// skip addition, ReLU and the BF16 rounding fused in the epilogue.  A CTA owns
// 64 output voxels of one sample and all output channels; per tap it stages
// the 64 gathered input rows and the tap's weight slice in shared memory.
// Transposed (up2) layers order their rows by (sample, parity, coarse voxel)
// so that one tile uses one weight slice.
//
// Backward (training only, FP32 CUDA cores): the input gradient is a gather
// over the taps that touched each input voxel, fused with the skip-gradient
// addition and the ReLU mask of the input activation; the weight gradient is
// a tiled reduction over output rows with FP32 atomics per chunk.
#include <cuda_bf16.h>

#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

#include "pmf_kernels.h"
#include "pmf_net.h"
#include "tune.h"

namespace pmf {

const NetLayer kNetLayers[NET_LAYERS] = {
    // type     cin cout s_in s_out relu skip in out
    {NL_CONV3, 16, 32, 16, 16, 1, -1, 0, 1},
    {NL_DOWN2, 32, 64, 16, 8, 1, -1, 1, 2},
    {NL_CONV3, 64, 64, 8, 8, 1, -1, 2, 3},
    {NL_DOWN2, 64, 96, 8, 4, 1, -1, 3, 4},
    {NL_CONV3, 96, 96, 4, 4, 1, -1, 4, 5},
    {NL_UP2, 96, 64, 4, 8, 1, 3, 5, 6},
    {NL_UP2, 64, 32, 8, 16, 1, 1, 6, 7},
    {NL_CONV3, 32, 32, 16, 16, 1, -1, 7, 8},
    {NL_CONV1, 32, 16, 16, 16, 0, -1, 8, 9},
};
const NetActShape kNetActs[NET_ACTS] = {{16, 16}, {16, 32}, {8, 64}, {8, 64}, {4, 96},
                                        {4, 96},  {8, 64},  {16, 32}, {16, 32}, {16, 16}};

namespace {

__device__ __forceinline__ int cube(int s) { return s * s * s; }

// Input voxel read by output voxel o through tap t (-1: zero padding / not this tap).
__device__ __forceinline__ int in_vox(int type, int s_in, int s_out, int o, int t) {
  int x = o % s_out, y = (o / s_out) % s_out, z = o / (s_out * s_out);
  if (type == NL_CONV3) {
    x += t % 3 - 1;
    y += (t / 3) % 3 - 1;
    z += t / 9 - 1;
    if (x < 0 || y < 0 || z < 0 || x >= s_in || y >= s_in || z >= s_in) return -1;
    return (z * s_in + y) * s_in + x;
  }
  if (type == NL_DOWN2) return ((2 * z + (t >> 2)) * s_in + 2 * y + ((t >> 1) & 1)) * s_in + 2 * x + (t & 1);
  if (type == NL_CONV1) return o;
  const int par = (x & 1) | ((y & 1) << 1) | ((z & 1) << 2);
  if (par != t) return -1;
  return ((z >> 1) * s_in + (y >> 1)) * s_in + (x >> 1);
}

// Fine voxel of coarse voxel v (edge s_in) and parity d.
__device__ __forceinline__ int up_vox(int v, int d, int s_in) {
  const int x = v % s_in, y = (v / s_in) % s_in, z = v / (s_in * s_in), s = 2 * s_in;
  return ((2 * z + (d >> 2)) * s + 2 * y + ((d >> 1) & 1)) * s + 2 * x + (d & 1);
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(addr));
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(addr));
}
__device__ __forceinline__ void mma_bf16(float* c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

struct FwdArgs {
  int type, cin, cout, s_in, s_out, relu;
  const __nv_bfloat16* in;
  const __nv_bfloat16* W;
  const float* bias;
  const __nv_bfloat16* skip;
  __nv_bfloat16* out;
  float* outf;
};

__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool valid) {
  // 16-byte global->shared copy; zero-filled when !valid (src-size 0)
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  const int n = valid ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(n));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

// ROWS output voxels of one sample per CTA (ROWS / (16 MT) warps, each MT
// 16-row tiles x all output channels, sharing the weight fragments); the
// gathered input rows and the weight slice of the next tap are copied with
// cp.async while the current tap is multiplied.
template <int NT, int ROWS, int MT>
__global__ void __launch_bounds__(ROWS * 2 / MT) k_net_fwd(FwdArgs a) {
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ int rowout[ROWS];
  const int lda = a.cin + 8, ldb = a.cout + 8;
  __nv_bfloat16* As0 = reinterpret_cast<__nv_bfloat16*>(smraw);
  __nv_bfloat16* Bs0 = As0 + 2 * ROWS * lda;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nthr = ROWS * 2 / MT;
  const int so3 = cube(a.s_out), si3 = cube(a.s_in);
  const long long r0 = (long long)blockIdx.x * ROWS;
  const int b = (int)(r0 / so3);
  const int rem0 = (int)(r0 % so3);
  const bool up = a.type == NL_UP2;
  const int d_tile = up ? rem0 / si3 : 0;
  for (int q = tid; q < ROWS; q += nthr) rowout[q] = up ? up_vox((rem0 + q) % si3, d_tile, a.s_in) : rem0 + q;
  __syncthreads();
  const int ntap = (up || a.type == NL_CONV1) ? 1 : net_taps(a.type);
  const int vin = a.cin >> 3, vout = a.cout >> 3;
  // Per-thread copy assignments, fixed for all taps: up to EA input-row
  // vectors and EB weight vectors, with their coordinates precomputed so the
  // per-tap gather needs no division.
  constexpr int NTHR = ROWS * 2 / MT;
  constexpr int EA = (ROWS * 12 + NTHR - 1) / NTHR;  // cin <= 96: 12 vectors per row
  constexpr int EB = (96 * 12 + NTHR - 1) / NTHR;
  int a_dst[EA], a_xyz[EA], a_src[EA];
  int b_dst[EB];
  const int sin = a.s_in;
#pragma unroll
  for (int j = 0; j < EA; ++j) {
    const int e = tid + j * nthr;
    a_dst[j] = -1;
    if (e < ROWS * vin) {
      const int rr = e / vin, cv = e % vin;
      a_dst[j] = rr * lda + cv * 8;
      if (up) {
        a_src[j] = ((rem0 + rr) % si3) * a.cin + cv * 8;
        a_xyz[j] = 0;
      } else {
        const int o = rowout[rr], so = a.s_out;
        int x = o % so, y = (o / so) % so, z = o / (so * so);
        if (a.type == NL_DOWN2) {
          x *= 2;
          y *= 2;
          z *= 2;
        }
        a_xyz[j] = x | (y << 10) | (z << 20);
        a_src[j] = ((z * sin + y) * sin + x) * a.cin + cv * 8;
      }
    }
  }
#pragma unroll
  for (int j = 0; j < EB; ++j) {
    const int e = tid + j * nthr;
    b_dst[j] = e < a.cin * vout ? (e / vout) * ldb + (e % vout) * 8 : -1;
  }
  const __nv_bfloat16* inb = a.in + (size_t)b * si3 * a.cin;
  auto stage = [&](int ti, int buf) {
    const int t = up ? d_tile : ti;
    __nv_bfloat16* As = As0 + buf * ROWS * lda;
    __nv_bfloat16* Bs = Bs0 + buf * a.cin * ldb;
    int dx = 0, dy = 0, dz = 0;
    if (a.type == NL_CONV3) {
      dx = t % 3 - 1;
      dy = (t / 3) % 3 - 1;
      dz = t / 9 - 1;
    } else if (a.type == NL_DOWN2) {
      dx = t & 1;
      dy = (t >> 1) & 1;
      dz = t >> 2;
    }
    const int off = ((dz * sin + dy) * sin + dx) * a.cin;
#pragma unroll
    for (int j = 0; j < EA; ++j) {
      if (a_dst[j] < 0) continue;
      bool ok = true;
      if (a.type == NL_CONV3) {
        const int x = (a_xyz[j] & 1023) + dx, y = ((a_xyz[j] >> 10) & 1023) + dy, z = (a_xyz[j] >> 20) + dz;
        ok = x >= 0 && y >= 0 && z >= 0 && x < sin && y < sin && z < sin;
      }
      const int src = ok ? a_src[j] + (up || a.type == NL_CONV1 ? 0 : off) : 0;
      cp_async16(As + a_dst[j], inb + src, ok);
    }
    const __nv_bfloat16* wt = a.W + (size_t)t * a.cin * a.cout;
#pragma unroll
    for (int j = 0; j < EB; ++j) {
      if (b_dst[j] < 0) continue;
      cp_async16(Bs + b_dst[j], wt + 8 * (tid + j * nthr), true);
    }
    cp_async_commit();
  };
  float acc[MT][NT][4];
#pragma unroll
  for (int mt = 0; mt < MT; ++mt)
#pragma unroll
    for (int n = 0; n < NT; ++n) acc[mt][n][0] = acc[mt][n][1] = acc[mt][n][2] = acc[mt][n][3] = 0.f;
  stage(0, 0);
  for (int ti = 0; ti < ntap; ++ti) {
    if (ti + 1 < ntap) {
      stage(ti + 1, (ti + 1) & 1);
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
    const __nv_bfloat16* As = As0 + (ti & 1) * ROWS * lda;
    const __nv_bfloat16* Bs = Bs0 + (ti & 1) * a.cin * ldb;
    for (int kc = 0; kc < a.cin; kc += 16) {
      uint32_t af[MT][4];
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
        ldsm_x4(smem_u32(As + ((warp * MT + mt) * 16 + (lane & 15)) * lda + kc + (lane >> 4) * 8), af[mt][0],
                af[mt][1], af[mt][2], af[mt][3]);
#pragma unroll
      for (int np = 0; np < NT / 2; ++np) {
        uint32_t b0, b1, b2, b3;
        ldsm_x4_t(smem_u32(Bs + (kc + (lane & 7) + ((lane >> 3) & 1) * 8) * ldb + np * 16 + (lane >> 4) * 8), b0, b1,
                  b2, b3);
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
          mma_bf16(acc[mt][2 * np], af[mt][0], af[mt][1], af[mt][2], af[mt][3], b0, b1);
          mma_bf16(acc[mt][2 * np + 1], af[mt][0], af[mt][1], af[mt][2], af[mt][3], b2, b3);
        }
      }
    }
    __syncthreads();  // the buffer just read is refilled two taps later
  }
  // epilogue: bias, skip, ReLU, store
#pragma unroll
  for (int mt = 0; mt < MT; ++mt)
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int rr = (warp * MT + mt) * 16 + (lane >> 2) + h * 8;
    const size_t rowbase = ((size_t)b * so3 + rowout[rr]) * a.cout;
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      const int col = n * 8 + (lane & 3) * 2;
      float v0 = acc[mt][n][2 * h] + a.bias[col];
      float v1 = acc[mt][n][2 * h + 1] + a.bias[col + 1];
      if (a.skip) {
        const __nv_bfloat162 s2 = *reinterpret_cast<const __nv_bfloat162*>(a.skip + rowbase + col);
        v0 += __bfloat162float(s2.x);
        v1 += __bfloat162float(s2.y);
      }
      if (a.relu) {
        v0 = fmaxf(v0, 0.f);
        v1 = fmaxf(v1, 0.f);
      }
      if (a.outf) {
        *reinterpret_cast<float2*>(a.outf + rowbase + col) = make_float2(v0, v1);
      } else {
        *reinterpret_cast<__nv_bfloat162*>(a.out + rowbase + col) = __floats2bfloat162_rn(v0, v1);
      }
    }
  }
}

// ---- 3x3x3 convolutions of 16^3 patches on the tcgen05 tensor cores ---------------------------
// One CTA (four warps) per patch marches through the 16 output z-planes.  The
// input planes z-1, z, z+1 sit with a one-voxel zero halo in a ring of four
// shared-memory slots ([slot][cin/8][18][18][8 channels] BF16) while plane
// z+2 is copied in with cp.async; all 27 taps' weights stay resident in the
// UMMA K-major layout ([tap][k-step][2][cout/8][8][8]).  An output plane is
// two 128-row tiles (rows y x 8 x-positions, one per x half), and for tap
// (dx, dy, dz) a tile's A operand is just a window of the haloed plane: a
// no-swizzle K-major descriptor whose 8-row groups step by one haloed row
// (288 B) and whose two 8-channel groups step by one channel plane, so the
// im2col gather costs nothing.  One thread issues the 27 x cin/16 x 2
// tcgen05.mma (kind::f16, BF16 in, FP32 accumulation in TMEM, M = 128,
// N = cout) and commits them to the plane's mbarrier; the accumulators are
// double-buffered across planes so that the epilogue of plane z-1
// (tcgen05.ld, bias, ReLU, BF16 store) overlaps the MMAs of plane z.  Every
// wait is bounded; a wait that runs out sets *err and skips the stores.
// Every load is a plain per-CTA cp.async (single-GPU code).
namespace {
constexpr int kTcPl = 18 * 18;                 // positions of one haloed plane
constexpr long long kTcSpin = 1LL << 24;      // mbarrier polls before giving up

__device__ __forceinline__ void tc_mbar_init(uint64_t* b) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(b)) : "memory");
}
__device__ __forceinline__ bool tc_mbar_try(uint64_t* b, uint32_t ph) {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n}"
               : "=r"(ok)
               : "r"(smem_u32(b)), "r"(ph)
               : "memory");
  return ok != 0;
}
// shared-memory matrix descriptor: no swizzle, K-major, sm_100 version bit
__device__ __forceinline__ uint64_t tc_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | ((uint64_t)1 << 46);
}
// instruction descriptor of kind::f16: BF16 A and B (K-major), FP32 D, M x N
__host__ __device__ constexpr uint32_t tc_idesc(int M, int N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}
template <int CIN, int COUT>
constexpr size_t tc_conv_smem() {
  return (size_t)27 * CIN * COUT * 2 + 4 * (CIN / 8) * kTcPl * 16 + 64;
}
}  // namespace

template <int CIN, int COUT>
__global__ void __launch_bounds__(128, 1) k_net_conv_tc(const __nv_bfloat16* in, const __nv_bfloat16* wpk,
                                                       const float* bias, __nv_bfloat16* out, int* err) {
  constexpr int VIN = CIN / 8, KS = CIN / 16;
  constexpr int WBYTES = 27 * CIN * COUT * 2;
  constexpr int SLOT = VIN * kTcPl * 16;
  constexpr int NCOL = 4 * COUT <= 32 ? 32 : (4 * COUT <= 64 ? 64 : (4 * COUT <= 128 ? 128 : 256));
  static_assert(CIN % 16 == 0 && COUT % 16 == 0 && 4 * COUT <= 256, "tile shape");
  extern __shared__ __align__(1024) unsigned char tc_sm[];
  unsigned char* slab = tc_sm + WBYTES;
  uint64_t* mbar = reinterpret_cast<uint64_t*>(slab + 4 * SLOT);
  uint32_t* taddr_s = reinterpret_cast<uint32_t*>(mbar + 2);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int b = blockIdx.x;
  const __nv_bfloat16* inb = in + (size_t)b * 4096 * CIN;
  const uint32_t wsa = smem_u32(tc_sm), sla = smem_u32(slab);
  for (int c = tid; c < WBYTES / 16; c += 128)
    cp_async16(tc_sm + c * 16, reinterpret_cast<const char*>(wpk) + c * 16, true);
  auto load_plane = [&](int zi) {
    unsigned char* base = slab + ((zi + 1) & 3) * SLOT;
    for (int e = tid; e < VIN * kTcPl; e += 128) {
      const int cg = e / kTcPl, pp = e % kTcPl, y = pp / 18 - 1, x = pp % 18 - 1;
      const bool ok = zi >= 0 && zi < 16 && y >= 0 && y < 16 && x >= 0 && x < 16;
      const __nv_bfloat16* src = ok ? inb + ((size_t)((zi * 16 + y) * 16 + x) * CIN + cg * 8) : inb;
      cp_async16(base + (cg * kTcPl + pp) * 16, src, ok);
    }
  };
  load_plane(-1);
  load_plane(0);
  cp_async_commit();
  load_plane(1);
  cp_async_commit();
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(taddr_s)),
                 "r"(NCOL));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
  }
  if (tid == 0) {
    tc_mbar_init(mbar);
    tc_mbar_init(mbar + 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *taddr_s;
  constexpr uint32_t idesc = tc_idesc(128, COUT);
  bool ok = true;
  auto wait_mma = [&](int zz) {
    for (long long s = 0; !tc_mbar_try(mbar + (zz & 1), (uint32_t)((zz >> 1) & 1)); ++s)
      if (s > kTcSpin) {
        ok = false;
        break;
      }
  };
  auto epilogue = [&](int zz) {
    const uint32_t buf = (uint32_t)((zz & 1) * 2 * COUT);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int m = 32 * warp + lane, y = m >> 3, x = 8 * h + (m & 7);
      __nv_bfloat16* op = out + ((size_t)b * 4096 + (zz * 16 + y) * 16 + x) * COUT;
#pragma unroll
      for (int c0 = 0; c0 < COUT; c0 += 16) {
        uint32_t r[16];
        const uint32_t ta = tmem + ((uint32_t)(32 * warp) << 16) + buf + (uint32_t)(h * COUT + c0);
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
              "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
            : "r"(ta));
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        uint32_t pk[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const float v0 = fmaxf(__uint_as_float(r[2 * q]) + bias[c0 + 2 * q], 0.f);
          const float v1 = fmaxf(__uint_as_float(r[2 * q + 1]) + bias[c0 + 2 * q + 1], 0.f);
          __nv_bfloat162 bb = __floats2bfloat162_rn(v0, v1);
          pk[q] = *reinterpret_cast<uint32_t*>(&bb);
        }
        uint4* dst = reinterpret_cast<uint4*>(op + c0);
        dst[0] = make_uint4(pk[0], pk[1], pk[2], pk[3]);
        dst[1] = make_uint4(pk[4], pk[5], pk[6], pk[7]);
      }
    }
  };
  for (int z = 0; z < 16; ++z) {
    cp_async_wait<0>();  // the weights and the planes up to z + 1 have landed
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (tid == 0) {
      const uint32_t dbuf = tmem + (uint32_t)((z & 1) * 2 * COUT);
      int cnt = 0;
      for (int t = 0; t < 27; ++t) {
        const int dx = t % 3 - 1, dy = (t / 3) % 3 - 1, dz = t / 9 - 1;
        const uint32_t pbase = sla + (uint32_t)(((z + dz + 1) & 3) * SLOT);
#pragma unroll
        for (int ks = 0; ks < KS; ++ks) {
          const uint64_t bd = tc_desc(wsa + (uint32_t)((t * KS + ks) * 16 * COUT * 2), (COUT / 8) * 128, 128);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const uint32_t a0 = pbase + (uint32_t)(((2 * ks) * kTcPl + (1 + dy) * 18 + (1 + dx + 8 * h)) * 16);
            const uint64_t ad = tc_desc(a0, kTcPl * 16, 18 * 16);
            const uint32_t acc = cnt >= 2 ? 1u : 0u;  // each half's first MMA starts from zero
            asm volatile(
                "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}\n" ::"r"(
                    dbuf + (uint32_t)(h * COUT)),
                "l"(ad), "l"(bd), "r"(idesc), "r"(acc), "r"(0u), "r"(0u), "r"(0u), "r"(0u));
            ++cnt;
          }
        }
      }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                       smem_u32(mbar + (z & 1)))
                   : "memory");
    }
    // plane z + 2 replaces plane z - 2, which the MMAs of plane z - 1 read last
    if (z >= 1) wait_mma(z - 1);
    if (z + 2 <= 16) load_plane(z + 2);
    cp_async_commit();
    if (z >= 1 && ok) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      epilogue(z - 1);
    }
  }
  wait_mma(15);
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (ok) epilogue(15);
  if (!ok) atomicOr(err, 1);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(NCOL));
}

// W[tap][cin][cout] (BF16) -> [tap][cin/16][2][cout/8][8 n][8 k], the B operand of k_net_conv_tc
__global__ void k_net_pack_tc(int cin, int cout, const __nv_bfloat16* w16, __nv_bfloat16* wpk) {
  const int n = 27 * cin * cout;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int co = i % cout, ci = (i / cout) % cin, t = i / (cin * cout);
    const int ks = ci / 16, k = ci % 16;
    const size_t blk = (size_t)(t * (cin / 16) + ks) * 16 * cout;
    wpk[blk + ((k / 8) * (cout / 8) + co / 8) * 64 + (co % 8) * 8 + k % 8] = w16[i];
  }
}

// layers k_net_conv_tc takes: 3x3x3 on 16^3 with ReLU, no skip, BF16 output
static bool conv_tc_layer(const NetLayer& L) {
  return L.type == NL_CONV3 && L.s_in == 16 && L.s_out == 16 && L.relu && L.skip < 0 &&
         ((L.cin == 16 && L.cout == 32) || (L.cin == 32 && L.cout == 32));
}

static void conv_tc_launch(const NetLayer& L, const __nv_bfloat16* in, const __nv_bfloat16* wpk, const float* bias,
                           __nv_bfloat16* out, int B, int* err, cudaStream_t st) {
  if (L.cin == 16) {
    constexpr size_t sm = tc_conv_smem<16, 32>();
    cudaFuncSetAttribute(k_net_conv_tc<16, 32>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    k_net_conv_tc<16, 32><<<B, 128, sm, st>>>(in, wpk, bias, out, err);
  } else {
    constexpr size_t sm = tc_conv_smem<32, 32>();
    cudaFuncSetAttribute(k_net_conv_tc<32, 32>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    k_net_conv_tc<32, 32><<<B, 128, sm, st>>>(in, wpk, bias, out, err);
  }
}

// ---- backward -------------------------------------------------------------------------------
struct DgradArgs {
  int type, cin, cout, s_in, s_out, B;
  const float* dz;                // pre-activation gradient of this layer's output [B][s_out^3][cout]
  const float* wt;                // W[tap][cout][cin] (FP32)
  const __nv_bfloat16* in_act;    // this layer's input activation (ReLU mask), may be null
  const float* add;               // gradient reaching the input through a skip, may be null
  float* din;                     // pre-activation gradient of the previous layer's output
};

// din[row][ci] = sum over taps t and output channels co of dz[out(row, t)][co] W[t][co][ci], masked by the
// input's ReLU, plus the skip gradient: an implicit GEMM in FP32 on the CUDA cores (the gradients are FP32
// and stay so), so bound by FP32 multiply-adds.  A CTA computes 128 rows x CIN channels, a thread TM x TN of
// them from shared-memory tiles of 16 channels of dz of one tap; the next tile is on its way in registers
// meanwhile.  The sum over (t, co) runs in the same order for every element as one thread per element would
// take it.  Rows are input voxels, for the stride-2 layer grouped by parity (one tap each).
// 64 patches, the 16^3 32 -> 32 layer: 3.33 ms with one thread per element, 0.53 ms.
template <int CIN, int TM, int TN>
__global__ void __launch_bounds__(256) k_net_dgrad(DgradArgs a) {
  constexpr int BM = 128, BK = 16, LDA = BM + 4;
  static_assert((BM / TM) * (CIN / TN) == 256, "one thread per TM x TN outputs");
  __shared__ __align__(16) float As[BK][LDA];
  __shared__ __align__(16) float Ws[BK][CIN];
  const int si = a.s_in, so = a.s_out, si3 = cube(si), so3 = cube(so);
  const bool down = a.type == NL_DOWN2;
  // rows of this tile: parity t0 of the stride-2 layer and output voxels, or input voxels
  const long long per = (long long)a.B * (down ? so3 : si3);
  const int tiles = (int)((per + BM - 1) / BM);
  const int t0 = down ? blockIdx.x / tiles : 0;
  const long long r0 = (long long)(blockIdx.x - t0 * tiles) * BM;
  // this thread's row of the dz tile (two threads a row, eight channels each)
  const int lr = threadIdx.x >> 1, lk = (threadIdx.x & 1) * 8;
  const bool lin = r0 + lr < per;
  const long long lrow = lin ? r0 + lr : 0;
  const int lb = (int)(lrow / (down ? so3 : si3)), lv = (int)(lrow % (down ? so3 : si3));
  const int lx = lv % (down ? so : si), ly = (lv / (down ? so : si)) % (down ? so : si),
            lz = lv / ((down ? so : si) * (down ? so : si));
  const float* dzb = a.dz + (size_t)lb * so3 * a.cout;
  const int ntap = a.type == NL_CONV3 ? 27 : a.type == NL_UP2 ? 8 : 1, nk = a.cout / BK, nchunk = ntap * nk;
  float4 ra[2], rw[2];
  constexpr int WV = BK * CIN / 4;  // float4s of a weight tile
  auto fetch = [&](int ch) {
    const int ti = ch / nk, k0 = (ch - ti * nk) * BK, t = down ? t0 : ti;
    int o = -1;
    if (lin) {
      if (a.type == NL_CONV3) {
        const int ox = lx - (t % 3 - 1), oy = ly - ((t / 3) % 3 - 1), oz = lz - (t / 9 - 1);
        if (ox >= 0 && oy >= 0 && oz >= 0 && ox < so && oy < so && oz < so) o = (oz * so + oy) * so + ox;
      } else {
        o = a.type == NL_UP2 ? up_vox(lv, t, si) : lv;
      }
    }
    ra[0] = ra[1] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (o >= 0) {
      const float4* src = reinterpret_cast<const float4*>(dzb + (size_t)o * a.cout + k0 + lk);
      ra[0] = src[0];
      ra[1] = src[1];
    }
    const float4* w = reinterpret_cast<const float4*>(a.wt + ((size_t)t * a.cout + k0) * CIN);
#pragma unroll
    for (int q = 0; q < 2; ++q)
      if (threadIdx.x + 256 * q < WV) rw[q] = w[threadIdx.x + 256 * q];
  };
  const int tn = threadIdx.x % (CIN / TN), tm = threadIdx.x / (CIN / TN);
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
  fetch(0);
  for (int ch = 0; ch < nchunk; ++ch) {
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      As[lk + 4 * q][lr] = ra[q].x;
      As[lk + 4 * q + 1][lr] = ra[q].y;
      As[lk + 4 * q + 2][lr] = ra[q].z;
      As[lk + 4 * q + 3][lr] = ra[q].w;
      if (threadIdx.x + 256 * q < WV) reinterpret_cast<float4*>(&Ws[0][0])[threadIdx.x + 256 * q] = rw[q];
    }
    __syncthreads();
    if (ch + 1 < nchunk) fetch(ch + 1);
#pragma unroll
    for (int k = 0; k < BK; ++k) {
      float av[TM], wv[TN];
#pragma unroll
      for (int i = 0; i < TM; i += 4) *reinterpret_cast<float4*>(av + i) = *reinterpret_cast<const float4*>(&As[k][tm * TM + i]);
#pragma unroll
      for (int j = 0; j < TN; j += 2) *reinterpret_cast<float2*>(wv + j) = *reinterpret_cast<const float2*>(&Ws[k][tn * TN + j]);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] += av[i] * wv[j];
    }
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const long long row = r0 + tm * TM + i;
    if (row >= per) continue;
    size_t vox = (size_t)row;  // input voxel (b, i)
    if (down) {
      const int b = (int)(row / so3), v = (int)(row % so3);
      vox = (size_t)b * si3 + up_vox(v, t0, so);
    }
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const size_t idx = vox * CIN + tn * TN + j;
      float v = 0.f;
      if (!a.in_act || __bfloat162float(a.in_act[idx]) > 0.f) v = acc[i][j] + (a.add ? a.add[idx] : 0.f);
      a.din[idx] = v;
    }
  }
}
static bool dgrad_launch(const DgradArgs& d, cudaStream_t st) {
  const int so3 = d.s_out * d.s_out * d.s_out, si3 = d.s_in * d.s_in * d.s_in;
  const long long per = (long long)d.B * (d.type == NL_DOWN2 ? so3 : si3);
  const int grid = (int)((per + 127) / 128) * (d.type == NL_DOWN2 ? 8 : 1);
  note_launch();
  if (d.cin == 32)
    k_net_dgrad<32, 4, 4><<<grid, 256, 0, st>>>(d);
  else if (d.cin == 64)
    k_net_dgrad<64, 8, 4><<<grid, 256, 0, st>>>(d);
  else if (d.cin == 96)
    k_net_dgrad<96, 8, 6><<<grid, 256, 0, st>>>(d);
  else
    return false;
  return true;
}

struct WgradArgs {
  int type, cin, cout, s_in, s_out, B, rows_per_chunk;
  const __nv_bfloat16* in;  // layer input activation
  const float* dz;          // pre-activation gradient of the output
  float* gw;                // [tap][cin][cout], accumulated
};

// dW[t][ci][co] = sum over output rows of in[gather(row, t)][ci] * dz[row][co], in FP32 on the CUDA cores.
// blockIdx.y = group of G taps, blockIdx.x = chunk of rows; a thread holds TA x TB outputs of each of the G
// taps, so that a row's dz is read from shared memory once for all of them (one tap of 32 x 32 channels alone
// gives a thread four multiply-adds for four reads, nine taps 36 for ten).  The rows' chunks are at least as many as
// fill the chip, their sums added atomically.
// 64 patches, the 16^3 32 -> 32 layer: 2.33 ms with one tap per CTA, 0.73 ms.
template <int CIN, int COUT, int TA, int TB, int G>
__global__ void __launch_bounds__((CIN / TA) * (COUT / TB)) k_net_wgrad(WgradArgs a) {
  constexpr int RT = 16, NT = (CIN / TA) * (COUT / TB), LX = CIN + 4, LZ = COUT + 4;
  __shared__ __align__(16) float xs[G][RT][LX];
  __shared__ __align__(16) float zs[RT][LZ];
  const int tg = blockIdx.y * G;
  const bool up = a.type == NL_UP2;
  const int so3 = cube(a.s_out), si3 = cube(a.s_in);
  const int rv = up ? si3 : so3;  // rows of a patch
  const long long nrows = (long long)a.B * rv;
  const long long rbeg = (long long)blockIdx.x * a.rows_per_chunk;
  const long long rend = min(nrows, rbeg + a.rows_per_chunk);
  const int tx = threadIdx.x % (COUT / TB), ty = threadIdx.x / (COUT / TB);
  float acc[G][TA][TB];
#pragma unroll
  for (int g = 0; g < G; ++g)
#pragma unroll
    for (int i = 0; i < TA; ++i)
#pragma unroll
      for (int j = 0; j < TB; ++j) acc[g][i][j] = 0.f;
  for (long long r0 = rbeg; r0 < rend; r0 += RT) {
    // input rows of the G taps, eight BF16 channels per load
#pragma unroll 2
    for (int e = threadIdx.x; e < G * RT * (CIN / 8); e += NT) {
      const int c8 = e % (CIN / 8), rr = (e / (CIN / 8)) % RT, g = e / (RT * (CIN / 8));
      const long long row = r0 + rr;
      uint4 v = make_uint4(0, 0, 0, 0);
      if (row < rend) {
        const int b = (int)(row / rv), o = (int)(row % rv);
        const int iv = up ? o : in_vox(a.type, a.s_in, a.s_out, o, tg + g);
        if (iv >= 0) v = *reinterpret_cast<const uint4*>(a.in + ((size_t)b * si3 + iv) * CIN + 8 * c8);
      }
      const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
      float2 f[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) f[q] = __bfloat1622float2(h[q]);
      float4* d = reinterpret_cast<float4*>(&xs[g][rr][8 * c8]);
      d[0] = make_float4(f[0].x, f[0].y, f[1].x, f[1].y);
      d[1] = make_float4(f[2].x, f[2].y, f[3].x, f[3].y);
    }
    for (int e = threadIdx.x; e < RT * (COUT / 4); e += NT) {
      const int c4 = e % (COUT / 4), rr = e / (COUT / 4);
      const long long row = r0 + rr;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (row < rend) {
        const int b = (int)(row / rv), i = (int)(row % rv);
        const int o = up ? up_vox(i, tg, a.s_in) : i;
        v = *reinterpret_cast<const float4*>(a.dz + ((size_t)b * so3 + o) * COUT + 4 * c4);
      }
      *reinterpret_cast<float4*>(&zs[rr][4 * c4]) = v;
    }
    __syncthreads();
#pragma unroll 4
    for (int rr = 0; rr < RT; ++rr) {
      float zv[TB];
#pragma unroll
      for (int j = 0; j < TB; j += 2) *reinterpret_cast<float2*>(zv + j) = *reinterpret_cast<const float2*>(&zs[rr][tx * TB + j]);
#pragma unroll
      for (int g = 0; g < G; ++g) {
        float xv[TA];
#pragma unroll
        for (int i = 0; i < TA; i += 2) *reinterpret_cast<float2*>(xv + i) = *reinterpret_cast<const float2*>(&xs[g][rr][ty * TA + i]);
#pragma unroll
        for (int i = 0; i < TA; ++i)
#pragma unroll
          for (int j = 0; j < TB; ++j) acc[g][i][j] += xv[i] * zv[j];
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int g = 0; g < G; ++g)
#pragma unroll
    for (int i = 0; i < TA; ++i)
#pragma unroll
      for (int j = 0; j < TB; ++j)
        atomicAdd(&a.gw[((size_t)(tg + g) * CIN + ty * TA + i) * COUT + tx * TB + j], acc[g][i][j]);
}
template <int CIN, int COUT, int TA, int TB, int G>
static void wgrad_launch(WgradArgs w, long long rows, int taps, cudaStream_t st) {
  // about four CTAs per SM, chunks of 64 rows at least and 2 048 at most: a chunk is one chain of FP32 additions
  const long long chunks = std::max<long long>(1, std::min<long long>(rows / 64, (148LL * 4 * G + taps - 1) / taps));
  w.rows_per_chunk = (int)std::min<long long>(2048, ((rows + chunks - 1) / chunks + 15) & ~15LL);
  const dim3 grid((unsigned)((rows + w.rows_per_chunk - 1) / w.rows_per_chunk), taps / G);
  note_launch();
  k_net_wgrad<CIN, COUT, TA, TB, G><<<grid, (CIN / TA) * (COUT / TB), 0, st>>>(w);
}

// gb[co] = sum over rows of dz[row][co]: a CTA sums a chunk of rows for all channels (a thread per channel and
// row class, coalesced), the last pass adds the chunks in order.  One CTA per channel, a strided column each,
// took 85 us a layer.
constexpr int kBgradCtas = 148;
__global__ void __launch_bounds__(256) k_net_bgrad(const float* dz, long long rows, int cout, double* part) {
  __shared__ double red[256];
  const int nr = 256 / cout, c = threadIdx.x % cout, q = threadIdx.x / cout;  // threads past nr * cout idle
  const long long per = (rows + gridDim.x - 1) / gridDim.x;
  const long long r1 = min(rows, (blockIdx.x + 1LL) * per);
  double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
  if (q < nr) {
    long long r = blockIdx.x * per + q;
    for (; r + 3LL * nr < r1; r += 4LL * nr) {
      s0 += dz[r * cout + c];
      s1 += dz[(r + nr) * cout + c];
      s2 += dz[(r + 2LL * nr) * cout + c];
      s3 += dz[(r + 3LL * nr) * cout + c];
    }
    for (; r < r1; r += nr) s0 += dz[r * cout + c];
  }
  red[threadIdx.x] = (s0 + s1) + (s2 + s3);
  __syncthreads();
  if (threadIdx.x < cout) {
    double s = 0.0;
    for (int i = 0; i < nr; ++i) s += red[i * cout + threadIdx.x];
    part[(long long)blockIdx.x * cout + threadIdx.x] = s;
  }
}
__global__ void k_net_bgrad_fin(const double* part, int nblk, int cout, float* gb) {
  if ((int)threadIdx.x >= cout) return;
  double s = 0.0;
#pragma unroll 8
  for (int b = 0; b < nblk; ++b) s += part[(long long)b * cout + threadIdx.x];
  gb[threadIdx.x] = (float)s;
}

__global__ void k_net_adam(long long n, float* w, const float* g, float* m, float* v, float lr, float b1, float b2,
                           float eps, float wd, float bc1, float bc2) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const float gi = g[i] + wd * w[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    w[i] -= lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
  }
}

// BF16 copy W16[t][ci][co] and FP32 transpose Wt[t][co][ci] of the master weights.
__global__ void k_net_refresh(int taps, int cin, int cout, const float* w, __nv_bfloat16* w16, float* wt) {
  const long long n = (long long)taps * cin * cout;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const int co = (int)(i % cout), ci = (int)((i / cout) % cin), t = (int)(i / ((long long)cin * cout));
    w16[i] = __float2bfloat16_rn(w[i]);
    wt[((size_t)t * cout + co) * cin + ci] = w[i];
  }
}

// ---- subspace loss ----------------------------------------------------------------------------
constexpr int kLossK = 8;

__global__ void __launch_bounds__(256) k_net_loss(const float* y, const float* V, const float* Mw, int k, int B,
                                                  float* loss, float* dy) {
  __shared__ double red[32], wred[8][2 * kLossK * kLossK];
  __shared__ double G[kLossK * kLossK], H[kLossK * kLossK], C[kLossK * kLossK];
  const int b = blockIdx.x;
  const float* yb = y + (size_t)b * NET_VOX * NET_COUT;
  const float* vb = V + (size_t)b * NET_VOX * k;
  const float* mb = Mw + (size_t)b * NET_VOX;
  // G and H in one pass: a thread keeps all entries of its voxels' sums (a pass per entry, k^2 block sums of a
  // strided read each, took 0.37 ms for 64 patches)
  {
    double g[kLossK * (kLossK + 1) / 2], h[kLossK * kLossK];
#pragma unroll
    for (int e = 0; e < kLossK * (kLossK + 1) / 2; ++e) g[e] = 0.0;
#pragma unroll
    for (int e = 0; e < kLossK * kLossK; ++e) h[e] = 0.0;
    for (int v = threadIdx.x; v < NET_VOX; v += blockDim.x) {
      const float m = mb[v];
      if (m == 0.f) continue;
      double yv[kLossK], vv[kLossK];
#pragma unroll
      for (int i = 0; i < kLossK; ++i) {
        yv[i] = i < k ? (double)yb[(size_t)v * NET_COUT + i] : 0.0;
        vv[i] = i < k ? (double)vb[(size_t)v * k + i] : 0.0;
      }
#pragma unroll
      for (int i = 0; i < kLossK; ++i) {
        const double my = (double)m * yv[i];
#pragma unroll
        for (int j = 0; j <= i; ++j) g[i * (i + 1) / 2 + j] += my * yv[j];
#pragma unroll
        for (int j = 0; j < kLossK; ++j) h[i * kLossK + j] += my * vv[j];
      }
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int i = 0; i < kLossK; ++i) {
#pragma unroll
      for (int j = 0; j < kLossK; ++j) {
        const double sg = j <= i ? warp_sum(g[i * (i + 1) / 2 + j]) : 0.0, sh = warp_sum(h[i * kLossK + j]);
        if (lane == 0) {
          wred[wid][i * kLossK + j] = sg;
          wred[wid][kLossK * kLossK + i * kLossK + j] = sh;
        }
      }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < 2 * kLossK * kLossK; e += blockDim.x) {
      double s = 0.0;
      for (int w = 0; w < 8; ++w) s += wred[w][e];
      const int i = (e % (kLossK * kLossK)) / kLossK, j = e % kLossK;
      if (e >= kLossK * kLossK)
        H[i * kLossK + j] = s;
      else if (j <= i)
        G[i * kLossK + j] = G[j * kLossK + i] = s;
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    // C = (G + eps I)^-1 H by Cholesky
    double tr = 0.0;
    for (int i = 0; i < k; ++i) tr += G[i * kLossK + i];
    const double eps = 1e-6 * tr / k + 1e-30;
    double L[kLossK * kLossK];
    for (int i = 0; i < k; ++i)
      for (int j = 0; j <= i; ++j) {
        double s = G[i * kLossK + j] + (i == j ? eps : 0.0);
        for (int q = 0; q < j; ++q) s -= L[i * kLossK + q] * L[j * kLossK + q];
        L[i * kLossK + j] = (i == j) ? sqrt(fmax(s, 1e-300)) : s / L[j * kLossK + j];
      }
    for (int c = 0; c < k; ++c) {
      double z[kLossK];
      for (int i = 0; i < k; ++i) {
        double s = H[i * kLossK + c];
        for (int q = 0; q < i; ++q) s -= L[i * kLossK + q] * z[q];
        z[i] = s / L[i * kLossK + i];
      }
      for (int i = k - 1; i >= 0; --i) {
        double s = z[i];
        for (int q = i + 1; q < k; ++q) s -= L[q * kLossK + i] * C[q * kLossK + c];
        C[i * kLossK + c] = s / L[i * kLossK + i];
      }
    }
  }
  __syncthreads();
  const float scale = -2.f / (float)(B * k);
  double lacc = 0.0;
  for (int v = threadIdx.x; v < NET_VOX; v += blockDim.x) {
    const float m = mb[v];
    float r[kLossK];
    for (int j = 0; j < k; ++j) {
      double p = 0.0;
      for (int i = 0; i < k; ++i) p += (double)yb[(size_t)v * NET_COUT + i] * C[i * kLossK + j];
      r[j] = vb[(size_t)v * k + j] - (float)p;
      lacc += (double)m * r[j] * r[j];
    }
    float* d = dy + ((size_t)b * NET_VOX + v) * NET_COUT;
    for (int i = 0; i < NET_COUT; ++i) {
      float s = 0.f;
      if (i < k)
        for (int j = 0; j < k; ++j) s += r[j] * (float)C[i * kLossK + j];
      d[i] = scale * m * s;
    }
  }
  lacc = block_sum(lacc, red);
  if (threadIdx.x == 0) loss[b] = (float)(lacc / k);
}

// ---- patches -------------------------------------------------------------------------------------
__global__ void k_net_features(Grid g, const SubInfo* subs, const double* kx, const double* ky, const double* kz,
                               int dmask, __nv_bfloat16* feats) {
  __shared__ double red[32];
  const SubInfo S = subs[blockIdx.x];
  const int nc = S.nx * S.ny * S.nz;
  double s = 0.0;
  for (int cl = threadIdx.x; cl < nc; cl += blockDim.x) {
    const int i = cl % S.nx, j = (cl / S.nx) % S.ny, q = cl / (S.nx * S.ny);
    const long long cg = ((long long)(S.z0 + q) * g.N + (S.y0 + j)) * g.M + (S.x0 + i);
    s += log(kx[cg]) + log(ky[cg]) + log(kz[cg]);
  }
  const double mean = block_sum(s, red) / (3.0 * nc);
  for (int v = threadIdx.x; v < NET_VOX; v += blockDim.x) {
    const int x = v % NET_S, y = (v / NET_S) % NET_S, z = v / (NET_S * NET_S);
    float f[NET_CIN];
#pragma unroll
    for (int c = 0; c < NET_CIN; ++c) f[c] = 0.f;
    if (x < S.nx && y < S.ny && z < S.nz) {
      const int ex = S.x0 + x, ey = S.y0 + y, ez = S.z0 + z;
      const long long cg = ((long long)ez * g.N + ey) * g.M + ex;
      f[0] = (float)((log(kx[cg]) - mean) * 0.25);
      f[1] = (float)((log(ky[cg]) - mean) * 0.25);
      f[2] = (float)((log(kz[cg]) - mean) * 0.25);
      const bool dir = ((dmask & 1) && ex == 0) || ((dmask & 2) && ex == g.M - 1) || ((dmask & 4) && ey == 0) ||
                       ((dmask & 8) && ey == g.N - 1) || ((dmask & 16) && ez == 0) || ((dmask & 32) && ez == g.P - 1);
      f[3] = dir ? 1.f : 0.f;
      f[4] = 1.f;
    }
    __nv_bfloat16* o = feats + ((size_t)blockIdx.x * NET_VOX + v) * NET_CIN;
#pragma unroll
    for (int c = 0; c < NET_CIN; c += 2)
      *reinterpret_cast<__nv_bfloat162*>(o + c) = __floats2bfloat162_rn(f[c], f[c + 1]);
  }
}

__device__ __forceinline__ double harm(double a, double b) { return 2.0 / (1.0 / a + 1.0 / b); }

// Mass diagonal of the local eigenproblem (src/PreMixFEM_3D.c:243-346), the same
// expression, term for term, as the batched eigensolver's.
__global__ void k_net_targets(NetTargetArgs a) {
  const SubInfo S = a.subs[blockIdx.x];
  const Grid g = a.g;
  for (int v = threadIdx.x; v < NET_VOX; v += blockDim.x) {
    const int i = v % NET_S, j = (v / NET_S) % NET_S, kk = v / (NET_S * NET_S);
    float* Vo = a.V + ((size_t)blockIdx.x * NET_VOX + v) * a.k;
    if (!(i < S.nx && j < S.ny && kk < S.nz)) {
      for (int c = 0; c < a.k; ++c) Vo[c] = 0.f;
      a.Mw[(size_t)blockIdx.x * NET_VOX + v] = 0.f;
      continue;
    }
    const int nx = S.nx, ny = S.ny, nz = S.nz;
    const int ex = S.x0 + i, ey = S.y0 + j, ez = S.z0 + kk;
    const long long cg = ((long long)ez * g.N + ey) * g.M + ex;
    double mv;
    if (a.eg_op == 1) {
      mv = a.kx[cg] + a.ky[cg] + a.kz[cg];
    } else if (a.eg_op == 2) {
      double dn = a.db[cg];
      if (i > 0) dn += a.tx[cg];
      if (i < nx - 1) dn += a.tx[cg + 1];
      if (j > 0) dn += a.ty[cg];
      if (j < ny - 1) dn += a.ty[cg + g.M];
      if (kk > 0) dn += a.tz[cg];
      if (kk < nz - 1) dn += a.tz[cg + g.MN];
      mv = dn;
    } else {
      mv = 0.0;
      if (i == 0 && ex >= 1) mv += 2.0 * harm(a.kx[cg - 1], a.kx[cg]) / a.Hx / a.Hx;
      if (ex + 1 != g.M) mv += 2.0 * harm(a.kx[cg], a.kx[cg + 1]) / a.Hx / a.Hx;
      if (ey >= 1) mv += 2.0 * harm(a.ky[cg - g.M], a.ky[cg]) / a.Hy / a.Hy;
      if (ey + 1 != g.N) mv += 2.0 * harm(a.ky[cg], a.ky[cg + g.M]) / a.Hy / a.Hy;
      if (ez >= 1) mv += 2.0 * harm(a.kz[cg - g.MN], a.kz[cg]) / a.Hz / a.Hz;
      if (ez + 1 != g.P) mv += 2.0 * harm(a.kz[cg], a.kz[cg + g.MN]) / a.Hz / a.Hz;
      if (i + 1 < nx) mv += 2.0 * harm(a.kx[cg], a.kx[cg + 1]) / a.Hx / a.Hx;
      const int dm = a.dirichlet_mask;
      if (dm & 1 && ex == 0) mv += 2.0 * (2.0 * a.kx[cg]) / a.Hx / a.Hx;
      if (dm & 2 && ex == g.M - 1) mv += 2.0 * (2.0 * a.kx[cg]) / a.Hx / a.Hx;
      if (dm & 4 && ey == 0) mv += 2.0 * (2.0 * a.ky[cg]) / a.Hy / a.Hy;
      if (dm & 8 && ey == g.N - 1) mv += 2.0 * (2.0 * a.ky[cg]) / a.Hy / a.Hy;
      if (dm & 16 && ez == 0) mv += 2.0 * (2.0 * a.kz[cg]) / a.Hz / a.Hz;
      if (dm & 32 && ez == g.P - 1) mv += 2.0 * (2.0 * a.kz[cg]) / a.Hz / a.Hz;
      mv *= a.meas;
    }
    a.Mw[(size_t)blockIdx.x * NET_VOX + v] = (float)mv;
    for (int c = 0; c < a.k; ++c)
      Vo[c] = a.phi_f32 ? reinterpret_cast<const float*>(a.phi)[cg * a.kmax + c]
                        : (float)reinterpret_cast<const double*>(a.phi)[cg * a.kmax + c];
  }
}

// Subdomains whose eigensolve did not converge (status 1), in index order.
__global__ void k_failed_list(const int* status, int nsub, int* list, int* count) {
  if (threadIdx.x != 0) return;
  int c = 0;
  for (int s = 0; s < nsub; ++s)
    if (status[s] == 1) list[c++] = s;
  *count = c;
}

}  // namespace

void launch_net_targets(const NetTargetArgs& a, cudaStream_t st) {
  { note_launch(); k_net_targets<<<a.nsub, 256, 0, st>>>(a); }
}

void launch_failed_list(const int* status, int nsub, int* list, int* count, cudaStream_t st) {
  { note_launch(); k_failed_list<<<1, 32, 0, st>>>(status, nsub, list, count); }
}

void launch_net_features(const Grid& g, const SubInfo* subs, int nsub, const double* kx, const double* ky,
                         const double* kz, int dirichlet_mask, __nv_bfloat16* feats, cudaStream_t st) {
  { note_launch(); k_net_features<<<nsub, 256, 0, st>>>(g, subs, kx, ky, kz, dirichlet_mask, feats); }
}

void launch_net_loss(const float* y, const float* V, const float* Mw, int B, int k, float* loss, float* dy,
                     cudaStream_t st) {
  { note_launch(); k_net_loss<<<B, 256, 0, st>>>(y, V, Mw, k, B, loss, dy); }
}

// ---- host side ---------------------------------------------------------------------------------
static size_t wcount(const NetLayer& L) { return (size_t)net_taps(L.type) * L.cin * L.cout; }
static size_t act_elems(int a) { return (size_t)kNetActs[a].s * kNetActs[a].s * kNetActs[a].s * kNetActs[a].c; }

Net::Net() {}

Net::~Net() {
  for (int l = 0; l < NET_LAYERS; ++l) {
    void* p[] = {w32_[l], b32_[l], w16_[l], wt_[l], wtc_[l], gw_[l], gb_[l], mw_[l], vw_[l], mb_[l], vb_[l]};
    for (void* q : p)
      if (q) cudaFree(q);
  }
  for (int a = 0; a < NET_ACTS; ++a) {
    if (a > 0 && act_[a]) cudaFree(act_[a]);
    if (dact_[a]) cudaFree(dact_[a]);
  }
  if (d_err_) cudaFree(d_err_);
  if (bpart_) cudaFree(bpart_);
  if (dyal_) cudaFree(dyal_);
}

int Net::take_error() {
  if (!d_err_) return 0;
  int f = 0;
  if (cudaMemcpy(&f, d_err_, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) {
    err = "reading the network's kernel flag failed";
    return 76;
  }
  if (!f) return 0;
  cudaMemset(d_err_, 0, sizeof(int));
  err = "a tensor-core convolution's wait for its MMAs ran out";
  return 76;
}

int Net::params() const {
  int n = 0;
  for (const NetLayer& L : kNetLayers) n += (int)wcount(L) + L.cout;
  return n;
}

int Net::alloc_params() {
  if (w32_[0]) return 0;
  for (int l = 0; l < NET_LAYERS; ++l) {
    const size_t nw = wcount(kNetLayers[l]), nb = kNetLayers[l].cout;
    bool ok = cudaMalloc(&w32_[l], nw * 4) == cudaSuccess && cudaMalloc(&b32_[l], nb * 4) == cudaSuccess &&
              cudaMalloc(&w16_[l], nw * 2) == cudaSuccess && cudaMalloc(&wt_[l], nw * 4) == cudaSuccess &&
              cudaMalloc(&gw_[l], nw * 4) == cudaSuccess && cudaMalloc(&gb_[l], nb * 4) == cudaSuccess &&
              cudaMalloc(&mw_[l], nw * 4) == cudaSuccess && cudaMalloc(&vw_[l], nw * 4) == cudaSuccess &&
              cudaMalloc(&mb_[l], nb * 4) == cudaSuccess && cudaMalloc(&vb_[l], nb * 4) == cudaSuccess;
    if (ok && conv_tc_layer(kNetLayers[l])) ok = cudaMalloc(&wtc_[l], nw * 2) == cudaSuccess;
    if (!ok) {
      err = "cudaMalloc of the network parameters failed";
      return 76;
    }
    cudaMemset(mw_[l], 0, nw * 4);
    cudaMemset(vw_[l], 0, nw * 4);
    cudaMemset(mb_[l], 0, nb * 4);
    cudaMemset(vb_[l], 0, nb * 4);
  }
  if (cudaMalloc(&d_err_, sizeof(int)) != cudaSuccess) {
    err = "cudaMalloc of the network parameters failed";
    return 76;
  }
  cudaMemset(d_err_, 0, sizeof(int));
  return 0;
}

void Net::refresh(int l, cudaStream_t st) {
  const NetLayer& L = kNetLayers[l];
  const long long n = (long long)wcount(L);
  { note_launch(); k_net_refresh<<<(int)std::min<long long>((n + 255) / 256, 4096), 256, 0, st>>>(net_taps(L.type), L.cin, L.cout, w32_[l], w16_[l], wt_[l]); }
  if (wtc_[l]) { note_launch(); k_net_pack_tc<<<(int)std::min<long long>((n + 255) / 256, 4096), 256, 0, st>>>(L.cin, L.cout, w16_[l], wtc_[l]); }
}

int Net::set_weights(int l, const float* w, const float* b) {
  if (l < 0 || l >= NET_LAYERS) {
    err = "layer index out of range";
    return 62;
  }
  if (int e = alloc_params()) return e;
  const NetLayer& L = kNetLayers[l];
  if (w) cudaMemcpy(w32_[l], w, wcount(L) * 4, cudaMemcpyHostToDevice);
  if (b) cudaMemcpy(b32_[l], b, L.cout * 4, cudaMemcpyHostToDevice);
  refresh(l, 0);
  if (cudaDeviceSynchronize() != cudaSuccess) {
    err = "set_weights failed";
    return 76;
  }
  return 0;
}

int Net::get_weights(int l, float* w, float* b) const {
  if (l < 0 || l >= NET_LAYERS || !w32_[l]) return 62;
  if (w) cudaMemcpy(w, w32_[l], wcount(kNetLayers[l]) * 4, cudaMemcpyDeviceToHost);
  if (b) cudaMemcpy(b, b32_[l], kNetLayers[l].cout * 4, cudaMemcpyDeviceToHost);
  return cudaDeviceSynchronize() == cudaSuccess ? 0 : 76;
}

int Net::get_grads(int l, float* gw, float* gb) const {
  if (l < 0 || l >= NET_LAYERS || !gw_[l]) return 62;
  if (gw) cudaMemcpy(gw, gw_[l], wcount(kNetLayers[l]) * 4, cudaMemcpyDeviceToHost);
  if (gb) cudaMemcpy(gb, gb_[l], kNetLayers[l].cout * 4, cudaMemcpyDeviceToHost);
  return cudaDeviceSynchronize() == cudaSuccess ? 0 : 76;
}

int Net::init(unsigned long long seed) {
  if (int e = alloc_params()) return e;
  std::mt19937_64 rng(seed);
  for (int l = 0; l < NET_LAYERS; ++l) {
    const NetLayer& L = kNetLayers[l];
    const int fan_in = (L.type == NL_UP2 ? 1 : net_taps(L.type)) * (l == 0 ? 5 : L.cin);
    std::normal_distribution<float> nd(0.f, std::sqrt((L.relu ? 2.f : 1.f) / fan_in));
    std::vector<float> w(wcount(L)), b(L.cout, 0.f);
    for (auto& x : w) x = nd(rng);
    if (int e = set_weights(l, w.data(), b.data())) return e;
  }
  step_ = 0;
  return 0;
}

static const char kMagic[8] = {'P', 'M', 'F', 'N', 'E', 'T', '0', '1'};

int Net::save(const char* path) const {
  FILE* f = fopen(path, "wb");
  if (!f) return 62;
  fwrite(kMagic, 1, 8, f);
  const int hdr[2] = {1, NET_LAYERS};
  fwrite(hdr, 4, 2, f);
  for (int l = 0; l < NET_LAYERS; ++l) {
    const NetLayer& L = kNetLayers[l];
    const int d[4] = {L.type, L.cin, L.cout, net_taps(L.type)};
    fwrite(d, 4, 4, f);
    std::vector<__nv_bfloat16> w(wcount(L));
    std::vector<float> b(L.cout);
    cudaMemcpy(w.data(), w16_[l], w.size() * 2, cudaMemcpyDeviceToHost);
    cudaMemcpy(b.data(), b32_[l], b.size() * 4, cudaMemcpyDeviceToHost);
    fwrite(w.data(), 2, w.size(), f);
    fwrite(b.data(), 4, b.size(), f);
  }
  const bool ok = fclose(f) == 0;
  return ok ? 0 : 76;
}

int Net::load(const char* path) {
  FILE* f = fopen(path, "rb");
  if (!f) {
    err = std::string("cannot open network weights ") + path;
    return 62;
  }
  auto fail = [&](const char* why) {
    fclose(f);
    err = std::string(path) + ": " + why;
    return 62;
  };
  char mg[8];
  int hdr[2];
  if (fread(mg, 1, 8, f) != 8 || memcmp(mg, kMagic, 8) != 0) return fail("not a weight file");
  if (fread(hdr, 4, 2, f) != 2 || hdr[0] != 1 || hdr[1] != NET_LAYERS) return fail("unsupported version or layout");
  if (int e = alloc_params()) {
    fclose(f);
    return e;
  }
  for (int l = 0; l < NET_LAYERS; ++l) {
    const NetLayer& L = kNetLayers[l];
    int d[4];
    if (fread(d, 4, 4, f) != 4 || d[0] != L.type || d[1] != L.cin || d[2] != L.cout || d[3] != net_taps(L.type))
      return fail("layer shapes differ from this build's network");
    std::vector<__nv_bfloat16> w(wcount(L));
    std::vector<float> w32(w.size()), b(L.cout);
    if (fread(w.data(), 2, w.size(), f) != w.size() || fread(b.data(), 4, b.size(), f) != b.size())
      return fail("truncated");
    for (size_t i = 0; i < w.size(); ++i) w32[i] = __bfloat162float(w[i]);
    if (int e = set_weights(l, w32.data(), b.data())) {
      fclose(f);
      return e;
    }
  }
  fclose(f);
  return 0;
}

int Net::ensure(int B) {
  if (B <= cap_) return 0;
  for (int a = 1; a < NET_ACTS; ++a) {
    if (act_[a]) cudaFree(act_[a]);
    if (dact_[a]) cudaFree(dact_[a]);
    act_[a] = nullptr;
    dact_[a] = nullptr;
  }
  for (int a = 1; a < NET_ACTS - 1; ++a)
    if (cudaMalloc(&act_[a], act_elems(a) * B * 2) != cudaSuccess) {
      err = "cudaMalloc of the network activations failed";
      cap_ = 0;
      return 76;
    }
  cap_ = B;
  return 0;
}

// One forward layer with ROWS-row tiles and MT 16-row m-tiles per warp.
template <int NT, int ROWS, int MT>
static bool fwd_launch_t(const FwdArgs& a, long long rows, cudaStream_t st) {
  const size_t smem = (2 * (size_t)ROWS * (a.cin + 8) + 2 * (size_t)a.cin * (a.cout + 8)) * 2;
  if (smem > 48 * 1024) cudaFuncSetAttribute(k_net_fwd<NT, ROWS, MT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  k_net_fwd<NT, ROWS, MT><<<(int)(rows / ROWS), ROWS * 2 / MT, smem, st>>>(a);
  return true;
}

template <int NT>
static bool fwd_launch_nt(int R, int MT, const FwdArgs& a, long long rows, cudaStream_t st) {
  if (R == 256 && MT == 2) return fwd_launch_t<NT, 256, 2>(a, rows, st);
  if (R == 128 && MT == 1) return fwd_launch_t<NT, 128, 1>(a, rows, st);
  if (R == 128 && MT == 2) return fwd_launch_t<NT, 128, 2>(a, rows, st);
  if (R == 64 && MT == 1) return fwd_launch_t<NT, 64, 1>(a, rows, st);
  return false;
}

static bool fwd_launch(int ntv, int R, int MT, const FwdArgs& a, long long rows, cudaStream_t st) {
  switch (ntv) {
    case 2: return fwd_launch_nt<2>(R, MT, a, rows, st);
    case 4: return fwd_launch_nt<4>(R, MT, a, rows, st);
    case 8: return fwd_launch_nt<8>(R, MT, a, rows, st);
    case 12: return fwd_launch_nt<12>(R, MT, a, rows, st);
  }
  return false;
}

int Net::forward(const __nv_bfloat16* x, int B, float* y, bool keep, cudaStream_t st) {
  if (!w32_[0]) {
    err = "network weights not initialised or loaded";
    return 73;
  }
  if (int e = ensure(B)) return e;
  x_ = x;
  for (int l = 0; l < NET_LAYERS; ++l) {
    const NetLayer& L = kNetLayers[l];
    FwdArgs a;
    a.type = L.type;
    a.cin = L.cin;
    a.cout = L.cout;
    a.s_in = L.s_in;
    a.s_out = L.s_out;
    a.relu = L.relu;
    a.in = L.in_act == 0 ? x : act_[L.in_act];
    a.W = w16_[l];
    a.bias = b32_[l];
    a.skip = L.skip >= 0 ? act_[L.skip] : nullptr;
    a.out = L.out_act == NET_ACTS - 1 ? nullptr : act_[L.out_act];
    a.outf = L.out_act == NET_ACTS - 1 ? y : nullptr;
    const long long rows = (long long)B * L.s_out * L.s_out * L.s_out;
    // tiles stay inside one sample (and one parity class for up2); candidate 0
    // is the built-in choice, the tuner may pick another for this layer and batch
    const int per = L.type == NL_UP2 ? L.s_in * L.s_in * L.s_in : L.s_out * L.s_out * L.s_out;
    static const int kTiles[4][2] = {{256, 2}, {128, 1}, {128, 2}, {64, 1}};
    int cand[5], nc = 0;
    const int def = per % 256 == 0 ? 0 : 3;
    cand[nc++] = def;
    for (int t = 0; t < 4; ++t)
      if (t != def && per % kTiles[t][0] == 0) cand[nc++] = t;
    const int ntv = L.cout / 8;
    if (ntv != 2 && ntv != 4 && ntv != 8 && ntv != 12) {
      err = "unsupported layer width";
      return 56;
    }
    // the tensor-core convolution (candidate index 4) where the layer fits it
    const bool tc = wtc_[l] && conv_tc_layer(L) && !a.outf;
    if (tc) cand[nc++] = 4;
    auto launch = [&](int c) -> bool {
      if (cand[c] == 4) {
        conv_tc_launch(L, a.in, wtc_[l], a.bias, a.out, B, d_err_, st);
        return true;
      }
      return fwd_launch(ntv, kTiles[cand[c]][0], kTiles[cand[c]][1], a, rows, st);
    };
    char key[96];
    snprintf(key, sizeof(key), tc ? "net_fwd|L%d|B%d|tc" : "net_fwd|L%d|B%d", l, B);
    const int c = tune_choose(key, nc, launch, st);
    note_launch();
    launch(c);
  }
  (void)keep;
  return 0;
}

int Net::backward(const float* dy, int B, cudaStream_t st) {
  if (B > cap_ || !x_) {
    err = "backward needs the activations of a forward pass of the same batch";
    return 73;
  }
  for (int a = 1; a < NET_ACTS - 1; ++a)
    if (!dact_[a] && cudaMalloc(&dact_[a], act_elems(a) * cap_ * 4) != cudaSuccess) {
      err = "cudaMalloc of the network gradients failed";
      return 76;
    }
  if (!bpart_ && cudaMalloc(&bpart_, sizeof(double) * kBgradCtas * 96) != cudaSuccess) {
    err = "cudaMalloc of the network gradients failed";
    return 76;
  }
  if (reinterpret_cast<uintptr_t>(dy) & 15) {  // the kernels read it 16 bytes at a time
    if (dyal_cap_ < B) {
      if (dyal_) cudaFree(dyal_);
      dyal_ = nullptr;
      dyal_cap_ = 0;
      if (cudaMalloc(&dyal_, sizeof(float) * (size_t)B * NET_VOX * NET_COUT) != cudaSuccess) {
        err = "cudaMalloc of the network gradients failed";
        return 76;
      }
      dyal_cap_ = B;
    }
    cudaMemcpyAsync(dyal_, dy, sizeof(float) * (size_t)B * NET_VOX * NET_COUT, cudaMemcpyDeviceToDevice, st);
    dy = dyal_;
  }
  // dpre[l]: pre-activation gradient of layer l's output; layer 8's is dy.
  auto dpre = [&](int l) -> float* {
    return l == NET_LAYERS - 1 ? const_cast<float*>(dy) : dact_[kNetLayers[l].out_act];
  };
  for (int l = NET_LAYERS - 1; l >= 0; --l) {
    const NetLayer& L = kNetLayers[l];
    const __nv_bfloat16* in = L.in_act == 0 ? x_ : act_[L.in_act];
    cudaMemsetAsync(gw_[l], 0, wcount(L) * 4, st);
    // weight gradient
    WgradArgs w;
    w.type = L.type;
    w.cin = L.cin;
    w.cout = L.cout;
    w.s_in = L.s_in;
    w.s_out = L.s_out;
    w.B = B;
    w.rows_per_chunk = 0;  // wgrad_launch
    w.in = in;
    w.dz = dpre(l);
    w.gw = gw_[l];
    const long long rows = (long long)B * (L.type == NL_UP2 ? L.s_in * L.s_in * L.s_in : L.s_out * L.s_out * L.s_out);
    const int taps = net_taps(L.type);
    const bool c3 = L.type == NL_CONV3;
    if (c3 && L.cin == 16 && L.cout == 32) wgrad_launch<16, 32, 2, 2, 9>(w, rows, taps, st);
    else if (c3 && L.cin == 32 && L.cout == 32) wgrad_launch<32, 32, 2, 2, 9>(w, rows, taps, st);
    else if (c3 && L.cin == 64 && L.cout == 64) wgrad_launch<64, 64, 4, 4, 3>(w, rows, taps, st);
    else if (c3 && L.cin == 96 && L.cout == 96) wgrad_launch<96, 96, 6, 6, 1>(w, rows, taps, st);
    else if (L.cin == 32 && L.cout == 64) wgrad_launch<32, 64, 4, 2, 1>(w, rows, taps, st);
    else if (L.cin == 64 && L.cout == 96) wgrad_launch<64, 96, 4, 6, 1>(w, rows, taps, st);
    else if (L.cin == 96 && L.cout == 64) wgrad_launch<96, 64, 6, 4, 1>(w, rows, taps, st);
    else if (L.cin == 64 && L.cout == 32) wgrad_launch<64, 32, 4, 2, 1>(w, rows, taps, st);
    else if (L.cin == 32 && L.cout == 16) wgrad_launch<32, 16, 2, 2, 1>(w, rows, taps, st);
    else {
      err = "unsupported layer shape in backward";
      return 56;
    }
    const long long orows = (long long)B * L.s_out * L.s_out * L.s_out;
    const int nb = (int)std::max<long long>(1, std::min<long long>(kBgradCtas, orows / 64));
    { note_launch(); k_net_bgrad<<<nb, 256, 0, st>>>(dpre(l), orows, L.cout, bpart_); }
    { note_launch(); k_net_bgrad_fin<<<1, 128, 0, st>>>(bpart_, nb, L.cout, gb_[l]); }
    if (l == 0) break;
    // gradient reaching the input activation, masked by its ReLU, plus skip gradients
    DgradArgs d;
    d.type = L.type;
    d.cin = L.cin;
    d.cout = L.cout;
    d.s_in = L.s_in;
    d.s_out = L.s_out;
    d.B = B;
    d.dz = dpre(l);
    d.wt = wt_[l];
    d.in_act = in;
    d.add = nullptr;
    for (int j = 0; j < NET_LAYERS; ++j)
      if (kNetLayers[j].skip == L.in_act) d.add = dpre(j);
    d.din = dact_[L.in_act];
    if (!dgrad_launch(d, st)) {
      err = "unsupported layer shape in backward";
      return 56;
    }
  }
  return 0;
}

void Net::adam(float lr, float b1, float b2, float eps, float wd, cudaStream_t st) {
  ++step_;
  const float bc1 = 1.f - powf(b1, (float)step_), bc2 = 1.f - powf(b2, (float)step_);
  for (int l = 0; l < NET_LAYERS; ++l) {
    const NetLayer& L = kNetLayers[l];
    const long long nw = (long long)wcount(L);
    { note_launch(); k_net_adam<<<(int)std::min<long long>((nw + 255) / 256, 4096), 256, 0, st>>>(nw, w32_[l], gw_[l], mw_[l], vw_[l], lr, b1, b2, eps, wd, bc1, bc2); }
    { note_launch(); k_net_adam<<<1, 256, 0, st>>>(L.cout, b32_[l], gb_[l], mb_[l], vb_[l], lr, b1, b2, eps, 0.f, bc1, bc2); }
    refresh(l, st);
  }
}

}  // namespace pmf
