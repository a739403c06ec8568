// Learned preconditioner: a gauge-covariant convolutional network approximating M~^-1.
//
// Fields live on the whole lattice in even-odd order (site j = parity * Vh + cb index) as
// [site][channel][colour] complex FP32.  A layer maps C_in to C_out channels:
//
//     out(x)[o][a] = sum_{d=0..8} sum_i W_d[o][i] (T_d h)(x)[i][a]
//     T_0 h(x) = h(x),  T_{+mu} h(x) = U_mu(x) h(x+mu),  T_{-mu} h(x) = U_mu(x-mu)^dag h(x-mu)
//
// W acts on channels only and the links on colour only, so every layer (and the network) is
// gauge covariant.  The channel mixing is a GEMM over the rows (site, colour): the gathered
// T_d h form a 9*C_in complex row, staged in shared memory as BF16 in the tensor cores' core-matrix
// layout, and tcgen05.mma (BF16 in, FP32 accumulate in tensor memory) multiplies it by the real
// form of W.  The network is linear; it takes the odd-site input as channels = spins with zero
// even sites and returns its odd sites.
//
// Backward: the input gradient of a layer is the same layer with W'_{+mu} = W_{-mu}^H,
// W'_{-mu} = W_{+mu}^H, W'_0 = W_0^H (T_{+mu}^dag = T_{-mu}), and the weight gradient is
// sum over rows of delta_out (x) conj(gathered input), with mma.sync m16n8k16 (a reduction over
// the rows into a small matrix, accumulated across blocks with atomics).
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <complex>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <fstream>
#include <random>
#include <string>
#include <vector>

#include "cnn.h"
#include "ctx.h"
#include "gbc_device.cuh"

namespace gbc {
namespace {

constexpr int SITES = 32;          // sites per block, one per lane -> 96 rows (site, colour)
constexpr int ROWS = SITES * 3;
constexpr int DIRS = 9;            // the site itself and 8 hops, one warp each
constexpr int CT = 32 * DIRS;      // threads per block

enum { IN_ODD = 1, OUT_ODD = 2 };  // layer input zero on the even sites; output wanted on the odd sites only

__host__ __device__ constexpr int kpad(int cin) { return ((9 * cin * 2 + 15) / 16) * 16; }
__host__ __device__ constexpr int npad(int cout) { return ((2 * cout + 7) / 8) * 8; }

// The GEMM's K index is (d * CIN + i) * 2 + re/im.  Its N index is comp(o, re/im), the order of the
// activation planes, (re_o, re_o+1, im_o, im_o+1) for even o, so an accumulator row is stored as it is.
__host__ __device__ constexpr int comp(int i, int im) { return (i >> 1) * 4 + 2 * im + (i & 1); }

__device__ __forceinline__ uint32_t bf16x2(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}

__device__ __forceinline__ Coord eo_coords(const Geom& g, int j) {
  const int par = j >= g.Vh ? 1 : 0;
  return cb_coords(g, j - par * g.Vh, par);
}

// Activations are planes of float4 over the even-odd site index: plane a * C/2 + i/2 holds
// (re, re, im, im) of channels i, i + 1 and colour a, so the 32 lanes of a warp (32 consecutive
// sites) read and write 512 contiguous bytes per plane.
__host__ __device__ constexpr int planes(int ch) { return 3 * ch / 2; }

// Byte offset of the 16-byte core-matrix row (row, 8-element column chunk) of a staged bf16 tile of
// COLS columns: the tensor cores' canonical K-major layout without swizzle, 8 x 8 core matrices
// (8 rows of 16 bytes, 128 contiguous bytes), 128 bytes apart along the columns (the descriptor's
// leading byte offset), row groups COLS * 16 bytes apart (its stride byte offset).  Rows are
// colour * 32 + site, so the 8 lanes of a quarter warp fill one core matrix: no bank conflicts.
template <int COLS>
__device__ __forceinline__ uint32_t core_row(int row, int chunk) {
  return (uint32_t)((row >> 3) * (COLS * 16) + chunk * 128 + (row & 7) * 16);
}

// The neighbour that direction d of site i (parity par) reads, as an even-odd index
__device__ __forceinline__ int neighbour(const Geom& g, int par, int i, int d) {
  if (d == 0) return par * g.Vh + i;
  Coord c = cb_coords(g, i, par);
  const int mu = (d - 1) >> 1;
  const bool bwd = ((d - 1) & 1) != 0;
#pragma unroll
  for (int m = 0; m < 4; ++m)
    if (m == mu) c.x[m] = bwd ? (c.x[m] == 0 ? g.L[m] - 1 : c.x[m] - 1) : (c.x[m] + 1 == g.L[m] ? 0 : c.x[m] + 1);
  return (1 - par) * g.Vh + cb_index(g, c);
}

// M_d of a site: U_mu(x) for +mu, U_mu(x - mu)^dag for -mu; links are planes [mu * 9 + entry][V]
__device__ __forceinline__ void load_transport(float2 (&m)[9], const float2* links, int V, int j, int n, int d) {
  const int mu = (d - 1) >> 1;
  if ((d - 1) & 1) {
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const float2 u = __ldg(links + (size_t)(mu * 9 + 3 * k + a) * V + n);
        m[3 * a + k] = make_float2(u.x, -u.y);
      }
  } else {
#pragma unroll
    for (int e = 0; e < 9; ++e) m[e] = __ldg(links + (size_t)(mu * 9 + e) * V + j);
  }
}

// One component of M x in FP32, (re, im) rounded to BF16.  The FMA order is spelled out: a last-bit
// change here flips BF16 roundings, which the following layers carry on.
__device__ __forceinline__ uint32_t transported(float2 u0, float2 u1, float2 u2, float x0r, float x0i, float x1r,
                                                float x1i, float x2r, float x2i) {
  float re = __fmaf_rn(u0.x, x0r, -__fmul_rn(u0.y, x0i));
  float im = __fmaf_rn(u0.x, x0i, __fmul_rn(u0.y, x0r));
  re = __fmaf_rn(-u1.y, x1i, __fmaf_rn(u1.x, x1r, re));
  im = __fmaf_rn(u1.y, x1r, __fmaf_rn(u1.x, x1i, im));
  re = __fmaf_rn(-u2.y, x2i, __fmaf_rn(u2.x, x2r, re));
  im = __fmaf_rn(u2.y, x2r, __fmaf_rn(u2.x, x2i, im));
  return bf16x2(re, im);
}

// One (site, direction) of the gathered tile: the channels of site n in chunks of four, transported
// by m (d > 0), rounded to BF16 and written as one 16-byte core-matrix row per colour and chunk.
// The transport stays in registers for all channels (and, in the callers, all right-hand sides).
template <int CIN>
__device__ __forceinline__ void gather_dir(unsigned char* G, int d, int s, const float2 (&m)[9], const float4* h,
                                           int V, int n) {
#pragma unroll
  for (int c = 0; c < CIN / 4; ++c) {
    float4 x[3][2];
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
      for (int q = 0; q < 2; ++q) x[k][q] = __ldg(h + (size_t)(k * (CIN / 2) + 2 * c + q) * V + n);
    const int chunk = d * (CIN / 4) + c;
    if (d == 0) {
#pragma unroll
      for (int a = 0; a < 3; ++a)
        *reinterpret_cast<uint4*>(G + core_row<kpad(CIN)>(a * 32 + s, chunk)) =
            make_uint4(bf16x2(x[a][0].x, x[a][0].z), bf16x2(x[a][0].y, x[a][0].w), bf16x2(x[a][1].x, x[a][1].z),
                       bf16x2(x[a][1].y, x[a][1].w));
      continue;
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const float2 u0 = m[3 * a], u1 = m[3 * a + 1], u2 = m[3 * a + 2];
      uint32_t w[4];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const float4 x0 = x[0][q], x1 = x[1][q], x2 = x[2][q];
        w[2 * q] = transported(u0, u1, u2, x0.x, x0.z, x1.x, x1.z, x2.x, x2.z);
        w[2 * q + 1] = transported(u0, u1, u2, x0.y, x0.w, x1.y, x1.w, x2.y, x2.w);
      }
      *reinterpret_cast<uint4*>(G + core_row<kpad(CIN)>(a * 32 + s, chunk)) = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
}

__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// ---- 5th-generation tensor cores (tcgen05) for the forward channel mixing ----------------------
// One thread issues tcgen05.mma (kind::f16, BF16 in, FP32 accumulate in tensor memory) on
// shared-memory descriptors of the gathered tile G (the MMA's M = 128 rows: the block's 96
// (site, colour) rows, then 32 rows that overlap the weights and are discarded) and the weights W
// (NU rows = output channels x re/im, padded to a multiple of 16); completion is signalled through
// an mbarrier by tcgen05.commit, and each warp reads its 32 accumulator lanes back with tcgen05.ld.

// shared-memory matrix descriptor, K-major without swizzle: start, leading byte offset (between
// K-adjacent core matrices), stride byte offset (between 8-row groups), descriptor version 1
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}
// instruction descriptor of kind::f16: FP32 accumulator, BF16 A and B, both K-major, N and M
__host__ __device__ constexpr uint32_t umma_idesc_bf16(int m, int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// waits for phase `parity` of the mbarrier, for about 1 s of SM clock at most
__device__ __forceinline__ bool mbar_wait(uint32_t addr, uint32_t parity) {
  const long long t0 = clock64();
  while (true) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(addr), "r"(parity)
        : "memory");
    if (ok) return true;
    if (clock64() - t0 > 2000000000LL) return false;
  }
}

template <int NU>
__device__ __forceinline__ void tmem_load_row(uint32_t taddr, float (&v)[NU]) {
  uint32_t r[NU];
  if constexpr (NU == 32) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
  } else {
    static_assert(NU == 16, "16 or 32 accumulator columns");
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
  }
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
  for (int q = 0; q < NU; ++q) v[q] = __uint_as_float(r[q]);
}

__host__ __device__ constexpr int nump(int cout) { return ((2 * cout + 15) / 16) * 16; }  // N of the MMA
constexpr int kTmemCols = 32;  // tensor-memory columns allocated per block (>= nump, power of 2)

// out[b] = (G W^T) for the right-hand sides b of this block: warp d gathers direction d of the
// block's 32 sites (all of one parity; lane = site) into the BF16 tile G, one thread issues the
// GEMM on the tensor cores, and warps 0..2 write colours 0..2 from their accumulator lanes.
// What bounds it: the gather's loads through L1/L2 (9 neighbours x C_in x 24 B per site and
// right-hand side).  Against one task per (site, direction, channel) with the transports in shared
// memory, this mapping reads whole 512-byte rows, keeps each transport in registers for every
// channel and right-hand side and writes 16 bytes per shared-memory store.  A 12 -> 12 layer at
// 16^3 x 32: 1772 -> 505 us for 12 right-hand sides, 217 -> 56 us for one (kernel time, cold L2).
// IN_ODD: only the self term of odd sites and the hops of even sites are non-zero; the others'
// columns of G are zeroed, and odd sites need only the K steps that cover the self term.
// A block walks its tiles: weights, tensor memory and barrier are set up once, and warps 3..8 gather
// the next tile while warps 0..2 still store this one (one right-hand side 60 -> 56 us; twelve, which
// fill the chip with a block per tile too, 492 -> 505).
// Every thread waits for the MMA on its own clock, so a warp votes on the outcome: it uses its
// accumulator rows (tcgen05.ld needs the whole warp) or counts one error (its network's, read by the
// host) and stores nothing.  Warp `quit` (-1: none) gives up its first wait at once, for tests of that path.
template <int CIN, int COUT>
__global__ void __launch_bounds__(CT, 3) layer_kernel(Geom g, int V, int tiles, int total, int batch, int per, int flags,
                                                      const float2* __restrict__ links, const float4* __restrict__ hin,
                                                      float4* __restrict__ hout, const uint4* __restrict__ Wc,
                                                      int* errors, int quit) {
  constexpr int KP = kpad(CIN), NP = npad(COUT), NU = nump(COUT);
  constexpr int MROWS = 128;  // the MMA's M: the 96 rows of the tile and 32 discarded rows
  static_assert(ROWS <= MROWS && NU <= kTmemCols, "tile does not fit the MMA");
  // G (96 rows), then W (NP rows); the MMA's rows 96..127 and weight rows NP..NU-1 read what
  // follows, inside the launch's 128 rows: their results are never read back
  extern __shared__ __align__(128) unsigned char smem[];
  unsigned char* G = smem;
  unsigned char* W = smem + ROWS * KP * 2;
  __shared__ __align__(8) uint64_t mbar;
  __shared__ uint32_t tmem_base;
  const int tid = threadIdx.x, d = tid >> 5, s = tid & 31;
  const int b0 = blockIdx.y * per, b1 = min(batch, b0 + per);
  for (int p = tid; p < NP * KP / 8; p += CT) reinterpret_cast<uint4*>(W)[p] = __ldg(Wc + p);
  if (d == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_base)),
                 "r"(kTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  }
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&mbar)));
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  constexpr int CH = CIN / 4;  // 16-byte chunks of a direction
  if (KP > 18 * CIN && d == 0) {
#pragma unroll
    for (int a = 0; a < 3; ++a)
      *reinterpret_cast<uint4*>(G + core_row<KP>(a * 32 + s, DIRS * CH)) = make_uint4(0, 0, 0, 0);
  }
  const uint64_t adesc = umma_desc(smem_u32(G), 128, KP * 16);
  const uint64_t bdesc = umma_desc(smem_u32(W), 128, KP * 16);
  constexpr uint32_t idesc = umma_idesc_bf16(MROWS, NU);
  bool ok = true, dead = false;
  uint32_t phase = 0;  // of the block's next MMA on the mbarrier
  for (int t = blockIdx.x; t < total && !dead; t += gridDim.x) {
    int tile = t, par = 1;
    if (!(flags & OUT_ODD)) {
      par = tile >= tiles ? 1 : 0;
      tile -= par * tiles;
    }
    const int i = tile * SITES + s;
    const bool valid = i < g.Vh;
    const int ic = valid ? i : g.Vh - 1;  // lanes past the end gather the last site, store nothing
    const int j = par * g.Vh + ic;
    const bool mine = !(flags & IN_ODD) || ((d == 0) == (par == 1));
    const int n = neighbour(g, par, ic, d);
    float2 m[9];
    if (mine && d > 0) load_transport(m, links, V, j, n, d);
    if (!mine && ok) {
#pragma unroll
      for (int c = 0; c < CH; ++c)
#pragma unroll
        for (int a = 0; a < 3; ++a)
          *reinterpret_cast<uint4*>(G + core_row<KP>(a * 32 + s, d * CH + c)) = make_uint4(0, 0, 0, 0);
    }
    const int ksteps = (flags & IN_ODD) && par == 1 ? (2 * CIN + 15) / 16 : KP / 16;
    for (int b = b0; b < b1; ++b) {
      if (mine && ok) gather_dir<CIN>(G, d, s, m, hin + (size_t)b * V * planes(CIN), V, n);
      // the tensor cores read G and W through the async proxy
      asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
      // every thread leaves together once a warp's wait for the previous MMA has given up
      if (!__syncthreads_and(ok)) {
        dead = true;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      const uint32_t tmem = tmem_base;
      if (tid == 0) {
        for (int ks = 0; ks < ksteps; ++ks) {
          // K steps of 16 elements: two core matrices along K, 256 bytes
          const uint64_t da = adesc + (uint64_t)((ks * 256) >> 4), db = bdesc + (uint64_t)((ks * 256) >> 4);
          const uint32_t acc = ks > 0 ? 1u : 0u;
          asm volatile(
              "{\n .reg .pred p;\n setp.ne.u32 p, %4, 0;\n"
              " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem),
              "l"(da), "l"(db), "r"(idesc), "r"(acc));
        }
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
                         smem_u32(&mbar))
                     : "memory");
      }
      // every thread waits: the MMA has read G (the next gather may overwrite it) and written its
      // accumulators
      ok = __all_sync(0xffffffffu, d != quit && mbar_wait(smem_u32(&mbar), phase));
      if (!ok) {
        if (s == 0) atomicAdd(errors, 1);
        // give the MMAs in flight one more bounded wait before their tensor memory is freed
        (void)mbar_wait(smem_u32(&mbar), phase);
      }
      phase ^= 1;
      if (!ok) continue;
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      if (d < 3) {  // warp = colour, lane = site
        float v[NU];
        tmem_load_row<NU>(tmem + ((uint32_t)(d * 32) << 16), v);
        if (valid) {
          float4* out = hout + (size_t)b * V * planes(COUT) + j;
#pragma unroll
          for (int q = 0; q < COUT / 2; ++q)
            out[(size_t)(d * (COUT / 2) + q) * V] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
        }
        asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
      }
    }
  }
  __syncthreads();
  if (d == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(kTmemCols));
}

__device__ __forceinline__ void ldmatrix4_trans(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ void ldmatrix2_trans(uint32_t (&r)[2], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];\n"
               : "=r"(r[0]), "=r"(r[1])
               : "r"(addr)
               : "memory");
}

// Gradient of the real-form weights: dW[n][k] += sum_rows delta[row][n] G[row][k], a reduction over
// every (site, colour, right-hand side).  Warp d gathers direction d of a 32-site tile as in
// layer_kernel and multiplies exactly the K columns it gathered (no other warp reads them) by the
// block's delta tile, both read through transposing ldmatrix from the core-matrix layout; the sums
// stay in registers while the block walks its tiles, so each block adds to global memory once
// (one atomic per weight and block instead of one per weight, tile and right-hand side, which took
// most of the time: 769 -> 242 us for 12 -> 12 channels and 4 right-hand sides at 16^3 x 32).  The
// delta tile is double buffered: one barrier per right-hand side.
template <int CIN, int COUT>
__global__ void __launch_bounds__(CT, 2) wgrad_kernel(Geom g, int V, int tiles, int batch, int per, int items, int flags,
                                                      const float2* __restrict__ links, const float4* __restrict__ hin,
                                                      const float4* __restrict__ delta, float* dW) {
  constexpr int KP = kpad(CIN), MT = (2 * COUT + 15) / 16, MP = MT * 16, CH = CIN / 4;
  extern __shared__ __align__(128) unsigned char smem[];
  unsigned char* G = smem;                   // ROWS x KP
  unsigned char* D = smem + ROWS * KP * 2;   // 2 x (ROWS x MP)
  const int tid = threadIdx.x, d = tid >> 5, s = tid & 31;
  if (d < 3) {  // the padding columns of both delta tiles
    for (int c = 2 * COUT / 8; c < MP / 8; ++c)
      for (int q = 0; q < 2; ++q)
        *reinterpret_cast<uint4*>(D + q * (ROWS * MP * 2) + core_row<MP>(d * 32 + s, c)) = make_uint4(0, 0, 0, 0);
  }
  float acc[CH][MT][4];
#pragma unroll
  for (int c = 0; c < CH; ++c)
#pragma unroll
    for (int t = 0; t < MT; ++t)
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[c][t][q] = 0.f;
  const int parts = (batch + per - 1) / per;
  int buf = 0;
  for (int item = blockIdx.x; item < items; item += gridDim.x) {
    int tile = item / parts, par = 1;
    const int b0 = (item - tile * parts) * per, b1 = min(batch, b0 + per);
    if (!(flags & OUT_ODD)) {
      par = tile >= tiles ? 1 : 0;
      tile -= par * tiles;
    }
    const int i = tile * SITES + s;
    const bool valid = i < g.Vh;
    const int ic = valid ? i : g.Vh - 1;
    const int j = par * g.Vh + ic;
    const bool mine = !(flags & IN_ODD) || ((d == 0) == (par == 1));
    const int n = neighbour(g, par, ic, d);
    float2 m[9];
    if (mine && d > 0) load_transport(m, links, V, j, n, d);
    for (int b = b0; b < b1; ++b, buf ^= 1) {
      unsigned char* Db = D + buf * (ROWS * MP * 2);
      if (d < 3) {  // warp = colour: a row of delta, zero past the lattice's end
        const float4* dl = delta + (size_t)b * V * planes(COUT) + j;
#pragma unroll
        for (int c = 0; c < COUT / 4; ++c) {
          const float4 p = __ldg(dl + (size_t)(d * (COUT / 2) + 2 * c) * V);
          const float4 q = __ldg(dl + (size_t)(d * (COUT / 2) + 2 * c + 1) * V);
          uint4 w = make_uint4(bf16x2(p.x, p.y), bf16x2(p.z, p.w), bf16x2(q.x, q.y), bf16x2(q.z, q.w));
          if (!valid) w = make_uint4(0, 0, 0, 0);
          *reinterpret_cast<uint4*>(Db + core_row<MP>(d * 32 + s, c)) = w;
        }
      }
      if (mine) gather_dir<CIN>(G, d, s, m, hin + (size_t)b * V * planes(CIN), V, n);
      __syncthreads();
      if (mine) {
        const uint32_t gs = smem_u32(G), ds = smem_u32(Db);
#pragma unroll
        for (int ks = 0; ks < ROWS / 16; ++ks) {
          uint32_t a[MT][4];
#pragma unroll
          for (int t = 0; t < MT; ++t)
            ldmatrix4_trans(a[t], ds + core_row<MP>(ks * 16 + (s >> 4) * 8 + (s & 7), t * 2 + ((s >> 3) & 1)));
#pragma unroll
          for (int c = 0; c < CH; ++c) {
            uint32_t bb[2];
            ldmatrix2_trans(bb, gs + core_row<KP>(ks * 16 + ((s >> 3) & 1) * 8 + (s & 7), d * CH + c));
#pragma unroll
            for (int t = 0; t < MT; ++t) mma_bf16(acc[c][t], a[t], bb);
          }
        }
        __syncwarp();  // all lanes have read this warp's columns of G before the next gather
      }
    }
  }
  const int gid = s >> 2, tig = s & 3;
#pragma unroll
  for (int c = 0; c < CH; ++c)
#pragma unroll
    for (int t = 0; t < MT; ++t)
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int nn = t * 16 + gid + 8 * half, k = (d * CH + c) * 8 + 2 * tig;
        if (nn < 2 * COUT) {
          atomicAdd(&dW[(size_t)nn * KP + k], acc[c][t][2 * half]);
          atomicAdd(&dW[(size_t)nn * KP + k + 1], acc[c][t][2 * half + 1]);
        }
      }
}

// spinor components (spin * 3 + colour) of one site <-> the 6 planes of a 4-channel activation
template <typename T>
__device__ __forceinline__ void put_site(float4* act, int V, int j, const cplx<T> (&v)[12]) {
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const cplx<T> x = v[(2 * q) * 3 + a], y = v[(2 * q + 1) * 3 + a];
      act[(size_t)(a * 2 + q) * V + j] = make_float4((float)x.re, (float)y.re, (float)x.im, (float)y.im);
    }
}
template <typename T>
__device__ __forceinline__ void get_site(const float4* act, int V, int j, cplx<T> (&v)[12]) {
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const float4 w = act[(size_t)(a * 2 + q) * V + j];
      v[(2 * q) * 3 + a] = {(T)w.x, (T)w.z};
      v[(2 * q + 1) * 3 + a] = {(T)w.y, (T)w.w};
    }
}

// odd-site spinor field (precision P) -> odd sites of the layer-0 activations
template <typename P>
__global__ void embed_kernel(Geom g, int V, Spinor f, float4* act) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int b = blockIdx.y;
  if (i >= g.Vh) return;
  cplx<typename P::real> v[12];
  load_spinor<P>(v, (const char*)f.v + (size_t)b * f.rhs_bytes, f.norm ? f.norm + (size_t)b * f.norm_rhs_stride : nullptr,
                 i, f.stride);
  put_site(act + (size_t)b * V * planes(4), V, g.Vh + i, v);
}

template <typename P>
__global__ void extract_kernel(Geom g, int V, const float4* act, Spinor f) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int b = blockIdx.y;
  if (i >= g.Vh) return;
  cplx<typename P::real> v[12];
  get_site(act + (size_t)b * V * planes(4), V, g.Vh + i, v);
  store_spinor<P>((char*)f.v + (size_t)b * f.rhs_bytes, f.norm ? f.norm + (size_t)b * f.norm_rhs_stride : nullptr, i,
                  f.stride, v);
}

// block sum of one double per thread (128 threads), valid in thread 0
__device__ __forceinline__ double block_sum_128(double v) {
  __shared__ double sh[4];
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  return threadIdx.x == 0 ? (sh[0] + sh[1]) + (sh[2] + sh[3]) : 0.0;
}

// canonical complex128 [V][12] (rhs b at offset b*V*12) -> activations, odd sites only;
// NORM: norm2[b] += |f_b|^2 over the odd sites, in FP64
template <bool NORM>
__global__ void __launch_bounds__(128) embed_canon_kernel(Geom g, int V, const double2* canon, float4* act,
                                                          double* norm2) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int b = blockIdx.y;
  double sum = 0.0;
  if (i < g.Vh) {
    const Coord c = cb_coords(g, i, 1);
    const double2* src = canon + ((size_t)b * V + full_index(g, c)) * 12;
    cplx<double> v[12];
#pragma unroll
    for (int k = 0; k < 12; ++k) {
      const double2 w = src[k];
      v[k] = {w.x, w.y};
      if (NORM) sum = fmadd(w.x, w.x, fmadd(w.y, w.y, sum));
    }
    put_site(act + (size_t)b * V * planes(4), V, g.Vh + i, v);
  }
  if constexpr (NORM) {
    sum = block_sum_128(sum);
    if (threadIdx.x == 0) atomicAdd(&norm2[b], sum);
  }
}

// One thread per (canonical site, component): consecutive threads write consecutive 16-byte
// components (one thread per site wrote 16 bytes of 32 different sectors per store instruction)
__global__ void extract_canon_kernel(Geom g, int V, const float4* act, double2* canon) {
  const long p = blockIdx.x * (long)blockDim.x + threadIdx.x;
  const int b = blockIdx.y;
  if (p >= (long)V * 12) return;
  const int site = (int)(p / 12), k = (int)(p - (long)site * 12);
  Coord c;
  int r = site;
  c.x[0] = r % g.L[0];
  r /= g.L[0];
  c.x[1] = r % g.L[1];
  r /= g.L[1];
  c.x[2] = r % g.L[2];
  c.x[3] = r / g.L[2];
  double2 v = make_double2(0.0, 0.0);
  if ((c.x[0] + c.x[1] + c.x[2] + c.x[3]) & 1) {
    const int spin = k / 3, a = k - spin * 3;
    const float* w = reinterpret_cast<const float*>(
        act + ((size_t)b * planes(4) + a * 2 + (spin >> 1)) * V + g.Vh + cb_index(g, c));
    v = make_double2((double)w[spin & 1], (double)w[2 + (spin & 1)]);
  }
  canon[(size_t)b * V * 12 + p] = v;
}

// loss = sum_b sum_odd |y - e|^2 / |e|^2 ; delta = 2 (y - e) / |e|^2, all on the odd sites
__global__ void __launch_bounds__(128) loss_kernel(Geom g, int V, const float4* y, const float4* e,
                                                   const double* enorm2, float4* delta, double* partial) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int b = blockIdx.y;
  double l = 0.0;
  if (i < g.Vh) {
    const float inv = (float)(1.0 / enorm2[b]);
#pragma unroll
    for (int q = 0; q < planes(4); ++q) {
      const size_t o = ((size_t)b * planes(4) + q) * V + g.Vh + i;
      const float4 p = y[o], t = e[o];
      const float4 d = make_float4(p.x - t.x, p.y - t.y, p.z - t.z, p.w - t.w);
      l += (double)(d.x * d.x + d.z * d.z) * inv;
      l += (double)(d.y * d.y + d.w * d.w) * inv;
      delta[o] = make_float4(2.f * d.x * inv, 2.f * d.y * inv, 2.f * d.z * inv, 2.f * d.w * inv);
    }
  }
  l = block_sum_128(l);
  if (threadIdx.x == 0) atomicAdd(partial, l);
}

// canonical links -> FP32 planes [mu * 9 + entry][even-odd site]
__global__ void links_kernel(Geom g, int V, const double2* canon, float2* links) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= V) return;
  const Coord c = eo_coords(g, j);
  const long s = full_index(g, c);
  for (int e = 0; e < 36; ++e) {
    const double2 v = canon[s * 36 + e];
    links[(size_t)e * V + j] = make_float2((float)v.x, (float)v.y);
  }
}

// Work split of a layer over the grid: a block is a 32-site tile of one parity and up to `per`
// right-hand sides, which share its transports and weights.  All of a batch in one block is best
// while the tiles alone fill the chip; with fewer tiles than two waves (152 SMs x 3 blocks) the
// batch is spread over more blocks.
struct Split {
  int tiles, blocks, per, parts;
};
Split split_of(const Geom& g, int batch, int flags) {
  Split w;
  w.tiles = (g.Vh + SITES - 1) / SITES;
  w.blocks = (flags & OUT_ODD) ? w.tiles : 2 * w.tiles;
  const int want = std::min(batch, std::max(1, 2 * 152 * 3 / w.blocks));
  w.per = (batch + want - 1) / want;
  w.parts = (batch + w.per - 1) / w.per;
  return w;
}

template <int CIN, int COUT>
void launch_layer(const Geom& g, int V, int batch, int flags, const float2* links, const float4* in, float4* out,
                  const __nv_bfloat16* W, int* errors, int quit, cudaStream_t s) {
  // G (96 rows) and W (npad rows) in the core-matrix layout, inside the 128 rows x kpad that the
  // MMA's A operand (and its B operand, ending at the same row) spans
  const size_t smem = (size_t)128 * kpad(CIN) * 2;
  GBC_CUDA(cudaFuncSetAttribute(layer_kernel<CIN, COUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const Split w = split_of(g, batch, flags);
  // three resident blocks per SM
  layer_kernel<CIN, COUT><<<dim3(std::min(w.blocks, 3 * 152), w.parts), CT, smem, s>>>(
      g, V, w.tiles, w.blocks, batch, w.per, flags, links, in, out, reinterpret_cast<const uint4*>(W), errors, quit);
  count_launch();
}

template <int CIN, int COUT>
void launch_wgrad(const Geom& g, int V, int batch, int flags, const float2* links, const float4* in,
                  const float4* delta, float* dW, cudaStream_t s) {
  constexpr int MP = ((2 * COUT + 15) / 16) * 16;
  const size_t smem = (size_t)ROWS * (kpad(CIN) + 2 * MP) * 2;
  GBC_CUDA(cudaFuncSetAttribute(wgrad_kernel<CIN, COUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const Split w = split_of(g, batch, flags);
  const int items = w.blocks * w.parts;
  // two resident blocks per SM walk the items (their sums live in registers)
  wgrad_kernel<CIN, COUT><<<std::min(items, 2 * 152), CT, smem, s>>>(g, V, w.tiles, batch, w.per, items, flags, links,
                                                                     in, delta, dW);
  count_launch();
}

void layer(const Geom& g, int V, int batch, int cin, int cout, int flags, const float2* links, const float4* in,
           float4* out, const __nv_bfloat16* W, int* errors, int quit, cudaStream_t s) {
  if (cin == 4 && cout == 12) launch_layer<4, 12>(g, V, batch, flags, links, in, out, W, errors, quit, s);
  else if (cin == 12 && cout == 12) launch_layer<12, 12>(g, V, batch, flags, links, in, out, W, errors, quit, s);
  else if (cin == 12 && cout == 4) launch_layer<12, 4>(g, V, batch, flags, links, in, out, W, errors, quit, s);
  else if (cin == 4 && cout == 4) launch_layer<4, 4>(g, V, batch, flags, links, in, out, W, errors, quit, s);
  else throw std::string("network layer shape not compiled");
}

void wgrad(const Geom& g, int V, int batch, int cin, int cout, int flags, const float2* links, const float4* in,
           const float4* delta, float* dW, cudaStream_t s) {
  if (cin == 4 && cout == 12) launch_wgrad<4, 12>(g, V, batch, flags, links, in, delta, dW, s);
  else if (cin == 12 && cout == 12) launch_wgrad<12, 12>(g, V, batch, flags, links, in, delta, dW, s);
  else if (cin == 12 && cout == 4) launch_wgrad<12, 4>(g, V, batch, flags, links, in, delta, dW, s);
  else if (cin == 4 && cout == 4) launch_wgrad<4, 4>(g, V, batch, flags, links, in, delta, dW, s);
  else throw std::string("network layer shape not compiled");
}

}  // namespace

// ---------------------------------------------------------------------------------------------
// host model
// ---------------------------------------------------------------------------------------------
using cf = std::complex<float>;

int Cnn::cin(int l) const { return l == 0 ? 4 : hidden; }
int Cnn::cout(int l) const { return l == nlayers - 1 ? 4 : hidden; }

void Cnn::init(int hidden_, int layers_, unsigned long long seed) {
  hidden = hidden_;
  nlayers = layers_;
  W.assign(nlayers, {});
  std::mt19937_64 rng(seed);
  std::normal_distribution<float> nd(0.f, 1.f);
  for (int l = 0; l < nlayers; ++l) {
    const int ci = cin(l), co = cout(l);
    W[l].assign((size_t)9 * co * ci, cf(0, 0));
    // start near the identity map through the self term, with small random hops (scaled so a
    // layer roughly preserves norms)
    const float sc = 0.1f / std::sqrt((float)(9 * ci));
    for (auto& w : W[l]) w = cf(sc * nd(rng), sc * nd(rng));
    for (int o = 0; o < co; ++o)
      for (int i = 0; i < ci; ++i)
        if (o % ci == i || (ci > co && i % co == o)) W[l][(size_t)o * ci + i] += cf(ci > co ? 1.0f / (ci / co) : 1.0f, 0);
  }
  m1.assign(nlayers, {});
  m2.assign(nlayers, {});
  for (int l = 0; l < nlayers; ++l) {
    m1[l].assign(W[l].size() * 2, 0.f);
    m2[l].assign(W[l].size() * 2, 0.f);
  }
  step = 0;
  dirty = true;
  // GBC_TC_QUIT_WARP=<warp>: that warp of every layer block gives up its waits (error-path tests)
  const char* q = getenv("GBC_TC_QUIT_WARP");
  quit = q && *q ? atoi(q) : -1;
}

// Real form of a layer's weights in the MMA's order (comp) and core-matrix layout: rows n = comp(o, .)
// of the outputs, columns k = (d * C_in + i) * 2 + re/im.
static void real_form(const std::vector<cf>& Wc, int ci, int co, bool adjoint, std::vector<__nv_bfloat16>& out) {
  // adjoint: out channels = ci, in channels = co, W'_d = (W_{swap d})^H
  const int oc = adjoint ? ci : co, ic = adjoint ? co : ci;
  const int KP = kpad(ic), NP = npad(oc);
  out.assign((size_t)NP * KP, __float2bfloat16(0.f));
  for (int d = 0; d < 9; ++d) {
    const int ds = adjoint ? (d == 0 ? 0 : (((d - 1) ^ 1) + 1)) : d;
    for (int o = 0; o < oc; ++o)
      for (int i = 0; i < ic; ++i) {
        cf w = adjoint ? std::conj(Wc[((size_t)ds * co + i) * ci + o]) : Wc[((size_t)d * co + o) * ci + i];
        auto at = [&](int no, int ki) -> __nv_bfloat16& {
          const int n = comp(o, no), k = (d * ic + i) * 2 + ki;
          return out[(size_t)(n >> 3) * (KP * 8) + (k >> 3) * 64 + (n & 7) * 8 + (k & 7)];
        };
        at(0, 0) = __float2bfloat16(w.real());
        at(0, 1) = __float2bfloat16(-w.imag());
        at(1, 0) = __float2bfloat16(w.imag());
        at(1, 1) = __float2bfloat16(w.real());
      }
  }
}

void Cnn::upload(cudaStream_t s) {
  if (!dirty) return;
  for (int l = 0; l < nlayers; ++l) {
    std::vector<__nv_bfloat16> a, b;
    real_form(W[l], cin(l), cout(l), false, a);
    real_form(W[l], cin(l), cout(l), true, b);
    if (!dW[l]) {
      GBC_CUDA(cudaMalloc(&dW[l], a.size() * 2));
      GBC_CUDA(cudaMalloc(&dWadj[l], b.size() * 2));
    }
    GBC_CUDA(cudaMemcpyAsync(dW[l], a.data(), a.size() * 2, cudaMemcpyHostToDevice, s));
    GBC_CUDA(cudaMemcpyAsync(dWadj[l], b.data(), b.size() * 2, cudaMemcpyHostToDevice, s));
  }
  GBC_CUDA(cudaStreamSynchronize(s));
  dirty = false;
}

void Cnn::release() {
  for (int l = 0; l < 8; ++l) {
    if (dW[l]) cudaFree(dW[l]);
    if (dWadj[l]) cudaFree(dWadj[l]);
    dW[l] = dWadj[l] = nullptr;
  }
  for (auto& p : act) if (p) cudaFree(p);
  act.clear();
  for (void* p : {(void*)links, (void*)delta[0], (void*)delta[1], (void*)target, (void*)dG, (void*)norms, (void*)errors})
    if (p) cudaFree(p);
  links = nullptr;
  delta[0] = delta[1] = target = nullptr;
  dG = nullptr;
  norms = nullptr;
  errors = nullptr;
  act_batch = train_batch = 0;
}

void Cnn::ensure(gbc_ctx* c, int batch) {
  const int V = (int)c->V;
  if (!errors) {
    GBC_CUDA(cudaMalloc(&errors, sizeof(int)));
    GBC_CUDA(cudaMemsetAsync(errors, 0, sizeof(int), c->stream));
  }
  if (!links || links_version != c->gauge_version) {
    if (!links) GBC_CUDA(cudaMalloc(&links, sizeof(float2) * (size_t)V * 36));
    links_kernel<<<(V + 127) / 128, 128, 0, c->stream>>>(c->g, V, reinterpret_cast<const double2*>(c->d_links), links);
    count_launch();
    links_version = c->gauge_version;
  }
  if (act_batch < batch) {
    act_batch = 0;
    for (auto& p : act) if (p) cudaFree(p);
    act.assign(nlayers + 1, nullptr);
    for (int l = 0; l <= nlayers; ++l)
      GBC_CUDA(cudaMalloc(&act[l], sizeof(float4) * (size_t)batch * V * planes(l == 0 ? 4 : cout(l - 1))));
    act_batch = batch;
  }
  upload(c->stream);
}

// Workspaces of the training step: targets, back-propagated deltas, the weight gradients of all
// layers in one buffer, and the target norms with the loss behind them.
void Cnn::ensure_train(gbc_ctx* c, int batch) {
  ensure(c, batch);
  if (!dG) GBC_CUDA(cudaMalloc(&dG, sizeof(float) * grad_offset(nlayers)));
  if (train_batch >= batch) return;
  train_batch = 0;
  for (float4** p : {&delta[0], &delta[1], &target}) {
    if (*p) cudaFree(*p);
    *p = nullptr;
  }
  if (norms) cudaFree(norms);
  norms = nullptr;
  const size_t V = (size_t)c->V;
  for (int q = 0; q < 2; ++q) GBC_CUDA(cudaMalloc(&delta[q], sizeof(float4) * batch * V * planes(hidden)));
  GBC_CUDA(cudaMalloc(&target, sizeof(float4) * batch * V * planes(4)));
  GBC_CUDA(cudaMalloc(&norms, sizeof(double) * (batch + 1)));
  train_batch = batch;
}

size_t Cnn::grad_offset(int l) const {
  size_t n = 0;
  for (int k = 0; k < l; ++k) n += (size_t)npad(cout(k)) * kpad(cin(k));
  return n;
}

// The network's input is zero on the even sites and only its odd output sites are wanted: the
// first layer skips the zero terms, the last the even sites.
void Cnn::forward(gbc_ctx* c, int batch) {
  const int V = (int)c->V;
  for (int l = 0; l < nlayers; ++l)
    layer(c->g, V, batch, cin(l), cout(l), (l == 0 ? IN_ODD : 0) | (l == nlayers - 1 ? OUT_ODD : 0), links, act[l],
          act[l + 1], dW[l], errors, quit, c->stream);
}

// A layer whose wait for its tensor-core results gave up (it then frees its tensor memory and
// returns) counts in `errors`: read and reset it, and fail the call that ran the layers.
void Cnn::check_waits(cudaStream_t s) {
  if (!errors) return;  // no layer has run
  int n = 0;
  GBC_CUDA(cudaMemcpyAsync(&n, errors, sizeof(int), cudaMemcpyDeviceToHost, s));
  GBC_CUDA(cudaStreamSynchronize(s));
  if (n) {
    GBC_CUDA(cudaMemsetAsync(errors, 0, sizeof(int), s));
    throw std::string("network layer: a wait for the tensor cores gave up");
  }
}

double Cnn::loss_and_grad(gbc_ctx* c, int batch) {
  const int V = (int)c->V;
  cudaStream_t s = c->stream;
  forward(c, batch);
  double* dl = norms + batch;
  GBC_CUDA(cudaMemsetAsync(dl, 0, sizeof(double), s));
  loss_kernel<<<dim3((c->g.Vh + 127) / 128, batch), 128, 0, s>>>(c->g, V, act[nlayers], target, norms, delta[0], dl);
  count_launch();
  GBC_CUDA(cudaMemsetAsync(dG, 0, sizeof(float) * grad_offset(nlayers), s));
  int cur = 0;
  for (int l = nlayers - 1; l >= 0; --l) {
    // delta of the last layer lives on the odd sites, the first layer's input too
    const bool last = l == nlayers - 1;
    wgrad(c->g, V, batch, cin(l), cout(l), (l == 0 ? IN_ODD : 0) | (last ? OUT_ODD : 0), links, act[l], delta[cur],
          dG + grad_offset(l), s);
    if (l > 0) {
      layer(c->g, V, batch, cout(l), cin(l), last ? IN_ODD : 0, links, delta[cur], delta[1 - cur], dWadj[l], errors, quit, s);
      cur = 1 - cur;
    }
  }
  double loss = 0;
  GBC_CUDA(cudaMemcpyAsync(&loss, dl, sizeof(double), cudaMemcpyDeviceToHost, s));
  check_waits(s);
  return loss;
}

// complex gradient dL/dRe W + i dL/dIm W from the real-form gradient
void Cnn::download_grad(cudaStream_t s, std::vector<std::vector<cf>>& grad) {
  grad.assign(nlayers, {});
  std::vector<float> all(grad_offset(nlayers));
  GBC_CUDA(cudaMemcpyAsync(all.data(), dG, all.size() * 4, cudaMemcpyDeviceToHost, s));
  GBC_CUDA(cudaStreamSynchronize(s));
  for (int l = 0; l < nlayers; ++l) {
    const int ci = cin(l), co = cout(l), KP = kpad(ci);
    const float* gr = all.data() + grad_offset(l);
    grad[l].assign((size_t)9 * co * ci, cf(0, 0));
    for (int d = 0; d < 9; ++d)
      for (int o = 0; o < co; ++o)
        for (int i = 0; i < ci; ++i) {
          auto at = [&](int no, int ki) { return gr[(size_t)comp(o, no) * KP + (d * ci + i) * 2 + ki]; };
          grad[l][((size_t)d * co + o) * ci + i] = cf(at(0, 0) + at(1, 1), at(1, 0) - at(0, 1));
        }
  }
}

void Cnn::adam(const std::vector<std::vector<cf>>& grad, double lr) {
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  ++step;
  const float c1 = 1.f - std::pow(b1, (float)step), c2 = 1.f - std::pow(b2, (float)step);
  for (int l = 0; l < nlayers; ++l)
    for (size_t q = 0; q < W[l].size(); ++q) {
      const float gq[2] = {grad[l][q].real(), grad[l][q].imag()};
      float wq[2] = {W[l][q].real(), W[l][q].imag()};
      for (int r = 0; r < 2; ++r) {
        float& m = m1[l][2 * q + r];
        float& v = m2[l][2 * q + r];
        m = b1 * m + (1 - b1) * gq[r];
        v = b2 * v + (1 - b2) * gq[r] * gq[r];
        wq[r] -= (float)lr * (m / c1) / (std::sqrt(v / c2) + eps);
      }
      W[l][q] = cf(wq[0], wq[1]);
    }
  dirty = true;
}

// file: "GBCW" u32 version=1, u32 layers, u32 hidden, then per layer u32 cin, u32 cout,
// 9*cout*cin complex float32, then u64 FNV-1a of everything before it
static uint64_t fnv1a(const unsigned char* p, size_t n) {
  uint64_t h = 1469598103934665603ULL;
  for (size_t i = 0; i < n; ++i) {
    h ^= p[i];
    h *= 1099511628211ULL;
  }
  return h;
}

bool Cnn::save(const std::string& path) const {
  std::vector<unsigned char> buf;
  auto put = [&](const void* p, size_t n) {
    const unsigned char* c = static_cast<const unsigned char*>(p);
    buf.insert(buf.end(), c, c + n);
  };
  const char magic[4] = {'G', 'B', 'C', 'W'};
  const uint32_t ver = 1, L = nlayers, H = hidden;
  put(magic, 4);
  put(&ver, 4);
  put(&L, 4);
  put(&H, 4);
  for (int l = 0; l < nlayers; ++l) {
    const uint32_t ci = cin(l), co = cout(l);
    put(&ci, 4);
    put(&co, 4);
    put(W[l].data(), W[l].size() * sizeof(cf));
  }
  const uint64_t h = fnv1a(buf.data(), buf.size());
  put(&h, 8);
  std::ofstream f(path, std::ios::binary);
  if (!f) return false;
  f.write(reinterpret_cast<const char*>(buf.data()), (std::streamsize)buf.size());
  return (bool)f;
}

int Cnn::load(const std::string& path) {
  std::ifstream f(path, std::ios::binary);
  if (!f) return GBC_ERR_PRECOND;
  std::vector<unsigned char> buf((std::istreambuf_iterator<char>(f)), std::istreambuf_iterator<char>());
  if (buf.size() < 16 + 8 || std::memcmp(buf.data(), "GBCW", 4) != 0) return GBC_ERR_PRECOND;
  uint64_t h;
  std::memcpy(&h, buf.data() + buf.size() - 8, 8);
  if (fnv1a(buf.data(), buf.size() - 8) != h) return GBC_ERR_PRECOND;
  uint32_t ver, L, H;
  std::memcpy(&ver, buf.data() + 4, 4);
  std::memcpy(&L, buf.data() + 8, 4);
  std::memcpy(&H, buf.data() + 12, 4);
  if (ver != 1 || L < 1 || L > 8 || (H != 4 && H != 12)) return GBC_ERR_PRECOND;
  init((int)H, (int)L, 0);
  size_t off = 16;
  for (int l = 0; l < nlayers; ++l) {
    uint32_t ci, co;
    if (off + 8 > buf.size() - 8) return GBC_ERR_PRECOND;
    std::memcpy(&ci, buf.data() + off, 4);
    std::memcpy(&co, buf.data() + off + 4, 4);
    off += 8;
    if ((int)ci != cin(l) || (int)co != cout(l)) return GBC_ERR_PRECOND;
    const size_t n = W[l].size() * sizeof(cf);
    if (off + n > buf.size() - 8) return GBC_ERR_PRECOND;
    std::memcpy(W[l].data(), buf.data() + off, n);
    off += n;
  }
  if (off != buf.size() - 8) return GBC_ERR_PRECOND;
  dirty = true;
  return GBC_OK;
}

void cnn_apply_spinor(gbc_ctx* c, Cnn& net, const Spinor& in, const Spinor& out) {
  const int V = (int)c->V;
  net.ensure(c, in.nrhs);
  const dim3 grid((c->g.Vh + 127) / 128, in.nrhs);
  if (in.prec == PREC_DOUBLE) embed_kernel<PrecD><<<grid, 128, 0, c->stream>>>(c->g, V, in, net.act[0]);
  else if (in.prec == PREC_SINGLE) embed_kernel<PrecS><<<grid, 128, 0, c->stream>>>(c->g, V, in, net.act[0]);
  else embed_kernel<PrecH><<<grid, 128, 0, c->stream>>>(c->g, V, in, net.act[0]);
  count_launch();
  net.forward(c, in.nrhs);
  if (out.prec == PREC_DOUBLE) extract_kernel<PrecD><<<grid, 128, 0, c->stream>>>(c->g, V, net.act[net.nlayers], out);
  else if (out.prec == PREC_SINGLE) extract_kernel<PrecS><<<grid, 128, 0, c->stream>>>(c->g, V, net.act[net.nlayers], out);
  else extract_kernel<PrecH><<<grid, 128, 0, c->stream>>>(c->g, V, net.act[net.nlayers], out);
  count_launch();
}

void cnn_embed_canon(gbc_ctx* c, Cnn& net, int batch, const double* canon_dev, float4* act, double* norm2) {
  const int V = (int)c->V;
  const dim3 grid((c->g.Vh + 127) / 128, batch);
  const double2* src = reinterpret_cast<const double2*>(canon_dev);
  if (norm2) {
    GBC_CUDA(cudaMemsetAsync(norm2, 0, sizeof(double) * batch, c->stream));
    embed_canon_kernel<true><<<grid, 128, 0, c->stream>>>(c->g, V, src, act, norm2);
  } else {
    embed_canon_kernel<false><<<grid, 128, 0, c->stream>>>(c->g, V, src, act, nullptr);
  }
  count_launch();
}

void cnn_extract_canon(gbc_ctx* c, Cnn& net, int batch, const float4* act, double* canon_dev) {
  const int V = (int)c->V;
  const dim3 grid((unsigned)(((long)V * 12 + 255) / 256), batch);
  extract_canon_kernel<<<grid, 256, 0, c->stream>>>(c->g, V, act, reinterpret_cast<double2*>(canon_dev));
  count_launch();
}

}  // namespace gbc
