// Clover term construction on the device, FP64:
//   F_{mu nu} = (1/8) (Q - Q^dag), Q = sum of the four plaquette leaves   (Chroma mesfield.cc:30-78)
//   A = diag_mass - sum_{mu<nu} c_{mu nu} gamma_mu gamma_nu F_{mu nu}, packed as Chroma's
//       PrimitiveClovTriang {diag[2][6], offd[2][15]}           (clover_term_qdp_w.h:244-294, 398-553)
//   A^-1 by LDL^dag factorisation of each 6x6 block + log|d_i| (clover_term_qdp_w.h:608-846)
#include "gbc_device.cuh"
#include "su3.cuh"

namespace gbc {

namespace {

struct Dims {
  int L[4];
};

// LDL^dag factorisation and inverse of one packed 6x6 block in place (diag d[6], offd o[15]);
// accumulates log|d_i| and the count of negative d_i.
__device__ __forceinline__ void ldl_invert_block(double* d, cplx<double>* o, double& logdet, int& nneg) {
  const int N = 6;
  cplx<double> v[6];
#pragma unroll
  for (int j = 0; j < N; ++j) {
#pragma unroll
    for (int i = 0; i < j; ++i) v[i] = d[i] * conj(o[j * (j - 1) / 2 + i]);
    v[j] = {d[j], 0.0};
#pragma unroll
    for (int k = 0; k < j; ++k) v[j] = v[j] - o[j * (j - 1) / 2 + k] * v[k];
    d[j] = v[j].re;
    const double inv = 1.0 / v[j].re;
#pragma unroll
    for (int k = j + 1; k < N; ++k) {
      const int ekj = k * (k - 1) / 2 + j;
#pragma unroll
      for (int l = 0; l < j; ++l) o[ekj] = o[ekj] - o[k * (k - 1) / 2 + l] * v[l];
      o[ekj] = inv * o[ekj];
    }
  }
  double dg[6];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    dg[i] = 1.0 / d[i];
    logdet += log(fabs(d[i]));
    if (d[i] < 0) ++nneg;
  }
  double inv_d[6];
  cplx<double> inv_o[15];
#pragma unroll
  for (int k = 0; k < N; ++k) {
#pragma unroll
    for (int i = 0; i < k; ++i) v[i] = {0.0, 0.0};
    v[k] = {dg[k], 0.0};
#pragma unroll
    for (int i = k + 1; i < N; ++i) {
      cplx<double> acc = {0.0, 0.0};
#pragma unroll
      for (int j = k; j < i; ++j) acc = acc - d[j] * (o[i * (i - 1) / 2 + j] * v[j]);
      v[i] = dg[i] * acc;
    }
#pragma unroll
    for (int i = N - 2; i >= k; --i)
#pragma unroll
      for (int j = i + 1; j < N; ++j) v[i] = v[i] - conj(o[j * (j - 1) / 2 + i]) * v[j];
    inv_d[k] = v[k].re;
#pragma unroll
    for (int i = k + 1; i < N; ++i) inv_o[i * (i - 1) / 2 + k] = v[i];
  }
#pragma unroll
  for (int i = 0; i < N; ++i) d[i] = inv_d[i];
#pragma unroll
  for (int i = 0; i < 15; ++i) o[i] = inv_o[i];
}

constexpr int kBuildSites = 32;

// f (Q - Q^dag) of plane (mu, nu) at site s, Q the sum of the four leaves.  Each leaf or its adjoint
// starts or ends with U_mu(x) or U_mu(x - mu), so Q - Q^dag = T - T^dag with
//   T = U_mu(x) [ U_nu(x+mu) U_mu^dag(x+nu) U_nu^dag(x) - U_nu^dag(x-nu+mu) U_mu^dag(x-nu) U_nu(x-nu) ]
//     + [ U_nu(x) U_mu^dag(x-mu+nu) U_nu^dag(x-mu) - U_nu^dag(x-nu) U_mu^dag(x-mu-nu) U_nu(x-mu-nu) ] U_mu(x-mu):
// 10 products instead of 12.
__device__ __forceinline__ M plane_field(const double2* u, long s, long up_m, long dn_m, long up_n, long dn_n, int mu,
                                         int nu, double f) {
  M a = mzero(), t = mzero(), r = mzero();
  mmac<false, true>(t, ld(u, s + up_m, nu), ld(u, s + up_n, mu));
  mmac<false, true>(a, t, ld(u, s, nu));
  t = mzero();
  mmac<true, true>(t, ld(u, s + dn_n + up_m, nu), ld(u, s + dn_n, mu));
  mmac<false, false, true>(a, t, ld(u, s + dn_n, nu));
  mmac<false, false>(r, ld(u, s, mu), a);
  a = t = mzero();
  mmac<false, true>(t, ld(u, s, nu), ld(u, s + dn_m + up_n, mu));
  mmac<false, true>(a, t, ld(u, s + dn_m, nu));
  t = mzero();
  mmac<true, true>(t, ld(u, s + dn_n, nu), ld(u, s + dn_m + dn_n, mu));
  mmac<false, false, true>(a, t, ld(u, s + dn_m + dn_n, nu));
  mmac<false, false>(r, a, ld(u, s + dn_m, mu));
  M o;
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j)
      o.a[3 * i + j] = make_double2(f * (r.a[3 * i + j].x - r.a[3 * j + i].x), f * (r.a[3 * i + j].y + r.a[3 * j + i].y));
  return o;
}

// A block builds 32 sites: warp k computes the field strength of plane k (lane = site), then warps 0
// and 1 assemble, store and invert chirality blocks 0 and 1; the block's sums of log|d| per parity and
// of the even sites' negative pivots.  Bound by the FP64 pipe: 1080 FP64 instructions per plane and site
// and about 1070 per chirality block.  One thread per site held six field strengths and both blocks at
// once and spilled them.
__global__ void __launch_bounds__(6 * kBuildSites, 2) clover_build_kernel(Dims D, const double2* canon, CloverCoeffs cc,
                                                                       double* clov, double* inv, int inv_parity, long V,
                                                                       double* sums, int sums_stride) {
  __shared__ double2 F[6][9][kBuildSites];
  const int l = threadIdx.x & 31, w = threadIdx.x >> 5;
  const long s = (long)blockIdx.x * kBuildSites + l;
  const bool valid = s < V;
  int x[4] = {0, 0, 0, 0};
  if (valid) {
    const Steps n = steps(D.L, s, x);
    const int mu = w < 3 ? 0 : w < 5 ? 1 : 2, nu = w < 3 ? w + 1 : w < 5 ? w - 1 : 3;  // planes 01,02,03,12,13,23
    double coef = cc.coef[0];
#pragma unroll
    for (int k = 1; k < 6; ++k)
      if (w == k) coef = cc.coef[k];
    const M o = plane_field(canon, s, pick(n.up, mu), pick(n.dn, mu), pick(n.up, nu), pick(n.dn, nu), mu, nu, 0.125 * coef);
#pragma unroll
    for (int e = 0; e < 9; ++e) F[w][e][l] = o.a[e];
  }
  __syncthreads();
  double v[3] = {0.0, 0.0, 0.0};
  if (w < 2 && valid) {
    const int b = w;
    auto f = [&](int k, int e) { return cplx<double>{F[k][e][l].x, F[k][e][l].y}; };
    // makeClov (clover_term_qdp_w.h:398-553)
    double diag[6];
    cplx<double> offd[15];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const double r = b == 0 ? (f(5, 4 * i) - f(0, 4 * i)).im : -(f(5, 4 * i) + f(0, 4 * i)).im;
      diag[i] = cc.diag_mass + r;
      diag[i + 3] = cc.diag_mass - r;
    }
#pragma unroll
    for (int i = 1; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < i; ++j) {
        const cplx<double> e0 = f(0, 3 * i + j), e5 = f(5, 3 * i + j);
        const cplx<double> e = timesI(b == 0 ? e0 - e5 : e5 + e0);
        offd[i * (i - 1) / 2 + j] = e;
        offd[(i + 3) * (i + 2) / 2 + j + 3] = -e;
      }
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const cplx<double> Em = timesI(f(2, 3 * i + j)) + f(4, 3 * i + j);
        const cplx<double> Bm = timesI(f(3, 3 * i + j)) - f(1, 3 * i + j);
        offd[(i + 3) * (i + 2) / 2 + j] = b == 0 ? Bm - Em : Em + Bm;
      }
    auto store = [&](double* p) {
#pragma unroll
      for (int i = 0; i < 6; ++i) p[6 * b + i] = diag[i];
#pragma unroll
      for (int i = 0; i < 15; ++i) {
        p[12 + 30 * b + 2 * i] = offd[i].re;
        p[12 + 30 * b + 2 * i + 1] = offd[i].im;
      }
    };
    store(clov + s * 72);
    const int par = (x[0] + x[1] + x[2] + x[3]) & 1;
    double logdet = 0.0;
    int nneg = 0;
    if (inv_parity == 2 || par == inv_parity) {
      ldl_invert_block(diag, offd, logdet, nneg);
    } else {
#pragma unroll
      for (int i = 0; i < 6; ++i) diag[i] = 0.0;
#pragma unroll
      for (int i = 0; i < 15; ++i) offd[i] = {0.0, 0.0};
    }
    store(inv + s * 72);
    v[0] = par ? 0.0 : logdet;
    v[1] = par ? logdet : 0.0;
    v[2] = par ? 0.0 : (double)nneg;
  }
  __shared__ double sh[3][2];
  if (w < 2) {
#pragma unroll
    for (int q = 0; q < 3; ++q) {
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) v[q] += __shfl_down_sync(0xffffffffu, v[q], off);
      if (l == 0) sh[q][w] = v[q];
    }
  }
  __syncthreads();
  if (threadIdx.x < 3) sums[(size_t)threadIdx.x * sums_stride + blockIdx.x] = sh[threadIdx.x][0] + sh[threadIdx.x][1];
}

__global__ void clover_invert_kernel(long n, double* packed, double* logdet, int* nneg) {
  const long s = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (s >= n) return;
  double* p = packed + s * 72;
  double d[2][6];
  cplx<double> o[2][15];
  for (int b = 0; b < 2; ++b) {
    for (int i = 0; i < 6; ++i) d[b][i] = p[6 * b + i];
    for (int i = 0; i < 15; ++i) o[b][i] = {p[12 + 30 * b + 2 * i], p[13 + 30 * b + 2 * i]};
  }
  double ld = 0.0;
  int nn = 0;
  for (int b = 0; b < 2; ++b) ldl_invert_block(d[b], o[b], ld, nn);
  for (int b = 0; b < 2; ++b) {
    for (int i = 0; i < 6; ++i) p[6 * b + i] = d[b][i];
    for (int i = 0; i < 15; ++i) {
      p[12 + 30 * b + 2 * i] = o[b][i].re;
      p[13 + 30 * b + 2 * i] = o[b][i].im;
    }
  }
  logdet[s] = ld;
  nneg[s] = nn;
}

}  // namespace

int clover_build(const int dims[4], const double* canon_links, const CloverCoeffs& cc, double* clov, double* inv,
                 double* sums, int sums_stride, int inv_parity, cudaStream_t s) {
  Dims D{{dims[0], dims[1], dims[2], dims[3]}};
  long V = (long)dims[0] * dims[1] * dims[2] * dims[3];
  const int nb = (int)((V + kBuildSites - 1) / kBuildSites);
  clover_build_kernel<<<nb, 6 * kBuildSites, 0, s>>>(D, reinterpret_cast<const double2*>(canon_links), cc, clov, inv,
                                                   inv_parity, V, sums, sums_stride);
  return nb;
}

// inv = A^-1 on the sites of parity `parity` (clov on all sites, canonical site order)
__global__ void clover_invert_parity_kernel(Dims D, const double* clov, double* inv, int parity, long V) {
  const long s = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (s >= V) return;
  long r = s;
  int sum = 0;
  for (int k = 0; k < 4; ++k) {
    sum += (int)(r % D.L[k]);
    r /= D.L[k];
  }
  if ((sum & 1) != parity) return;
  const double* p = clov + s * 72;
  double* q = inv + s * 72;
  double d[2][6];
  cplx<double> o[2][15];
  for (int b = 0; b < 2; ++b) {
    for (int i = 0; i < 6; ++i) d[b][i] = p[6 * b + i];
    for (int i = 0; i < 15; ++i) o[b][i] = {p[12 + 30 * b + 2 * i], p[13 + 30 * b + 2 * i]};
  }
  double ld = 0.0;
  int nn = 0;
  for (int b = 0; b < 2; ++b) ldl_invert_block(d[b], o[b], ld, nn);
  for (int b = 0; b < 2; ++b) {
    for (int i = 0; i < 6; ++i) q[6 * b + i] = d[b][i];
    for (int i = 0; i < 15; ++i) {
      q[12 + 30 * b + 2 * i] = o[b][i].re;
      q[13 + 30 * b + 2 * i] = o[b][i].im;
    }
  }
}

void clover_invert(long nsites, double* packed, double* logdet, int* nneg, cudaStream_t s) {
  clover_invert_kernel<<<(unsigned)((nsites + 63) / 64), 64, 0, s>>>(nsites, packed, logdet, nneg);
}

void clover_invert_parity(const int dims[4], const double* clov, double* inv, int parity, cudaStream_t s) {
  Dims D{{dims[0], dims[1], dims[2], dims[3]}};
  long V = (long)dims[0] * dims[1] * dims[2] * dims[3];
  clover_invert_parity_kernel<<<(unsigned)((V + 63) / 64), 64, 0, s>>>(D, clov, inv, parity, V);
}

}  // namespace gbc
