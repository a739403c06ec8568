// Stout smearing of the gauge field on the device, FP64 (setup of smeared-link actions).
//
//   C_mu(x) = rho sum_{nu != mu, smeared} [ U_nu(x) U_mu(x+nu) U_nu^dag(x+mu)
//                                          + U_nu^dag(x-nu) U_mu(x-nu) U_nu(x-nu+mu) ]
//   Omega = C U^dag,  Q = (i/2) (Omega^dag - Omega) - (i/6) tr(Omega^dag - Omega),
//   U'_mu(x) = exp(i Q) U_mu(x)
// (Chroma lib/util/gauge/stout_utils.cc:105-180 getQsandCs, :936-966 smear_links), with exp(iQ) =
// f0 + f1 Q + f2 Q^2 by Cayley-Hamilton (Q^3 = c1 Q + c0, c0 = det Q, c1 = tr(Q^2)/2): the closed
// form of Morningstar & Peardon, PRD 69 (2004) 054501 (stout_utils.cc:415-700) for c1 >= 0.75, and
// below it the Taylor series with every power of Q reduced to the same three coefficients.
//
// One thread per link (site, mu) of the canonical layout [V][4][3][3] complex: a block is 32
// consecutive sites, one warp per mu, so the loop over nu does not diverge; the staples read their
// links through L1/L2 (each link is read by up to 18 staples).  Links of directions that are not
// smeared are copied.
// What bounds it: the FP64 pipe (about two lane operations per SM and clock), with 1296 FP64
// instructions per link in the staples and about 480 in the rest.  So each staple's second product
// accumulates into the sum, Q and Q^2 are kept as the 3 real and 3 complex numbers of a Hermitian
// matrix, and the Taylor coefficients are scalar recursions (8 instructions a term).
#include <cuda_runtime.h>

#include <string>

#include "ctx.h"
#include "hostmem.h"
#include "su3.cuh"

namespace gbc {
namespace {

// Hermitian 3x3: diagonal d, upper off-diagonals o[0] = 01, o[1] = 02, o[2] = 12
struct Herm {
  double d[3];
  double2 o[3];
};

// terms FIRST .. LAST of sum_n (i Q)^n / n! as f0 + f1 Q + f2 Q^2; (a, b, c) is Q^n / n! on entry of
// term n + 1
template <int FIRST, int LAST>
__device__ __forceinline__ void taylor(double& a, double& b, double& c, double c0, double c1, double2 (&f)[3]) {
#pragma unroll
  for (int n = FIRST; n <= LAST; ++n) {
    const double inv = 1.0 / n;
    const double an = c * c0 * inv, bn = fma(c, c1, a) * inv;
    c = b * inv;
    a = an;
    b = bn;
    const double v[3] = {a, b, c};
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      if (n % 4 == 0) f[q].x += v[q];
      if (n % 4 == 1) f[q].y += v[q];
      if (n % 4 == 2) f[q].x -= v[q];
      if (n % 4 == 3) f[q].y -= v[q];
    }
  }
}

// f of exp(iQ) = f0 + f1 Q + f2 Q^2 for traceless Hermitian Q with c0 = det Q, c1 = tr(Q^2) / 2
__device__ __forceinline__ void exp_coef(double c0, double c1, double2 (&f)[3]) {
  // the eigenvalues of Q are at most 2 sqrt(c1 / 3): 0.26 for c1 = 0.05, where the 13th term is
  // below 4e-18, and 1 for c1 = 0.75, where the 21st is below 2e-20
  if (c1 < 0.75) {
    double a = 1.0, b = 0.0, c = 0.0;
    f[0] = make_double2(1.0, 0.0);
    f[1] = f[2] = make_double2(0.0, 0.0);
    taylor<1, 12>(a, b, c, c0, c1, f);
    if (!(c1 < 0.05)) taylor<13, 20>(a, b, c, c0, c1, f);
    return;
  }
  const bool neg = c0 < 0;
  const double c0a = fabs(c0);
  const double c0max = 2.0 * (c1 / 3.0) * sqrt(c1 / 3.0);
  const double theta = acos(fmin(1.0, c0a / c0max));
  const double u = sqrt(c1 / 3.0) * cos(theta / 3.0);
  const double w = sqrt(c1) * sin(theta / 3.0);
  const double u2 = u * u, w2 = w * w;
  const double xi0 = fabs(w) < 0.05 ? 1.0 - w2 / 6.0 * (1.0 - w2 / 20.0 * (1.0 - w2 / 42.0)) : sin(w) / w;
  const double cw = cos(w);
  double s2u, c2u, su, cu;
  sincos(2.0 * u, &s2u, &c2u);
  sincos(u, &su, &cu);
  const double2 e2iu = make_double2(c2u, s2u), emiu = make_double2(cu, -su);
  auto cm = [](double2 x, double2 y) { return make_double2(x.x * y.x - x.y * y.y, x.x * y.y + x.y * y.x); };
  // h0 = (u2 - w2) e2iu + emiu (8 u2 cw + 2i u (3u2 + w2) xi0)
  const double2 t0 = cm(emiu, make_double2(8.0 * u2 * cw, 2.0 * u * (3.0 * u2 + w2) * xi0));
  const double2 h0 = make_double2((u2 - w2) * e2iu.x + t0.x, (u2 - w2) * e2iu.y + t0.y);
  // h1 = 2u e2iu - emiu (2u cw - i (3u2 - w2) xi0)
  const double2 t1 = cm(emiu, make_double2(2.0 * u * cw, -(3.0 * u2 - w2) * xi0));
  const double2 h1 = make_double2(2.0 * u * e2iu.x - t1.x, 2.0 * u * e2iu.y - t1.y);
  // h2 = e2iu - emiu (cw + 3i u xi0)
  const double2 t2 = cm(emiu, make_double2(cw, 3.0 * u * xi0));
  const double2 h2 = make_double2(e2iu.x - t2.x, e2iu.y - t2.y);
  const double den = 1.0 / (9.0 * u2 - w2);
  f[0] = make_double2(h0.x * den, h0.y * den);
  f[1] = make_double2(h1.x * den, h1.y * den);
  f[2] = make_double2(h2.x * den, h2.y * den);
  if (neg) {
    f[0].y = -f[0].y;
    f[1].x = -f[1].x;
    f[2].y = -f[2].y;
  }
}

// f1 q + f2 s
__device__ __forceinline__ double2 lin(double2 f1, double2 q, double2 f2, double2 s) {
  double2 r = make_double2(0.0, 0.0);
  mac(r, f1, q);
  mac(r, f2, s);
  return r;
}

// exp(iQ) for traceless Hermitian Q
__device__ __forceinline__ M exp_iQ(const Herm& q) {
  const double n01 = fma(q.o[0].x, q.o[0].x, q.o[0].y * q.o[0].y);
  const double n02 = fma(q.o[1].x, q.o[1].x, q.o[1].y * q.o[1].y);
  const double n12 = fma(q.o[2].x, q.o[2].x, q.o[2].y * q.o[2].y);
  Herm s;  // Q^2
  s.d[0] = fma(q.d[0], q.d[0], n01 + n02);
  s.d[1] = fma(q.d[1], q.d[1], n01 + n12);
  s.d[2] = fma(q.d[2], q.d[2], n02 + n12);
  const double t01 = q.d[0] + q.d[1], t02 = q.d[0] + q.d[2], t12 = q.d[1] + q.d[2];
  s.o[0] = make_double2(t01 * q.o[0].x, t01 * q.o[0].y);
  s.o[1] = make_double2(t02 * q.o[1].x, t02 * q.o[1].y);
  s.o[2] = make_double2(t12 * q.o[2].x, t12 * q.o[2].y);
  mac(s.o[0], q.o[1], cj(q.o[2]));
  double2 p = make_double2(0.0, 0.0);  // q01 q12
  mac(p, q.o[0], q.o[2]);
  s.o[1].x += p.x;
  s.o[1].y += p.y;
  mac(s.o[2], cj(q.o[0]), q.o[1]);
  const double c1 = 0.5 * (s.d[0] + s.d[1] + s.d[2]);
  // det Q = d0 d1 d2 + 2 Re(q01 q12 conj(q02)) - d0 |q12|^2 - d1 |q02|^2 - d2 |q01|^2
  double c0 = 2.0 * fma(p.x, q.o[1].x, p.y * q.o[1].y);
  c0 = fma(q.d[0], fma(q.d[1], q.d[2], -n12), c0);
  c0 = fma(-q.d[1], n02, c0);
  c0 = fma(-q.d[2], n01, c0);
  double2 f[3];
  exp_coef(c0, c1, f);
  M r;
#pragma unroll
  for (int i = 0; i < 3; ++i)
    r.a[4 * i] = make_double2(fma(f[2].x, s.d[i], fma(f[1].x, q.d[i], f[0].x)), fma(f[2].y, s.d[i], fma(f[1].y, q.d[i], f[0].y)));
  r.a[1] = lin(f[1], q.o[0], f[2], s.o[0]);
  r.a[2] = lin(f[1], q.o[1], f[2], s.o[1]);
  r.a[5] = lin(f[1], q.o[2], f[2], s.o[2]);
  r.a[3] = lin(f[1], cj(q.o[0]), f[2], cj(s.o[0]));
  r.a[6] = lin(f[1], cj(q.o[1]), f[2], cj(s.o[1]));
  r.a[7] = lin(f[1], cj(q.o[2]), f[2], cj(s.o[2]));
  return r;
}

struct Lat {
  int L[4];
  long V;
};

__global__ void __launch_bounds__(128) stout_kernel(Lat g, const double2* __restrict__ cur, double2* __restrict__ nxt,
                                                    double rho, int4 dirs) {
  const long s = (long)blockIdx.x * 32 + (threadIdx.x & 31);
  const int mu = threadIdx.x >> 5;
  if (s >= g.V) return;
  const int on[4] = {dirs.x, dirs.y, dirs.z, dirs.w};
  M out;
  if (!on[mu]) {
    out = ld(cur, s, mu);
  } else {
    int x[4];
    const Steps n = steps(g.L, s, x);
    const long up_mu = pick(n.up, mu);
    M C = mzero();
#pragma unroll 1
    for (int nu = 0; nu < 4; ++nu) {
      if (nu == mu || !on[nu]) continue;
      const long un = pick(n.up, nu), dnn = pick(n.dn, nu);
      // a step in nu leaves the mu coordinate alone: x - nu + mu is s + dnn + up_mu
      M t = mzero();
      mmac<false, false>(t, ld(cur, s, nu), ld(cur, s + un, mu));
      mmac<false, true>(C, t, ld(cur, s + up_mu, nu));
      t = mzero();
      mmac<true, false>(t, ld(cur, s + dnn, nu), ld(cur, s + dnn, mu));
      mmac<false, false>(C, t, ld(cur, s + dnn + up_mu, nu));
    }
    const M U = ld(cur, s, mu);
    M Om = mzero();
    mmac<false, true>(Om, C, U);
    // Q = (i/2)(Omega^dag - Omega - trace / 3): real diagonal Im Omega_ii - mean, and
    // Q_ij = (Im Omega_ij + Im Omega_ji, Re Omega_ji - Re Omega_ij) / 2
    Herm Q;
    const double mean = (Om.a[0].y + Om.a[4].y + Om.a[8].y) / 3.0, h = 0.5 * rho;
#pragma unroll
    for (int i = 0; i < 3; ++i) Q.d[i] = rho * (Om.a[4 * i].y - mean);
    Q.o[0] = make_double2(h * (Om.a[1].y + Om.a[3].y), h * (Om.a[3].x - Om.a[1].x));
    Q.o[1] = make_double2(h * (Om.a[2].y + Om.a[6].y), h * (Om.a[6].x - Om.a[2].x));
    Q.o[2] = make_double2(h * (Om.a[5].y + Om.a[7].y), h * (Om.a[7].x - Om.a[5].x));
    out = mzero();
    mmac<false, false>(out, exp_iQ(Q), U);
  }
  double2* p = nxt + (s * 4 + mu) * 9;
#pragma unroll
  for (int k = 0; k < 9; ++k) p[k] = out.a[k];
}

}  // namespace
}  // namespace gbc

using namespace gbc;

extern "C" int gbc_stout_smear(const gbc_geom* geom, int n_steps, double rho, const int smear_dirs[4],
                               const double* links_in, double* links_out) {
  if (!geom || !links_in || !links_out || n_steps < 0) return GBC_ERR_ARGS;
  Lat g;
  g.V = 1;
  for (int k = 0; k < 4; ++k) {
    if (geom->dims[k] < 2) return GBC_ERR_ARGS;
    g.L[k] = geom->dims[k];
    g.V *= geom->dims[k];
  }
  const int all[4] = {1, 1, 1, 1};
  const int* d = smear_dirs ? smear_dirs : all;
  const int4 dirs = make_int4(d[0] != 0, d[1] != 0, d[2] != 0, d[3] != 0);
  const size_t bytes = sizeof(double) * 72 * (size_t)g.V;
  double2* buf[2] = {nullptr, nullptr};
  cudaStream_t s = nullptr;
  int rc = GBC_OK;
  PageTouch touch;
  if (cudaMalloc(&buf[0], bytes) != cudaSuccess || cudaMalloc(&buf[1], bytes) != cudaSuccess ||
      cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) != cudaSuccess) {
    rc = GBC_ERR_CUDA;
    (void)cudaGetLastError();  // reported here: the thread's next call must not find it
  } else {
    try {
      touch.populate({{links_out, bytes}}, nullptr, PageTouch::kThreads);
    } catch (...) {  // no host memory for the helpers: the copy meets the page faults itself
    }
    cudaMemcpyAsync(buf[0], links_in, bytes, cudaMemcpyHostToDevice, s);
    for (int i = 0; i < n_steps; ++i) {
      stout_kernel<<<(unsigned)((g.V + 31) / 32), 128, 0, s>>>(g, buf[i & 1], buf[(i + 1) & 1], rho, dirs);
      count_launch();
    }
    touch.join();
    cudaMemcpyAsync(links_out, buf[n_steps & 1], bytes, cudaMemcpyDeviceToHost, s);
    if (cudaStreamSynchronize(s) != cudaSuccess || cudaGetLastError() != cudaSuccess) rc = GBC_ERR_CUDA;
  }
  if (buf[0]) cudaFree(buf[0]);
  if (buf[1]) cudaFree(buf[1]);
  if (s) cudaStreamDestroy(s);
  return rc;
}
