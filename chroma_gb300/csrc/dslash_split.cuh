// FP64 hopping term with fused clover epilogues, the 8 hops of a site split over 8 threads.
//
// What bounds it: the FP64 pipe.  GB300 retires about two FP64 lane operations per SM and clock, so
// a 32-site tile of A_ee^-1 D_eo (1136 FP64 instructions per site) keeps one SM busy for about 9 us
// however many warps it has, and a lattice is fast only when its sites are spread evenly over all
// 152 SMs.  One thread per site in blocks of 128 (hop_kernel) leaves a 4096-site checkerboard on 32
// SMs; splitting the hops makes blocks of 8 to 32 sites that still have 2 to 8 warps.
//
// Thread (s, q) of a block of S sites: hop q of site s (projection and colour product, written to
// shared memory), then three of the site's 24 real output components (the sum over the hops and its
// row of the clover block).  The hop's direction only selects data (which spins, which link element,
// which signs), so the lanes of a warp may hold different hops.  Every component is summed in the
// order of hop_kernel's scalar FP64 code.
#pragma once
#include "gbc_device.cuh"

namespace gbc {

// Field access of the context's fields (planes, dslash.cuh); noalloc.cu has the canonical one.
struct SplitPlanes {
  const HopArgs& a;
  int rhs;
  __device__ __forceinline__ const Geom& geom() const { return a.g; }
  __device__ __forceinline__ int parity() const { return a.out_parity; }
  __device__ __forceinline__ double2 in(const Coord& n, int ni, int k) const {
    (void)n;
    return ldw(reinterpret_cast<const double2*>((const char*)a.in + (size_t)rhs * a.in_rhs_bytes) +
               (size_t)k * a.g.stride + ni);
  }
  // element e of U_mu(x) (fwd) or U_mu(x - mu)
  __device__ __forceinline__ double2 link(const Coord& c, int idx, const Coord& n, int ni, int mu, bool fwd, int e) const {
    (void)c;
    (void)n;
    const void* p = fwd ? a.gauge_fwd[mu] : a.gauge_bwd[mu];
    return ldg(reinterpret_cast<const double2*>(p) + (size_t)e * a.g.stride + (fwd ? idx : ni));
  }
  __device__ __forceinline__ double diag(const Coord&, int idx, int b, int i) const {
    const double* p = reinterpret_cast<const double*>(a.clov);
    return ldg(p + 2 * ((size_t)(18 * b + (i >> 1)) * a.g.stride + idx) + (i & 1));
  }
  __device__ __forceinline__ double2 offd(const Coord&, int idx, int b, int k) const {
    return ldg(reinterpret_cast<const double2*>(a.clov) + (size_t)(18 * b + 3 + k) * a.g.stride + idx);
  }
  __device__ __forceinline__ double2 self(const Coord&, int idx, int k) const {
    return ldw(reinterpret_cast<const double2*>((const char*)a.self + (size_t)rhs * a.self_rhs_bytes) +
               (size_t)k * a.g.stride + idx);
  }
  __device__ __forceinline__ double2 aux(int idx, int k) const {  // an FP32 field, two complex per plane
    const float2 v = ldw(reinterpret_cast<const float2*>((const char*)a.aux + (size_t)rhs * a.aux_rhs_bytes) +
                         2 * ((size_t)(k >> 1) * a.g.stride + idx) + (k & 1));
    return make_double2(v.x, v.y);
  }
  __device__ __forceinline__ void out(const Coord&, int idx, int k, int im, double v) const {
    reinterpret_cast<double*>((char*)a.out + (size_t)rhs * a.out_rhs_bytes)[2 * ((size_t)k * a.g.stride + idx) + im] = v;
  }
};

// -v if neg, on the integer side: a negation that no instruction can absorb as an operand modifier
// is an FP64 instruction (45 of them per thread made the kernel 1.4 times slower)
__device__ __forceinline__ double flip_if(bool neg, double v) {
  return __hiloint2double(__double2hiint(v) ^ (neg ? (int)0x80000000 : 0), __double2loint(v));
}

// The three real components (spin * 3 + colour, re/im) r = 3 q .. 3 q + 2 of the output at the
// block's site s; sum[] receives this thread's part of the REDUCE sums.
template <class A, int MODE, bool DAG, int REDUCE, int S>
__device__ __forceinline__ void split_site(const A& f, double coef, double twist, int sblock, double (&sum)[3]) {
  __shared__ double2 uh[8][6][S];
  constexpr bool kClovOfHop = MODE == HOP_CLOV || MODE == HOP_SYM;  // the clover block acts on the hops' sum
  __shared__ double xs[kClovOfHop ? 24 : 1][S];
  const int s = threadIdx.x % S, q = threadIdx.x / S;
  const auto& g = f.geom();
  const int idx = sblock * S + s;
  const bool valid = idx < g.Vh;
  Coord c{};
  if (valid) {
    c = cb_coords(g, idx, f.parity());
    const int mu = q >> 1;
    const bool fwd = (q & 1) == 0;
    const bool neg = fwd ? !DAG : DAG;  // s = -1: forward (1 - isign gamma), backward (1 + isign gamma)
    Coord n = c;
#pragma unroll
    for (int d = 0; d < 4; ++d)
      if (mu == d) n.x[d] = fwd ? (c.x[d] + 1 == g.L[d] ? 0 : c.x[d] + 1) : (c.x[d] == 0 ? g.L[d] - 1 : c.x[d] - 1);
    const int ni = cb_index(g, n);
    double2 p[12], u[9];
#pragma unroll
    for (int k = 0; k < 12; ++k) p[k] = f.in(n, ni, k);
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        u[3 * r + k] = f.link(c, idx, n, ni, mu, fwd, fwd ? 3 * r + k : 3 * k + r);
        u[3 * r + k].y = flip_if(!fwd, u[3 * r + k].y);
      }
    // h = p_top + s A p_bot: the lower spin each upper spin takes, times i (mu = 0, 2) and a sign
    cplx<double> h[2][3];
    const bool swap = mu < 2;       // upper spin 0 takes spin 3 (and 1 takes 2), else 0 takes 2
    const bool times_i = !(mu & 1);
    const bool neg0 = neg != (mu == 1), neg1 = neg != (mu == 2);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const double2 b0 = swap ? p[9 + k] : p[6 + k], b1 = swap ? p[6 + k] : p[9 + k];
      h[0][k] = {p[k].x + flip_if(neg0 != times_i, times_i ? b0.y : b0.x), p[k].y + flip_if(neg0, times_i ? b0.x : b0.y)};
      h[1][k] = {p[3 + k].x + flip_if(neg1 != times_i, times_i ? b1.y : b1.x),
                 p[3 + k].y + flip_if(neg1, times_i ? b1.x : b1.y)};
    }
#pragma unroll
    for (int t = 0; t < 2; ++t)
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        cplx<double> v = {0.0, 0.0};
#pragma unroll
        for (int k = 0; k < 3; ++k) cmac(v, cplx<double>{u[3 * r + k].x, u[3 * r + k].y}, h[t][k]);
        uh[q][3 * t + r][s] = make_double2(v.re, v.im);
      }
  }
  __syncthreads();
  double acc[3];
  if (valid) {
#pragma unroll
    for (int t = 0; t < 3; ++t) {
      const int r = 3 * q + t, im = r & 1, spin = r / 6, col = (r >> 1) - 3 * spin;
      double v;
#pragma unroll
      for (int hp = 0; hp < 8; ++hp) {
        const int mu = hp >> 1;
        const bool neg = (hp & 1) == 0 ? !DAG : DAG;
        // upper spins: uh itself; lower: s B uh (the tables of reconstruct<>)
        bool hi = spin & 1, cross = false, minus = false;
        if (spin >= 2) {
          hi = (spin == 2) == (mu < 2);
          cross = !(mu & 1);  // times -i, or +i for (mu = 2, spin 3)
          minus = mu == 1 ? spin == 3 : cross ? ((im != 0) != (mu == 2 && spin == 3)) : false;
          minus = minus != neg;
        }
        const double2 w = uh[hp][3 * (hi ? 1 : 0) + col][s];
        const double x = flip_if(minus, (im != 0) != cross ? w.y : w.x);
        v = hp == 0 ? x : v + x;
      }
      acc[t] = v;
      if (kClovOfHop) xs[r][s] = coef == 1.0 ? v : coef * v;
    }
  }
  double2 x[6];
  const int b = q >> 2;  // chirality block of this thread's components
  if (MODE == HOP_XPAY && valid) {
#pragma unroll
    for (int j = 0; j < 6; ++j) x[j] = f.self(c, idx, 6 * b + j);
  }
  // xs is complete; and a caller's out may be self: the site's threads have read it before any writes
  if (MODE != HOP_PLAIN) __syncthreads();
  if (!valid) return;
  if (kClovOfHop) {
#pragma unroll
    for (int j = 0; j < 6; ++j) x[j] = make_double2(xs[12 * b + 2 * j][s], xs[12 * b + 2 * j + 1][s]);
  }
#pragma unroll
  for (int t = 0; t < 3; ++t) {
    const int r = 3 * q + t, im = r & 1, k = r >> 1, i = k - 6 * b;
    double v, sr = 0.0, sx = 0.0;  // sr: the same real component of self, sx: the other one
    if (MODE == HOP_PLAIN) {
      v = coef * acc[t];
    } else {
      double2 xi = x[0];
#pragma unroll
      for (int j = 1; j < 6; ++j)
        if (i == j) xi = x[j];
      sr = im ? xi.y : xi.x;
      sx = im ? xi.x : xi.y;
      v = f.diag(c, idx, b, i) * sr;
#pragma unroll
      for (int j = 0; j < 6; ++j) {
        if (j == i) continue;
        const bool low = j < i;
        const double2 o = f.offd(c, idx, b, low ? i * (i - 1) / 2 + j : j * (j - 1) / 2 + i);
        v = fmadd(o.x, im ? x[j].y : x[j].x, v);
        v = fmadd(flip_if(low != (im != 0), o.y), im ? x[j].x : x[j].y, v);
      }
      if (MODE == HOP_SYM) {
        const double2 xk = f.self(c, idx, k);
        sr = im ? xk.y : xk.x;
        sx = im ? xk.x : xk.y;
        v = sr - v;
      }
      if (MODE == HOP_XPAY) v = fmadd(coef, acc[t], v);
      if (MODE == HOP_XPAY || MODE == HOP_SYM) {
        // + isign i mu gamma_5 self, gamma_5 = diag(1, 1, -1, -1)
        if (twist != 0.0) v += flip_if((im == 0) != (b != 0), DAG ? -twist : twist) * sx;
      }
    }
    f.out(c, idx, k, im, v);
    if constexpr (REDUCE == RED_NORM) sum[0] = fmadd(v, v, sum[0]);
    if constexpr (REDUCE == RED_DOT_SELF) {  // (out, self), |out|^2
      sum[0] = fmadd(v, sr, sum[0]);
      sum[1] = fmadd(flip_if(im != 0, v), sx, sum[1]);
      sum[2] = fmadd(v, v, sum[2]);
    }
    if constexpr (REDUCE == RED_DOT_AUX) {  // (aux, out)
      const double2 ax = f.aux(idx, k);
      sum[0] = fmadd(im ? ax.y : ax.x, v, sum[0]);
      sum[1] = fmadd(flip_if(im == 0, im ? ax.x : ax.y), v, sum[1]);
    }
  }
}

}  // namespace gbc
