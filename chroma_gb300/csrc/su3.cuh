// FP64 3x3 complex matrices for the setup kernels (clover term, stout): products accumulate into their
// sum, so a chain of them costs no separate additions (GB300's FP64 pipe is what bounds these kernels).
#pragma once
#include <cuda_runtime.h>

namespace gbc {

struct M {
  double2 a[9];
};

// r += x y
__device__ __forceinline__ void mac(double2& r, double2 x, double2 y) {
  r.x = fma(x.x, y.x, r.x);
  r.x = fma(-x.y, y.y, r.x);
  r.y = fma(x.x, y.y, r.y);
  r.y = fma(x.y, y.x, r.y);
}
template <bool NEG>
__device__ __forceinline__ double2 sgn(double2 x) { return NEG ? make_double2(-x.x, -x.y) : x; }
__device__ __forceinline__ double2 cj(double2 x) { return make_double2(x.x, -x.y); }

// r += X Y (NEG: r -= X Y) with X = x or x^dag, Y = y or y^dag
template <bool XD, bool YD, bool NEG = false>
__device__ __forceinline__ void mmac(M& r, const M& x, const M& y) {
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
      for (int k = 0; k < 3; ++k)
        mac(r.a[3 * i + j], sgn<NEG>(XD ? cj(x.a[3 * k + i]) : x.a[3 * i + k]),
            YD ? cj(y.a[3 * j + k]) : y.a[3 * k + j]);
}
__device__ __forceinline__ M mzero() {
  M r;
#pragma unroll
  for (int k = 0; k < 9; ++k) r.a[k] = make_double2(0.0, 0.0);
  return r;
}
__device__ __forceinline__ M ld(const double2* u, long site, int mu) {
  M r;
  const double2* p = u + (site * 4 + mu) * 9;
#pragma unroll
  for (int k = 0; k < 9; ++k) r.a[k] = __ldg(p + k);
  return r;
}

// steps from canonical site s to its neighbours: s + up[k], s + dn[k]
struct Steps {
  long up[4], dn[4];
};
__device__ __forceinline__ Steps steps(const int (&L)[4], long s, int (&x)[4]) {
  Steps st;
  long stride = 1;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    x[k] = (int)(s % L[k]);
    s /= L[k];
    st.up[k] = x[k] + 1 == L[k] ? -stride * (L[k] - 1) : stride;
    st.dn[k] = x[k] == 0 ? stride * (L[k] - 1) : -stride;
    stride *= L[k];
  }
  return st;
}
__device__ __forceinline__ long pick(const long (&v)[4], int k) {
  return k == 0 ? v[0] : k == 1 ? v[1] : k == 2 ? v[2] : v[3];
}

}  // namespace gbc
