// The end of a reduction inside the kernel that produced its partial sums: the last block of a
// right-hand side to arrive sums that side's partials (fixed order: bitwise repeatable) and applies
// the solver's scalar step to them.  A reduction that ends in launches of its own (one to sum, one for
// the scalars) costs two launches of some 2 us each in an iteration whose kernels take 5 to 15 us on
// lattices of up to 16^3 x 32; see finish_in_kernel() for where the line lies.
#pragma once
#include "../../include/gbclover.h"
#include "gbc_device.cuh"

namespace gbc {

__device__ __forceinline__ double2 cdiv(double2 a, double2 b) {
  const double d = b.x * b.x + b.y * b.y;
  return make_double2((a.x * b.x + a.y * b.y) / d, (a.y * b.x - a.x * b.y) / d);
}
__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// The scalar step of right-hand side r on its sums v.
// InvCG2 (invcg2.cc:153-221): alpha after |M p|^2 (or p^dag A p), beta after |r|^2; a converged right-hand
// side gets alpha = beta = 0.
__device__ inline void scalar_step(const Finish& f, int r, const double* v) {
  if (f.kind == FIN_CG_ALPHA) {
    CGScalars s = static_cast<CGScalars*>(f.sc)[r];
    s.d = v[0];
    s.a = (s.active && s.d > 0.0) ? s.c / s.d : 0.0;
    f.coef[r] = s.a;
    static_cast<CGScalars*>(f.sc)[r] = s;
  } else if (f.kind == FIN_CG_BETA) {
    CGScalars s = static_cast<CGScalars*>(f.sc)[r];
    if (s.active) {
      s.cp = v[0];
      s.iters += 1;
      if (!(s.cp > s.rsd_sq)) s.active = 0;  // converged (or non-finite: stops and is reported)
      s.b = (s.active && s.c > 0.0) ? s.cp / s.c : 0.0;
      s.c_prev = s.c;
      s.c = s.cp;
    } else {
      s.b = 0.0;
    }
    f.coef[r] = s.b;
    static_cast<CGScalars*>(f.sc)[r] = s;
  } else if (f.kind == FIN_BI_ALPHA) {  // alpha = rho / (r0, v)
    BiScal q = static_cast<BiScal*>(f.sc)[r];
    q.alpha = make_double2(0.0, 0.0);
    if (q.active) {
      const double2 d = make_double2(v[0], v[1]);
      if (d.x * d.x + d.y * d.y > 0.0 && isfinite(d.x) && isfinite(d.y)) {
        q.alpha = cdiv(q.rho, d);
      } else {
        q.active = 0;
        q.status = GBC_ERR_BREAKDOWN;
      }
    }
    static_cast<BiScal*>(f.sc)[r] = q;
  } else if (f.kind == FIN_BI_OMEGA) {  // omega = (t, s) / (t, t)
    BiScal q = static_cast<BiScal*>(f.sc)[r];
    const double tt = v[2];
    q.omega = (q.active && tt > 0.0) ? make_double2(v[0] / tt, v[1] / tt) : make_double2(0.0, 0.0);
    static_cast<BiScal*>(f.sc)[r] = q;
  } else if (f.kind == FIN_BI_BETA) {  // |r|^2, rho' = (r0, r); beta = (rho' / rho)(alpha / omega)
    BiScal q = static_cast<BiScal*>(f.sc)[r];
    q.beta = make_double2(0.0, 0.0);
    if (q.active) {
      q.iters += 1;
      q.rr = v[0];
      const double2 rho1 = make_double2(v[1], v[2]);
      if (!isfinite(q.rr)) {
        q.active = 0;
        q.status = GBC_ERR_NONFINITE;
      } else if (!(q.rr > q.rsd_sq)) {
        q.active = 0;  // converged
      } else if (q.omega.x == 0.0 && q.omega.y == 0.0) {
        q.active = 0;
        q.status = GBC_ERR_BREAKDOWN;
      } else {
        q.beta = cmul(cdiv(rho1, q.rho), cdiv(q.alpha, q.omega));
      }
      q.rho = rho1;
    }
    static_cast<BiScal*>(f.sc)[r] = q;
  }
}

// Sums of the NQ partial rows of right-hand side r by a block of NT threads, then the scalar step
template <int NQ, int NT>
__device__ __forceinline__ void sum_partials(const Finish& f, const double* partials, int part_stride, int nrhs, int r,
                                             int nblk) {
  __shared__ double fs[NQ][NT / 32];
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    const double* p = partials + ((size_t)q * nrhs + r) * part_stride;
    double s = 0.0;
#pragma unroll 8
    for (int i = threadIdx.x; i < nblk; i += NT) s += __ldcg(p + i);  // written by other SMs: from L2
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
    if ((threadIdx.x & 31) == 0) fs[q][threadIdx.x >> 5] = s;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double v[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
#pragma unroll
      for (int w = 0; w < NT / 32; ++w) v[q] += fs[q][w];
      f.result[q * nrhs + r] = v[q];
    }
    scalar_step(f, r, v);
  }
}

// Called by every thread of a block after threads of its first warp wrote the block's partials of
// right-hand side r; nblk blocks of that right-hand side take part.  Nobody waits: the block that finds
// every other one counted is the last.  It leaves the counter at zero for the next launch on the
// stream.  Only the first warp fences: a fence waits for all of its thread's stores, and the block's
// field stores need not be ordered before its arrival.
template <int NQ, int NT>
__device__ __forceinline__ void finish_reduction(const Finish& f, const double* partials, int part_stride, int nrhs,
                                                 int r, int nblk) {
  if (f.kind == FIN_NONE) return;
  __shared__ bool last;
  if (threadIdx.x < 32) __threadfence();  // this block's partials before its arrival
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(&f.count[r], 1u) == (unsigned)(nblk - 1);
  __syncthreads();
  if (!last) return;
  __threadfence();  // the other blocks' arrivals before their partials
  sum_partials<NQ, NT>(f, partials, part_stride, nrhs, r, nblk);
  if (threadIdx.x == 0) f.count[r] = 0;
}

}  // namespace gbc
