// Multi-shift CG on the normal equations, (M~^dag M~ + sigma_s) psi_s = chi for every shift at
// once: the RHMC solver behind Chroma's MdagMMultiSysSolverCG (multi_syssolver_mdagm_cg.h:58-80)
// -> MInvCG2 (minvcg2.cc:70-357), Jegerlehner's recursion (hep-lat/9708029).  With a sloppy
// precision (HALF or SINGLE) the recursion runs in FP32 and each shift is then refined by an FP64
// defect correction whose corrections come from CG on the shifted system in the sloppy operator,
// Chroma's multiprec pattern (a single-precision MInvCG2 followed by per-shift refinement).  One Krylov space of
// the unshifted M~^dag M~ is built; each shifted solution follows from the ratios zeta_s of its
// residual to the unshifted one, so an iteration costs one M~^dag M~ plus one fused update of all
// shifted search vectors and one of all solutions.  Fields and sums in FP64, the scalar recursion
// on the host (two reductions per iteration).  The recursion, its sign conventions and its
// convergence test (|r| zeta_s <= RsdCG_s |chi|) are the reference's, so iteration counts agree.
#include <algorithm>
#include <cmath>
#include <string>
#include <cstring>
#include <vector>

#include "ctx.h"
#include "hostmem.h"
#include "launch.cuh"

namespace gbc {
namespace {

enum { MS_CHI = 700, MS_R, MS_MP, MS_MMP, MS_TE, MS_P, MS_X, MS_T1, MS_T2 };

// the first finalized sum of red(c) -> host (synchronises)
double fetch(gbc_ctx* c) {
  GBC_CUDA(cudaMemcpyAsync(c->h_result, c->d_result, sizeof(double), cudaMemcpyDeviceToHost, c->stream));
  sync(c);
  return c->h_result[0];
}
double norm2(gbc_ctx* c, const Spinor& x) {
  blas_norm2(c->g, x, red(c), c->stream);
  return fetch(c);
}

// every right-hand-side index of the view reads the same field x
Spinor broadcast(const Spinor& x, int n) {
  Spinor t = x;
  t.nrhs = n;
  t.rhs_bytes = 0;
  t.norm_rhs_stride = 0;
  return t;
}

struct Coefs {
  std::vector<double2> h;  // [2][n]
  double2* d = nullptr;
  int n = 0;
  explicit Coefs(int n_) : h(2 * (size_t)n_), n(n_) { GBC_CUDA(cudaMalloc(&d, sizeof(double2) * 2 * n_)); }
  ~Coefs() {
    if (d) cudaFree(d);
  }
  // upload a[s], b[s] and run y_s = a_s x_s + b_s y_s (then wait, the host vector is reused)
  void axpby(gbc_ctx* c, const Spinor& x, const Spinor& y) {
    GBC_CUDA(cudaMemcpyAsync(d, h.data(), sizeof(double2) * 2 * n, cudaMemcpyHostToDevice, c->stream));
    blas_axpby(c->g, d, x, d + n, y, c->stream);
    sync(c);
  }
};

// The recursion's scalars on the device, so that iterations run without a host round trip.  Arrays of
// ns entries behind it: shift, rsd_sq (|chi|^2 target^2), zeta, zeta of the step before, b zeta; conv;
// and the coefficient arrays of the three updates.
struct MsScal {
  double cp, cc, a, b, bp;
  int done, status, iters, ns;
  double *shift, *rsd_sq, *z, *zprev, *bs;
  int* conv;
  double2* cp_;  // [2][ns + 1]: p_s = zeta_s r + a_s p_s, and p0 = r + a p0 in the last place
  double2* cr;   // [2]: r = b A p0 + r
  double2* cx;   // [2][ns]: psi_s -= bs_s p_s
};

// a = |r|^2 / |r_prev|^2 and the direction coefficients (converged shifts keep p_s: 0, 1)
__global__ void ms_directions(MsScal* m) {
  pdl_begin();
  const int n = m->ns, q = threadIdx.x;
  const bool done = m->done;
  const double a = done ? 0.0 : m->cc / m->cp, b = m->b;
  __syncthreads();
  for (int k = q; k < n; k += blockDim.x) {
    const bool keep = done || m->conv[k];
    m->cp_[k] = make_double2(keep ? 0.0 : m->z[k], 0.0);
    m->cp_[n + 1 + k] = make_double2(keep ? 1.0 : a * m->z[k] * m->bs[k] / (m->zprev[k] * b), 0.0);
  }
  if (q == 0) {
    m->cp_[n] = make_double2(done ? 0.0 : 1.0, 0.0);
    m->cp_[2 * n + 1] = make_double2(done ? 1.0 : a, 0.0);
    m->a = a;
    if (!done) m->cp = m->cc;
  }
}

// b = -|r|^2 / <p0, A p0>
__global__ void ms_step(MsScal* m, const double* d) {
  pdl_begin();
  if (!m->done) {
    m->bp = m->b;
    m->b = -m->cp / d[0];
  }
  m->cr[0] = make_double2(m->done ? 0.0 : m->b, 0.0);
  m->cr[1] = make_double2(1.0, 0.0);
}

// zeta_next = zeta zeta_prev bp / (b a (zeta_prev - zeta) + zeta_prev bp (1 - sigma b)), the solution
// coefficients, and convergence of each shift (one block)
__global__ void ms_solution(MsScal* m, const double* rr) {
  pdl_begin();
  const int n = m->ns, q = threadIdx.x;
  const bool done = m->done;
  const double cc = rr[0], a = m->a, b = m->b, bp = m->bp;
  int open = 0;
  for (int k = q; k < n; k += blockDim.x) {
    const bool skip = done || m->conv[k];
    if (!skip) {
      const double z = m->z[k], zp = m->zprev[k];
      const double zn = z * zp * bp / (b * a * (zp - z) + zp * bp * (1.0 - m->shift[k] * b));
      m->bs[k] = b * zn / z;
      m->zprev[k] = z;
      m->z[k] = zn;
      m->conv[k] = cc * zn * zn < m->rsd_sq[k];
    }
    m->cx[k] = make_double2(skip ? 0.0 : -m->bs[k], 0.0);
    m->cx[n + k] = make_double2(1.0, 0.0);
    open |= !m->conv[k];
  }
  open = __syncthreads_or(open);
  if (q == 0 && !done) {
    m->cc = cc;
    m->iters += 1;
    if (!isfinite(cc)) m->status = GBC_ERR_NONFINITE;
    m->done = !open || !isfinite(cc);
  }
}

// the device side of MsScal, one allocation
struct MsDevice {
  MsScal h{};
  MsScal* d = nullptr;
  void upload(gbc_ctx* c, int ns, const std::vector<double>& shift, const std::vector<double>& rsd_sq,
              const std::vector<double>& z, const std::vector<double>& zprev, const std::vector<double>& bs) {
    const size_t nd = 5 * (size_t)ns, n2 = 2 * (ns + 1) + 2 + 2 * (size_t)ns;
    const size_t head = (sizeof(MsScal) + 15) / 16 * 16, bytes = head + n2 * 16 + nd * 8 + (size_t)ns * 4;
    GBC_CUDA(cudaMalloc(&d, bytes));
    char* p = reinterpret_cast<char*>(d) + head;
    h.cp_ = reinterpret_cast<double2*>(p);
    h.cr = h.cp_ + 2 * (ns + 1);
    h.cx = h.cr + 2;
    h.shift = reinterpret_cast<double*>(h.cx + 2 * (size_t)ns);
    h.rsd_sq = h.shift + ns;
    h.z = h.rsd_sq + ns;
    h.zprev = h.z + ns;
    h.bs = h.zprev + ns;
    h.conv = reinterpret_cast<int*>(h.bs + ns);
    h.ns = ns;
    std::vector<char> img(bytes, 0);
    std::memcpy(img.data(), &h, sizeof h);
    const std::vector<double>* src[5] = {&shift, &rsd_sq, &z, &zprev, &bs};
    char* base = img.data() + (reinterpret_cast<char*>(h.shift) - reinterpret_cast<char*>(d));
    for (int k = 0; k < 5; ++k) std::memcpy(base + sizeof(double) * ns * k, src[k]->data(), sizeof(double) * ns);
    GBC_CUDA(cudaMemcpyAsync(d, img.data(), bytes, cudaMemcpyHostToDevice, c->stream));
    sync(c);  // img goes out of scope
  }
  ~MsDevice() {
    if (d) cudaFree(d);
  }
};

}  // namespace

int solve_multishift(gbc_ctx* c, const gbc_solve_params* pp, int ns, const double* shifts, const double* rsd,
                     double* const* psi_canon, const double* chi_canon, gbc_result* res) {
  const int D = PREC_DOUBLE;
  const Geom& g = c->g;
  cudaStream_t s = c->stream;
  const int max_iter = pp->max_iter > 0 ? pp->max_iter : 10000;
  // mixed precision (sloppy_precision HALF or SINGLE): the shared-Krylov recursion runs on FP32
  // fields and the FP32 operator to a relative 1e-6 (near FP32's floor), then every shift is
  // refined by the FP64 defect correction of refine_shifted (batched over the shifts, corrections
  // from CG in the sloppy operator); else the recursion runs in FP64 to the targets
  const int sp = pp->sloppy_precision;
  const bool mixed = sp == PREC_HALF || sp == PREC_SINGLE;
  const int W = mixed ? PREC_SINGLE : D;
  ensure_prec(c, D);
  if (mixed) {
    ensure_prec(c, PREC_SINGLE);
    ensure_prec(c, sp);
  }
  const double t0 = now();
  cudaEvent_t ev0, ev1;
  GBC_CUDA(cudaEventCreate(&ev0));
  GBC_CUDA(cudaEventCreate(&ev1));
  GBC_CUDA(cudaEventRecord(ev0, s));
  const long long launches0 = launch_count();

  const int o = 20 * pidx(W);  // workspace slots per recursion precision
  Spinor chid = sub(workspace(c, MS_CHI, D, 1), 0, 1);
  Spinor chi = mixed ? sub(workspace(c, MS_CHI + o, W, 1), 0, 1) : chid;
  Spinor r = sub(workspace(c, MS_R + o, W, 1), 0, 1);
  Spinor mp = sub(workspace(c, MS_MP + o, W, 1), 0, 1);
  Spinor mmp = sub(workspace(c, MS_MMP + o, W, 1), 0, 1);
  Spinor te = sub(workspace(c, MS_TE + o, W, 1), 0, 1);
  Spinor Pall = sub(workspace(c, MS_P + o, W, ns + 1), 0, ns + 1);  // p_s, then p0
  Spinor P = sub(Pall, 0, ns), p0 = sub(Pall, ns, 1);
  Spinor X = sub(workspace(c, MS_X + o, W, ns), 0, ns);
  const size_t rs = (size_t)c->V * 24;
  ensure_stage(c, ns);
  GBC_CUDA(cudaMemcpyAsync(c->d_stage[0], chi_canon, rs * sizeof(double), cudaMemcpyHostToDevice, s));
  import_spinor(g, c->d_stage[0], rs, 1, chid, s);
  // the solutions go back through d_stage[1], one slot per shift (the even sites of psi_s are kept)
  std::vector<HostResult::Item> items(ns);
  for (int q = 0; q < ns; ++q) items[q] = {psi_canon[q], c->d_stage[1] + q * rs, rs * sizeof(double)};
  HostResult out(s, copy_stream(c), std::move(items), HostResult::kLoad);
  if (mixed) blas_copy(g, chi, chid, s);
  Coefs co(ns), one(1);

  std::vector<double> shift(shifts, shifts + ns), rsd_sq(ns);
  int k = 0, iters = 0, status = GBC_OK;
  const double chi2 = norm2(c, chi);
  blas_zero(g, X, s);
  if (!(chi2 > 0.0)) {
    status = std::isfinite(chi2) ? GBC_OK : GBC_ERR_NONFINITE;
  } else {
    for (int q = 0; q < ns; ++q) {
      const double t = mixed ? std::max(rsd[q], 1e-6) : rsd[q];
      rsd_sq[q] = chi2 * t * t;
    }
    const int smallest = (int)(std::min_element(shift.begin(), shift.end()) - shift.begin());
    // r = p0 = p_s = chi
    blas_copy(g, r, chi, s);
    blas_copy(g, p0, chi, s);
    blas_copy(g, P, broadcast(chi, ns), s);
    // b = -|r|^2 / <p0, A p0>,  r += b A p0
    double cp = chi2;
    apply_meo(c, W, false, p0, mp, te, true);
    double d = fetch(c);
    apply_meo(c, W, true, mp, mmp, te, false);
    double b = -cp / d;
    one.h[0] = make_double2(b, 0.0);
    one.h[1] = make_double2(1.0, 0.0);
    one.axpby(c, mmp, r);
    // zeta_prev = 1, zeta = 1 / (1 - sigma b), bs = b zeta; psi_s = -bs chi
    std::vector<double> zprev(ns, 1.0), z(ns), bs(ns);
    for (int q = 0; q < ns; ++q) {
      z[q] = 1.0 / (1.0 - shift[q] * b);
      bs[q] = b * z[q];
      co.h[q] = make_double2(-bs[q], 0.0);
      co.h[ns + q] = make_double2(0.0, 0.0);
    }
    co.axpby(c, broadcast(chi, ns), X);
    double cc = norm2(c, r);
    bool done = cc < rsd_sq[smallest];
    if (!done && !std::isfinite(cc)) status = GBC_ERR_NONFINITE;
    if (!done && status == GBC_OK) {
      MsDevice ms;
      ms.h.cp = cp;
      ms.h.cc = cc;
      ms.h.b = b;
      ms.upload(c, ns, shift, rsd_sq, z, zprev, bs);
      const int nth = std::min(256, (ns + 31) / 32 * 32);
      auto body = [&]() {
        launch_pdl(ms_directions, 1, nth, s, ms.d);
        // p0 = r + a p0 and p_s = zeta_s r + as_s p_s in one pass over r
        blas_axpby(g, ms.h.cp_, broadcast(r, ns + 1), ms.h.cp_ + ns + 1, Pall, s);
        apply_meo(c, W, false, p0, mp, te, true);
        launch_pdl(ms_step, 1, 1, s, ms.d, c->d_result);
        apply_meo(c, W, true, mp, mmp, te, false);
        blas_axpby_norm2(g, ms.h.cr, mmp, ms.h.cr + 1, r, red(c), s);  // r += b A p0
        launch_pdl(ms_solution, 1, nth, s, ms.d, c->d_result);
        blas_axpby(g, ms.h.cx, P, ms.h.cx + ns, X, s);
        count_launch(3);
      };
      // blocks of iterations between host checks, replayed from a graph after the first (uncaptured,
      // tuning) iteration; once every shift has converged an iteration changes nothing
      constexpr int kBlock = 4;
      cudaGraphExec_t exec = nullptr;
      struct ExecScope {
        cudaGraphExec_t& e;
        ~ExecScope() {
          if (e) cudaGraphExecDestroy(e);
        }
      } scope{exec};
      long long graph_launches = 0;
      MsScal now_{};
      while (!now_.done && k < max_iter) {
        const int steps = k == 0 ? 1 : std::min(kBlock, max_iter - k);
        if (k > 0 && steps == kBlock && c->use_graphs) {
          if (!exec) {
            cudaGraph_t graph;
            const long long l0 = launch_count();
            GBC_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
            for (int q = 0; q < kBlock; ++q) body();
            GBC_CUDA(cudaStreamEndCapture(s, &graph));
            GBC_CUDA(cudaGraphInstantiate(&exec, graph, 0));
            cudaGraphDestroy(graph);
            graph_launches = launch_count() - l0;
            count_launch(-graph_launches);
          }
          GBC_CUDA(cudaGraphLaunch(exec, s));
          count_launch(graph_launches);
        } else {
          for (int q = 0; q < steps; ++q) body();
        }
        k += steps;
        GBC_CUDA(cudaMemcpyAsync(&now_, ms.d, sizeof now_, cudaMemcpyDeviceToHost, s));
        sync(c);
      }
      iters = now_.iters;
      status = now_.status;
      done = now_.done && status == GBC_OK;
    }
    if (!done && status == GBC_OK) status = GBC_ERR_NOT_CONVERGED;
  }
  // mixed precision: FP64 copies of the solutions, refined shift by shift (batched)
  std::vector<int> refine_iters(ns, 0), refine_status(ns, GBC_OK);
  std::vector<double> refine_rr;
  bool rr_final = false;
  Spinor XD = X;
  if (mixed) {
    XD = sub(workspace(c, MS_X, D, ns), 0, ns);
    blas_copy(g, XD, X, s);
    if (status == GBC_OK || status == GBC_ERR_NOT_CONVERGED) {
      double* d_shift = nullptr;
      GBC_CUDA(cudaMalloc(&d_shift, sizeof(double) * ns));
      GBC_CUDA(cudaMemcpyAsync(d_shift, shift.data(), sizeof(double) * ns, cudaMemcpyHostToDevice, s));
      refine_rr.resize(ns);
      rr_final = true;
      try {
        // the context's scalars and partial sums are sized for max_rhs right-hand sides
        for (int q0 = 0; q0 < ns; q0 += c->max_rhs) {
          const int m = std::min(c->max_rhs, ns - q0);
          std::vector<double> rr;
          std::vector<int> st;
          bool last = false;
          const std::vector<int> it = refine_shifted(c, sp, chid, d_shift + q0, sub(XD, q0, m),
                                                     std::vector<double>(rsd + q0, rsd + q0 + m),
                                                     std::max(1, max_iter - iters), rr, st, last);
          std::copy(it.begin(), it.end(), refine_iters.begin() + q0);
          std::copy(st.begin(), st.end(), refine_status.begin() + q0);
          std::copy(rr.begin(), rr.end(), refine_rr.begin() + q0);
          rr_final = rr_final && last;
        }
      } catch (...) {
        cudaFree(d_shift);
        throw;
      }
      cudaFree(d_shift);
      status = GBC_OK;
    }
  }
  GBC_CUDA(cudaEventRecord(ev1, s));
  GBC_CUDA(cudaEventSynchronize(ev1));
  float ms = 0.f;
  cudaEventElapsedTime(&ms, ev0, ev1);
  const long long launches = launch_count() - launches0;

  // the odd sites of each solution to the host, beside the true FP64 residual of every shifted system
  out.ready();
  for (int q = 0; q < ns; ++q) {
    export_spinor(g, c->d_stage[1] + q * rs, rs, 1, sub(XD, q, 1), s);
    out.send(q);
  }
  Spinor t1 = sub(workspace(c, MS_T1, D, 1), 0, 1);
  Spinor t2 = sub(workspace(c, MS_T2, D, 1), 0, 1);
  Spinor ted = sub(workspace(c, MS_TE, D, 1), 0, 1);
  for (int q = 0; q < ns; ++q) {
    double rr = 0.0;
    if (rr_final) {
      rr = refine_rr[q];  // the refinement ended on this residual of this solution
    } else {
      Spinor xq = sub(XD, q, 1);
      apply_meo(c, D, false, xq, t1, ted, false);
      apply_meo(c, D, true, t1, t2, ted, false);
      one.h[0] = make_double2(shift[q], 0.0);
      one.h[1] = make_double2(1.0, 0.0);
      one.axpby(c, xq, t2);  // t2 = (M~^dag M~ + sigma) psi
      blas_xmy_norm2(g, chid, t2, red(c), s);
      rr = fetch(c);
    }
    gbc_result& o = res[q];
    o = gbc_result{};
    o.n_count = iters + refine_iters[q];
    o.n_outer = mixed ? 1 : 0;
    o.resid = std::sqrt(rr);
    o.rel_resid = chi2 > 0 ? std::sqrt(rr / chi2) : 0.0;
    o.status = mixed && status == GBC_OK ? refine_status[q] : status;
    if (o.status == GBC_ERR_NOT_CONVERGED) o.status = GBC_OK;  // judged by the tolerance factor below
    if (o.status == GBC_OK && !(o.rel_resid <= pp->rsd_tolerance_factor * rsd[q])) o.status = GBC_ERR_NOT_CONVERGED;
    o.device_seconds = ms * 1e-3;
    o.launches = (int)launches;
  }
  sync(c);
  out.wait();
  cudaEventDestroy(ev0);
  cudaEventDestroy(ev1);
  const double t1s = now();
  int worst = GBC_OK;
  for (int q = 0; q < ns; ++q) {
    res[q].seconds = t1s - t0;
    if (res[q].status != GBC_OK && worst == GBC_OK) worst = res[q].status;
  }
  return worst;
}

}  // namespace gbc

using namespace gbc;

extern "C" int gbc_solve_multishift(gbc_ctx* c, const gbc_solve_params* p, int nshift, const double* shifts,
                                    const double* rsd_targets, double* const* psi, const double* chi,
                                    gbc_result* res) {
  if (!c || !p || nshift < 1 || !shifts || !psi || !chi || !res) return GBC_ERR_ARGS;
  for (int q = 0; q < nshift; ++q)
    if (!psi[q] || !std::isfinite(shifts[q]) || shifts[q] < 0.0) return GBC_ERR_ARGS;
  if (!c->have_gauge) {
    c->err = "load the gauge field first";
    return GBC_ERR_STATE;
  }
  std::vector<double> rsd(nshift);
  for (int q = 0; q < nshift; ++q) {
    rsd[q] = rsd_targets ? rsd_targets[q] : p->rsd_target;
    if (!(rsd[q] > 0)) rsd[q] = 1e-10;
  }
  gbc_solve_params pp = *p;
  if (!(pp.rsd_tolerance_factor > 0)) pp.rsd_tolerance_factor = 10.0;
  try {
    return solve_multishift(c, &pp, nshift, shifts, rsd.data(), psi, chi, res);
  } catch (const CudaError& e) {
    c->err = std::string(e.where) + ": " + cudaGetErrorString(e.e);
    return GBC_ERR_CUDA;
  } catch (const std::string& m) {
    c->err = m;
    return GBC_ERR_STATE;
  } catch (const std::bad_alloc&) {
    c->err = "host allocation failed";
    return GBC_ERR_CUDA;
  }
}
