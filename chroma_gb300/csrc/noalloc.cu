// gbc_apply_meo_noalloc: the even-odd clover operator M~ in FP64 with no device allocation.
//
// Some callers cannot allocate device memory while they run.  Chroma built on QDP-JIT is the
// main one here: QDP-JIT's pool allocator reserves most of the GPU's memory when it starts, so a
// cudaMalloc issued later from a library may fail, and a cudaMalloc/cudaFree pair can also
// synchronise the device in the middle of a caller's pipelined stream work.  The ordinary entry
// points allocate their workspaces inside a gbc_ctx.  This one takes every input and output as a
// caller-owned device pointer in the canonical layouts of gbclover.h, and the only temporary it
// needs -- the even-parity intermediate A_ee^-1 D_eo psi_o -- lives in a file-scope static
// __device__ array of fixed size, which every GPU that loads the library holds until exit.
//
// The two kernels follow the same algebra as apply_meo (Chroma eoprec_clover_linop_w.cc:142-187)
// but read the canonical array-of-structures layout directly.
#include <cstdio>
#include <mutex>

#include "../../include/gbclover.h"
#include "dslash.cuh"
#include "dslash_split.cuh"

namespace gbc {
namespace {

// Even-parity intermediate, GBC_NOALLOC_MAX_VH sites x 12 complex doubles (12 MiB).
static __device__ __align__(256) double2 noalloc_scratch[(size_t)GBC_NOALLOC_MAX_VH * 12];

constexpr int kMaxDevices = 64;
std::mutex g_mu;
double2* g_scratch_ptr[kMaxDevices] = {nullptr};

// Field access of split_site (dslash_split.cuh) in the canonical layouts; the even intermediate is
// the scratch array, indexed by checkerboard site.
template <int PARITY>
struct CanonField {
  Geom g;
  const double2* links;
  const double* clov;
  const double2* psi;
  double2* scratch;
  double2* dst;
  __device__ __forceinline__ const Geom& geom() const { return g; }
  __device__ __forceinline__ int parity() const { return PARITY; }
  __device__ __forceinline__ double2 in(const Coord& n, int ni, int k) const {
    return PARITY == 0 ? psi[(size_t)full_index(g, n) * 12 + k] : scratch[(size_t)ni * 12 + k];
  }
  __device__ __forceinline__ double2 link(const Coord& c, int, const Coord& n, int, int mu, bool fwd, int e) const {
    return links[((size_t)full_index(g, fwd ? c : n) * 4 + mu) * 9 + e];
  }
  __device__ __forceinline__ double diag(const Coord& c, int, int b, int i) const {
    return clov[(size_t)full_index(g, c) * 72 + 6 * b + i];
  }
  __device__ __forceinline__ double2 offd(const Coord& c, int, int b, int k) const {
    const double* p = clov + (size_t)full_index(g, c) * 72 + 12 + 30 * b + 2 * k;  // 8-byte aligned
    return make_double2(p[0], p[1]);
  }
  __device__ __forceinline__ double2 self(const Coord& c, int, int k) const {
    return psi[(size_t)full_index(g, c) * 12 + k];
  }
  __device__ __forceinline__ double2 aux(int, int) const { return make_double2(0.0, 0.0); }
  __device__ __forceinline__ void out(const Coord& c, int idx, int k, int im, double v) const {
    double2* p = PARITY == 0 ? scratch + (size_t)idx * 12 : dst + (size_t)full_index(g, c) * 12;
    reinterpret_cast<double*>(p + k)[im] = v;
  }
};

// even sites: scratch[cb] = A_ee^-1 D'_eo psi_o
template <bool DAG, int S>
__global__ void __launch_bounds__(8 * S) noalloc_even(const CanonField<0> f) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");  // the odd kernel may be placed
  double sum[3];
  split_site<CanonField<0>, HOP_CLOV, DAG, RED_NONE, S>(f, 1.0, 0.0, blockIdx.x, sum);
}

// odd sites: out = A_oo psi_o - 1/4 D'_oe scratch  (+ isign i mu gamma_5 psi_o)
template <bool DAG, int S>
__global__ void __launch_bounds__(8 * S) noalloc_odd(const CanonField<1> f, double twist) {
  pdl_begin();
  double sum[3];
  split_site<CanonField<1>, HOP_XPAY, DAG, RED_NONE, S>(f, -0.25, twist, blockIdx.x, sum);
}

template <bool DAG, int S>
void noalloc_launch(const CanonField<0>& fe, const CanonField<1>& fo, double twist, cudaStream_t s) {
  const unsigned blocks = (unsigned)((fe.g.Vh + S - 1) / S);
  noalloc_even<DAG, S><<<blocks, 8 * S, 0, s>>>(fe);
  // up to two blocks per SM the odd kernel is placed beside the even one (8^4: 24.6 -> 22.5 us); larger
  // grids would lose their even spread over the SMs
  launch_pdl_if(blocks <= 2 * 152, noalloc_odd<DAG, S>, blocks, 8 * S, s, fo, twist);
}
template <bool DAG>
void noalloc_launch(const CanonField<0>& fe, const CanonField<1>& fo, double twist, cudaStream_t s) {
  switch (hop_split_sites(fe.g.Vh, 1)) {
    case 8: return noalloc_launch<DAG, 8>(fe, fo, twist, s);
    case 16: return noalloc_launch<DAG, 16>(fe, fo, twist, s);
    default: return noalloc_launch<DAG, 32>(fe, fo, twist, s);
  }
}

}  // namespace

// Device address of the scratch array on the current device; looked up once per device.  The
// lookup is also what makes the array exist there: under CUDA's default lazy module loading
// (CUDA_MODULE_LOADING=LAZY) this file's module, with its static array, is loaded on the first
// use of one of its symbols, not when the library is loaded.
int noalloc_scratch_for_current_device(double2** out) {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return GBC_ERR_CUDA;
  std::lock_guard<std::mutex> lock(g_mu);
  if (!g_scratch_ptr[dev]) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, noalloc_scratch);
    if (e != cudaSuccess || !p) {
      fprintf(stderr, "gbc_apply_meo_noalloc: cudaGetSymbolAddress failed on device %d: %s\n", dev,
              cudaGetErrorString(e));
      return GBC_ERR_CUDA;
    }
    g_scratch_ptr[dev] = static_cast<double2*>(p);
  }
  *out = g_scratch_ptr[dev];
  return GBC_OK;
}

int noalloc_reserve() {
  double2* p = nullptr;
  return noalloc_scratch_for_current_device(&p);
}

}  // namespace gbc

extern "C" int gbc_apply_meo_noalloc(const gbc_geom* geom, const gbc_action* act, const double* links_dev,
                                     const double* clov_dev, const double* invclov_dev, int isign, double* out_dev,
                                     const double* in_dev, void* stream) {
  using namespace gbc;
  if (!geom || !act || !links_dev || !clov_dev || !invclov_dev || !out_dev || !in_dev) return GBC_ERR_ARGS;
  if (isign != 1 && isign != -1) return GBC_ERR_ARGS;
  // every extent even: with an odd extent the wrap-around neighbour has the site's own parity
  for (int m = 0; m < 4; ++m)
    if (geom->dims[m] < 2 || geom->dims[m] % 2) return GBC_ERR_ARGS;
  const long V = (long)geom->dims[0] * geom->dims[1] * geom->dims[2] * geom->dims[3];
  if (V / 2 > GBC_NOALLOC_MAX_VH) {
    fprintf(stderr,
            "gbc_apply_meo_noalloc: %ld sites per checkerboard exceed the static scratch of %d; "
            "use gbc_apply for this lattice\n",
            V / 2, GBC_NOALLOC_MAX_VH);
    return GBC_ERR_ARGS;
  }
  double2* scratch = nullptr;
  int rc = noalloc_scratch_for_current_device(&scratch);
  if (rc != GBC_OK) return rc;
  Geom g{};
  for (int m = 0; m < 4; ++m) g.L[m] = geom->dims[m];
  g.Lxh = g.L[0] / 2;
  g.Vh = (int)(V / 2);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const double2* links = reinterpret_cast<const double2*>(links_dev);
  const double2* in = reinterpret_cast<const double2*>(in_dev);
  double2* out = reinterpret_cast<double2*>(out_dev);
  const double twist = act->twisted ? act->twisted_m : 0.0;
  // the scratch is fully overwritten by the first kernel on every call: nothing to clear
  const CanonField<0> fe{g, links, invclov_dev, in, scratch, nullptr};
  const CanonField<1> fo{g, links, clov_dev, in, scratch, out};
  if (isign > 0) noalloc_launch<false>(fe, fo, twist, s);
  else noalloc_launch<true>(fe, fo, twist, s);
  return cudaGetLastError() == cudaSuccess ? GBC_OK : GBC_ERR_CUDA;
}
