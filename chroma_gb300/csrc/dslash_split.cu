// FP64 hopping kernels with the hops of a site split over threads (dslash_split.cuh): launch and dispatch.
#include "dslash.cuh"
#include "dslash_split.cuh"

namespace gbc {
namespace {

// Grid: one dimension, right-hand sides fastest (blocks that share links run together).
template <int MODE, bool DAG, int REDUCE, int S>
__global__ void __launch_bounds__(8 * S) hop_kernel_split(const HopArgs a) {
  pdl_begin();
  const int sblock = blockIdx.x / a.nrhs, rhs = blockIdx.x - sblock * a.nrhs;
  double sum[3] = {0.0, 0.0, 0.0};
  if (!a.active || a.active[(size_t)rhs * a.active_stride])
    split_site<SplitPlanes, MODE, DAG, REDUCE, S>(SplitPlanes{a, rhs}, a.a, a.twist, sblock, sum);
  if constexpr (REDUCE != RED_NONE)
    block_sums_1rhs<red_count<REDUCE>(), 8 * S>(a, Sums3<double>{{sum[0], sum[1], sum[2]}}, rhs, sblock,
                                                (a.g.Vh + S - 1) / S);
}

template <int MODE, bool DAG, int REDUCE>
int launch(const HopArgs& a, int sites, cudaStream_t s) {
  const int nb = (a.g.Vh + sites - 1) / sites;
  const unsigned grid = (unsigned)nb * a.nrhs;
  if (sites == 8) launch_pdl(hop_kernel_split<MODE, DAG, REDUCE, 8>, grid, 64, s, a);
  else if (sites == 16) launch_pdl(hop_kernel_split<MODE, DAG, REDUCE, 16>, grid, 128, s, a);
  else launch_pdl(hop_kernel_split<MODE, DAG, REDUCE, 32>, grid, 256, s, a);
  return nb;
}

}  // namespace

int hop_split_launch(int mode, bool dag, int reduce, const HopArgs& a, int sites, cudaStream_t s) {
  switch (mode) {
    case HOP_SYM:
      if (dag) return -1;
      switch (reduce) {
        case RED_NONE: return launch<HOP_SYM, false, RED_NONE>(a, sites, s);
        case RED_NORM: return launch<HOP_SYM, false, RED_NORM>(a, sites, s);
        case RED_DOT_SELF: return launch<HOP_SYM, false, RED_DOT_SELF>(a, sites, s);
        default: return launch<HOP_SYM, false, RED_DOT_AUX>(a, sites, s);
      }
    case HOP_PLAIN:
      if (reduce) return -1;
      return dag ? launch<HOP_PLAIN, true, RED_NONE>(a, sites, s) : launch<HOP_PLAIN, false, RED_NONE>(a, sites, s);
    case HOP_CLOV:
      if (reduce) return -1;
      return dag ? launch<HOP_CLOV, true, RED_NONE>(a, sites, s) : launch<HOP_CLOV, false, RED_NONE>(a, sites, s);
    case HOP_XPAY:
      if (reduce == RED_NONE)
        return dag ? launch<HOP_XPAY, true, RED_NONE>(a, sites, s) : launch<HOP_XPAY, false, RED_NONE>(a, sites, s);
      if (reduce == RED_NORM)
        return dag ? launch<HOP_XPAY, true, RED_NORM>(a, sites, s) : launch<HOP_XPAY, false, RED_NORM>(a, sites, s);
      // BiCGStab applies M~ itself, never its dagger
      if (dag) return -1;
      return reduce == RED_DOT_SELF ? launch<HOP_XPAY, false, RED_DOT_SELF>(a, sites, s)
                                    : launch<HOP_XPAY, false, RED_DOT_AUX>(a, sites, s);
  }
  return -1;
}

}  // namespace gbc
