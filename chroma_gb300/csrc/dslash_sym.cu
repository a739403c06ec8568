// Second step of the symmetric operator, FP32 and FP64, and its dispatch on the precision.
#include "dslash_inst.cuh"

namespace gbc {
int hop_sym_launch_h(int recon, int reduce, const HopArgs& a, HopShape sh, cudaStream_t s);

int hop_sym_launch(int prec, int recon, bool dag, int reduce, const HopArgs& a, HopShape sh, cudaStream_t s) {
  if (dag || (recon != 12 && recon != 18)) return -1;
  switch (prec) {
    case PREC_DOUBLE: return recon == 18 ? hop_sym_reduce<PrecD, 18>(reduce, a, sh, s) : -1;
    case PREC_SINGLE:
      return recon == 18 ? hop_sym_reduce<PrecS, 18>(reduce, a, sh, s) : hop_sym_reduce<PrecS, 12>(reduce, a, sh, s);
    case PREC_HALF: return hop_sym_launch_h(recon, reduce, a, sh, s);
  }
  return -1;
}
}  // namespace gbc
