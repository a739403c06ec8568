// Second step of the symmetric operator, fp16 storage.
#include "dslash_inst.cuh"

namespace gbc {
int hop_sym_launch_h(int recon, int reduce, const HopArgs& a, HopShape sh, cudaStream_t s) {
  return recon == 18 ? hop_sym_reduce<PrecH, 18>(reduce, a, sh, s) : hop_sym_reduce<PrecH, 12>(reduce, a, sh, s);
}
}  // namespace gbc
