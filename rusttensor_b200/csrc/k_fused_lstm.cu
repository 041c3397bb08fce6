// Chains of recurrent networks: the LSTM cell, its gradient, the input of the gates' product.
#include "fused_known.cuh"

namespace {
constexpr KnownProgram kPrograms[] = {
#include "fused_programs_recurrent.inc"
};
}  // namespace

const fused::KnownProgram* fused::known_recurrent_programs(int* n) {
  *n = (int)(sizeof(kPrograms) / sizeof(kPrograms[0]));
  return kPrograms;
}
