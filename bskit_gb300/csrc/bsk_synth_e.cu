// Field synthesis passes of some compiled lengths (one translation unit of several).
#include "bsk_synth_warp.cuh"

namespace bsk {
namespace synth {

bool run_compiled_e(int N, const SynthArgs& A, const FftPlan& pl, cudaStream_t st) {
  return run_one_of<360, 48, 160, 256, 64>(N, A, pl, st);
}

}  // namespace synth
}  // namespace bsk
