// Field synthesis passes of some compiled lengths (one translation unit of several).
#include "bsk_synth_warp.cuh"

namespace bsk {
namespace synth {

bool run_compiled_d(int N, const SynthArgs& A, const FftPlan& pl, cudaStream_t st) {
  return run_one_of<384, 40, 144, 240, 72>(N, A, pl, st);
}

}  // namespace synth
}  // namespace bsk
