// Field synthesis passes of some compiled lengths (one translation unit of several).
#include "bsk_synth_warp.cuh"

namespace bsk {
namespace synth {

bool run_compiled_f(int N, const SynthArgs& A, const FftPlan& pl, cudaStream_t st) {
  return run_one_of<320, 288, 300, 60, 80>(N, A, pl, st);
}

}  // namespace synth
}  // namespace bsk
