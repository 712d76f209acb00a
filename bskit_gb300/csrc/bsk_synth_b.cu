// Field synthesis passes of some compiled lengths (one translation unit of several).
#include "bsk_synth_warp.cuh"

namespace bsk {
namespace synth {

bool run_compiled_b(int N, const SynthArgs& A, const FftPlan& pl, cudaStream_t st) {
  return run_one_of<480, 32, 100, 120, 192>(N, A, pl, st);
}

}  // namespace synth
}  // namespace bsk
