// The persistent PCG kernels: single precision.
#include "qedf_pcg_kernel.cuh"

namespace qedf {

int launch_pcg_f32(PcgParams& p, const BandTaps& taps, int by, cudaStream_t st) {
  return launch_pcg_by<float, float, float, float>(p, taps, by, st);
}

}  // namespace qedf
